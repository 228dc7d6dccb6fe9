// Host side of the decode engine and its C ABI (include/b200moe.h).
//
// What the reference does in aegist_rs/src/hybrid.rs is done here with a different plan:
//   * every tensor, the embedding table and all experts included, is resident in HBM (a slot table
//     [layer][expert] -> device address replaces the LRU pool of hybrid.rs:190-390);
//   * a decode step is one CUDA graph of 6 launches per layer with no host synchronisation inside:
//     token ids, positions, router picks and the arg-max stay on the device (the reference crosses
//     the host boundary 82 times per token, hybrid.rs:743-758, 875, 919, 1000);
//   * the KV cache is paged (64-token pages through a page table) and stored as bf16 or fp32.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nccl.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/b200moe.h"
#include "kernels.cuh"
#include "step1.cuh"
#include "nxfile.hpp"

namespace b2 {

#define CU(call)                                                                                       \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return fail("%s: %s", #call, cudaGetErrorString(e_));                   \
    } while (0)

// From this many sequences (or prompt tokens) on a step runs on the tcgen05 GEMM family; below it on the GEMV family,
// which re-reads the weights once per four sequences. Not 5, where the GEMM family is the faster one (4-layer full-width case at
// context 1000, 0.50 ms per step against 0.65): its three digit planes hold an activation to 2^-22 of a row's largest
// value, the GEMV family's four to 2^-31, and a sequence of five keeps the precision it has in a batch of four. In ms per step: 0.41
// at 4 and 0.65 at 5 sequences on the GEMV family, 0.53 at 6 on the GEMM family.
constexpr int BATCH_GEMM_MIN = 6;

struct Cfg {
    int V = 0, D = 0, L = 0;
    std::vector<int> attn;
    int H = 0, KV = 0, HD = 0, RD = 0;
    double theta = 0;
    int HK = 0, HV = 0, DK = 0, DV = 0, CK = 0;
    int E = 0, TOPK = 0, I = 0, SH = 0, G = 0;
    float eps = 1e-6f;
    int n1 = 0, n2 = 0, rank = 0, cores_active = 0;
    int C() const { return 2 * HK * DK + HV * DV; }
    int VD() const { return HV * DV; }
    int n_attn() const { int n = 0; for (int a : attn) n += a; return n; }
    int n_delta() const { return L - n_attn(); }
    size_t gu_q() const { return (size_t)2 * I * (D / 2); }
    size_t gu_sm() const { return (size_t)2 * I * (D / G) * 2; }
    size_t dn_q() const { return (size_t)D * (I / 2); }
    size_t dn_sm() const { return (size_t)D * (I / G) * 2; }
    size_t off_gu_s() const { return gu_q(); }
    size_t off_gu_m() const { return gu_q() + gu_sm(); }
    size_t off_dn_q() const { return gu_q() + 2 * gu_sm(); }
    size_t off_dn_s() const { return off_dn_q() + dn_q(); }
    size_t off_dn_m() const { return off_dn_s() + dn_sm(); }
    size_t expert_bytes() const { size_t n = off_dn_m() + dn_sm(); return (n + 63) / 64 * 64; }
};

struct DevTensor {
    void* p = nullptr;
    size_t nbytes = 0;
    std::string dtype;
    std::vector<int64_t> shape;
};

struct QWd { const int8_t* w = nullptr; const uint16_t* s = nullptr; int n = 0, k = 0; };

struct LayerW {
    bool attn = false;
    int slot = 0;
    const uint16_t *norm1 = nullptr, *norm2 = nullptr;
    // attention
    QWd q, k, v, o;
    const uint16_t *q_norm = nullptr, *k_norm = nullptr;
    // DeltaNet
    QWd in_qkv, in_z, out;
    const uint16_t *in_a = nullptr, *in_b = nullptr, *conv = nullptr, *a_log = nullptr, *dt_bias = nullptr, *gnorm = nullptr;
    // MoE
    const uint16_t* router = nullptr;
    QWd sh_gate, sh_up, sh_down;
    const uint16_t* sh_gw = nullptr;
    const uint8_t* experts = nullptr;       // [local experts][expert_bytes]
    const uint8_t** eptr = nullptr;         // device [E]
    float* router_bias = nullptr;           // device [E] or null
    // core engine + the layer's live switchable cores (live_bank, aegist_rs/src/hybrid.rs:1122-1150)
    const uint16_t *key1 = nullptr, *key2 = nullptr;      // [n1][D], [n2][D]; null: the brain has no core engine tensors
    int* live = nullptr;                    // device [n1 * n2]: core id -> index into the bank, or -1
    int n_live = 0;
    const uint16_t *cg = nullptr, *cu = nullptr, *cd = nullptr;   // bank: gate, up [n][D][r], down [n][r][D]
};

static size_t dtype_size(const std::string& d) {
    if (d == "bf16" || d == "f16") return 2;
    if (d == "f32") return 4;
    if (d == "i8" || d == "u8") return 1;
    if (d == "i64") return 8;
    return 0;
}

// places for `picks` sorted picks of up to `experts` experts, every expert's list starting at a multiple of UQ_G; bytes of their planes
static size_t q4_slots(int picks, int experts) { return ((size_t)picks + (size_t)(UQ_G - 1) * std::min(experts, picks) + UQ_G - 1) / UQ_G * UQ_G; }
static size_t q4_plane_bytes(size_t slots, int K) { return (size_t)((K + UQ_KB - 1) / UQ_KB) * (slots / UQ_G) * UQ_GBYTES; }
constexpr int g_tc_warps = 16;   // compute warps per block of k_tcgemv
static int down_row_blocks(int D) { return (D + DOWN_ROWS - 1) / DOWN_ROWS; }

}  // namespace b2

using namespace b2;

constexpr int STEP1_AHEAD = 2;      // steps that an engine queues while others take turns with it on its device

struct b2_engine {
    Cfg c;
    int device = 0, B = 1, cap = 0, nsm = 148;
    bool kv_f32 = false;
    int ep_rank = 0, ep_world = 1;
    std::string err, desc;
    std::map<std::string, DevTensor> t;
    std::vector<LayerW> layers;
    const uint16_t *embed = nullptr, *norm = nullptr;
    QWd lm_head;
    bool finished = false;
    size_t weight_bytes = 0;
    std::string gpu_name;

    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int launches = 0;

    // state
    float *conv = nullptr, *state = nullptr;
    size_t conv_bytes = 0, state_bytes = 0;
    float* snap_conv[2] = {nullptr, nullptr};
    float* snap_state[2] = {nullptr, nullptr};
    long snap_pos[2] = {-1, -1};
    void *kpool = nullptr, *vpool = nullptr;
    int* page_table = nullptr;
    int pages_per_seq = 0;
    float *rope_cos = nullptr, *rope_sin = nullptr;
    int length = 0;
    // the tokens fed so far (one sequence), for saved states; unknown after steps whose tokens stayed on the device
    std::vector<uint32_t> toks;
    bool toks_known = true;
    std::string fingerprint;      // names the weights (NxFile::fingerprint); empty when built from tensors

    // per-step device scalars and work buffers
    int *d_tok = nullptr, *d_next = nullptr, *d_pos = nullptr, *d_err = nullptr;
    int* d_hist = nullptr;                  // [cap][B] the arg-max after every position
    unsigned int* d_counter = nullptr;      // [B] gemv finishers
    unsigned int* d_acounter = nullptr;     // [B][KV] attention merge
    float *x = nullptr, *big = nullptr, *zbuf = nullptr, *kraw = nullptr, *vraw = nullptr, *beta = nullptr, *gdec = nullptr;
    float *obuf = nullptr, *att = nullptr, *rlogits = nullptr, *sh_act = nullptr, *sgate = nullptr, *act = nullptr, *logits = nullptr;
    int* top_idx = nullptr;                  // [L][B][TOPK]
    float* top_w = nullptr;
    float* part_val = nullptr;
    int* part_idx = nullptr;
    float* attn_part = nullptr;
    __half* xh = nullptr;                    // [Tpad][2][4096] fp16 activations for the tensor-core path
    int xh_tpad = 0;
    int8_t* uq_i = nullptr;                  // [passes][3][64][4096] int8 digit planes for the tcgen05 GEMM
    uint16_t* uq_b = nullptr;                // [passes][3][64][4096] bf16 planes
    float* uq_scale = nullptr;               // [passes * 64]
    int uq_passes = 0;
    // grouped expert GEMM: picks sorted by expert, chunk table, fp16 expert activations, group sums
    int *g_list = nullptr, *g_slot = nullptr, *g_chunk = nullptr;
    __half* acth = nullptr;
    float *xsum_tok = nullptr, *xsum_act = nullptr;
    uint8_t* sq = nullptr; float *sq_scale = nullptr, *sq_sum = nullptr;   // planes of the sorted picks (k_umma_q4)
    int cap_small = 0, cap_big = 0;
    const uint8_t** top_ptr = nullptr;       // [B][TOPK] expert blobs of the current layer's picks (k_moe_gu1 -> k_moe_down1)
    int8_t* actq = nullptr;                  // [B * TOPK][4][I] digit planes of act
    float *asc = nullptr, *asum = nullptr;   // [B * TOPK][I / 32] scale and sum of each 32-value group of act
    unsigned long long* d_trace = nullptr;   // step timeline slots, allocated by the first b2_debug_trace_step
    float* ypart = nullptr;                  // [B][TOPK + 1][D]
    unsigned int* d_dcounter = nullptr;      // [B][row blocks of the expert down projection]
    int nsplit = 1, head_grid = 1;
    int attn_tiles = 1;                      // 64-position tiles a slice of the longest context spans
    uint32_t* h_pin = nullptr;               // pinned staging [B]
    std::vector<int> tap_layers;
    float* tap_buf = nullptr;
    uint64_t hits = 0;
    // core engine: switch-on counts per layer and core, the picks of the current layer, its score rows, the live cores' output
    int* d_counts = nullptr;                 // [L][n1 * n2]
    int* csel = nullptr; float* cselw = nullptr;      // [B][cores_active]
    float *cscore = nullptr, *core_y = nullptr;       // [B][n1 + n2], [B][D]
    int live_cores = 0;
    // expert parallelism (ep_world > 1): NCCL is resolved at run time from the library the process
    // already has loaded (torch's), so that one process never holds two NCCL versions
    void* nccl_lib = nullptr;
    ncclComm_t comm = nullptr;
    ncclResult_t (*p_ncclGetUniqueId)(ncclUniqueId*) = nullptr;
    ncclResult_t (*p_ncclCommInitRank)(ncclComm_t*, int, ncclUniqueId, int) = nullptr;
    ncclResult_t (*p_ncclCommDestroy)(ncclComm_t) = nullptr;
    ncclResult_t (*p_ncclAllGather)(const void*, void*, size_t, ncclDataType_t, ncclComm_t, cudaStream_t) = nullptr;
    ncclResult_t (*p_ncclSend)(const void*, size_t, ncclDataType_t, int, ncclComm_t, cudaStream_t) = nullptr;
    ncclResult_t (*p_ncclRecv)(void*, size_t, ncclDataType_t, int, ncclComm_t, cudaStream_t) = nullptr;
    ncclResult_t (*p_ncclGroupStart)() = nullptr;
    ncclResult_t (*p_ncclGroupEnd)() = nullptr;
    const char* (*p_ncclGetErrorString)(ncclResult_t) = nullptr;
    float *rec_local = nullptr, *rec_all = nullptr, *recv_y = nullptr;
    // exchange by peer stores: rec_all | recv_y | flags are one block that the other ranks map (cudaIpc)
    float* ep_block = nullptr;
    size_t ep_block_floats = 0, ep_flag_off = 0;
    float* ep_peer[EP_MAX_WORLD] = {};
    bool ep_peer_ready = false;
    int* d_ep_seq = nullptr;
    unsigned long long* d_ep_rows = nullptr;
    long ep_steps = 0;
    int load_nccl();
    int ep_exchange_records(cudaStream_t st);
    int ep_exchange_outputs(cudaStream_t st);

    // Prompt chunks (b2_feed of 16 or more tokens): the step's kernels with the chunk's tokens as the columns, on a work
    // buffer set of its own, allocated for the longest chunk that has come in so far.
    struct ChunkBufs {
        int W = 0;                                  // tokens the buffers hold
        char* arena = nullptr;                      // the allocation they all lie in
        int *tok = nullptr, *vpos = nullptr;        // [W] token ids, positions pos0 + t
        float *x = nullptr, *big = nullptr, *qkv = nullptr, *zbuf = nullptr, *kraw = nullptr, *vraw = nullptr, *beta = nullptr, *gdec = nullptr;
        float *obuf = nullptr, *att = nullptr, *rlogits = nullptr, *sh_act = nullptr, *sgate = nullptr, *act = nullptr;
        int* top_idx = nullptr; float* top_w = nullptr;
        float *ypart = nullptr, *attn_part = nullptr;
        unsigned int *dcounter = nullptr, *counter = nullptr;
        __half *xh = nullptr, *acth = nullptr;
        int xh_tpad = 0;
        int8_t* uq_i = nullptr; uint16_t* uq_b = nullptr; float* uq_scale = nullptr; int uq_passes = 0;
        int *g_list = nullptr, *g_slot = nullptr, *g_chunk = nullptr;
        float *xsum_tok = nullptr, *xsum_act = nullptr;
        uint8_t* sq = nullptr; float *sq_scale = nullptr, *sq_sum = nullptr;
        int cap_small = 0, cap_big = 0, nsplit = 1, attn_tiles = 1;
        int* csel = nullptr; float *cselw = nullptr, *cscore = nullptr, *core_y = nullptr;
    } pc;
    void free_chunk_bufs();
    int ensure_chunk_bufs(int T);
    int feed_chunk(const uint32_t* ids, int T, bool want_head);

    // The persistent launch that runs a whole step of one sequence (step1.cuh), where the shapes allow it
    struct Step1 {
        const void* kernel = nullptr;               // null: steps run as one launch per stage
        size_t smem = 0;
        bool off = false;                           // the tapped layers do not allow it
        int stages = 0;                             // stages of a step: rows of its timeline
        Step1Layer* layers = nullptr;
        uint32_t *tiles = nullptr, *epoch = nullptr;
        S1Copy* copies = nullptr;
        uint64_t* ll = nullptr;
        cudaEvent_t done[STEP1_AHEAD] = {};         // behind this engine's latest steps, in turn
        unsigned steps = 0;
        Step1Args args{};
    } s1;
    int plan_step1();
    int upload_step1();
    int launch_step1(cudaStream_t st);
    cudaError_t run_graph(cudaGraphExec_t g);
    cudaError_t await_turn();
    bool use_step1() const { return s1.kernel && !s1.off && !profiling; }

    // per-kernel timing (b2_profile_step): one event after every launch of an un-graphed step
    bool profiling = false;
    std::vector<cudaEvent_t> prof_ev;
    std::vector<int> prof_class;
    size_t prof_used = 0;
    void mark(int cls, cudaStream_t st) {
        if (!profiling) return;
        if (prof_used == prof_ev.size()) { cudaEvent_t e; cudaEventCreate(&e); prof_ev.push_back(e); prof_class.push_back(0); }
        prof_class[prof_used] = cls;
        cudaEventRecord(prof_ev[prof_used++], st);
    }
    void class_bytes(double out[8]) const;

    int fail(const char* fmt, ...) {
        char buf[1024];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        err = buf;
        return 1;
    }
    ~b2_engine();
    int parse_config(const JValue& j);
    int put(const std::string& name, const std::string& dtype, const std::vector<int64_t>& shape, const void* data,
            size_t nbytes, bool on_device);
    int finish();
    int need(const std::string& name, const std::string& dtype, std::vector<int64_t> shape, const void** out);
    int qw(const std::string& prefix, int n, int k, QWd* out);
    int build_graph();
    int enqueue_step(cudaStream_t st, bool count, int chunk_T = 0, bool chunk_head = false);
    int run_steps(int n);
    int check_device_error();
    int reset_state();
    std::string state_key() const;
    struct Piece { char* p; size_t bytes; };
    std::vector<Piece> state_pieces(int n) const;
};

static void enter_step1(b2_engine* e);
static void leave_step1(b2_engine* e);
b2_engine::~b2_engine() {
    if (t.empty() && !finished) return;   // nothing was ever allocated (e.g. creation was refused)
    cudaSetDevice(device);
    leave_step1(this);
    if (ep_peer_ready) for (int p = 0; p < ep_world; p++) if (p != ep_rank && ep_peer[p]) cudaIpcCloseMemHandle(ep_peer[p]);
    if (graph) cudaGraphExecDestroy(graph);
    for (auto& kv : t) cudaFree(kv.second.p);
    for (auto& l : layers) { cudaFree((void*)l.eptr); cudaFree(l.router_bias); cudaFree(l.live); }
    void* bufs[] = {conv, state, snap_conv[0], snap_conv[1], snap_state[0], snap_state[1], kpool, vpool, page_table, rope_cos,
                    rope_sin, d_tok, d_next, d_pos, d_err, d_hist, d_counter, d_acounter, x, big, zbuf, kraw, vraw, beta, gdec, obuf, att,
                    rlogits, sh_act, sgate, act, logits, top_idx, top_w, part_val, part_idx, attn_part, tap_buf, ypart, d_dcounter, rec_local, ep_block, d_ep_seq, d_ep_rows, xh, g_list, g_slot, g_chunk, acth, xsum_tok, xsum_act, sq, sq_scale, sq_sum, d_trace, (void*)top_ptr, actq, asc, asum, uq_i, uq_b, uq_scale, d_counts, csel, cselw, cscore, core_y,
                    s1.layers, s1.tiles, s1.copies, s1.epoch, s1.ll};
    for (void* p : bufs) cudaFree(p);
    free_chunk_bufs();
    if (h_pin) cudaFreeHost(h_pin);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    for (cudaEvent_t e : s1.done) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : prof_ev) cudaEventDestroy(e);
    if (comm && p_ncclCommDestroy) p_ncclCommDestroy(comm);
    if (stream) cudaStreamDestroy(stream);
}

// HConfig::from_header + check (aegist_rs/src/hybrid.rs:53-120), with this engine's own shape limits.
int b2_engine::parse_config(const JValue& j) {
    auto num = [&](const char* k, double* out) -> bool {
        const JValue* v = j.get(k);
        if (!v || !v->is_num()) { fail("config is missing %s", k); return false; }
        *out = v->num;
        return true;
    };
    double d;
#define GETI(field, key) if (!num(key, &d)) return 1; c.field = (int)d;
    GETI(V, "vocab_size") GETI(D, "d_model") GETI(L, "n_layers") GETI(H, "n_heads") GETI(KV, "n_kv_heads")
    GETI(HD, "head_dim") GETI(RD, "rotary_dim") GETI(HK, "lin_k_heads") GETI(HV, "lin_v_heads") GETI(DK, "lin_k_dim")
    GETI(DV, "lin_v_dim") GETI(CK, "conv_kernel") GETI(E, "n_experts") GETI(TOPK, "experts_active")
    GETI(I, "expert_hidden") GETI(SH, "shared_hidden") GETI(G, "expert_group") GETI(rank, "core_rank")
    GETI(cores_active, "cores_active")
#undef GETI
    if (!num("rope_theta", &c.theta)) return 1;
    if (!num("norm_eps", &d)) return 1;
    c.eps = (float)d;
    const JValue* lt = j.get("layer_types");
    if (!lt || lt->type != JValue::Arr) return fail("config is missing layer_types");
    for (auto& k : lt->arr) c.attn.push_back(k.type == JValue::Str && k.str == "attn");
    const JValue* grid = j.get("core_grid");
    if (!grid || grid->type != JValue::Arr || grid->arr.size() != 2) return fail("config is missing core_grid");
    c.n1 = (int)grid->arr[0].num;
    c.n2 = (int)grid->arr[1].num;
    const JValue* tie = j.get("tie_embeddings");
    if (tie && tie->type == JValue::Bool && tie->b) return fail("this engine build needs an untied output head");
    const JValue* arch = j.get("arch");
    if (arch && arch->type == JValue::Str && arch->str != "hybrid-moe") return fail("arch %s is not hybrid-moe", arch->str.c_str());
    for (const char* k : {"hc_count"}) {
        const JValue* v = j.get(k);
        if (v && v->is_num() && v->num > 1) return fail("this engine does not run brains with hyper-connections (hc_count > 1)");
    }
    const JValue* ef = j.get("expert_format");
    if (ef && ef->type == JValue::Str && ef->str != "q4") return fail("expert_format %s is not q4", ef->str.c_str());

    std::string bad;
    auto add = [&](const std::string& s) { bad += (bad.empty() ? "" : "; ") + s; };
    if ((int)c.attn.size() != c.L) add("layer_types length");
    if (c.V < 1 || c.L < 1) add("empty model");
    if (c.D % 64 != 0 || c.D < 64 || c.D > 2048) add("d_model must be a multiple of 64, at most 2048");
    if (!(c.HD == 64 || c.HD == 128 || c.HD == 256) || c.RD > c.HD || c.RD % 2 != 0 || c.RD < 2) add("head_dim must be 64/128/256 and rotary_dim even <= head_dim");
    if (c.KV < 1 || c.H % std::max(c.KV, 1) != 0 || c.H / std::max(c.KV, 1) > 8) add("n_heads must be a multiple of n_kv_heads with at most 8 query heads per KV head");
    if (!(c.DK == 64 || c.DK == 128) || c.DV % 32 != 0 || c.DV > 256 || c.HK < 1 || c.HV % std::max(c.HK, 1) != 0 || c.CK != 4) add("DeltaNet needs lin_k_dim 64/128, lin_v_dim a multiple of 32, hv % hk == 0, conv kernel 4");
    if (c.H * c.HD > 4096 || c.VD() > 4096 || (c.H * c.HD) % 32 != 0 || c.VD() % 32 != 0) add("mixer width above 4096");
    if (c.C() % 2 != 0) add("odd conv width");
    if (c.E > 256 || c.E < 1 || c.TOPK > 8 || c.TOPK < 1 || c.TOPK > c.E || c.G != 64 || c.I % 64 != 0 || c.I > 512 || c.I < 64) add("experts need n_experts <= 256, top-k <= 8, group 64, hidden a multiple of 64 up to 512");
    if (c.SH % 16 != 0 || c.SH > 512 || c.SH < 16) add("shared_hidden must be a multiple of 16 up to 512");
    if (c.E % ep_world != 0) add("n_experts not divisible by the number of expert-parallel ranks");
    if (c.n1 < 1 || c.n2 < 1 || c.n1 > 128 || c.n2 > 128 || c.cores_active < 1 || c.cores_active > 8 || c.rank < 1 || c.rank > 256)
        add("core engine needs a grid of at most 128 x 128, 1 to 8 active cores, rank up to 256");
    if (!bad.empty()) return fail("this engine build does not support this brain's shape: %s", bad.c_str());
    return 0;
}

int b2_engine::put(const std::string& name, const std::string& dtype, const std::vector<int64_t>& shape, const void* data,
                   size_t nbytes, bool on_device) {
    if (finished) return fail("b2_put_tensor after b2_finish");
    size_t es = dtype_size(dtype);
    if (!es) return fail("%s: unsupported dtype %s", name.c_str(), dtype.c_str());
    size_t n = es;
    for (auto s : shape) n *= (size_t)s;
    if (n != nbytes) return fail("%s: %zu bytes given, shape says %zu", name.c_str(), nbytes, n);
    CU(cudaSetDevice(device));
    DevTensor d;
    d.dtype = dtype;
    d.shape = shape;
    const char* src = (const char*)data;
    // expert-parallel: keep only this rank's rows of the packed experts
    bool is_experts = name.size() > 15 && name.rfind(".moe.experts.q4") == name.size() - 15;
    if (is_experts && ep_world > 1) {
        if (shape.size() != 2 || shape[0] != c.E) return fail("%s: expected [%d, expert_bytes]", name.c_str(), c.E);
        size_t per = (size_t)c.E / ep_world;
        src += per * ep_rank * (size_t)shape[1];
        nbytes = per * (size_t)shape[1];
        d.shape[0] = (int64_t)per;
    }
    d.nbytes = nbytes;
    if (t.count(name)) { cudaFree(t[name].p); weight_bytes -= t[name].nbytes; }
    CU(cudaMalloc(&d.p, std::max<size_t>(nbytes, 16)));
    if (nbytes) CU(cudaMemcpy(d.p, src, nbytes, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
    weight_bytes += nbytes;
    t[name] = d;
    return 0;
}

int b2_engine::need(const std::string& name, const std::string& dtype, std::vector<int64_t> shape, const void** out) {
    auto it = t.find(name);
    if (it == t.end()) return fail("the brain has no tensor %s", name.c_str());
    const DevTensor& d = it->second;
    bool same = d.dtype == dtype && d.shape.size() == shape.size();
    for (size_t i = 0; same && i < shape.size(); i++) same = d.shape[i] == shape[i];
    if (!same) {
        std::string got = d.dtype + " [", want = dtype + " [";
        for (auto s : d.shape) got += std::to_string(s) + ",";
        for (auto s : shape) want += std::to_string(s) + ",";
        return fail("%s is %s], expected %s]", name.c_str(), got.c_str(), want.c_str());
    }
    *out = d.p;
    return 0;
}

int b2_engine::qw(const std::string& prefix, int n, int k, QWd* out) {
    const void *w, *s;
    if (need(prefix + ".qweight", "i8", {n, k}, &w)) return 1;
    if (need(prefix + ".scale", "bf16", {n, 1}, &s)) return 1;
    out->w = (const int8_t*)w;
    out->s = (const uint16_t*)s;
    out->n = n;
    out->k = k;
    return 0;
}

// (zeroed on the default stream: whoever uses it on another one waits for that first)
template <typename T>
static cudaError_t dalloc(T** p, size_t n, bool zero = true) {
    cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(n * sizeof(T), 16));
    if (e == cudaSuccess && zero) e = cudaMemset(*p, 0, std::max<size_t>(n * sizeof(T), 16));
    return e;
}

int b2_engine::finish() {
    if (finished) return fail("b2_finish called twice");
    CU(cudaSetDevice(device));
    cudaDeviceProp prop;
    CU(cudaGetDeviceProperties(&prop, device));
    nsm = prop.multiProcessorCount;
    gpu_name = prop.name;
    const void* p;
#define NEED(dst, name, dtype, ...) if (need(name, dtype, {__VA_ARGS__}, &p)) return 1; dst = (decltype(dst))p;
    NEED(embed, "embed.weight", "bf16", c.V, c.D)
    NEED(norm, "norm.weight", "bf16", c.D)
    if (qw("lm_head", c.V, c.D, &lm_head)) return 1;
    int n_attn = 0, n_delta = 0;
    const int per = c.E / ep_world;
    for (int i = 0; i < c.L; i++) {
        LayerW l;
        std::string b = "blocks." + std::to_string(i) + ".";
        l.attn = c.attn[i];
        NEED(l.norm1, b + "norm1.weight", "bf16", c.D)
        NEED(l.norm2, b + "norm2.weight", "bf16", c.D)
        if (l.attn) {
            l.slot = n_attn++;
            NEED(l.q_norm, b + "mixer.q_norm.weight", "bf16", c.HD)
            NEED(l.k_norm, b + "mixer.k_norm.weight", "bf16", c.HD)
            if (qw(b + "mixer.q", 2 * c.H * c.HD, c.D, &l.q) || qw(b + "mixer.k", c.KV * c.HD, c.D, &l.k) ||
                qw(b + "mixer.v", c.KV * c.HD, c.D, &l.v) || qw(b + "mixer.o", c.D, c.H * c.HD, &l.o)) return 1;
        } else {
            l.slot = n_delta++;
            NEED(l.in_a, b + "mixer.in_a.weight", "bf16", c.HV, c.D)
            NEED(l.in_b, b + "mixer.in_b.weight", "bf16", c.HV, c.D)
            NEED(l.conv, b + "mixer.conv", "bf16", c.C(), c.CK)
            NEED(l.a_log, b + "mixer.A_log", "bf16", c.HV)
            NEED(l.dt_bias, b + "mixer.dt_bias", "bf16", c.HV)
            NEED(l.gnorm, b + "mixer.norm.weight", "bf16", c.DV)
            if (qw(b + "mixer.in_qkv", c.C(), c.D, &l.in_qkv) || qw(b + "mixer.in_z", c.VD(), c.D, &l.in_z) ||
                qw(b + "mixer.out", c.D, c.VD(), &l.out)) return 1;
        }
        NEED(l.router, b + "moe.router.weight", "bf16", c.E, c.D)
        NEED(l.sh_gw, b + "moe.shared_gate.weight", "bf16", 1, c.D)
        if (qw(b + "moe.shared.gate", c.SH, c.D, &l.sh_gate) || qw(b + "moe.shared.up", c.SH, c.D, &l.sh_up) ||
            qw(b + "moe.shared.down", c.D, c.SH, &l.sh_down)) return 1;
        NEED(l.experts, b + "moe.experts.q4", "u8", per, (int64_t)c.expert_bytes())
        // the slot table: every expert of this rank is resident at a fixed address
        std::vector<const uint8_t*> tab(c.E, nullptr);
        for (int e = 0; e < per; e++) tab[ep_rank * per + e] = l.experts + (size_t)e * c.expert_bytes();
        CU(cudaMalloc((void**)&l.eptr, c.E * sizeof(void*)));
        CU(cudaMemcpy((void*)l.eptr, tab.data(), c.E * sizeof(void*), cudaMemcpyHostToDevice));
        CU(dalloc(&l.router_bias, c.E));   // zeros: adding them changes no logit; b2_set_router_bias fills them
        if (t.count(b + "engine.key1.weight")) {
            NEED(l.key1, b + "engine.key1.weight", "bf16", c.n1, c.D)
            NEED(l.key2, b + "engine.key2.weight", "bf16", c.n2, c.D)
            // the sparse bank: ids [n] name the cores that are stored; everything else adds nothing
            const int nc = c.n1 * c.n2;
            std::vector<int> map(nc, -1);
            auto it = t.find(b + "cores.ids");
            int n = 0;
            if (it != t.end() && it->second.nbytes) {
                if (it->second.dtype != "i64") return fail("%scores.ids must be i64", b.c_str());
                n = (int)(it->second.nbytes / 8);
                std::vector<int64_t> ids(n);
                CU(cudaMemcpy(ids.data(), it->second.p, (size_t)n * 8, cudaMemcpyDeviceToHost));
                for (int j = 0; j < n; j++) {
                    if (ids[j] < 0 || ids[j] >= nc) return fail("%scores.ids: core id %lld is outside the %d x %d grid", b.c_str(), (long long)ids[j], c.n1, c.n2);
                    map[(size_t)ids[j]] = j;
                }
                NEED(l.cg, b + "cores.gate", "bf16", n, c.D, c.rank)
                NEED(l.cu, b + "cores.up", "bf16", n, c.D, c.rank)
                NEED(l.cd, b + "cores.down", "bf16", n, c.rank, c.D)
            }
            l.n_live = n;
            live_cores += n;
            CU(dalloc(&l.live, nc, false));
            CU(cudaMemcpy(l.live, map.data(), (size_t)nc * 4, cudaMemcpyHostToDevice));
        }
        layers.push_back(l);
    }
#undef NEED
    // context, recurrent state, snapshots (aegist_rs/src/hybrid.rs:606-625)
    if (cap <= 0) cap = 32768;
    pages_per_seq = (cap + KV_PAGE - 1) / KV_PAGE;
    const size_t kv_elems = (size_t)std::max(n_attn, 1) * B * pages_per_seq * c.KV * KV_PAGE * c.HD;
    const size_t kvb = kv_f32 ? 4 : 2;
    cudaError_t e1 = cudaMalloc(&kpool, kv_elems * kvb), e2 = cudaMalloc(&vpool, kv_elems * kvb);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return fail("KV cache for %d tokens x %d sequences: %s", cap, B, cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
    CU(cudaMemset(kpool, 0, kv_elems * kvb));
    CU(cudaMemset(vpool, 0, kv_elems * kvb));
    {
        // identity page table: sequence b owns pages [b * pages_per_seq, (b+1) * pages_per_seq) of each layer's pool
        std::vector<int> pt((size_t)B * pages_per_seq);
        for (size_t i = 0; i < pt.size(); i++) pt[i] = (int)i;
        CU(dalloc(&page_table, pt.size(), false));
        CU(cudaMemcpy(page_table, pt.data(), pt.size() * 4, cudaMemcpyHostToDevice));
    }
    conv_bytes = (size_t)std::max(n_delta, 1) * B * c.C() * 3 * 4;
    state_bytes = (size_t)std::max(n_delta, 1) * B * c.HV * c.DK * c.DV * 4;
    CU(dalloc((char**)&conv, conv_bytes));
    CU(dalloc((char**)&state, state_bytes));
    for (int s = 0; s < 2; s++) {
        CU(dalloc((char**)&snap_conv[s], conv_bytes));
        CU(dalloc((char**)&snap_state[s], state_bytes));
    }
    {
        // RoPE tables as the Python reference builds them (aegist/hybrid.py:152-157): fp32 angle =
        // fp32(position) * fp32(1 / fp32(theta^(2j/rd))); the power in double reproduces torch's fp32 pow.
        const int hr = c.RD / 2;
        std::vector<float> cs((size_t)cap * hr), sn((size_t)cap * hr);
        for (int j = 0; j < hr; j++) {
            const float ex = (float)(2 * j) / (float)c.RD;
            const float pw = (float)std::pow((double)(float)c.theta, (double)ex);
            const float inv = 1.0f / pw;
            for (int pos = 0; pos < cap; pos++) {
                const float ang = (float)pos * inv;
                cs[(size_t)pos * hr + j] = (float)std::cos((double)ang);
                sn[(size_t)pos * hr + j] = (float)std::sin((double)ang);
            }
        }
        CU(dalloc(&rope_cos, cs.size(), false));
        CU(dalloc(&rope_sin, sn.size(), false));
        CU(cudaMemcpy(rope_cos, cs.data(), cs.size() * 4, cudaMemcpyHostToDevice));
        CU(cudaMemcpy(rope_sin, sn.data(), sn.size() * 4, cudaMemcpyHostToDevice));
    }
    // work buffers
    const int bigw = std::max(2 * c.H * c.HD, c.C());
    CU(dalloc(&d_tok, B)); CU(dalloc(&d_next, B)); CU(dalloc(&d_pos, B)); CU(dalloc(&d_err, 1)); CU(dalloc(&d_hist, (size_t)cap * B));
    CU(dalloc(&d_counter, B)); CU(dalloc(&d_acounter, (size_t)B * c.KV));
    CU(dalloc(&x, (size_t)B * c.D)); CU(dalloc(&big, (size_t)B * bigw)); CU(dalloc(&zbuf, (size_t)B * c.VD()));
    CU(dalloc(&kraw, (size_t)B * c.KV * c.HD)); CU(dalloc(&vraw, (size_t)B * c.KV * c.HD));
    CU(dalloc(&beta, (size_t)B * c.HV)); CU(dalloc(&gdec, (size_t)B * c.HV));
    CU(dalloc(&obuf, (size_t)B * c.VD())); CU(dalloc(&att, (size_t)B * c.H * c.HD));
    CU(dalloc(&rlogits, (size_t)B * c.E)); CU(dalloc(&sh_act, (size_t)B * c.SH)); CU(dalloc(&sgate, B));
    const size_t Bg = (size_t)B * ep_world;   // sequences whose picks may land on this GPU's experts
    CU(dalloc(&act, Bg * c.TOPK * c.I)); CU(dalloc(&logits, (size_t)B * c.V));
    CU(dalloc(&top_idx, (size_t)c.L * B * c.TOPK)); CU(dalloc(&top_w, (size_t)c.L * B * c.TOPK));
    CU(dalloc(&top_ptr, (size_t)B * c.TOPK));
    CU(dalloc(&actq, (size_t)B * c.TOPK * M1_PLANES * c.I));
    CU(dalloc(&asc, (size_t)B * c.TOPK * std::max(1, c.I / 32))); CU(dalloc(&asum, (size_t)B * c.TOPK * std::max(1, c.I / 32)));
    head_grid = std::min((c.V + 31) / 32, nsm);
    CU(dalloc(&part_val, (size_t)B * head_grid)); CU(dalloc(&part_idx, (size_t)B * head_grid));
    // attention: enough slices to fill the GPU, but at least 64 positions each at full context. With many sequences the
    // GPU is full anyway; slices of about 8 tiles then keep the blocks short, so that they spread evenly over the SMs
    // (an SM holds one block: 2 x 64 x 2 blocks of 64 tiles each were two uneven waves, 295 us per layer at context 8192)
    nsplit = std::max(1, std::min({64, std::max((2 * nsm) / std::max(1, c.KV * B), (cap + 8 * AM_TILE - 1) / (8 * AM_TILE)), (cap + 63) / 64}));
    if (const char* v = getenv("B2_ATTN_SPLITS")) nsplit = std::max(1, std::min(64, atoi(v)));   // for tests: long slices at short contexts
    attn_tiles = ((cap + nsplit - 1) / nsplit + AM_TILE - 1) / AM_TILE;
    CU(dalloc(&attn_part, (size_t)B * c.KV * nsplit * (c.H / c.KV) * (c.HD + 2)));
    if ((int)Bg >= BATCH_GEMM_MIN) {
        xh_tpad = ((int)Bg + MM_TOK - 1) / MM_TOK * MM_TOK;
        CU(dalloc((uint16_t**)&xh, (size_t)xh_tpad * 2 * 4096));
        uq_passes = ((int)Bg + UM_TOK - 1) / UM_TOK;
        CU(dalloc(&uq_i, (size_t)uq_passes * UM_PI * UM_TOK * 4096));
        CU(dalloc(&uq_b, (size_t)uq_passes * UM_PB * UM_TOK * 4096));
        CU(dalloc(&uq_scale, (size_t)uq_passes * UM_TOK));
        const size_t P = Bg * c.TOPK;
        cap_small = (int)std::min<size_t>(P, c.E / ep_world);
        cap_big = (int)(P / (GQ_SMALL + 1)) + 1;
        CU(dalloc(&g_list, q4_slots((int)P, c.E / ep_world))); CU(dalloc(&g_slot, P));
        CU(dalloc(&g_chunk, (size_t)3 * (cap_small + cap_big) + 2));
        CU(dalloc((uint16_t**)&acth, P * 2 * c.I));
        CU(dalloc(&xsum_tok, Bg * (c.D / 64)));
        CU(dalloc(&xsum_act, P * std::max(1, c.I / 64)));
        const size_t slots = q4_slots((int)P, c.E / ep_world);
        CU(dalloc(&sq, q4_plane_bytes(slots, std::max(c.D, c.I))));
        CU(dalloc(&sq_scale, slots)); CU(dalloc(&sq_sum, slots * (size_t)(std::max(c.D, c.I) / 64 + 1)));
    }
    CU(dalloc(&ypart, Bg * (c.TOPK + 1) * c.D));
    CU(dalloc(&d_dcounter, Bg * down_row_blocks(c.D)));
    CU(dalloc(&d_counts, (size_t)c.L * c.n1 * c.n2));
    CU(dalloc(&csel, (size_t)B * c.cores_active)); CU(dalloc(&cselw, (size_t)B * c.cores_active));
    CU(dalloc(&cscore, (size_t)B * (c.n1 + c.n2))); CU(dalloc(&core_y, (size_t)B * c.D));
    if (ep_world > 1) {
        const size_t rw = c.D + 2 * c.TOPK;
        CU(dalloc(&rec_local, (size_t)B * rw));
        const size_t nrec = (Bg * rw + 63) / 64 * 64, ny = Bg * (c.TOPK + 1) * c.D;
        ep_flag_off = nrec + ny;
        ep_block_floats = ep_flag_off + 2 * EP_MAX_WORLD * EP_MAX_BLOCKS;
        CU(dalloc(&ep_block, ep_block_floats));
        CU(cudaMemset(ep_block, 0, ep_block_floats * sizeof(float)));
        rec_all = ep_block; recv_y = ep_block + nrec;
        CU(dalloc(&d_ep_seq, 2)); CU(dalloc(&d_ep_rows, 1));
    }
    CU(cudaMallocHost((void**)&h_pin, (std::max(B, 1) * 2 + 1) * sizeof(uint32_t)));   // ids | arg-max | device error word
    CU(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    CU(cudaEventCreate(&ev0));
    CU(cudaEventCreate(&ev1));
    finished = true;
    char buf[512];
    size_t kv_bytes = 2 * kv_elems * kvb;
    snprintf(buf, sizeof(buf), "%s: %.2f GB of weights in HBM (%d of %d experts resident%s), %d live cores, context %d tokens x %d, KV %s %.2f GB",
             gpu_name.c_str(), weight_bytes / 1e9, c.L * per, c.L * c.E, ep_world > 1 ? " on this rank" : "", live_cores, cap, B,
             kv_f32 ? "fp32" : "bf16", kv_bytes / 1e9);
    desc = buf;
    if (ep_world == 1 && plan_step1()) return 1;
    // everything so far came over the default stream, which the engine's does not wait for. (A wait for the whole device would also be for streams
    // that other threads capture on, which is an error here and breaks their captures)
    CU(cudaStreamSynchronize(cudaStreamLegacy));
    if (ep_world > 1) return 0;   // the step graph holds NCCL calls: it is built by b2_ep_init
    return build_graph();
}


static thread_local int g_launch_count = 0;   // kernels that this thread has launched so far (a step's count is the difference)

// Step timeline (b2_debug_trace_step): while g_trace_base is set, the launch with index i since g_trace_first
// gets the slot g_trace_base + 16 i in its argument struct (structs with a `trace` member; null otherwise). A thread's own: another
// engine's capture meanwhile must not take slots, nor keep pointers to them.
static thread_local unsigned long long* g_trace_base = nullptr;
static thread_local int g_trace_first = 0;
constexpr int TRACE_MAX_LAUNCHES = 4096;
template <typename T>
static auto with_trace(const T& a, int) -> decltype((void)a.trace, T()) {
    T c = a;
    const int i = g_launch_count - 1 - g_trace_first;
    c.trace = (g_trace_base && i >= 0 && i < TRACE_MAX_LAUNCHES) ? g_trace_base + (size_t)16 * i : nullptr;
    return c;
}
template <typename T>
static const T& with_trace(const T& a, long) { return a; }

// `cluster` blocks in a row share a cluster (1: none)
template <typename... KArgs, typename... Args>
static cudaError_t launch_kc(int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    g_launch_count++;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;   // programmatic dependent launch for every kernel of a step
    return cudaLaunchKernelEx(&cfg, kernel, with_trace(args, 0)...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    return launch_kc(1, kernel, grid, block, smem, st, args...);
}

// The limit belongs to the kernel on its device, and engines of several threads ask for different sizes: always all there is. (Set every time: a
// host program may have reset the device between two engines.)
template <typename F>
static cudaError_t opt_in_smem(F* f, size_t bytes) {
    if (bytes <= 32 * 1024) return cudaSuccess;        // the 48 KB that need no opting in hold the kernel's static arrays too
    static std::mutex mutex;
    static std::map<const void*, int> limits;
    std::unique_lock<std::mutex> lock(mutex);
    int& limit = limits[(const void*)f];
    if (!limit) {
        cudaFuncAttributes fa;
        const cudaError_t e = cudaFuncGetAttributes(&fa, (const void*)f);
        if (e != cudaSuccess) return e;
        limit = 227 * 1024 - (int)fa.sharedSizeBytes;
    }
    const int all = limit;
    lock.unlock();
    return cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, all);
}

// k_mma_i8 over `passes` groups of MM_TOK sequences. A grid that gives an SM at most one block (the out projections,
// the MoE-in matrices) is bound by the latency of its K chunks, one after the other: it takes the deeper ring.
static cudaError_t launch_mma_i8(const MmaArgs& m, int passes, int nsm, cudaStream_t st) {
    const dim3 grid(m.total_blocks, passes), block(MM_THREADS);
    const bool deep = m.total_blocks * passes <= nsm && m.K / MM_KC >= MM_STAGES_DEEP;
    const size_t smem = (size_t)(deep ? MM_STAGES_DEEP : MM_STAGES) * MM_STAGE_BYTES;
    cudaError_t e;
    if (deep) { if ((e = opt_in_smem(k_mma_i8<MM_STAGES_DEEP>, smem)) == cudaSuccess) e = launch_k(k_mma_i8<MM_STAGES_DEEP>, grid, block, smem, st, m); }
    else { if ((e = opt_in_smem(k_mma_i8<MM_STAGES>, smem)) == cudaSuccess) e = launch_k(k_mma_i8<MM_STAGES>, grid, block, smem, st, m); }
    return e;
}

// Tensor-core paths for BATCH_GEMM_MIN or more tokens: scratch for the fp16 activations of k_mma_i8, and for the activation planes of
// the tcgen05 GEMM (k_umma: int8 digit planes qi, bf16 planes qb, per-token scales; `passes_max` groups of 64 tokens).
// one_order: every fp32 sum in one order however many tokens there are (prompt chunks: the cut of a prompt changes no bit)
struct BatchCtx { __half* xh; int Tpad; int8_t* qi; uint16_t* qb; float* xscale; int passes_max; bool one_order; };

// cuTensorMapEncodeTiled through the runtime's driver entry point table (no link against libcuda)
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        cudaGetLastError();
        return (PFN_cuTensorMapEncodeTiled_v12000)p;
    }();
    return fn;
}
static thread_local bool g_refuse_maps = false;      // b2_debug_refuse_tensor_maps
static bool encode_byte_map(CUtensorMap* m, int rank, const void* p, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    auto enc = tensor_map_encoder();
    const cuuint32_t es[3] = {1, 1, 1};
    return enc && !g_refuse_maps &&
           enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(p), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// a [rows][row_bytes] byte matrix as a 2-D tensor of bytes; box = 128 bytes x box_rows, 128-byte swizzle, zeros outside
static bool byte_matrix_map(CUtensorMap* m, const void* p, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
    if (!p || ((uintptr_t)p & 15) || row_bytes % 128 != 0 || box_rows > 256) return false;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {UM_BK, box_rows};
    return encode_byte_map(m, 2, p, dims, strides, box);
}
static bool umma_kind(int k) {
    return k == SEG_I8 || k == SEG_I8_CONV || k == SEG_I8_SILU || k == SEG_I8_ACC || k == SEG_I8_GATEUP || k == SEG_I8_ARGMAX ||
           k == SEG_BF || k == SEG_BF_SIGMOID || k == SEG_BF_DECAY;
}
// All segments of a GEMV group for T tokens on the tcgen05 GEMM: planes, then one persistent launch. false = this group
// does not fit it (the caller takes another path); *err carries a launch error.
static long g_umma_launches = 0;      // how many GEMV groups went to k_umma (tests check that the tcgen05 path is the one that runs)
// clusters of `sk` blocks of k_umma<true> that the current GPU runs at the same time
static int split_clusters(int sk) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sk * 64);
    cfg.blockDim = dim3(UM_THREADS);
    cfg.dynamicSmemBytes = UM_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)sk;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (opt_in_smem(k_umma<true>, UM_SMEM) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, k_umma<true>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}

static bool launch_umma(const GemvArgs& a, int T, int nsm, cudaStream_t st, const BatchCtx& bc, cudaError_t* err) {
    *err = cudaSuccess;
    const int passes = (T + UM_TOK - 1) / UM_TOK;
    if (!bc.qi || passes > bc.passes_max || a.K % UM_BK != 0 || a.K > 4096 || a.nseg > GEMV_MAX_SEG || !tensor_map_encoder()) return false;
    UmmaArgs u{};
    bool any_i8 = false, any_bf = false, any_conv = false;
    for (int i = 0; i < a.nseg; i++) {
        const Seg& g = a.seg[i];
        if (!umma_kind(g.kind)) return false;
        any_conv |= g.kind == SEG_I8_CONV;
        const bool isbf = g.kind == SEG_BF || g.kind == SEG_BF_SIGMOID || g.kind == SEG_BF_DECAY;
        const bool pair = g.kind == SEG_I8_GATEUP;
        (isbf ? any_bf : any_i8) = true;
        UmmaSeg& d = u.seg[i];
        d.s = g.s; d.s2 = g.s2; d.bias = g.bias; d.out = g.out; d.rows = g.rows; d.out_stride = g.out_stride;
        d.kind = g.kind == SEG_I8_ARGMAX ? (int)SEG_I8 : g.kind;
        d.units = pair ? (g.rows + 63) / 64 : (g.rows + UM_M - 1) / UM_M;
        u.total_units += d.units;
        const uint64_t rb = isbf ? 2ull * a.K : (uint64_t)a.K;
        if (!byte_matrix_map(&u.wmap[i], g.w, g.rows, rb, 64)) return false;
        if (pair && !byte_matrix_map(&u.wmap2[i], g.w2, g.rows, rb, 64)) return false;
    }
    u.nseg = a.nseg;
    // tokens per unit: a block pulls about 110 GB/s out of L2, so few row blocks are split over the tokens too
    int tt = UM_TOK;
    while (tt > 16 && tt / 2 >= T) tt /= 2;      // no wider than the tokens need: narrow tiles move two K chunks per stage
    while (tt > 16 && u.total_units * passes * ((std::min(T, (int)UM_TOK) + tt - 1) / tt) * 2 <= nsm && T > tt / 2) tt /= 2;
    u.tt = tt;
    if (!byte_matrix_map(&u.xmap_i8, bc.qi, (uint64_t)passes * UM_PI * UM_TOK, a.K, tt)) return false;
    if (!byte_matrix_map(&u.xmap_bf, bc.qb, (uint64_t)passes * UM_PB * UM_TOK, 2ull * a.K, tt)) return false;
    PrepQArgs p{};
    p.x = a.x; p.x_stride = a.x_stride; p.norm_w = a.norm_w; p.gn_w = a.gn_w; p.z = a.z; p.DV = a.DV; p.eps = a.eps;
    p.K = a.K; p.T = T; p.qi = any_i8 ? bc.qi : nullptr; p.qb = any_bf ? bc.qb : nullptr; p.xscale = bc.xscale;
    if ((*err = launch_k(k_prep_q, dim3(passes * UM_TOK), dim3(256), 0, st, p)) != cudaSuccess) return true;
    u.K = a.K; u.T = T; u.passes = passes; u.xscale = bc.xscale;
    u.conv_w = a.conv_w; u.conv_state = a.conv_state; u.a_log = a.a_log; u.dt_bias = a.dt_bias; u.err = a.err;
    const int nsub = passes == 1 ? (std::min(T, (int)UM_TOK) + tt - 1) / tt : UM_TOK / tt;      // as the kernel counts them
    const int items = u.total_units * passes * nsub;
    // Clusters share a unit along K when all of them fit the GPU at once, with at least a stage (two chunks) to a block: with
    // fewer SMs than twice the units a block would have two turns, and the barrier costs more than the shorter K loop saves
    // (bf16 rows are summed in fp32: split, their order follows the token count)
    int sk = 1;
    if (tt == UM_SK_TOK && passes == 1 && !any_conv && !(any_bf && bc.one_order)) {
        static const int fit[3] = {split_clusters(2), split_clusters(4), split_clusters(8)};
        for (int i = 2; i >= 0 && sk == 1; i--) {
            const int c = 2 << i, chunks = a.K / UM_BK;
            if (items * c <= nsm && items <= fit[i] && chunks % c == 0 && chunks / c >= um_kc(UM_SK_TOK)) sk = c;
        }
    }
    if (sk > 1) {
        u.sk = sk;
        if ((*err = opt_in_smem(k_umma<true>, UM_SMEM)) != cudaSuccess) return true;
        *err = launch_kc(sk, k_umma<true>, dim3(items * sk), dim3(UM_THREADS), UM_SMEM, st, u);
    } else {
        if ((*err = opt_in_smem(k_umma<false>, UM_SMEM)) != cudaSuccess) return true;
        *err = launch_k(k_umma<false>, dim3(std::max(1, std::min(items, nsm))), dim3(UM_THREADS), UM_SMEM, st, u);
    }
    g_umma_launches++;
    return true;
}
static void seal(GemvArgs& a, int K);

static cudaError_t launch_gemv(const GemvArgs& a0, int B, int nsm, cudaStream_t st, int grid_override = 0,
                               const BatchCtx* bc = nullptr) {
    GemvArgs a = a0;
    if (a.x_stride == 0) a.x_stride = a.K;
    cudaError_t e;
    if (bc && B >= BATCH_GEMM_MIN && launch_umma(a, B, nsm, st, *bc, &e)) {
        // every matrix of the group went to the tcgen05 GEMM; the head's arg-max and the router's top-8 are launches of their own
        if (e != cudaSuccess) return e;
        for (int i = 0; i < a.nseg; i++)
            if (a.seg[i].kind == SEG_I8_ARGMAX && a.finisher == FIN_ARGMAX) {
                e = launch_k(k_argmax_rows, dim3(B), dim3(1024), 0, st, (const float*)a.seg[i].out, a.seg[i].rows, a.seg[i].out_stride, a.next_tok, a.pos, a.hist, a.tok);
                if (e != cudaSuccess) return e;
            }
        if (a.finisher == FIN_TOPK)
            e = launch_k(k_router_topk, dim3((B + 3) / 4), dim3(256), 0, st, (const float*)a.seg[0].out, a.seg[0].out_stride, a.E, a.topk,
                         a.top_idx, a.top_w, B, a.core);
        return e;
    }
    if (bc && bc->xh && B >= BATCH_GEMM_MIN && B <= bc->Tpad && a.K % MM_KC == 0) {
        // int8 matrices (except the head with its arg-max) go to the tensor cores; bf16 rows stay on k_rowgemv
        MmaArgs m{};
        GemvArgs rest = a;
        rest.nseg = 0;
        const float* argmax_logits = nullptr;
        int argmax_rows = 0, argmax_stride = 0;
        bool topk_moved = false;
        for (int i = 0; i < a.nseg; i++) {
            const Seg& g = a.seg[i];
            // the head's rows are multiplied like any int8 matrix; its arg-max runs as a kernel of its own over the logits
            const bool i8 = g.kind == SEG_I8 || g.kind == SEG_I8_CONV || g.kind == SEG_I8_SILU || g.kind == SEG_I8_ACC || g.kind == SEG_I8_GATEUP ||
                            (g.kind == SEG_I8_ARGMAX && a.finisher == FIN_ARGMAX) ||
                            // bf16 rows (router, DeltaNet a/b, shared gate) are widened to fp16 in registers; the router's
                            // top-8 then runs as a launch of its own
                            ((g.kind == SEG_BF_SIGMOID || g.kind == SEG_BF_DECAY || g.kind == SEG_BF) && a.K % (MM_KC / 2) == 0);
            if (i8 && m.nseg < 4) {
                if (g.kind == SEG_BF && a.finisher == FIN_TOPK && i == 0) topk_moved = true;
                MmaSeg& d = m.seg[m.nseg++];
                d.w = (const int8_t*)g.w; d.s = g.s; d.w2 = (const int8_t*)g.w2; d.s2 = g.s2; d.out = g.out; d.rows = g.rows; d.bias = g.bias;
                d.kind = g.kind == SEG_I8_ARGMAX ? (int)SEG_I8 : g.kind; d.out_stride = g.out_stride;
                if (g.kind == SEG_I8_ARGMAX) { argmax_logits = g.out; argmax_rows = g.rows; argmax_stride = g.out_stride; }
                const int rpb = g.kind == SEG_I8_GATEUP ? MM_ROWS / 2 : MM_ROWS;
                d.blocks = (g.rows + rpb - 1) / rpb;
                m.total_blocks += d.blocks;
            } else {
                rest.seg[rest.nseg++] = g;
            }
        }
        if (m.nseg > 0) {
            PrepArgs p{};
            p.x = a.x; p.x_stride = a.x_stride; p.norm_w = a.norm_w; p.gn_w = a.gn_w; p.z = a.z; p.DV = a.DV; p.eps = a.eps;
            p.K = a.K; p.T = B; p.out = bc->xh; p.Tpad = (B + MM_TOK - 1) / MM_TOK * MM_TOK;
            e = launch_k(k_prep_x, dim3(p.Tpad), dim3(256), 0, st, p);
            if (e != cudaSuccess) return e;
            m.xh = bc->xh; m.K = a.K; m.T = B; m.conv_w = a.conv_w; m.conv_state = a.conv_state; m.a_log = a.a_log; m.dt_bias = a.dt_bias;
            e = launch_mma_i8(m, p.Tpad / MM_TOK, nsm, st);
            if (e != cudaSuccess) return e;
            if (argmax_logits) {
                e = launch_k(k_argmax_rows, dim3(B), dim3(1024), 0, st, argmax_logits, argmax_rows, argmax_stride, a.next_tok, a.pos, a.hist, a.tok);
                if (e != cudaSuccess) return e;
            }
            if (topk_moved) {
                // the picks need every score row: what this kernel did not take (beyond its four matrices) is multiplied first
                if (rest.nseg > 0) {
                    rest.finisher = FIN_NONE;
                    rest.core.score = nullptr;
                    seal(rest, a.K);
                    if ((e = launch_gemv(rest, B, nsm, st, 0, nullptr)) != cudaSuccess) return e;
                }
                return launch_k(k_router_topk, dim3((B + 3) / 4), dim3(256), 0, st, (const float*)a.seg[0].out, a.seg[0].out_stride, a.E, a.topk,
                                a.top_idx, a.top_w, B, a.core);
            }
            if (rest.nseg == 0) return cudaSuccess;
            seal(rest, a.K);
            a = rest;
            grid_override = 0;
        }
    }
    if (tc_shape_ok(a.K, g_tc_warps)) {
        // int8 products on the tensor cores; one block per SM, NB sequences per pass. Rows per tile (r for
        // 2048-byte slots, r / 2 for wide rows and pairs) such that the longest block has the least to stream.
        int best_r = 32;
        long best_cost = -1;
        for (int r = B >= 3 ? 30 : 32; r >= 16; r -= 2) {    // beside the planes of four sequences two stages of at most 30 rows fit
            int T = 0;
            for (int i = 0; i < a.nseg; i++) {
                const int tr = rl_tile_rows(a.seg[i].kind, a.K) == 32 ? r : r / 2;
                T += (a.seg[i].rows + tr - 1) / tr;
            }
            const int G = grid_override ? grid_override : std::max(1, std::min(T, nsm));
            const long cost = (long)((T + G - 1) / G) * r;
            if (best_cost < 0 || cost < best_cost) { best_cost = cost; best_r = r; }
        }
        a.total_jobs = 0;
        for (int i = 0; i < a.nseg; i++) {
            Seg& g = a.seg[i];
            g.tr = rl_tile_rows(g.kind, a.K) == 32 ? best_r : best_r / 2;
            g.jobs = (g.rows + g.tr - 1) / g.tr;
            a.total_jobs += g.jobs;
        }
        const int grid = grid_override ? grid_override : std::max(1, std::min(a.total_jobs, nsm));
        a.jq = a.total_jobs / grid; a.jr = a.total_jobs % grid;
        const int per_block = (a.total_jobs + grid - 1) / grid;
        // three or four sequences share a pass; a stage more would not fit beside their planes. (Two passes of two re-read
        // the weights: 3 sequences 0.46 ms per step of the 4-layer case)
        const int NBsel = B >= 3 ? 4 : B;
        int nst = std::max(1, std::min(per_block, TC_MAX_STAGES));         // stages: what the longest block needs
        while (nst > 1 && tc_smem_bytes(a, NBsel, nst, 16) > 226 * 1024) nst--;
#define TCG(NBv, Wv)                                                                                            \
    {                                                                                                           \
        const size_t smem = tc_smem_bytes(a, NBv, nst, Wv);                                                     \
        e = opt_in_smem(k_tcgemv<NBv, Wv>, smem);                                                               \
        if (e == cudaSuccess)                                                                                   \
            e = launch_k(k_tcgemv<NBv, Wv>, dim3(grid, (B + NBv - 1) / NBv), dim3((Wv + TC_EPI) * 32), smem, st, a, B, nst, tc_stage_bytes(a)); \
    }
        if (B >= 3) TCG(4, 16) else if (B == 2) TCG(2, 16) else TCG(1, 16)
#undef TCG
        return e;
    }
    {
        // shapes the tensor-core kernel does not take: one block of 1024 threads per SM, NB sequences per pass
        const int grid = grid_override ? grid_override : std::max(1, std::min(a.total_jobs, nsm));
        if (B >= 2) {
            const size_t smem = (size_t)2 * RL_STAGE_BYTES + (size_t)4 * a.K * 4 + (size_t)2 * 4 * RL_WARPS * 32 * 4;
            e = opt_in_smem(k_rowgemv<4, 2>, smem);
            if (e == cudaSuccess) e = launch_k(k_rowgemv<4, 2>, dim3(grid, (B + 3) / 4), RL_THREADS, smem, st, a, B);
        } else {
            const size_t smem = (size_t)3 * RL_STAGE_BYTES + (size_t)a.K * 4 + (size_t)2 * RL_WARPS * 32 * 4;
            e = opt_in_smem(k_rowgemv<1, 3>, smem);
            if (e == cudaSuccess) e = launch_k(k_rowgemv<1, 3>, dim3(grid, 1), RL_THREADS, smem, st, a, B);
        }
        return e;
    }
}

static Seg make_seg(int kind, const void* w, const uint16_t* s, int rows, float* out, int out_stride) {
    Seg g{};
    g.w = w; g.s = s; g.rows = rows; g.kind = kind; g.out = out; g.out_stride = out_stride;
    g.jobs = 0;   // tiles: filled by seal(), which knows K
    return g;
}
static void seal(GemvArgs& a, int K) {
    a.K = K;
    a.total_jobs = 0;
    for (int i = 0; i < a.nseg; i++) {
        Seg& g = a.seg[i];
        g.jobs = (g.rows + rl_tile_rows(g.kind, K) - 1) / rl_tile_rows(g.kind, K);
        a.total_jobs += g.jobs;
    }
}

static void seal(GemvArgs& a, int K);
static Seg make_seg(int kind, const void* w, const uint16_t* s, int rows, float* out, int out_stride);

static void launch_proj(const ProjArgs& a, int B, int nsm, cudaStream_t st, const BatchCtx* bc = nullptr) {
    GemvArgs g{};
    g.seg[0] = make_seg(SEG_I8_ACC, a.w, a.s, a.N, a.x, a.N);
    g.nseg = 1;
    seal(g, a.K);
    g.x = a.in; g.x_stride = a.K; g.norm_w = nullptr; g.eps = a.eps;
    if (a.mode == 0) { g.gn_w = a.gn_w; g.z = a.z; g.DV = a.DV; }
    launch_gemv(g, B, nsm, st, 0, bc);
}

static void launch_delta(const DeltaArgs& a, int DK, int B, cudaStream_t st) {
    dim3 g(a.HV * (a.DV / 32), B);
    if (DK == 64) launch_k(k_delta_step<64>, g, THREADS, 0, st, a);
    else launch_k(k_delta_step<128>, g, THREADS, 0, st, a);
}

static void launch_experts(const ExpertArgs& a, int B, int nsm, cudaStream_t st, b2_engine* prof = nullptr) {
    const int picks = B * a.topk;
    // whole rows per warp: I / 8 warps / blocks; 32 blocks give two rows per warp at I = 512
    const int gx = std::max(1, (a.I + GU_RPW * WARPS - 1) / (GU_RPW * WARPS));   // every warp gets its GU_RPW row pairs
    if (a.D <= 1024) launch_k(k_expert_gu<1>, dim3(gx, picks), THREADS, 0, st, a);
    else launch_k(k_expert_gu<2>, dim3(gx, picks), THREADS, 0, st, a);
    if (prof) prof->mark(5, st);
    launch_k(k_expert_down, dim3(down_row_blocks(a.D), a.topk + 1, B), THREADS, 0, st, a);
    if (prof) prof->mark(6, st);
}

// The experts of one layer for T tokens as a grouped tensor-core GEMM: group the picks, gate/up, down into
// ypart, the shared expert's down projection into ypart's last slot. The caller combines.
struct ExpertMmaCtx {
    int* list; int* slot; int* chunk; int cap_small, cap_big;
    __half* xh; __half* acth; float* xsum_tok; float* xsum_act;
    // the tcgen05 kernel's operands: planes of the sorted picks, and where this GPU's expert blobs lie
    uint8_t* sq; float* sq_scale; float* sq_sum; int slots;
    const uint8_t* experts; size_t expert_bytes; int per, e0;
};
static void chunk_tables(const ExpertMmaCtx& m, ChunkTable& small, ChunkTable& big) {
    int* p = m.chunk;
    small.expert = p; small.start = p + m.cap_small; small.n = p + 2 * m.cap_small; small.cap = m.cap_small;
    p += 3 * m.cap_small;
    big.expert = p; big.start = p + m.cap_big; big.n = p + 2 * m.cap_big; big.cap = m.cap_big;
    p += 3 * m.cap_big;
    small.count = p; big.count = p + 1;
}
static cudaError_t launch_q4(Q4Args q, const ChunkTable& small, const ChunkTable& big, int row_blocks, int nsm, cudaStream_t st) {
    cudaError_t e;
    const size_t sm1 = (size_t)Q4_STAGES * q4_stage_bytes(1), sm4 = (size_t)Q4_STAGES * q4_stage_bytes(4);
    if ((e = opt_in_smem(k_mma_q4<1>, sm1)) != cudaSuccess) return e;
    if ((e = opt_in_smem(k_mma_q4<4>, sm4)) != cudaSuccess) return e;
    // blocks per row block: what fills the SMs at the occupancy each variant reaches (5 and 2 blocks per SM)
    const int gs = std::max(1, std::min(small.cap, (5 * nsm + row_blocks - 1) / row_blocks));
    const int gb = std::max(1, std::min(big.cap, (2 * nsm + row_blocks - 1) / row_blocks));
    q.chunks = small;
    if ((e = launch_k(k_mma_q4<1>, dim3(row_blocks, gs), dim3(Q4_THREADS), sm1, st, q)) != cudaSuccess) return e;
    q.chunks = big;
    return launch_k(k_mma_q4<4>, dim3(row_blocks, gb), dim3(Q4_THREADS), sm4, st, q);
}
// The shapes k_umma_q4 takes, and the tensor maps of its two launches (gate/up pairs, down): the pick lists are cut for the kernel
// that reads them, so whether it can run, in this build too (uq_regs_suffice), is known before they are.
static bool umma_q4_maps(const ExpertArgs& a, const ExpertMmaCtx& m, int P, UmmaQ4Args (&u)[2]) {
    if (!m.sq || !m.experts || q4_slots(P, m.per) > m.slots || m.expert_bytes % 16 != 0 || a.I > 512) return false;       // k_prep_q_slots<2>: 512 values
    cudaFuncAttributes built;
    if (cudaFuncGetAttributes(&built, k_umma_q4) != cudaSuccess) { cudaGetLastError(); return false; }
    if (!uq_regs_suffice(built.numRegs)) return false;
    for (int i = 0; i < 2; i++) {
        const bool pair = i == 0;
        const int K = pair ? a.D : a.I, row_blocks = pair ? a.I : a.D / 2;
        const uint8_t* base = m.experts + (pair ? 0 : a.off_dn_q);
        u[i].off_s = pair ? a.off_gu_s : a.off_dn_s; u[i].off_m = pair ? a.off_gu_m : a.off_dn_m;
        if (K % UQ_KB != 0 || K > 64 * UQ_MAXG || row_blocks % UM_M != 0 || ((uintptr_t)base & 15) || (u[i].off_s | u[i].off_m) % 8 != 0) return false;
        const cuuint64_t dims[3] = {(cuuint64_t)K / 2, (cuuint64_t)(pair ? 2 * a.I : a.D), (cuuint64_t)m.per};
        const cuuint64_t strides[2] = {(cuuint64_t)K / 2, (cuuint64_t)m.expert_bytes};
        const cuuint32_t box[3] = {UQ_KB / 2, UM_M, 1};
        if (!encode_byte_map(&u[i].wmap, 3, base, dims, strides, box)) return false;
        u[i].wide = (K / 64) % 8 == 0 && (u[i].off_s | u[i].off_m) % 16 == 0;
    }
    return true;
}
// One matrix of the experts (gate/up pairs, or down) on k_umma_q4: planes of the sorted picks, then the grouped GEMM.
static cudaError_t launch_umma_q4(const ExpertArgs& a, const ExpertMmaCtx& m, const GroupArgs& g, bool pair, int P, UmmaQ4Args& u, int nsm, cudaStream_t st) {
    cudaError_t e;
    const int K = pair ? a.D : a.I, rows = pair ? a.I : a.D;
    PrepSlotsArgs p{};
    p.src = pair ? a.x : a.act; p.stride = pair ? a.x_stride : a.I; p.by_pick = pair ? 0 : 1; p.topk = a.topk;
    p.norm_w = pair ? a.norm_w : nullptr; p.eps = a.eps; p.K = K; p.rows = pair ? P / a.topk : P; p.slot = g.slot; p.planes = m.sq; p.slots = m.slots;
    p.xscale = m.sq_scale; p.xsum = m.sq_sum;
    e = pair ? launch_k(k_prep_q_slots<8>, dim3(p.rows), dim3(256), 0, st, p) : launch_k(k_prep_q_slots<2>, dim3((P + 3) / 4), dim3(256), 0, st, p);
    if (e != cudaSuccess) return e;
    u.eptr = a.eptr; u.list = g.list; u.small = g.small; u.big = g.big; u.topk = a.topk; u.pair = pair ? 1 : 0; u.rows = rows; u.K = K;
    u.up_row0 = a.I; u.e0 = m.e0;
    u.slots = m.slots; u.planes = m.sq; u.xscale = m.sq_scale; u.xsum = m.sq_sum; u.out = pair ? a.act : a.ypart; u.err = a.err;
    if ((e = opt_in_smem(k_umma_q4, UQ_SMEM)) != cudaSuccess) return e;
    g_umma_launches++;
    return launch_k(k_umma_q4, dim3(nsm), dim3(UQ_THREADS), UQ_SMEM, st, u);
}

static cudaError_t launch_experts_mma(const ExpertArgs& a, int T, const ExpertMmaCtx& m, int nsm, cudaStream_t st, b2_engine* prof) {
    cudaError_t e;
    const int P = T * a.topk;
    GroupArgs g{};
    g.top_idx = a.top_idx; g.idx_stride = a.idx_stride; g.T = T; g.topk = a.topk; g.E = a.E; g.eptr = a.eptr;
    g.list = m.list; g.slot = m.slot;
    chunk_tables(m, g.small, g.big);
    UmmaQ4Args u[2] = {};
    const bool q4_umma = umma_q4_maps(a, m, P, u);            // else (K not a multiple of 256, no tensor maps): k_mma_q4
    g.small_n = q4_umma ? UQ_SMALL : GQ_SMALL;
    g.big_n = q4_umma ? UQ_TT : GQ_BIG;
    g.align = q4_umma ? UQ_G : 1;
    if ((e = launch_k(k_group_picks, dim3(1), dim3(1024), 0, st, g)) != cudaSuccess) return e;
    if (q4_umma) {
        if ((e = launch_umma_q4(a, m, g, true, P, u[0], nsm, st)) != cudaSuccess) return e;
        if (prof) prof->mark(5, st);
        if ((e = launch_umma_q4(a, m, g, false, P, u[1], nsm, st)) != cudaSuccess) return e;
    } else {
        Q4Args q{};
        q.eptr = a.eptr; q.list = g.list; q.topk = a.topk;
        PrepArgs p{};
        p.x = a.x; p.x_stride = a.x_stride; p.norm_w = a.norm_w; p.eps = a.eps; p.K = a.D; p.T = T; p.Tpad = T; p.out = m.xh;
        p.xsum = m.xsum_tok; p.perm8 = 1;
        if ((e = launch_k(k_prep_x, dim3(T), dim3(256), 0, st, p)) != cudaSuccess) return e;
        q.pair = 1; q.rows = a.I; q.K = a.D; q.off_q = 0; q.off_s = a.off_gu_s; q.off_m = a.off_gu_m; q.up_row0 = a.I;
        q.xh = m.xh; q.xsum = m.xsum_tok; q.by_pick = 0; q.out = a.act; q.row_tiles = 1;
        if ((e = launch_q4(q, g.small, g.big, (a.I + 31) / 32, nsm, st)) != cudaSuccess) return e;
        if (prof) prof->mark(5, st);
        PrepArgs p2{};
        p2.x = a.act; p2.x_stride = a.I; p2.K = a.I; p2.T = P; p2.Tpad = P; p2.out = m.acth; p2.xsum = m.xsum_act; p2.perm8 = 1;
        if ((e = launch_k(k_prep_x, dim3(P), dim3(256), 0, st, p2)) != cudaSuccess) return e;
        q.pair = 0; q.rows = a.D; q.K = a.I; q.off_q = a.off_dn_q; q.off_s = a.off_dn_s; q.off_m = a.off_dn_m; q.up_row0 = 0;
        q.xh = m.acth; q.xsum = m.xsum_act; q.by_pick = 1; q.out = a.ypart;
        q.row_tiles = std::max(1, std::min(4, 2048 / a.I));      // keep about 8 ring steps per block
        if ((e = launch_q4(q, g.small, g.big, (a.D + Q4_ROWS * q.row_tiles - 1) / (Q4_ROWS * q.row_tiles), nsm, st)) != cudaSuccess) return e;
    }
    // shared expert down for this GPU's own tokens: int8 [D][SH] on the dense tensor-core kernel. Its input is a product of
    // activations with a long tail: fp16 hi + lo keeps 2^-22 of every value, digit planes would keep it of a row's largest only
    PrepArgs p3{};
    p3.x = a.sh_act; p3.x_stride = a.SH; p3.K = a.SH; p3.T = a.nlocal; p3.Tpad = (a.nlocal + MM_TOK - 1) / MM_TOK * MM_TOK; p3.out = m.xh;
    if ((e = launch_k(k_prep_x, dim3(p3.Tpad), dim3(256), 0, st, p3)) != cudaSuccess) return e;
    MmaArgs d{};
    d.seg[0].w = a.shd_w; d.seg[0].s = a.shd_s; d.seg[0].rows = a.D; d.seg[0].kind = SEG_I8;
    d.seg[0].out = a.ypart + ((size_t)a.local0 * (a.topk + 1) + a.topk) * a.D; d.seg[0].out_stride = (a.topk + 1) * a.D;
    d.seg[0].blocks = (a.D + MM_ROWS - 1) / MM_ROWS;
    d.nseg = 1; d.total_blocks = d.seg[0].blocks; d.xh = m.xh; d.K = a.SH; d.T = a.nlocal;
    if ((e = launch_mma_i8(d, p3.Tpad / MM_TOK, nsm, st)) != cudaSuccess) return e;
    if (prof) prof->mark(6, st);
    return cudaSuccess;
}

static bool attn_mma_ok(const AttnArgs& a, int HD, bool f32) {
    const int hr = a.RD / 2;
    const bool rope_ok = hr % 32 == 0 || (hr > 0 && hr < 32 && (hr & (hr - 1)) == 0);   // pairs in one lane, or a power of two lanes apart
    return !f32 && a.H / a.KV <= 8 && rope_ok && (HD == 256 || HD == 128 || HD == 64);
}
static cudaError_t launch_attn(const AttnArgs& a, int HD, bool f32, int B, cudaStream_t st, int tiles_per_slice, int nsm, b2_engine* prof = nullptr) {
    const int G = a.H / a.KV;
    const size_t smem = (size_t)WARPS * G * HD * 4;
    dim3 g(a.nsplit, a.KV, B);
#define ATT(hd, f)                                                                     \
    {                                                                                  \
        cudaError_t e = opt_in_smem(k_attn<hd, f>, smem);                              \
        if (e != cudaSuccess) return e;                                                \
        launch_k(k_attn<hd, f>, g, THREADS, smem, st, a);                              \
    }
    if (attn_mma_ok(a, HD, f32)) {
        // bf16 cache: both contractions on the tensor cores; two tile buffers when a slice can span several tiles
        // with two or more blocks per SM to choose from, two single-buffered blocks on an SM (registers allow two) hide a
        // tile's latency behind each other's products better than one double-buffered block does
        const int nbuf = (tiles_per_slice > 1 && (long)a.nsplit * a.KV * B < 2L * nsm) ? 2 : 1;
        cudaError_t e;
#define ATM(hd)                                                                                     \
    {                                                                                               \
        e = opt_in_smem(k_attn_mma<hd>, am_smem<hd>(nbuf));                                         \
        if (e == cudaSuccess) e = launch_k(k_attn_mma<hd>, g, THREADS, am_smem<hd>(nbuf), st, a, nbuf); \
    }
        if (HD == 256) ATM(256) else if (HD == 128) ATM(128) else ATM(64)
#undef ATM
        if (e != cudaSuccess) return e;
        if (!a.append_only) launch_k(k_attn_merge, dim3(a.H, B), THREADS, 0, st, a, HD);
        return cudaSuccess;
    }
    if (HD == 64) { if (f32) ATT(64, true) else ATT(64, false) }
    else if (HD == 128) { if (f32) ATT(128, true) else ATT(128, false) }
    else { if (f32) ATT(256, true) else ATT(256, false) }
#undef ATT
    if (!a.append_only) launch_k(k_attn_merge, dim3(a.H, B), THREADS, 0, st, a, HD);
    return cudaSuccess;
}
// Attention of a prompt chunk of T tokens. Every token's key and value row goes into the cache first: a token's blocks then find
// the rows of the chunk's earlier tokens there (in the decode kernel they write their own row again, with the same bytes).
// Tiles of tokens that share their reads of the context when a block per token would take more than one turn of the GPU (two
// blocks to an SM); the results are the same bits. 40 layers behind 2000 tokens of context: 290 tokens 19.1 ms a block per
// token and 18.4 in tiles, 512 tokens 27.5 and 24.5; 160 tokens 15.4 either way.
static cudaError_t launch_attn_chunk(AttnArgs a, int HD, bool f32, int T, cudaStream_t st, int tiles_per_slice, int nsm) {
    const bool tiled = attn_mma_ok(a, HD, f32) && a.nsplit == 1 && (long)T * a.KV > 2L * nsm;
    AttnArgs ap = a;
    ap.append_only = tiled ? 2 : 1;
    cudaError_t e = launch_attn(ap, HD, f32, T, st, tiles_per_slice, nsm);
    if (e != cudaSuccess) return e;
    if (!tiled) return launch_attn(a, HD, f32, T, st, tiles_per_slice, nsm);
    const int tpt = AP_ROWS / (a.H / a.KV);
    const dim3 g((T + tpt - 1) / tpt, a.KV);
#define APR(hd)                                                                                       \
    {                                                                                                 \
        e = opt_in_smem(k_attn_prompt<hd>, ap_smem<hd>());                                            \
        if (e == cudaSuccess) e = launch_k(k_attn_prompt<hd>, g, dim3(256), ap_smem<hd>(), st, a, T); \
    }
    if (HD == 256) APR(256) else if (HD == 128) APR(128) else APR(64)
#undef APR
    return e;
}

// The expert kernels for fewer than BATCH_GEMM_MIN tokens (moe1.cuh): shapes they take, and their two launches. `x_in` rows are
// normalised with `norm_w` when it is given; the result is added into `xout`.
static bool moe1_shape_ok(const Cfg& c) {
    return (c.D == 512 || c.D == 1024 || c.D == 2048 || c.D == 4096) && c.I >= 128 && c.I <= 2048 && (c.I & (c.I - 1)) == 0 &&
           c.SH % 128 == 0 && c.TOPK <= 8 && c.E <= 256;
}
// what the grouped expert GEMM takes (k_umma_q4 or k_mma_q4)
static bool grouped_shape_ok(const Cfg& c, int T) {
    return T * c.TOPK <= GQ_MAXP && c.D % MM_KC == 0 && c.I % MM_KC == 0 && c.SH % MM_KC == 0 && c.D <= 2048 && c.I <= 2048 && c.E <= 256;
}
struct Moe1Ctx { const uint8_t** top_ptr; int8_t* actq; float* asc; float* asum; };
static cudaError_t launch_moe1(const Cfg& c, const float* rlogits, const float* x_in, const uint16_t* norm_w, const uint8_t* const* eptr,
                               int* top_idx, float* top_w, const Moe1Ctx& m, const float* sh_act, const float* sgate, const int8_t* shd_w,
                               const uint16_t* shd_s, float* xout, int* err, int B, cudaStream_t st, b2_engine* prof,
                               const CoreRoute* core = nullptr, const CoresLiveArgs* live = nullptr, const LayerW* next = nullptr) {
    Gu1Args g{};
    if (core) g.core = *core;
    g.logits = rlogits; g.x = x_in; g.norm_w = norm_w; g.eps = c.eps; g.eptr = eptr;
    g.off_gu_s = c.off_gu_s(); g.off_gu_m = c.off_gu_m(); g.off_dn = c.off_dn_q(); g.dn_bytes = (int)(c.off_dn_m() + c.dn_sm() - c.off_dn_q()); g.D = c.D; g.I = c.I; g.E = c.E; g.topk = c.TOPK;
    g.top_idx = top_idx; g.top_w = top_w; g.top_ptr = m.top_ptr; g.actq = m.actq; g.asc = m.asc; g.asum = m.asum; g.err = err;
    const int gx = c.TOPK * c.I / M1_GU_PAIRS;
    cudaError_t ce = opt_in_smem(k_moe_gu1, m1_gu_smem(c.D));
    if (ce == cudaSuccess) ce = launch_k(k_moe_gu1, dim3(gx, B), dim3(M1_GU_THREADS), m1_gu_smem(c.D), st, g);
    if (prof) prof->mark(5, st);
    // the gate/up kernel has made the core engine's picks; the live cores read x before the down kernel writes it
    if (live && ce == cudaSuccess) ce = launch_k(k_cores_live, dim3(B), dim3(256), (size_t)(live->D + live->r) * 4, st, *live);
    Down1Args d{};
    d.top_ptr = m.top_ptr; d.top_w = top_w; d.actq = m.actq; d.asc = m.asc; d.asum = m.asum; d.sh_act = sh_act; d.sg = sgate;
    d.shd_w = shd_w; d.shd_s = shd_s;
    d.off_dn_q = c.off_dn_q(); d.off_dn_s = c.off_dn_s(); d.off_dn_m = c.off_dn_m();
    d.D = c.D; d.I = c.I; d.SH = c.SH; d.topk = c.TOPK; d.xout = xout;
    if (next) {
        const QWd* w[3] = {next->attn ? &next->q : &next->in_qkv, next->attn ? &next->k : &next->in_z, next->attn ? &next->v : nullptr};
        for (int i = 0; i < 3; i++)
            if (w[i]) { d.pf[i] = w[i]->w; d.pf_bytes[i] = (size_t)w[i]->n * w[i]->k; }
    }
    const size_t dsm = m1_down_smem(c.I, c.SH, c.TOPK);
    if (ce == cudaSuccess) ce = opt_in_smem(k_moe_down1, dsm);
    if (ce == cudaSuccess)
        ce = launch_k(k_moe_down1, dim3((c.D + M1_DOWN_ROWS - 1) / M1_DOWN_ROWS, B), dim3(2 * (c.TOPK + 1) * 32), dsm, st, d);
    if (prof) prof->mark(6, st);
    return ce;
}

// One decode step for all B sequences: token ids in d_tok, positions in d_pos.
// chunk_T > 0: a prompt chunk of chunk_T tokens of the engine's one sequence instead (the tokens are the columns of
// every matrix product; conv, delta rule and attention walk them in order; the head runs for the last token only,
// and only when chunk_head is set).
int b2_engine::enqueue_step(cudaStream_t st, bool count, int chunk_T, bool chunk_head) {
    if (chunk_T == 0 && use_step1()) {
        if (count) launches = 1;
        return launch_step1(st);
    }
    int n = 0;
    const int launches0 = g_launch_count;
    const bool chunk = chunk_T > 0;
    const int NSEQ = this->B;                     // sequences: what the recurrent state, the conv taps and the KV pages are laid out by
    const int B = chunk ? chunk_T : this->B;      // columns of this step's matrix products
    // the work buffers of this step: the members, or the chunk's own set under the same names
    int* const d_tok = chunk ? pc.tok : this->d_tok;
    int* const d_pos = chunk ? pc.vpos : this->d_pos;
    float* const x = chunk ? pc.x : this->x;
    float* const big = chunk ? pc.big : this->big;
    float* const zbuf = chunk ? pc.zbuf : this->zbuf;
    float* const kraw = chunk ? pc.kraw : this->kraw;
    float* const vraw = chunk ? pc.vraw : this->vraw;
    float* const beta = chunk ? pc.beta : this->beta;
    float* const gdec = chunk ? pc.gdec : this->gdec;
    float* const obuf = chunk ? pc.obuf : this->obuf;
    float* const att = chunk ? pc.att : this->att;
    float* const rlogits = chunk ? pc.rlogits : this->rlogits;
    float* const sh_act = chunk ? pc.sh_act : this->sh_act;
    float* const sgate = chunk ? pc.sgate : this->sgate;
    float* const act = chunk ? pc.act : this->act;
    float* const ypart = chunk ? pc.ypart : this->ypart;
    float* const attn_part = chunk ? pc.attn_part : this->attn_part;
    unsigned int* const d_dcounter = chunk ? pc.dcounter : this->d_dcounter;
    unsigned int* const d_counter = chunk ? pc.counter : this->d_counter;
    __half* const xh = chunk ? pc.xh : this->xh;
    __half* const acth = chunk ? pc.acth : this->acth;
    int* const g_list = chunk ? pc.g_list : this->g_list;
    int* const g_slot = chunk ? pc.g_slot : this->g_slot;
    int* const g_chunk = chunk ? pc.g_chunk : this->g_chunk;
    float* const xsum_tok = chunk ? pc.xsum_tok : this->xsum_tok;
    float* const xsum_act = chunk ? pc.xsum_act : this->xsum_act;
    const int cap_small = chunk ? pc.cap_small : this->cap_small, cap_big = chunk ? pc.cap_big : this->cap_big;
    const int nsplit = chunk ? pc.nsplit : this->nsplit, attn_tiles = chunk ? pc.attn_tiles : this->attn_tiles;
    const BatchCtx bctx = chunk ? BatchCtx{pc.xh, pc.xh_tpad, pc.uq_i, pc.uq_b, pc.uq_scale, pc.uq_passes, true}
                                : BatchCtx{this->xh, xh_tpad, uq_i, uq_b, uq_scale, uq_passes, false};
    const BatchCtx* bc = xh ? &bctx : nullptr;
    cudaGetLastError();   // a stale error of an earlier, unrelated call must not be blamed on these launches
    mark(-1, st);
    launch_k(k_embed, dim3(B), dim3(256), 0, st, embed, (const int*)d_tok, x, c.D, c.V, d_err);
    if (chunk) launch_k(k_iota_from, dim3((B + 255) / 256), dim3(256), 0, st, d_pos, (const int*)this->d_pos, B);
    mark(0, st);
    n++;
    const size_t kv_layer = (size_t)NSEQ * pages_per_seq * c.KV * KV_PAGE * c.HD * (kv_f32 ? 4 : 2);
    for (int li = 0; li < c.L; li++) {
        const LayerW& l = layers[li];
        if (l.attn) {
            GemvArgs a{};
            a.seg[0] = make_seg(SEG_I8, l.q.w, l.q.s, l.q.n, big, 2 * c.H * c.HD);
            a.seg[1] = make_seg(SEG_I8, l.k.w, l.k.s, l.k.n, kraw, c.KV * c.HD);
            a.seg[2] = make_seg(SEG_I8, l.v.w, l.v.s, l.v.n, vraw, c.KV * c.HD);
            a.nseg = 3; seal(a, c.D);
            a.x = x; a.norm_w = l.norm1; a.eps = c.eps; a.K = c.D; a.err = d_err;
            launch_gemv(a, B, nsm, st, 0, bc);
            mark(1, st);
            AttnArgs t{};
            t.qraw = big; t.kraw = kraw; t.vraw = vraw; t.qn_w = l.q_norm; t.kn_w = l.k_norm;
            t.rope_cos = rope_cos; t.rope_sin = rope_sin; t.pos = d_pos;
            t.kpool = (char*)kpool + kv_layer * l.slot; t.vpool = (char*)vpool + kv_layer * l.slot;
            t.page_table = page_table; t.pt_stride = chunk ? 0 : pages_per_seq;
            t.H = c.H; t.KV = c.KV; t.RD = c.RD; t.eps = c.eps; t.scale = 1.0f / std::sqrt((float)c.HD);
            t.part = attn_part; t.out = att; t.nsplit = nsplit;
            const cudaError_t e = chunk ? launch_attn_chunk(t, c.HD, kv_f32, B, st, attn_tiles, nsm) : launch_attn(t, c.HD, kv_f32, B, st, attn_tiles, nsm);
            if (e != cudaSuccess) return fail("attention launch: %s", cudaGetErrorString(e));
            mark(3, st);
            ProjArgs p{};
            p.in = att; p.mode = 1; p.w = l.o.w; p.s = l.o.s; p.x = x; p.N = c.D; p.K = c.H * c.HD; p.eps = c.eps; p.DV = c.DV;
            launch_proj(p, B, nsm, st, bc);
        } else {
            GemvArgs a{};
            a.seg[0] = make_seg(chunk ? SEG_I8 : SEG_I8_CONV, l.in_qkv.w, l.in_qkv.s, l.in_qkv.n, big, c.C());
            a.seg[1] = make_seg(SEG_I8_SILU, l.in_z.w, l.in_z.s, l.in_z.n, zbuf, c.VD());
            a.seg[2] = make_seg(SEG_BF_SIGMOID, l.in_b, nullptr, c.HV, beta, c.HV);
            a.seg[3] = make_seg(SEG_BF_DECAY, l.in_a, nullptr, c.HV, gdec, c.HV);
            a.nseg = 4; seal(a, c.D);
            a.x = x; a.norm_w = l.norm1; a.eps = c.eps; a.K = c.D; a.err = d_err;
            a.conv_w = l.conv; a.conv_state = conv + (size_t)l.slot * NSEQ * c.C() * 3;
            a.a_log = l.a_log; a.dt_bias = l.dt_bias;
            launch_gemv(a, B, nsm, st, 0, bc);
            mark(1, st);
            float* const lstate = state + (size_t)l.slot * NSEQ * c.HV * c.DK * c.DV;
            if (chunk) {
                ConvPromptArgs cs{big, pc.qkv, l.conv, a.conv_state, c.C(), B, c.HK * c.DK};
                const dim3 gc((c.C() + 1023) / 1024, (B + CONV_TOK - 1) / CONV_TOK);
                if (c.DK == 64) launch_k(k_conv_prompt<64>, gc, dim3(256), 0, st, cs);
                else launch_k(k_conv_prompt<128>, gc, dim3(256), 0, st, cs);
                DeltaPromptArgs ds{pc.qkv, beta, gdec, lstate, obuf, c.C(), c.HK, c.HV, c.DV, B};
                const dim3 g(c.HV * (c.DV / 32));
                cudaError_t e = c.DK == 64 ? opt_in_smem(k_delta_prompt<64>, DP_SMEM) : opt_in_smem(k_delta_prompt<128>, DP_SMEM);
                if (e == cudaSuccess) e = c.DK == 64 ? launch_k(k_delta_prompt<64>, g, dim3(DP_THREADS), DP_SMEM, st, ds)
                                                     : launch_k(k_delta_prompt<128>, g, dim3(DP_THREADS), DP_SMEM, st, ds);
                if (e != cudaSuccess) return fail("delta rule of a prompt chunk: %s", cudaGetErrorString(e));
            } else {
            DeltaArgs d{};
            d.y = big; d.beta = beta; d.g = gdec; d.state = lstate;
            d.o = obuf; d.C = c.C(); d.HK = c.HK; d.HV = c.HV; d.DV = c.DV; d.prenormed = 0;
            launch_delta(d, c.DK, B, st);
            }
            mark(2, st);
            ProjArgs p{};
            p.in = obuf; p.z = zbuf; p.gn_w = l.gnorm; p.eps = c.eps; p.DV = c.DV; p.mode = 0;
            p.w = l.out.w; p.s = l.out.s; p.x = x; p.N = c.D; p.K = c.VD();
            launch_proj(p, B, nsm, st, bc);
        }
        mark(4, st);
        n += l.attn ? 4 : 3;
        {
            GemvArgs a{};
            a.seg[0] = make_seg(SEG_BF, l.router, nullptr, c.E, rlogits, c.E);
            a.seg[0].bias = l.router_bias;
            a.seg[1] = make_seg(SEG_I8_GATEUP, l.sh_gate.w, l.sh_gate.s, c.SH, sh_act, c.SH);
            a.seg[1].w2 = l.sh_up.w; a.seg[1].s2 = l.sh_up.s;
            a.seg[2] = make_seg(SEG_BF_SIGMOID, l.sh_gw, nullptr, 1, sgate, 1);
            a.nseg = 3;
            // the core engine's two key tables ride along: their scores, then the picks where the router's are made
            float* const cscore = chunk ? pc.cscore : this->cscore;
            int* const csel = chunk ? pc.csel : this->csel;
            float* const cselw = chunk ? pc.cselw : this->cselw;
            float* const core_y = chunk ? pc.core_y : this->core_y;
            CoreRoute cr{};
            if (l.key1) {
                a.seg[3] = make_seg(SEG_BF, l.key1, nullptr, c.n1, cscore, c.n1 + c.n2);
                a.seg[4] = make_seg(SEG_BF, l.key2, nullptr, c.n2, cscore + c.n1, c.n1 + c.n2);
                a.nseg = 5;
                cr.score = cscore; cr.n1 = c.n1; cr.n2 = c.n2; cr.k = c.cores_active;
                cr.counts = d_counts + (size_t)li * c.n1 * c.n2; cr.sel = csel; cr.selw = cselw;
            }
            seal(a, c.D);
            a.core = cr;
            // the layer's live cores: their output goes to core_y once the picks are known and before the experts write x
            CoresLiveArgs cl{};
            const bool has_live = l.key1 && l.n_live > 0;
            if (has_live) {
                cl.x = x; cl.norm_w = l.norm2; cl.eps = c.eps; cl.live = l.live; cl.cg = l.cg; cl.cu = l.cu; cl.cd = l.cd;
                cl.sel = csel; cl.selw = cselw; cl.y = core_y; cl.D = c.D; cl.r = c.rank; cl.k = c.cores_active;
            }
            auto launch_live = [&]() {
                if (has_live) launch_k(k_cores_live, dim3(B), dim3(256), (size_t)(c.D + c.rank) * 4, st, cl);
            };
            a.x = x; a.norm_w = l.norm2; a.eps = c.eps; a.K = c.D; a.err = d_err;
            // fewer than BATCH_GEMM_MIN tokens on one GPU: the top-8 moves into the expert kernel and the experts are spread over all SMs
            const bool moe1 = ep_world == 1 && B < BATCH_GEMM_MIN && moe1_shape_ok(c);
            a.finisher = moe1 ? FIN_NONE : FIN_TOPK; a.counter = d_counter; a.E = c.E; a.topk = c.TOPK;
            // a chunk's picks live in its own scratch; the last token's are kept where a decode step's are (b2_debug_router)
            a.top_idx = chunk ? pc.top_idx : top_idx + (size_t)li * B * c.TOPK;
            a.top_w = chunk ? pc.top_w : top_w + (size_t)li * B * c.TOPK;
            launch_gemv(a, B, nsm, st, 0, bc);
            if (chunk) {
                cudaMemcpyAsync(top_idx + (size_t)li * NSEQ * c.TOPK, pc.top_idx + (size_t)(B - 1) * c.TOPK, c.TOPK * sizeof(int), cudaMemcpyDeviceToDevice, st);
                cudaMemcpyAsync(top_w + (size_t)li * NSEQ * c.TOPK, pc.top_w + (size_t)(B - 1) * c.TOPK, c.TOPK * sizeof(float), cudaMemcpyDeviceToDevice, st);
            }
            mark(1, st);
            if (!moe1) launch_live();              // the picks were made by the launch above (its finisher, or k_router_topk)
            if (moe1) {
                const Moe1Ctx mc{top_ptr, actq, asc, asum};
                cudaError_t ce = launch_moe1(c, rlogits, x, l.norm2, l.eptr, a.top_idx, a.top_w, mc, sh_act, sgate, (const int8_t*)l.sh_down.w,
                                             l.sh_down.s, x, d_err, B, st, this, &cr, has_live ? &cl : nullptr, li + 1 < c.L ? &layers[li + 1] : nullptr);
                if (ce != cudaSuccess) return fail("expert kernels: %s", cudaGetErrorString(ce));
                n += 3;
            } else {
            ExpertArgs x2{};
            x2.eptr = l.eptr; x2.topk = c.TOPK; x2.E = c.E; x2.D = c.D; x2.I = c.I;
            x2.off_gu_s = c.off_gu_s(); x2.off_gu_m = c.off_gu_m(); x2.off_dn_q = c.off_dn_q(); x2.off_dn_s = c.off_dn_s(); x2.off_dn_m = c.off_dn_m();
            x2.norm_w = l.norm2; x2.eps = c.eps; x2.act = act; x2.sh_act = sh_act; x2.sg = sgate;
            x2.shd_w = l.sh_down.w; x2.shd_s = l.sh_down.s; x2.SH = c.SH; x2.xout = x; x2.err = d_err;
            x2.ypart = ypart; x2.counter = d_dcounter; x2.null_is_error = ep_world == 1;
            const int Tg = B * ep_world;
            const bool grouped = xh && Tg >= BATCH_GEMM_MIN && grouped_shape_ok(c, Tg);
            const ExpertMmaCtx mctx{g_list, g_slot, g_chunk, cap_small, cap_big, xh, acth, xsum_tok, xsum_act,
                                    chunk ? pc.sq : sq, chunk ? pc.sq_scale : sq_scale, chunk ? pc.sq_sum : sq_sum, (int)q4_slots(Tg * c.TOPK, c.E / ep_world),
                                    l.experts, c.expert_bytes(), c.E / ep_world, ep_rank * (c.E / ep_world)};
            if (ep_world == 1) {
                x2.x = x; x2.x_stride = c.D; x2.top_idx = a.top_idx; x2.top_w = a.top_w; x2.idx_stride = c.TOPK;
                x2.combine = 1; x2.local0 = 0; x2.nlocal = B;
                if (grouped) {
                    cudaError_t ce = launch_experts_mma(x2, B, mctx, nsm, st, this);
                    if (ce != cudaSuccess) return fail("grouped expert GEMM: %s", cudaGetErrorString(ce));
                    EpArgs ep{};
                    ep.x = x; ep.top_idx = a.top_idx; ep.top_w = a.top_w; ep.recv_y = ypart; ep.sg = sgate; ep.xout = x;
                    ep.D = c.D; ep.topk = c.TOPK; ep.B = B; ep.E = c.E; ep.world = 1; ep.rank = 0; ep.has_shared = 1;
                    launch_k(k_ep_combine, dim3((c.D + 1023) / 1024, B), dim3(256), 0, st, ep);
                } else {
                    launch_experts(x2, B, nsm, st, this);
                }
            } else {
                const int rw = c.D + 2 * c.TOPK;
                EpArgs ep{};
                ep.x = x; ep.top_idx = a.top_idx; ep.top_w = a.top_w; ep.rec = rec_local; ep.recv_y = recv_y; ep.sg = sgate; ep.xout = x;
                ep.D = c.D; ep.topk = c.TOPK; ep.B = B; ep.E = c.E; ep.world = ep_world; ep.rank = ep_rank; ep.has_shared = 1;
                EpPushArgs pa{};
                if (ep_peer_ready) {
                    for (int p = 0; p < ep_world; p++) pa.peers.base[p] = ep_peer[p];
                    pa.peers.rec_off = 0; pa.peers.y_off = (size_t)(recv_y - ep_block); pa.peers.flag_off = ep_flag_off;
                    pa.x = x; pa.top_idx = a.top_idx; pa.top_w = a.top_w; pa.ypart = ypart; pa.D = c.D; pa.topk = c.TOPK; pa.B = B; pa.E = c.E;
                    pa.world = ep_world; pa.rank = ep_rank; pa.seq = d_ep_seq; pa.rows_sent = d_ep_rows; pa.err = d_err;
                    const int nb0 = std::min(B, EP_MAX_BLOCKS);
                    launch_k(k_ep_push_records, dim3(nb0), dim3(256), 0, st, pa);
                    launch_k(k_ep_wait, dim3(1), dim3(EP_MAX_WORLD * EP_MAX_BLOCKS), 0, st, EpWaitArgs{nullptr, (int*)ep_block + ep_flag_off, d_ep_seq, 0, ep_world, ep_rank, nb0, 1 << 21, d_err});
                } else {
                    launch_k(k_ep_pack, dim3(B), dim3(256), 0, st, ep);
                    if (ep_exchange_records(st)) return 1;
                }
                x2.x = rec_all; x2.x_stride = rw; x2.top_idx = (const int*)(rec_all + c.D); x2.top_w = rec_all + c.D + c.TOPK; x2.idx_stride = rw;
                x2.combine = 0; x2.local0 = ep_rank * B; x2.nlocal = B;
                if (grouped) {
                    cudaError_t ce = launch_experts_mma(x2, Tg, mctx, nsm, st, this);
                    if (ce != cudaSuccess) return fail("grouped expert GEMM: %s", cudaGetErrorString(ce));
                } else {
                    launch_experts(x2, Tg, nsm, st, this);
                }
                if (ep_peer_ready) {
                    launch_k(k_ep_push_outputs, dim3(EP_MAX_BLOCKS), dim3(256), 0, st, pa);
                    launch_k(k_ep_wait, dim3(1), dim3(EP_MAX_WORLD * EP_MAX_BLOCKS), 0, st, EpWaitArgs{nullptr, (int*)ep_block + ep_flag_off, d_ep_seq, 1, ep_world, ep_rank, EP_MAX_BLOCKS, 1 << 21, d_err});
                } else if (ep_exchange_outputs(st)) return 1;
                launch_k(k_ep_combine, dim3((c.D + 1023) / 1024, B), dim3(256), 0, st, ep);
                n += 2;
            }
            n += 3;
            }
        }
        if (l.key1 && l.n_live > 0) {
            float* const cy = chunk ? pc.core_y : this->core_y;
            launch_k(k_add_rows, dim3((B * c.D + 255) / 256), dim3(256), 0, st, x, (const float*)cy, B * c.D);
        }
        for (size_t j = 0; j < tap_layers.size(); j++)
            if (tap_layers[j] == li) {
                // the hidden state after this layer, of every sequence's token; of a chunk's last token
                if (chunk) cudaMemcpyAsync(tap_buf + j * (size_t)NSEQ * c.D, x + (size_t)(B - 1) * c.D, (size_t)c.D * 4, cudaMemcpyDeviceToDevice, st);
                else cudaMemcpyAsync(tap_buf + j * (size_t)B * c.D, x, (size_t)B * c.D * 4, cudaMemcpyDeviceToDevice, st);
            }
    }
    if (!chunk || chunk_head) {
        GemvArgs a{};
        a.seg[0] = make_seg(SEG_I8_ARGMAX, lm_head.w, lm_head.s, c.V, logits, c.V);
        a.nseg = 1; seal(a, c.D);
        a.x = chunk ? x + (size_t)(B - 1) * c.D : x; a.norm_w = norm; a.eps = c.eps; a.K = c.D; a.err = d_err;
        a.finisher = FIN_ARGMAX; a.counter = this->d_counter; a.part_val = part_val; a.part_idx = part_idx;
        a.next_tok = d_next; a.pos = chunk ? nullptr : d_pos;
        a.hist = TokHist{d_hist, cap, NSEQ}; a.tok = this->d_tok;
        // a chunk's head runs for its last token alone (the decode GEMV), and leaves the residual row where a decode step does
        launch_gemv(a, chunk ? 1 : B, nsm, st, head_grid, chunk ? nullptr : bc);
        mark(7, st);
        n++;
    }
    if (chunk) {
        cudaMemcpyAsync(this->x, x + (size_t)(B - 1) * c.D, (size_t)c.D * 4, cudaMemcpyDeviceToDevice, st);
        k_add_i32<<<1, 32, 0, st>>>(this->d_pos, B, NSEQ);                  // the sequence is B positions further
    }
    (void)n;
    if (count) launches = g_launch_count - launches0;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail("kernel launch: %s", cudaGetErrorString(e));
    return 0;
}

// ---- prompt chunks ------------------------------------------------------------------------------------------------
// Tokens per chunk: the more, the fewer times the experts' 450 MB per layer cross HBM (128 tokens already touch them all)
// and the fuller the expert GEMM's pick lists; 1024 x 8 picks is what the pick grouping handles at once (GQ_MAXP).
constexpr int CHUNK_TOKENS = 1024;
constexpr int CHUNK_MIN = 16;            // shorter feeds go token by token

void b2_engine::free_chunk_bufs() {
    cudaFree(pc.arena);
    pc = ChunkBufs();
}

// buffers for T tokens, in steps of a power of two (64 .. CHUNK_TOKENS), so that a program's feeds grow them a few times at most. One
// allocation for all of them: 38 separate ones made a prompt that grows them wait up to 90 ms for the driver
int b2_engine::ensure_chunk_bufs(int T) {
    if (pc.W >= T) return 0;
    CU(cudaStreamSynchronize(stream));
    free_chunk_bufs();
    int W = 64;
    while (W < T) W *= 2;
    const int bigw = std::max(2 * c.H * c.HD, c.C());
    const size_t P = (size_t)W * c.TOPK;
    std::vector<std::pair<void**, size_t>> parts;
    auto want = [&](auto** p, size_t n) { parts.push_back({(void**)p, std::max<size_t>(n * sizeof(**p), 16)}); };
    want(&pc.tok, W); want(&pc.vpos, W);
    want(&pc.x, (size_t)W * c.D); want(&pc.big, (size_t)W * bigw); want(&pc.qkv, (size_t)W * c.C()); want(&pc.zbuf, (size_t)W * c.VD());
    want(&pc.kraw, (size_t)W * c.KV * c.HD); want(&pc.vraw, (size_t)W * c.KV * c.HD);
    want(&pc.beta, (size_t)W * c.HV); want(&pc.gdec, (size_t)W * c.HV);
    want(&pc.obuf, (size_t)W * c.VD()); want(&pc.att, (size_t)W * c.H * c.HD);
    want(&pc.rlogits, (size_t)W * c.E); want(&pc.sh_act, (size_t)W * c.SH); want(&pc.sgate, W);
    want(&pc.act, P * c.I); want(&pc.top_idx, P); want(&pc.top_w, P);
    want(&pc.ypart, (size_t)W * (c.TOPK + 1) * c.D);
    want(&pc.dcounter, (size_t)W * down_row_blocks(c.D)); want(&pc.counter, W);
    // the tokens fill the GPU: few, long slices. By the cache's size alone, never by W: a token's sums keep their order
    pc.nsplit = std::max(1, std::min({64, (2 * nsm) / std::max(1, c.KV * 128), (cap + 63) / 64}));
    pc.attn_tiles = ((cap + pc.nsplit - 1) / pc.nsplit + AM_TILE - 1) / AM_TILE;
    want(&pc.attn_part, (size_t)W * c.KV * pc.nsplit * (c.H / c.KV) * (c.HD + 2));
    pc.xh_tpad = (W + MM_TOK - 1) / MM_TOK * MM_TOK;
    want((uint16_t**)&pc.xh, (size_t)pc.xh_tpad * 2 * 4096);
    pc.uq_passes = (W + UM_TOK - 1) / UM_TOK;
    want(&pc.uq_i, (size_t)pc.uq_passes * UM_PI * UM_TOK * 4096);
    want(&pc.uq_b, (size_t)pc.uq_passes * UM_PB * UM_TOK * 4096);
    want(&pc.uq_scale, (size_t)pc.uq_passes * UM_TOK);
    pc.cap_small = (int)std::min<size_t>(P, c.E);
    pc.cap_big = (int)(P / (GQ_SMALL + 1)) + 1;
    want(&pc.g_list, q4_slots((int)P, c.E)); want(&pc.g_slot, P);
    want(&pc.g_chunk, (size_t)3 * (pc.cap_small + pc.cap_big) + 2);
    want((uint16_t**)&pc.acth, P * 2 * c.I);
    want(&pc.xsum_tok, (size_t)W * (c.D / 64));
    want(&pc.xsum_act, P * std::max(1, c.I / 64));
    const size_t slots = q4_slots((int)P, c.E);
    want(&pc.sq, q4_plane_bytes(slots, std::max(c.D, c.I))); want(&pc.sq_scale, slots); want(&pc.sq_sum, slots * (size_t)(std::max(c.D, c.I) / 64 + 1));
    want(&pc.csel, (size_t)W * c.cores_active); want(&pc.cselw, (size_t)W * c.cores_active);
    want(&pc.cscore, (size_t)W * (c.n1 + c.n2)); want(&pc.core_y, (size_t)W * c.D);
    size_t total = 0;
    const size_t align = 1024;
    for (auto& part : parts) total += (part.second + align - 1) / align * align;
    if (const cudaError_t e = dalloc(&pc.arena, total); e != cudaSuccess) {
        free_chunk_bufs();
        cudaGetLastError();
        return fail("no memory for prompt chunks of %d tokens: %s", W, cudaGetErrorString(e));
    }
    total = 0;
    for (auto& part : parts) { *part.first = pc.arena + total; total += (part.second + align - 1) / align * align; }
    CU(cudaStreamSynchronize(cudaStreamLegacy));         // the buffers' zeroes (default stream) before the engine's stream uses them
    pc.W = W;
    return 0;
}

// T (CHUNK_MIN .. pc.W) tokens of the sequence in one pass over the layers (forward_chunk, aegist_rs/src/hybrid.rs:1023-1025)
int b2_engine::feed_chunk(const uint32_t* ids, int T, bool want_head) {
    CU(cudaMemcpyAsync(pc.tok, ids, (size_t)T * 4, cudaMemcpyHostToDevice, stream));
    if (enqueue_step(stream, false, T, want_head)) return 1;
    length += T;
    hits += (uint64_t)T * c.TOPK * c.L;
    toks.insert(toks.end(), ids, ids + T);
    return 0;
}

// ---- the persistent launch of a step of one sequence (step1.cuh) ---------------------------------------------------
struct Step1Shape { int sd, so, dk, hd, gh; const void* kernel; int smem_rest; };
#define S1_SHAPE(sd, so, dk, hd, gh) {sd, so, dk, hd, gh, (const void*)k_step1<sd, so, dk, hd, gh>, Step1Smem<sd, so, hd, gh>::TOTAL}
// widths the kernel is built for: d_model / 16, the mixers' output width / 16, key width of the delta rule, head width, expert
// hidden / 128. d_model from 1024 on: a stage takes 4 to 5 us whatever its width, which is what a launch of 512 values takes. Microseconds a
// token of eight layers, one launch against a launch per stage: d_model 512 235, 226; 1024 222, 275 (its head has fewer rows); 2048
// with mixers as wide 250, 290; with mixers of 4096 315, 368.
static const Step1Shape STEP1_SHAPES[] = {S1_SHAPE(64, 128, 128, 128, 2), S1_SHAPE(128, 128, 128, 128, 4), S1_SHAPE(128, 256, 128, 256, 4)};

// Rows of several matrices dealt out to G blocks in one go: block b owns the rows that start in its share of all bytes, in order, cut into
// tiles of at most seg.maxn rows. False if a block gets more tiles than it has room for.
struct Step1Seg { int rows, unit, maxn; };
static bool deal_tiles(const std::vector<Step1Seg>& segs, int G, int kind, std::vector<uint32_t>& tiles) {
    long total = 0, at = 0;
    for (const Step1Seg& s : segs) total += (long)s.rows * s.unit;
    std::vector<int> n(G, 0), last(G, -1);
    for (size_t si = 0; si < segs.size(); si++)
        for (int r = 0; r < segs[si].rows; r++, at += segs[si].unit) {
            int b = (int)(at * G / total);
            while (b + 1 < G && (long)(b + 1) * total / G <= at) b++;
            while (b > 0 && (long)b * total / G > at) b--;
            uint32_t* t = &tiles[(size_t)b * S1_TILES + s1_at(kind)];
            if (n[b] > 0 && last[b] == (int)si && (int)((t[n[b] - 1] >> 24) & 31) < segs[si].maxn) { t[n[b] - 1] += 1u << 24; continue; }
            if (n[b] == s1_cap(kind)) return false;
            t[n[b]++] = s1_tile((int)si, 1, r);
            last[b] = (int)si;
        }
    return true;
}

// The same where a few rows (`heavy`) take long to multiply: whole tiles of them go to blocks far apart, and the other rows fill the blocks up
// to an even height.
static bool deal_spread(const std::vector<Step1Seg>& heavy, const std::vector<Step1Seg>& rest, int G, int kind, std::vector<uint32_t>& tiles) {
    std::vector<int> n(G, 0);
    std::vector<long> used(G, 0);
    int nt = 0, at = 0;
    for (const Step1Seg& s : heavy) nt += (s.rows + s.maxn - 1) / s.maxn;
    for (size_t si = 0; si < heavy.size(); si++)
        for (int r = 0; r < heavy[si].rows; r += heavy[si].maxn, at++) {
            const int b = (int)((long)at * G / nt), m = std::min(heavy[si].maxn, heavy[si].rows - r);
            if (n[b] == s1_cap(kind)) return false;
            tiles[(size_t)b * S1_TILES + s1_at(kind) + n[b]++] = s1_tile((int)si, m, r);
            used[b] += (long)m * heavy[si].unit;
        }
    long rows = 0;
    for (const Step1Seg& s : rest) rows += s.rows;
    long height = 0, room = 0;
    while (room < rows) {
        height++;
        room = 0;
        for (int b = 0; b < G; b++) room += std::max(0L, height - used[b]);
    }
    int b = 0;
    for (size_t si = 0; si < rest.size(); si++)
        for (int r = 0; r < rest[si].rows;) {
            while (b < G && used[b] >= height) b++;
            if (b == G || n[b] == s1_cap(kind)) return false;
            const int m = (int)std::min<long>({(long)rest[si].maxn, (long)rest[si].rows - r, height - used[b]});
            tiles[(size_t)b * S1_TILES + s1_at(kind) + n[b]++] = s1_tile((int)(heavy.size() + si), m, r);
            used[b] += m;
            r += m;
        }
    return true;
}

// Which rows every one of G blocks multiplies, and the copies that fetch them: host arithmetic on the widths. n1, n2: rows of the core engine's
// tables (0, 0: this brain has none). False where the kernel is not built for the shape.
struct Step1Plan {
    const Step1Shape* sh = nullptr;
    int n8, h8, hb, ho, hp, hs, stage;             // rows of an int8 tile; where the second half of a tile's rows begins, by matrix; bytes of a tile
    std::vector<uint32_t> tiles;
    std::vector<S1Copy> copies;
};
static bool lay_out_step1(const Cfg& c, int G, int n1, int n2, bool kv_f32, Step1Plan& p) {
    const int hr = c.RD / 2;
    const bool rope_ok = c.RD > 0 && c.RD <= c.HD && hr % std::max(1, c.HD / 32) == 0;
    if (c.G != 64 || c.CK != 4 || c.TOPK > 8 || c.E > 256 || c.E % 8 || c.SH % 32 || c.SH > 512 || c.I % 128 || !rope_ok || c.H % c.KV || c.H / c.KV > 8 || c.KV > G ||
        c.HV % std::max(c.HK, 1) || (c.DV != 64 && c.DV != 128) || c.H * c.HD != c.VD() || c.D < G || (c.D + G - 1) / G > 16 || c.TOPK * c.I < G ||
        (c.TOPK * c.I + G - 1) / G > 32 || (c.n1 + c.n2) % 2 || c.V < G || c.V >= 1 << 24 ||
        c.V % 8 || c.C() % 8 || c.VD() % 8 || c.HV % 8 || (c.KV * c.HD) % 8 || c.SH % 8 || c.D % 8) return false;       // (the last: 16-byte pieces of their scales)
    for (const Step1Shape& s : STEP1_SHAPES)
        if (s.sd * 16 == c.D && s.so * 16 == c.VD() && s.dk == c.DK && s.hd == c.HD && s.gh * 128 == c.I) p.sh = &s;
    if (!p.sh) return false;
    // tiles: as many rows as make the longest share of the DeltaNet in-projections (the largest stage) a whole number of them
    const int VD = c.VD(), KO = VD, rd = (c.D + G - 1) / G, gp = (c.TOPK * c.I + G - 1) / G;
    const long u = ((long)c.C() + VD + 4L * c.HV + G - 1) / G;
    const int r = (int)((u + (u + 15) / 16 - 1) / ((u + 15) / 16));
    const int n8 = r, nb = std::max(1, std::min(8, r / 2)), no = std::max(1, std::min(8, (rd + 1) / 2)), np = std::max(1, std::min(8, r / 2 / 2 * 2));
    const int h8 = s1_half_at(n8, c.D), hb = s1_half_at(nb, 2 * c.D), ho = s1_half_at(no, KO), hp = s1_half_at(np, c.D), hs = s1_half_at(rd, c.SH);
    const int stage = (std::max({h8 + n8 / 2 * c.D, hb + nb / 2 * 2 * c.D, ho + no / 2 * KO, 3 * hp + np / 2 * c.D, hs + rd / 2 * c.SH,
                                 gp * (c.D / 2) + 64, c.TOPK * s1_dn_stride(rd, c.I / 2), 16 * c.HD * (kv_f32 ? 4 : 2), 4 * s1_gsc_stride(c.D) + 2 * c.TOPK * s1_dsc_stride(c.I)}) + 15) / 16 * 16;
    std::vector<uint32_t> tiles((size_t)G * S1_TILES, S1_NONE);
    if (!deal_spread({{c.HV, 2, nb}, {c.HV, 2, nb}}, {{c.C(), 1, n8}, {VD, 1, n8}}, G, S1_IN_DELTA, tiles) ||
        !deal_tiles({{2 * c.H * c.HD, 1, n8}, {c.KV * c.HD, 1, n8}, {c.KV * c.HD, 1, n8}}, G, S1_IN_ATTN, tiles) ||
        !deal_tiles({{c.D, 1, no}}, G, S1_OUT, tiles) ||
        !deal_tiles({{c.E, 1, nb}, {n1, 1, nb}, {n2, 1, nb}, {1, 1, nb}, {c.SH, 1, np}}, G, S1_MOE, tiles) ||
        !deal_tiles({{c.D, 1, 16}}, G, S1_SHD, tiles)) return false;
    // every block has its rows of the residual stream where the kernel expects them
    for (int b = 0; b < G; b++) {
        const uint32_t t = tiles[(size_t)b * S1_TILES + s1_at(S1_SHD)];
        const int r0 = (int)((long)b * c.D / G), r1 = (int)((long)(b + 1) * c.D / G);
        if (t != s1_tile(0, r1 - r0, r0) || (int)(tiles[(size_t)b * S1_TILES + s1_at(S1_OUT)] & 0xffffff) != r0) return false;
    }
    // the copies that fetch a tile: its two halves (four of a tile of gate-up pairs) and what the epilogue needs of its rows
    std::vector<S1Copy> copies((size_t)G * S1_TILES * S1_COPIES, S1Copy{0, 0});
    bool fits = true;
    for (int b = 0; b < G; b++)
        for (int kind = 0; kind < S1_KINDS; kind++)
            for (int i = 0; i < s1_cap(kind); i++) {
                const size_t ti = (size_t)b * S1_TILES + s1_at(kind) + i;
                if (tiles[ti] == S1_NONE) break;
                const int seg = tiles[ti] >> 29, n = (tiles[ti] >> 24) & 31, row0 = tiles[ti] & 0xffffff, h = (n + 1) / 2;
                S1Copy* to = &copies[ti * S1_COPIES];
                auto put = [&](int ptr, size_t from, size_t bytes, int at) {
                    if (bytes == 0) return;
                    if (from % 16 || bytes % 16 || at % 16 || bytes / 16 >= 4096 || at / 16 >= 2048 || from / 16 > 0xffffffffull || to == &copies[(ti + 1) * S1_COPIES]) { fits = false; return; }
                    *to++ = S1Copy{(uint32_t)ptr | (uint32_t)(at / 16) << 5 | (uint32_t)(bytes / 16) << 16, (uint32_t)(from / 16)};
                };
                const bool pair = kind == S1_MOE && seg == 4;
                const size_t rb = s1_is_bf(kind, seg) ? 2 * c.D : (kind == S1_OUT ? KO : (kind == S1_SHD ? c.SH : c.D));
                const int half = s1_is_bf(kind, seg) ? hb : (kind == S1_OUT ? ho : (kind == S1_SHD ? hs : (pair ? hp : h8)));
                const int ptr = kind <= S1_IN_ATTN ? seg : (kind == S1_OUT ? W_OUT : (kind == S1_MOE ? W_ROUTER + seg : W_SHD));
                for (int u = 0; u < (pair ? 2 : 1); u++) {
                    put(u ? (int)W_UP : ptr, row0 * rb, h * rb, u * 2 * hp);
                    put(u ? (int)W_UP : ptr, (row0 + h) * rb, (n - h) * rb, u * 2 * hp + half);
                }
                auto op = [&](int ptr, size_t size, int at) {
                    const size_t from = row0 * size / 16 * 16, end = ((row0 + n) * size + 15) / 16 * 16;
                    put(ptr, from, end - from, stage + at);
                };
                if (kind == S1_IN_DELTA && seg == 1) { op(Q_A_LOG, 2, 0); op(Q_DT, 2, 64); }
                if (kind == S1_IN_DELTA && seg >= 2) op(S_IN + seg - 2, 2, 0);
                if (kind == S1_IN_DELTA && seg == 2) { op(Q_CONV_W, 8, 128); op(Q_CONV_STATE, 12, 272); }
                if (kind == S1_IN_ATTN) op(S_IN + seg, 2, 0);
                if (kind == S1_OUT) op(S_OUT, 2, 0);
                if (kind == S1_SHD) op(S_SHD, 2, 0);
                if (kind == S1_MOE && seg == 0) op(Q_BIAS, 4, 64);
                if (pair) { op(S_GATE, 2, 0); op(S_UP, 2, 64); }
            }
    if (!fits) return false;
    p.n8 = n8; p.h8 = h8; p.hb = hb; p.ho = ho; p.hp = hp; p.hs = hs; p.stage = stage;
    p.tiles = std::move(tiles); p.copies = std::move(copies);
    return true;
}

// Decides whether steps of this engine run as one persistent launch, and lays out what that needs. Not an error if they do not.
int b2_engine::plan_step1() {
    const int G = nsm;
    if (B != 1 || ep_world != 1 || live_cores > 0 || getenv("B2_NO_STEP1")) return 0;
    bool keys = false;
    for (const LayerW& l : layers) keys = keys || l.key1;
    const int n1 = keys ? c.n1 : 0, n2 = keys ? c.n2 : 0;
    Step1Plan p;
    if (!lay_out_step1(c, G, n1, n2, kv_f32, p)) return 0;
    const Step1Shape* sh = p.sh;
    const int ns = G / c.KV, chunk = std::max(16, (cap + ns - 1) / ns), stage = p.stage;
    if ((chunk + KV_PAGE - 1) / KV_PAGE + 1 > S1_PAGES) return 0;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, sh->kernel) != cudaSuccess) { cudaGetLastError(); return 0; }
    if (!s1_regs_suffice(fa.numRegs)) return 0;
    const long room = 227 * 1024 - (long)fa.sharedSizeBytes - sh->smem_rest;
    const int nst = (int)std::min<long>(S1_MAXST, room / (stage + S1_OPS));
    if (nst < 5) return 0;         // the attention looks at two tiles of keys while their values are on their way, the experts at three of four
    const size_t smem = (size_t)nst * (stage + S1_OPS) + sh->smem_rest;
    int per_sm = 0;
    if (opt_in_smem(sh->kernel, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sh->kernel, S1_THREADS, smem) != cudaSuccess || per_sm < 1) { cudaGetLastError(); return 0; }
    Step1Args& a = s1.args;
    uint32_t at = 0;
    auto part = [&](uint32_t n) { const uint32_t o = at; at += (n + 15) / 16 * 16; return o; };
    a.o_xa = part(c.D); a.o_xb = part(c.D); a.o_q = part(std::max(c.C(), (2 * c.H + 2 * c.KV) * c.HD)); a.o_z = part(c.VD()); a.o_bg = part(2 * c.HV);
    a.o_og = part(c.VD()); a.o_rl = part(c.E); a.o_sa = part(c.SH); a.o_sg = part(1); a.o_act = part(c.TOPK * c.I);
    a.ll_set = at;
    at *= 2;
    a.o_ap = part(c.KV * ns * 8 * (c.HD + 2)); a.cs_words = (n1 + n2 + 15) / 16 * 16; a.o_cs = part(c.L * a.cs_words);
    CU(dalloc(&s1.ll, at));
    CU(dalloc(&s1.tiles, p.tiles.size(), false));
    CU(cudaMemcpy(s1.tiles, p.tiles.data(), p.tiles.size() * 4, cudaMemcpyHostToDevice));
    CU(dalloc(&s1.copies, p.copies.size(), false));
    CU(cudaMemcpy(s1.copies, p.copies.data(), p.copies.size() * sizeof(S1Copy), cudaMemcpyHostToDevice));
    CU(dalloc(&s1.epoch, 1));
    CU(dalloc(&s1.layers, c.L, false));
    if (G > head_grid) {                       // the arg-max' scratch: one place per block
        cudaFree(part_val); cudaFree(part_idx);
        part_val = nullptr; part_idx = nullptr;
        CU(dalloc(&part_val, G)); CU(dalloc(&part_idx, G));
    }
    a.layers = s1.layers; a.tiles = s1.tiles; a.embed = embed; a.norm = norm; a.head_w = lm_head.w; a.head_s = lm_head.s; a.logits = logits; a.x = x; a.ll = s1.ll;
    a.epoch = s1.epoch; a.rope_cos = rope_cos; a.rope_sin = rope_sin; a.page_table = page_table; a.scale = 1.0f / std::sqrt((float)c.HD); a.eps = c.eps;
    a.L = c.L; a.V = c.V; a.E = c.E; a.topk = c.TOPK; a.I = c.I; a.SH = c.SH; a.HK = c.HK; a.HV = c.HV; a.DV = c.DV; a.H = c.H; a.KV = c.KV; a.RD = c.RD; a.C = c.C();
    a.n1 = n1; a.n2 = n2; a.cores_k = c.cores_active; a.kv_f32 = kv_f32; a.half_i8 = p.h8; a.half_bf = p.hb; a.half_out = p.ho; a.half_pair = p.hp; a.half_shd = p.hs; a.copies = s1.copies; a.kv_tile = std::min(64, stage / (c.HD * (kv_f32 ? 4 : 2))); a.head_rows = p.n8; a.nst = nst; a.stage_bytes = stage + S1_OPS;
    a.expert_bytes = c.expert_bytes(); a.off_gu_s = c.off_gu_s(); a.off_gu_m = c.off_gu_m(); a.off_dn_q = c.off_dn_q(); a.off_dn_s = c.off_dn_s(); a.off_dn_m = c.off_dn_m();
    a.cscore = cscore; a.csel = csel; a.cselw = cselw; a.part_val = part_val; a.part_idx = part_idx; a.next_tok = d_next; a.pos = d_pos; a.tok = d_tok;
    a.hist = TokHist{d_hist, cap, 1}; a.counter = d_counter; a.err = d_err; a.polls = S1_SPINS;
    s1.smem = smem;
    s1.stages = 1;
    for (const LayerW& l : layers) s1.stages += l.attn ? 7 : 6;
    if (s1.stages > TRACE_MAX_LAUNCHES) return 0;
    for (cudaEvent_t& e : s1.done) CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    s1.kernel = sh->kernel;
    enter_step1(this);
    return 0;
}

// The table of the layers' pointers; again whenever the tapped layers change. A layer tapped twice has one place only: launches per stage then.
int b2_engine::upload_step1() {
    if (!s1.layers) return 0;
    s1.off = false;
    std::vector<Step1Layer> tab(c.L);
    const size_t kv_layer = (size_t)pages_per_seq * c.KV * KV_PAGE * c.HD * (kv_f32 ? 4 : 2);
    for (int i = 0; i < c.L; i++) {
        const LayerW& l = layers[i];
        Step1Layer& t = tab[i];
        t = Step1Layer{};
        auto put = [&](int wi, int si, const QWd& q) { t.w[wi] = q.w; if (si >= 0) t.s[si] = q.s; };
        if (l.attn) {
            put(0, 0, l.q); put(1, 1, l.k); put(2, 2, l.v); put(4, 3, l.o);
            t.n_a = l.q_norm; t.n_b = l.k_norm;
            t.kpool = (char*)kpool + kv_layer * l.slot; t.vpool = (char*)vpool + kv_layer * l.slot;
        } else {
            t.w[0] = l.in_b; t.w[1] = l.in_a; put(2, 0, l.in_qkv); put(3, 1, l.in_z); put(4, 3, l.out);
            t.n_a = l.gnorm; t.conv_w = l.conv; t.a_log = l.a_log; t.dt_bias = l.dt_bias;
            t.conv_state = conv + (size_t)l.slot * c.C() * 3; t.state = state + (size_t)l.slot * c.HV * c.DK * c.DV;
        }
        t.w[5] = l.router; t.w[6] = l.key1; t.w[7] = l.key2; t.w[8] = l.sh_gw;      // (a layer without keys among layers with them: nothing is copied)
        put(9, 4, l.sh_gate); put(10, 5, l.sh_up); put(11, 6, l.sh_down);
        t.norm1 = l.norm1; t.norm2 = l.norm2; t.bias = l.router_bias; t.experts = l.experts;
        t.counts = l.key1 ? d_counts + (size_t)i * c.n1 * c.n2 : nullptr;
        t.top_idx = top_idx + (size_t)i * c.TOPK; t.top_w = top_w + (size_t)i * c.TOPK; t.attn = l.attn;
        int taps = 0;
        for (size_t j = 0; j < tap_layers.size(); j++)
            if (tap_layers[j] == i) { t.tap = tap_buf + j * (size_t)c.D; taps++; }
        if (taps > 1) s1.off = true;
    }
    CU(cudaMemcpyAsync(s1.layers, tab.data(), tab.size() * sizeof(Step1Layer), cudaMemcpyHostToDevice, stream));       // (the steps' own stream)
    CU(cudaStreamSynchronize(stream));
    return 0;
}

int b2_engine::launch_step1(cudaStream_t st) {
    Step1Args a = s1.args;
    a.trace = g_trace_base;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nsm);
    cfg.blockDim = dim3(S1_THREADS);
    cfg.dynamicSmemBytes = s1.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;       // its blocks wait on one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* p[] = {&a};
    g_launch_count++;
    const cudaError_t e = cudaLaunchKernelExC(&cfg, s1.kernel, p);
    if (e != cudaSuccess) return fail("step launch: %s", cudaGetErrorString(e));
    return 0;
}

// Persistent launches of two engines of a process must not hold half of a GPU's SMs each and wait for the other half: an engine that
// follows another one on a device waits for the event behind that one's last step. Every engine records its own: its stream belongs to its
// thread, which may be capturing on it. Where there are several, a greedy loop queues no more than STEP1_AHEAD steps: who asks for one step
// beside a loop of a thousand gets its turn after two of them. Two are enough to keep the GPU busy: a step is longer than a launch.
// Beside a loop of 1000 steps of 40 layers a step took 1201 ms and takes 3.8 ms (as launches, which share the GPU: 2.6). Engines that decode at
// the same time get no more tokens between them than one alone, 1.29 ms a token; as launches of their own 1.23 ms for two, 1.13 for three.
struct Step1Turns { b2_engine* last = nullptr; int engines = 0; };
static std::mutex g_step1_mutex;
static std::map<int, Step1Turns> g_step1_turns;         // by device
cudaError_t b2_engine::run_graph(cudaGraphExec_t g) {
    if (!use_step1()) return cudaGraphLaunch(g, stream);
    std::lock_guard<std::mutex> lock(g_step1_mutex);
    Step1Turns& turns = g_step1_turns[device];
    const Step1* before = turns.last && turns.last != this ? &turns.last->s1 : nullptr;
    cudaError_t e = before ? cudaStreamWaitEvent(stream, before->done[(before->steps - 1) % STEP1_AHEAD], 0) : cudaSuccess;
    if (e == cudaSuccess) e = cudaGraphLaunch(g, stream);
    if (e != cudaSuccess) return e;
    turns.last = this;
    return cudaEventRecord(s1.done[s1.steps++ % STEP1_AHEAD], stream);
}
// before one more step of a loop
cudaError_t b2_engine::await_turn() {
    if (!use_step1()) return cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_step1_mutex);
        if (g_step1_turns[device].engines < 2) return cudaSuccess;
    }
    return cudaEventSynchronize(s1.done[s1.steps % STEP1_AHEAD]);
}
static void enter_step1(b2_engine* e) {
    std::lock_guard<std::mutex> lock(g_step1_mutex);
    g_step1_turns[e->device].engines++;
}
static void leave_step1(b2_engine* e) {
    if (!e->s1.kernel) return;
    std::lock_guard<std::mutex> lock(g_step1_mutex);
    Step1Turns& turns = g_step1_turns[e->device];
    turns.engines--;
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (turns.last == e) turns.last = nullptr;
}

int b2_engine::build_graph() {
    CU(cudaSetDevice(device));
    if (graph) { cudaGraphExecDestroy(graph); graph = nullptr; }
    if (upload_step1()) return 1;
    cudaGraph_t g;
    CU(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue_step(stream, true);
    cudaError_t e = cudaStreamEndCapture(stream, &g);
    if (rc) return rc;
    if (e != cudaSuccess) return fail("graph capture: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail("graph instantiate: %s", cudaGetErrorString(e));
    return 0;
}

// The device error word travels to page-locked memory on the stream, so a feed pays one synchronisation for its
// results and the check together.
int b2_engine::check_device_error() {
    uint32_t* slot = h_pin + 2 * std::max(B, 1);
    CU(cudaMemcpyAsync(slot, d_err, 4, cudaMemcpyDeviceToHost, stream));
    CU(cudaStreamSynchronize(stream));
    const int h = (int)*slot;
    if (h) {
        cudaMemsetAsync(d_err, 0, 4, stream);
        cudaStreamSynchronize(stream);
        if (h == 1) return fail("a token id is outside the vocabulary (%d)", c.V);
        if (h == 3) return fail("a bulk copy into shared memory did not complete (bounded wait gave up)");
        if (h == 4) return fail("a block waited too long for another block's results (bounded wait gave up)");
        if (h == 5) return fail("another rank's part of the expert exchange did not arrive (bounded wait gave up)");
        return fail("router returned an expert outside 0..%d", c.E - 1);
    }
    return 0;
}

int b2_engine::run_steps(int n) {
    for (int i = 0; i < n; i++) {
        if (i >= STEP1_AHEAD) CU(await_turn());
        CU(run_graph(graph));
    }
    if (ep_world > 1) ep_steps += n;
    length += n;
    hits += (uint64_t)n * B * c.TOPK * c.L;
    return 0;
}

int b2_engine::reset_state() {
    CU(cudaMemsetAsync(conv, 0, conv_bytes, stream));
    CU(cudaMemsetAsync(state, 0, state_bytes, stream));
    CU(cudaMemsetAsync(d_pos, 0, B * 4, stream));
    length = 0;
    toks.clear();
    toks_known = true;
    snap_pos[0] = snap_pos[1] = -1;
    return 0;
}

int b2_engine::load_nccl() {
    if (p_ncclAllGather) return 0;
    const char* names[] = {getenv("B2_NCCL_LIB"), "libnccl.so.2", "libnccl.so"};
    for (const char* n : names) {
        if (!n) continue;
        nccl_lib = dlopen(n, RTLD_NOW | RTLD_NOLOAD);        // the copy this process already uses, if any
        if (!nccl_lib) nccl_lib = dlopen(n, RTLD_NOW | RTLD_GLOBAL);
        if (nccl_lib) break;
    }
    if (!nccl_lib) return fail("cannot load NCCL (libnccl.so.2): %s", dlerror());
#define SYM(name) *(void**)(&p_##name) = dlsym(nccl_lib, #name); if (!p_##name) return fail("NCCL has no %s", #name);
    SYM(ncclGetUniqueId) SYM(ncclCommInitRank) SYM(ncclCommDestroy) SYM(ncclAllGather) SYM(ncclSend) SYM(ncclRecv)
    SYM(ncclGroupStart) SYM(ncclGroupEnd) SYM(ncclGetErrorString)
#undef SYM
    return 0;
}
#define NC(call)                                                                                   \
    do {                                                                                           \
        ncclResult_t r_ = (call);                                                                  \
        if (r_ != ncclSuccess) return fail("%s: %s", #call, p_ncclGetErrorString(r_));             \
    } while (0)

// every GPU's records [B][D + 2 topk] -> all records, in rank order
int b2_engine::ep_exchange_records(cudaStream_t st) {
    const size_t n = (size_t)B * (c.D + 2 * c.TOPK);
    NC(p_ncclAllGather(rec_local, rec_all, n, ncclFloat32, comm, st));
    return 0;
}
// block p of ypart (the picks of GPU p's sequences computed here) goes to GPU p; block q of recv_y comes from GPU q
int b2_engine::ep_exchange_outputs(cudaStream_t st) {
    const size_t blk = (size_t)B * (c.TOPK + 1) * c.D;
    NC(p_ncclGroupStart());
    for (int p = 0; p < ep_world; p++) {
        NC(p_ncclSend(ypart + p * blk, blk, ncclFloat32, p, comm, st));
        NC(p_ncclRecv(recv_y + p * blk, blk, ncclFloat32, p, comm, st));
    }
    NC(p_ncclGroupEnd());
    return 0;
}

// Algorithmic bytes of one decode step by kernel class (0 embed, 1 norm+GEMV groups, 2 delta step,
// 3 attention, 4 output projections, 5 expert gate/up, 6 expert down + shared down, 7 head):
// every weight byte once per step, recurrent state read and written, KV read up to the current length,
// min(B * top-k, E) experts per layer. Activations are not counted.
void b2_engine::class_bytes(double out[8]) const {
    for (int i = 0; i < 8; i++) out[i] = 0;
    auto qwb = [](double n, double k) { return n * k + 2 * n; };
    const double nb = B;
    const double uniq = std::min<double>(nb * c.TOPK, c.E / ep_world);
    out[0] = nb * c.D * 2.0;
    for (int i = 0; i < c.L; i++) {
        if (c.attn[i]) {
            out[1] += c.D * 2.0 + qwb(2 * c.H * c.HD, c.D) + 2 * qwb(c.KV * c.HD, c.D);
            out[3] += 2.0 * c.HD * 2 + nb * 2.0 * c.KV * c.HD * (kv_f32 ? 4 : 2) * (length + 1);
            out[4] += qwb(c.D, c.H * c.HD);
        } else {
            out[1] += c.D * 2.0 + qwb(c.C(), c.D) + qwb(c.VD(), c.D) + 2.0 * c.HV * c.D * 2 + c.C() * c.CK * 2.0 + c.HV * 4.0 +
                      nb * 2.0 * c.C() * 3 * 4;
            out[2] += nb * 2.0 * c.HV * c.DK * c.DV * 4;
            out[4] += qwb(c.D, c.VD()) + c.DV * 2.0;
        }
        out[1] += c.D * 2.0 + (double)c.E * c.D * 2 + c.D * 2.0 + 2 * qwb(c.SH, c.D) + (layers[i].key1 ? (c.n1 + c.n2) * c.D * 2.0 : 0.0);
        out[5] += uniq * (double)(c.gu_q() + 2 * c.gu_sm()) + c.D * 2.0;
        out[6] += uniq * (double)(c.dn_q() + 2 * c.dn_sm()) + qwb(c.D, c.SH);
    }
    out[7] = c.D * 2.0 + qwb(c.V, c.D);
}

// ------------------------------------------------------------------------------------------
extern "C" {

int b2_create(const char* config_json, int max_context, int device, int batch, int kv_dtype, int ep_rank, int ep_world,
              b2_engine** out) {
    if (!out) return 1;
    b2_engine* e = new b2_engine();
    *out = e;
    e->device = device;
    e->B = batch < 1 ? 1 : batch;
    e->cap = max_context;
    e->kv_f32 = kv_dtype == B2_KV_F32;
    e->ep_rank = ep_rank;
    e->ep_world = ep_world < 1 ? 1 : ep_world;
    if (ep_rank < 0 || ep_rank >= e->ep_world) return e->fail("expert-parallel rank %d outside 0..%d", ep_rank, e->ep_world - 1);
    int ndev = 0;
    cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev == 0) return e->fail("no CUDA device: %s (this engine has no CPU path)", cudaGetErrorString(ce));
    if (device < 0 || device >= ndev) return e->fail("CUDA device %d does not exist (%d visible)", device, ndev);
    JValue j;
    std::string jerr;
    JParser parser(config_json, strlen(config_json));
    if (!parser.parse(j, jerr)) return e->fail("bad config JSON: %s", jerr.c_str());
    return e->parse_config(j);
}

int b2_put_tensor(b2_engine* e, const char* name, const char* dtype, const int64_t* shape, int ndim, const void* data,
                  size_t nbytes, int data_on_device) {
    if (!e) return 1;
    return e->put(name, dtype, std::vector<int64_t>(shape, shape + ndim), data, nbytes, data_on_device != 0);
}

int b2_finish(b2_engine* e) { return e ? e->finish() : 1; }

int b2_ep_unique_id(b2_engine* e, void* id_out, size_t len) {
    if (!e) return 1;
    if (len < sizeof(ncclUniqueId)) return e->fail("the id buffer needs %zu bytes", sizeof(ncclUniqueId));
    if (e->load_nccl()) return 1;
    ncclUniqueId id;
    ncclResult_t r = e->p_ncclGetUniqueId(&id);
    if (r != ncclSuccess) return e->fail("ncclGetUniqueId: %s", e->p_ncclGetErrorString(r));
    memcpy(id_out, &id, sizeof(id));
    return 0;
}

int b2_ep_init(b2_engine* e, const void* id_in, size_t len) {
    if (!e || !e->finished) return 1;
    if (e->ep_world <= 1) return e->fail("this engine was created for a single GPU");
    if (len < sizeof(ncclUniqueId)) return e->fail("the id buffer needs %zu bytes", sizeof(ncclUniqueId));
    if (e->load_nccl()) return 1;
    cudaError_t ce = cudaSetDevice(e->device);
    if (ce != cudaSuccess) return e->fail("cudaSetDevice: %s", cudaGetErrorString(ce));
    ncclUniqueId id;
    memcpy(&id, id_in, sizeof(id));
    ncclResult_t r = e->p_ncclCommInitRank(&e->comm, e->ep_world, id, e->ep_rank);
    if (r != ncclSuccess) return e->fail("ncclCommInitRank: %s", e->p_ncclGetErrorString(r));
    // one exchange of each kind outside the graph: NCCL sets up its channels on first use
    if (e->ep_exchange_records(e->stream) || e->ep_exchange_outputs(e->stream)) return 1;
    ce = cudaStreamSynchronize(e->stream);
    if (ce != cudaSuccess) return e->fail("first exchange: %s", cudaGetErrorString(ce));
    return e->build_graph();
}

int b2_ep_ipc_handle(b2_engine* e, void* out, size_t len) {
    if (!e || !e->finished) return 1;
    if (e->ep_world <= 1 || !e->ep_block) return e->fail("this engine was created for a single GPU");
    if (len < sizeof(cudaIpcMemHandle_t)) return e->fail("the handle buffer needs %zu bytes", sizeof(cudaIpcMemHandle_t));
    cudaIpcMemHandle_t h;
    cudaError_t ce = cudaSetDevice(e->device);
    if (ce == cudaSuccess) ce = cudaIpcGetMemHandle(&h, e->ep_block);
    if (ce != cudaSuccess) return e->fail("cudaIpcGetMemHandle: %s", cudaGetErrorString(ce));
    memcpy(out, &h, sizeof(h));
    return 0;
}

int b2_ep_ipc_attach(b2_engine* e, const void* handles, size_t len_each, int n) {
    if (!e || !e->finished) return 1;
    if (e->ep_world <= 1 || !e->ep_block) return e->fail("this engine was created for a single GPU");
    if (n != e->ep_world || n > EP_MAX_WORLD || len_each < sizeof(cudaIpcMemHandle_t))
        return e->fail("expected %d handles of %zu bytes (at most %d ranks)", e->ep_world, sizeof(cudaIpcMemHandle_t), EP_MAX_WORLD);
    if (e->ep_peer_ready) return e->fail("the peers' blocks are mapped already");
    if (e->c.D % 4 != 0 || (2 * e->c.TOPK) % 4 != 0) return e->fail("the peer-store exchange needs d_model and 2 x experts_active to be multiples of 4 (16-byte rows)");
    cudaError_t ce = cudaSetDevice(e->device);
    if (ce != cudaSuccess) return e->fail("cudaSetDevice: %s", cudaGetErrorString(ce));
    for (int p = 0; p < n; p++) {
        if (p == e->ep_rank) { e->ep_peer[p] = e->ep_block; continue; }
        cudaIpcMemHandle_t h;
        memcpy(&h, (const char*)handles + (size_t)p * len_each, sizeof(h));
        void* ptr = nullptr;
        ce = cudaIpcOpenMemHandle(&ptr, h, cudaIpcMemLazyEnablePeerAccess);
        if (ce != cudaSuccess) {
            for (int q = 0; q < p; q++) if (q != e->ep_rank && e->ep_peer[q]) { cudaIpcCloseMemHandle(e->ep_peer[q]); e->ep_peer[q] = nullptr; }
            cudaGetLastError();
            return e->fail("cudaIpcOpenMemHandle (rank %d): %s", p, cudaGetErrorString(ce));
        }
        e->ep_peer[p] = (float*)ptr;
    }
    e->ep_peer_ready = true;
    return e->comm ? e->build_graph() : 0;          // the step graph holds the exchange's launches
}

int b2_open(const char* nx_path, int max_context, int device, int batch, int kv_dtype, b2_engine** out) {
    if (!out) return 1;
    *out = nullptr;
    NxFile nx;
    std::string err;
    if (!nx.open(nx_path, err)) {
        b2_engine* e = new b2_engine();
        *out = e;
        return e->fail("%s", err.c_str());
    }
    const JValue* cfg = nx.header.get("config");
    // re-serialise the config object: find it in the raw header is not needed, rebuild minimal JSON
    std::string js = "{";
    if (cfg && cfg->type == JValue::Obj) {
        bool first = true;
        for (auto& kv : cfg->obj) {
            const JValue& v = kv.second;
            std::string s;
            char buf[64];
            if (v.type == JValue::Num) { snprintf(buf, sizeof(buf), "%.17g", v.num); s = buf; }
            else if (v.type == JValue::Bool) s = v.b ? "true" : "false";
            else if (v.type == JValue::Str) s = "\"" + v.str + "\"";
            else if (v.type == JValue::Arr) {
                s = "[";
                for (size_t i = 0; i < v.arr.size(); i++) {
                    if (i) s += ",";
                    if (v.arr[i].type == JValue::Num) { snprintf(buf, sizeof(buf), "%.17g", v.arr[i].num); s += buf; }
                    else if (v.arr[i].type == JValue::Str) s += "\"" + v.arr[i].str + "\"";
                    else s += "null";
                }
                s += "]";
            } else s = "null";
            js += std::string(first ? "" : ",") + "\"" + kv.first + "\":" + s;
            first = false;
        }
    }
    js += "}";
    int rc = b2_create(js.c_str(), max_context, device, batch, kv_dtype, 0, 1, out);
    if (rc) return rc;
    b2_engine* e = *out;
    e->fingerprint = nx.fingerprint();
    for (auto& kv : nx.tensors) {
        const NxTensor& t = kv.second;
        if (e->put(kv.first, t.dtype, t.shape, nx.data(t), t.nbytes, false)) return 1;
    }
    return e->finish();
}

int b2_verify_file(const char* nx_path, int ok[3], char* err, size_t err_len) {
    NxFile nx;
    std::string msg;
    if (!nx.open(nx_path, msg)) {
        if (err && err_len) snprintf(err, err_len, "%s", msg.c_str());
        return 1;
    }
    auto r = nx.verify();
    ok[0] = r["base"]; ok[1] = r["engine"]; ok[2] = r["cores"];
    return 0;
}

void b2_close(b2_engine* e) { delete e; }

static int feed_checks(b2_engine* e, int n) {
    if (!e) return 1;
    if (!e->finished) return e->fail("the engine is not loaded (b2_finish has not succeeded)");
    if (e->length + n > e->cap) return e->fail("context full: %d + %d tokens > %d", e->length, n, e->cap);
    cudaError_t ce = cudaSetDevice(e->device);
    if (ce != cudaSuccess) return e->fail("cudaSetDevice: %s", cudaGetErrorString(ce));
    return 0;
}
#define CUE(call)                                                                                      \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return e->fail("%s: %s", #call, cudaGetErrorString(e_));                \
    } while (0)

int b2_feed(b2_engine* e, const uint32_t* ids, int n, float* logits_out) {
    if (e && e->B != 1) return e->fail("b2_feed needs an engine opened with batch 1 (this one has %d)", e->B);
    if (e && n < 1) return e->fail("b2_feed needs at least one token");
    if (feed_checks(e, n)) return 1;
    for (int i = 0; i < n; i++)
        if (ids[i] >= (uint32_t)e->c.V) return e->fail("token id %u is outside the vocabulary (%d)", ids[i], e->c.V);
    int i0 = 0;
    // a prompt goes through the layers in chunks of equal length (no short rest); a feed of fewer than CHUNK_MIN tokens token by token
    if (n >= CHUNK_MIN && e->ep_world == 1) {
        // shorter chunks where the GPU has no room for the buffers of the longest (0.4 MB a token at the 35B shape)
        int nchunk = (n + CHUNK_TOKENS - 1) / CHUNK_TOKENS;
        for (int t = CHUNK_TOKENS; e->ensure_chunk_bufs((n + nchunk - 1) / nchunk); nchunk = (n + t - 1) / t) {
            t /= 2;
            if (t < 64) return 1;
        }
        for (int k = 0; k < nchunk; k++) {
            const int i1 = (int)((long)n * (k + 1) / nchunk);
            if (e->feed_chunk(ids + i0, i1 - i0, i1 == n)) return 1;
            i0 = i1;                 // (the caller's ids are read by stream-ordered copies; the stream is drained before we return)
        }
    }
    for (int i = i0; i < n; i++) {
        // the id travels as a kernel-independent 4-byte copy ordered on the stream
        CUE(cudaMemcpyAsync(e->d_tok, ids + i, 4, cudaMemcpyHostToDevice, e->stream));
        if (e->run_steps(1)) return 1;
        e->toks.push_back(ids[i]);
    }
    if (logits_out) CUE(cudaMemcpyAsync(logits_out, e->logits, (size_t)e->c.V * 4, cudaMemcpyDeviceToHost, e->stream));
    return e->check_device_error();
}

void* b2_host_alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}
void b2_host_free(void* p) {
    if (p) cudaFreeHost(p);
}

int b2_feed_batch(b2_engine* e, const uint32_t* ids, uint32_t* next_greedy, float* logits_out) {
    if (feed_checks(e, 1)) return 1;
    for (int b = 0; b < e->B; b++)
        if (ids[b] >= (uint32_t)e->c.V) return e->fail("token id %u is outside the vocabulary (%d)", ids[b], e->c.V);
    memcpy(e->h_pin, ids, (size_t)e->B * 4);
    CUE(cudaMemcpyAsync(e->d_tok, e->h_pin, (size_t)e->B * 4, cudaMemcpyHostToDevice, e->stream));
    if (e->run_steps(1)) return 1;
    if (e->B == 1) e->toks.push_back(ids[0]); else e->toks_known = false;
    if (next_greedy) CUE(cudaMemcpyAsync(e->h_pin + e->B, e->d_next, (size_t)e->B * 4, cudaMemcpyDeviceToHost, e->stream));
    if (logits_out) CUE(cudaMemcpyAsync(logits_out, e->logits, (size_t)e->B * e->c.V * 4, cudaMemcpyDeviceToHost, e->stream));
    if (e->check_device_error()) return 1;
    if (next_greedy) memcpy(next_greedy, e->h_pin + e->B, (size_t)e->B * 4);
    return 0;
}

int b2_decode_greedy(b2_engine* e, const uint32_t* first, int steps, uint32_t* tokens_out, float* device_ms) {
    if (e && steps < 1) return e->fail("b2_decode_greedy needs at least one step");
    if (feed_checks(e, steps)) return 1;
    const int B = e->B;
    for (int b = 0; b < B; b++)
        if (first[b] >= (uint32_t)e->c.V) return e->fail("token id %u is outside the vocabulary (%d)", first[b], e->c.V);
    memcpy(e->h_pin, first, (size_t)B * 4);
    CUE(cudaMemcpyAsync(e->d_tok, e->h_pin, (size_t)B * 4, cudaMemcpyHostToDevice, e->stream));
    const int p0 = e->length;
    CUE(cudaEventRecord(e->ev0, e->stream));
    if (e->run_steps(steps)) return 1;   // a step leaves its arg-max where the next one reads its input, and in the history
    CUE(cudaEventRecord(e->ev1, e->stream));
    CUE(cudaMemcpyAsync(tokens_out, e->d_hist + (size_t)p0 * B, (size_t)steps * B * 4, cudaMemcpyDeviceToHost, e->stream));
    CUE(cudaStreamSynchronize(e->stream));
    if (B == 1) {                       // fed: the first token, then every arg-max but the last
        e->toks.push_back(first[0]);
        for (int s = 0; s + 1 < steps; s++) e->toks.push_back(tokens_out[s]);
    } else e->toks_known = false;
    if (device_ms) CUE(cudaEventElapsedTime(device_ms, e->ev0, e->ev1));
    return e->check_device_error();
}

// Lm::crop (aegist_rs/src/hybrid.rs:1029-1059)
int b2_crop(b2_engine* e, int n) {
    if (!e || !e->finished) return -1;
    if (n >= e->length) return e->length;
    cudaSetDevice(e->device);
    int best = -1;
    for (int i = 0; i < 2; i++)
        if (e->snap_pos[i] >= 0 && e->snap_pos[i] <= n && (best < 0 || e->snap_pos[i] > e->snap_pos[best])) best = i;
    bool ok = false;
    if (best >= 0) {
        ok = cudaMemcpyAsync(e->conv, e->snap_conv[best], e->conv_bytes, cudaMemcpyDeviceToDevice, e->stream) == cudaSuccess &&
             cudaMemcpyAsync(e->state, e->snap_state[best], e->state_bytes, cudaMemcpyDeviceToDevice, e->stream) == cudaSuccess;
    }
    if (ok) {
        const int p = (int)e->snap_pos[best];
        e->length = p;
        if ((int)e->toks.size() >= p) e->toks.resize(p);
        k_fill_i32<<<(e->B + 255) / 256, 256, 0, e->stream>>>(e->d_pos, p, e->B);
        for (int i = 0; i < 2; i++) if (e->snap_pos[i] > p) e->snap_pos[i] = -1;
    } else {
        e->reset_state();
    }
    cudaStreamSynchronize(e->stream);
    return e->length;
}

// Lm::snapshot (aegist_rs/src/hybrid.rs:1061-1072)
int b2_snapshot(b2_engine* e) {
    if (!e || !e->finished) return 1;
    for (int i = 0; i < 2; i++) if (e->snap_pos[i] == e->length) return 0;
    int i = (e->snap_pos[0] <= e->snap_pos[1]) ? 0 : 1;   // an empty slot (-1), else the oldest
    CUE(cudaSetDevice(e->device));
    CUE(cudaMemcpyAsync(e->snap_conv[i], e->conv, e->conv_bytes, cudaMemcpyDeviceToDevice, e->stream));
    CUE(cudaMemcpyAsync(e->snap_state[i], e->state, e->state_bytes, cudaMemcpyDeviceToDevice, e->stream));
    CUE(cudaStreamSynchronize(e->stream));
    e->snap_pos[i] = e->length;
    return 0;
}

// ---- saved states (trait Lm::state_key / save_state / load_state, aegist_rs/src/model.rs:375-387) ----
// File format of the reference's engines that save states (aegist_rs/src/next.rs:2442-2548): "AEGSTATE", u64 LE
// header length, JSON {"key", "toks"}, then layer by layer what the first n tokens left behind: an attention
// layer's keys and values per KV head (n rows each), a DeltaNet layer's conv taps [C][3] and state [HV][DK][DV].
std::string b2_engine::state_key() const {
    char buf[96];
    snprintf(buf, sizeof(buf), "-%dx%dx%d%s", c.L, c.KV, c.HD, kv_f32 ? "-kvf32" : "");
    return (fingerprint.empty() ? std::string("tensors") : fingerprint) + buf;
}
// (device address, bytes) of every piece in file order; the KV rows of a head are contiguous within a 64-token page
std::vector<b2_engine::Piece> b2_engine::state_pieces(int n) const {
    std::vector<Piece> v;
    const size_t esz = kv_f32 ? 4 : 2;
    const size_t kv_layer = (size_t)B * pages_per_seq * c.KV * KV_PAGE * c.HD * esz;
    for (const LayerW& l : layers) {
        if (l.attn) {
            for (int h = 0; h < c.KV; h++)
                for (int which = 0; which < 2; which++)
                    for (int p0 = 0; p0 < n; p0 += KV_PAGE) {
                        const int rows = std::min(KV_PAGE, n - p0);
                        char* pool = (char*)(which ? vpool : kpool) + kv_layer * l.slot;
                        v.push_back({pool + (((size_t)(p0 / KV_PAGE) * c.KV + h) * KV_PAGE) * c.HD * esz, (size_t)rows * c.HD * esz});
                    }
        } else {
            v.push_back({(char*)(conv + (size_t)l.slot * B * c.C() * 3), (size_t)c.C() * 3 * 4});
            v.push_back({(char*)(state + (size_t)l.slot * B * c.HV * c.DK * c.DV), (size_t)c.HV * c.DK * c.DV * 4});
        }
    }
    return v;
}

const char* b2_state_key(const b2_engine* e) {
    static thread_local std::string k;
    k = e ? e->state_key() : "";
    return k.c_str();
}

int b2_save_state(b2_engine* e, const char* path) {
    if (!e || !e->finished) return 1;
    if (e->B != 1) return e->fail("states are saved for one sequence (this engine has %d)", e->B);
    if (!e->toks_known || (int)e->toks.size() != e->length) return e->fail("the tokens of this context are not all known to the host (device-side steps were run)");
    CUE(cudaSetDevice(e->device));
    CUE(cudaStreamSynchronize(e->stream));
    const int n = e->length;
    std::string head = "{\"key\":\"" + e->state_key() + "\",\"toks\":[";
    for (int i = 0; i < n; i++) head += (i ? "," : "") + std::to_string(e->toks[i]);
    head += "]}";
    const std::string tmp = std::string(path) + ".tmp";
    FILE* f = fopen(tmp.c_str(), "wb");
    if (!f) return e->fail("%s: %s", tmp.c_str(), strerror(errno));
    const uint64_t hl = head.size();
    bool ok = fwrite("AEGSTATE", 1, 8, f) == 8 && fwrite(&hl, 8, 1, f) == 1 && fwrite(head.data(), 1, head.size(), f) == head.size();
    std::vector<char> buf;
    for (auto& pc : e->state_pieces(n)) {
        if (!ok) break;
        buf.resize(pc.bytes);
        if (cudaMemcpy(buf.data(), pc.p, pc.bytes, cudaMemcpyDeviceToHost) != cudaSuccess) { ok = false; break; }
        ok = fwrite(buf.data(), 1, pc.bytes, f) == pc.bytes;
    }
    ok = (fclose(f) == 0) && ok;
    if (!ok) { remove(tmp.c_str()); cudaGetLastError(); return e->fail("%s: could not write the state", tmp.c_str()); }
    if (rename(tmp.c_str(), path) != 0) return e->fail("%s: %s", path, strerror(errno));
    return 0;
}

int b2_load_state(b2_engine* e, const char* path, uint32_t* toks_out, int cap_toks, int* n_out) {
    if (!e || !e->finished) return 1;
    if (e->B != 1) return e->fail("states are loaded for one sequence (this engine has %d)", e->B);
    CUE(cudaSetDevice(e->device));
    // on any error the engine is left empty (model.rs:383-384)
    e->reset_state();
    cudaStreamSynchronize(e->stream);
    FILE* f = fopen(path, "rb");
    if (!f) return e->fail("%s: %s", path, strerror(errno));
    char magic[16];
    if (fread(magic, 1, 16, f) != 16 || memcmp(magic, "AEGSTATE", 8) != 0) { fclose(f); return e->fail("%s: not a saved state", path); }
    uint64_t hl;
    memcpy(&hl, magic + 8, 8);
    if (hl > (1ull << 30)) { fclose(f); return e->fail("%s: not a saved state", path); }
    std::string head(hl, 0);
    if (fread(&head[0], 1, hl, f) != hl) { fclose(f); return e->fail("%s: truncated", path); }
    JValue j;
    std::string jerr;
    JParser parser(head.data(), head.size());
    if (!parser.parse(j, jerr)) { fclose(f); return e->fail("%s: %s", path, jerr.c_str()); }
    const JValue* key = j.get("key");
    if (!key || key->type != JValue::Str || key->str != e->state_key()) { fclose(f); return e->fail("%s: saved by another brain", path); }
    std::vector<uint32_t> toks;
    if (const JValue* t = j.get("toks")) for (auto& x : t->arr) toks.push_back((uint32_t)x.num);
    const int n = (int)toks.size();
    if (n == 0 || n >= e->cap) { fclose(f); return e->fail("%s: %d tokens do not fit a context of %d", path, n, e->cap); }
    std::vector<char> buf;
    for (auto& pc : e->state_pieces(n)) {
        buf.resize(pc.bytes);
        if (fread(buf.data(), 1, pc.bytes, f) != pc.bytes) { fclose(f); e->reset_state(); return e->fail("%s: truncated", path); }
        if (cudaMemcpyAsync(pc.p, buf.data(), pc.bytes, cudaMemcpyHostToDevice, e->stream) != cudaSuccess || cudaStreamSynchronize(e->stream) != cudaSuccess) { fclose(f); cudaGetLastError(); e->reset_state(); return e->fail("%s: upload failed", path); }
    }
    fclose(f);
    k_fill_i32<<<1, 32, 0, e->stream>>>(e->d_pos, n, 1);
    CUE(cudaStreamSynchronize(e->stream));
    e->length = n;
    e->toks = toks;
    e->toks_known = true;
    e->snap_pos[0] = e->snap_pos[1] = -1;
    if (b2_snapshot(e)) return 1;
    if (n_out) *n_out = n;
    if (toks_out) memcpy(toks_out, toks.data(), (size_t)std::min(n, cap_toks) * 4);
    return 0;
}

int b2_length(const b2_engine* e) { return e ? e->length : 0; }
int b2_cap(const b2_engine* e) { return e ? e->cap : 0; }
int b2_vocab(const b2_engine* e) { return e ? e->c.V : 0; }
int b2_d_model(const b2_engine* e) { return e ? e->c.D : 0; }

int b2_set_taps(b2_engine* e, const int* layers, int n) {
    if (!e || !e->finished) return 1;
    for (int i = 0; i < n; i++)
        if (layers[i] < 0 || layers[i] >= e->c.L) return e->fail("tap layer %d out of range (the brain has %d layers)", layers[i], e->c.L);
    CUE(cudaSetDevice(e->device));
    CUE(cudaStreamSynchronize(e->stream));
    cudaFree(e->tap_buf);
    e->tap_buf = nullptr;
    e->tap_layers.assign(layers, layers + n);
    if (n) {
        CUE(dalloc(&e->tap_buf, (size_t)n * e->B * e->c.D, false));
        CUE(cudaMemsetAsync(e->tap_buf, 0, (size_t)n * e->B * e->c.D * sizeof(float), e->stream));
    }
    return e->build_graph();
}

int b2_taps(b2_engine* e, float* out) {
    if (!e || !e->finished) return 1;
    if (e->tap_layers.empty()) return 0;
    CUE(cudaSetDevice(e->device));
    CUE(cudaMemcpyAsync(out, e->tap_buf, e->tap_layers.size() * (size_t)e->B * e->c.D * 4, cudaMemcpyDeviceToHost, e->stream));
    CUE(cudaStreamSynchronize(e->stream));
    return 0;
}

int b2_core_counts(b2_engine* e, int32_t* out) {
    if (!e || !e->finished) return 1;
    CUE(cudaSetDevice(e->device));
    CUE(cudaStreamSynchronize(e->stream));
    CUE(cudaMemcpy(out, e->d_counts, (size_t)e->c.L * e->c.n1 * e->c.n2 * 4, cudaMemcpyDeviceToHost));
    return 0;
}
int b2_reset_counts(b2_engine* e) {
    if (!e || !e->finished) return 1;
    CUE(cudaSetDevice(e->device));
    CUE(cudaMemsetAsync(e->d_counts, 0, (size_t)e->c.L * e->c.n1 * e->c.n2 * 4, e->stream));
    CUE(cudaStreamSynchronize(e->stream));
    return 0;
}

void b2_expert_counters(const b2_engine* e, uint64_t* hits, uint64_t* page_ins) {
    if (hits) *hits = e ? e->hits : 0;
    if (page_ins) *page_ins = 0;
}

const char* b2_describe(const b2_engine* e) { return e ? e->desc.c_str() : ""; }
const char* b2_last_error(const b2_engine* e) { return e ? e->err.c_str() : "no engine"; }

int b2_debug_router(b2_engine* e, int layer, int32_t* idx, float* wts) {
    if (!e || !e->finished) return 1;
    if (layer < 0 || layer >= e->c.L) return e->fail("layer %d out of range", layer);
    CUE(cudaSetDevice(e->device));
    const size_t n = (size_t)e->B * e->c.TOPK;
    CUE(cudaStreamSynchronize(e->stream));
    if (idx) CUE(cudaMemcpy(idx, e->top_idx + layer * n, n * 4, cudaMemcpyDeviceToHost));
    if (wts) CUE(cudaMemcpy(wts, e->top_w + layer * n, n * 4, cudaMemcpyDeviceToHost));
    return 0;
}

int b2_debug_hidden(b2_engine* e, float* out) {
    if (!e || !e->finished) return 1;
    CUE(cudaSetDevice(e->device));
    CUE(cudaStreamSynchronize(e->stream));
    CUE(cudaMemcpy(out, e->x, (size_t)e->B * e->c.D * 4, cudaMemcpyDeviceToHost));
    return 0;
}

int b2_set_router_bias(b2_engine* e, int layer, const float* bias) {
    if (!e || !e->finished) return 1;
    if (layer < 0 || layer >= e->c.L) return e->fail("layer %d out of range", layer);
    CUE(cudaSetDevice(e->device));
    LayerW& l = e->layers[layer];
    if (!bias) CUE(cudaMemsetAsync(l.router_bias, 0, (size_t)e->c.E * 4, e->stream));
    else CUE(cudaMemcpyAsync(l.router_bias, bias, (size_t)e->c.E * 4, cudaMemcpyHostToDevice, e->stream));
    CUE(cudaStreamSynchronize(e->stream));
    return 0;
}

int b2_launches_per_step(const b2_engine* e) { return e ? e->launches : 0; }
int b2_kernels_per_step(const b2_engine* e) { return b2_launches_per_step(e); }
int b2_stages_per_step(const b2_engine* e) { return !e ? 0 : (e->use_step1() ? e->s1.stages : e->launches); }
long b2_debug_umma_launches(void) { return g_umma_launches; }
void b2_debug_refuse_tensor_maps(int on) { g_refuse_maps = on != 0; }

int b2_debug_seek(b2_engine* e, int n) {
    if (!e || !e->finished) return 1;
    if (n < 0 || n > e->cap) return e->fail("cannot seek to %d (context holds %d)", n, e->cap);
    CUE(cudaSetDevice(e->device));
    k_fill_i32<<<(e->B + 255) / 256, 256, 0, e->stream>>>(e->d_pos, n, e->B);
    CUE(cudaStreamSynchronize(e->stream));
    e->length = n;
    e->toks_known = false;
    return 0;
}

double b2_step_bytes(const b2_engine* e) {
    if (!e) return 0;
    double cls[8];
    e->class_bytes(cls);
    double s = 0;
    for (double v : cls) s += v;
    return s;
}

double b2_ep_bytes_per_step(const b2_engine* e) {
    if (!e || e->ep_world <= 1) return 0;
    const Cfg& c = e->c;
    const double peers = e->ep_world - 1;
    const double gather = peers * e->B * (c.D + 2.0 * c.TOPK) * 4;       // this GPU's records, to every peer
    if (e->ep_peer_ready) {
        // peer stores: only the rows of picks computed here for other ranks' tokens travel; counted on the device
        unsigned long long rows = 0;
        cudaMemcpy(&rows, e->d_ep_rows, sizeof(rows), cudaMemcpyDeviceToHost);
        return c.L * gather + (e->ep_steps > 0 ? (double)rows * c.D * 4 / e->ep_steps : 0.0);
    }
    const double back = peers * e->B * (c.TOPK + 1.0) * c.D * 4;         // pick outputs computed here, to their owners
    return c.L * (gather + back);
}

int b2_debug_step1_plan(const char* config_json, int sms, int has_keys, int kv_dtype, int64_t* out, int cap) {
    b2_engine e;                       // (for its config only: no device is touched)
    JValue j;
    std::string err;
    JParser parser(config_json, strlen(config_json));
    if (!parser.parse(j, err) || e.parse_config(j) || sms < 1) return -1;
    const Cfg& c = e.c;
    Step1Plan p;
    if (!lay_out_step1(c, sms, has_keys ? c.n1 : 0, has_keys ? c.n2 : 0, kv_dtype == B2_KV_F32, p)) return 0;
    int n = 0;
    for (int b = 0; b < sms; b++)
        for (int kind = 0; kind < S1_KINDS; kind++)
            for (int i = 0; i < s1_cap(kind); i++) {
                const size_t ti = (size_t)b * S1_TILES + s1_at(kind) + i;
                const uint32_t t = p.tiles[ti];
                if (t == S1_NONE) break;
                for (int k = 0; k < S1_COPIES; k++) {
                    const S1Copy& y = p.copies[ti * S1_COPIES + k];
                    if (!(y.what >> 16)) continue;
                    const int64_t r[9] = {b, kind, (int64_t)(t >> 29), (int64_t)((t >> 24) & 31), (int64_t)(t & 0xffffff), (int64_t)(y.what & 31), (int64_t)y.from * 16,
                                          (int64_t)(y.what >> 16) * 16, (int64_t)((y.what >> 5) & 2047) * 16 - p.stage};
                    if (n < cap) std::copy(r, r + 9, out + (size_t)9 * n);
                    n++;
                }
            }
    return n;
}

int b2_debug_step1_polls(b2_engine* e, int polls) {
    if (!e || !e->finished) return 1;
    if (polls < 0 || polls > S1_SPINS) return e->fail("polls outside 0..%d", S1_SPINS);
    CUE(cudaSetDevice(e->device));
    CUE(cudaStreamSynchronize(e->stream));
    e->s1.args.polls = polls ? polls : S1_SPINS;
    return e->build_graph();
}

int b2_debug_trace_step(b2_engine* e, unsigned long long* out, int cap_launches, int* n_launches) {
    if (feed_checks(e, 1)) return 1;
    if (!e->d_trace && cudaMalloc(&e->d_trace, (size_t)TRACE_MAX_LAUNCHES * 128) != cudaSuccess) return e->fail("trace buffer: out of memory");
    std::vector<unsigned long long> init((size_t)TRACE_MAX_LAUNCHES * 16, 0ull);
    for (int i = 0; i < TRACE_MAX_LAUNCHES; i++) init[(size_t)16 * i] = ~0ull;
    cudaMemcpyAsync(e->d_trace, init.data(), init.size() * 8, cudaMemcpyHostToDevice, e->stream);
    cudaStreamSynchronize(e->stream);
    // the same step as the decode graph, captured once more with the time stamp slots handed out
    cudaGraph_t g;
    cudaGraphExec_t ge = nullptr;
    g_trace_base = e->d_trace;
    g_trace_first = g_launch_count;
    cudaError_t ce = cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal);
    int rc = ce == cudaSuccess ? e->enqueue_step(e->stream, false) : 1;
    const int n = e->use_step1() ? e->s1.stages : g_launch_count - g_trace_first;
    g_trace_base = nullptr;
    cudaError_t ce2 = cudaStreamEndCapture(e->stream, &g);
    if (rc || ce != cudaSuccess || ce2 != cudaSuccess) return e->fail("trace step: capture failed");
    ce = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) return e->fail("trace step: %s", cudaGetErrorString(ce));
    ce = e->run_graph(ge);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
    cudaGraphExecDestroy(ge);
    if (ce != cudaSuccess) return e->fail("trace step: %s", cudaGetErrorString(ce));
    e->length += 1;
    e->toks_known = false;
    const int m = std::min(std::min(n, cap_launches), TRACE_MAX_LAUNCHES);
    cudaMemcpy(out, e->d_trace, (size_t)m * 128, cudaMemcpyDeviceToHost);
    *n_launches = m;
    return 0;
}

int b2_profile_step(b2_engine* e, int iters, float ms[8], double bytes[8], int launches[8]) {
    if (feed_checks(e, iters)) return 1;
    for (int i = 0; i < 8; i++) { ms[i] = 0; launches[i] = 0; }
    e->class_bytes(bytes);
    e->profiling = true;
    for (int it = 0; it < iters; it++) {
        e->prof_used = 0;
        if (e->enqueue_step(e->stream, false)) { e->profiling = false; return 1; }
        cudaError_t ce = cudaStreamSynchronize(e->stream);
        if (ce != cudaSuccess) { e->profiling = false; return e->fail("profile step: %s", cudaGetErrorString(ce)); }
        e->length += 1;
        e->toks_known = false;
        for (size_t k = 1; k < e->prof_used; k++) {
            float t = 0;
            cudaEventElapsedTime(&t, e->prof_ev[k - 1], e->prof_ev[k]);
            ms[e->prof_class[k]] += t;
            launches[e->prof_class[k]] += 1;
        }
    }
    e->profiling = false;
    for (int i = 0; i < 8; i++) { ms[i] /= iters; launches[i] /= iters; }
    return 0;
}

}  // extern "C"

#include "ops.cuh"
#include "noalloc.cuh"
#include "sampler.hpp"
