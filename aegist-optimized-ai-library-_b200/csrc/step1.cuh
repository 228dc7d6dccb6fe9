// k_step1: a whole decode step of one sequence (embedding, every layer, head, arg-max) as one persistent launch.
//
// What bounds a step of one sequence is not its bytes but the six dependent stages of every layer: as launches of their own
// (k_tcgemv, k_delta_step, k_moe_gu1, ...) each pays a hand-over, an activation prologue, the first tiles' way from HBM and a
// tail. Here one block per SM stays for the whole step and
//   * a producer warp streams this block's rows of every weight matrix, in the order of their use and across stages and layers,
//     into a ring in shared memory: the dense weights of a stage wait there before its activations exist, the rows of the picked
//     experts are asked for by the block itself as soon as it knows the picks;
//   * a value that other blocks need is stored once as 8 bytes, the fp32 value and the layer's tag, and a reader polls the very
//     words it needs until they carry the tag: no counter, no fence, no grid-wide barrier between a value and its use;
//   * every warp owns a slice of the contraction of all rows in the ring; one block barrier per stage where the slices meet.
// 40 layers at context 4096: 1.36 ms a token, 1.61 ms as one launch per stage; at 190 (every token through the host) 1.38 and 1.71. A layer of
// 50 MB takes 27 us, 8 of which HBM would need: the rest is the way of six dependent values from SM to SM (0.9 us each: a store and two
// polls of L2) and what lies between their coming and the products, in every warp.
//
// Every sum is added in the order and with the roundings of the kernels that run steps of two to five sequences, so that a sequence has
// the same bits beside others as alone: slices, chunks and groups below are cut as there. (A sixteenth of the contraction per warp, with
// the rms behind the products and a scale for every slice, is 1.1x faster.) Only the attention's split of the context differs.
// The launch is cooperative: its blocks wait on one another, so all of them must be resident, and it begins when they can be (behind a
// kernel that held one SM for 2.5 s it took 2.5 s and no wait ran out). Every wait is bounded; one that runs out sets the error
// word and lets the step run to its end.
//
// Buffers that carry tagged words are used again two layers later. A block that writes for layer l + 2 has read all rows of
// layer l + 1's output, and every block owns some of those (rows are spread over all blocks), written after that block's last
// read of layer l. The attention's partial results have one place for all layers: who writes them for layer l + 1 has read all of layer
// l's output, which every block wrote after its last read of that layer's.
#pragma once

namespace b2 {

constexpr int S1_WARPS = 16;                      // warps that compute; one more feeds the ring
constexpr int S1_CONS = S1_WARPS * 32;
constexpr int S1_THREADS = S1_CONS + 128;
// Registers: a block is launched with 96 a thread; the producer's four warps (three of them idle) give some back for the others
// (setmaxnreg). The wait for them knows no bound: the kernel is launched only where the built one's count makes the hand-over work out.
constexpr int S1_REGS_LOW = 32, S1_REGS_HIGH = 112;
constexpr bool s1_regs_suffice(int regs) {
    return regs >= S1_REGS_LOW && regs <= S1_REGS_HIGH && regs * S1_THREADS >= S1_REGS_LOW * (S1_THREADS - S1_CONS) + S1_REGS_HIGH * S1_CONS;
}
constexpr int S1_MAXT = 7;                        // tiles of one stage in one block (epilogue: a thread per row slot, 16 slots a tile)
constexpr int S1_ROWS = S1_MAXT * 16;
constexpr int S1_MAXST = 12;                      // ring stages
constexpr int S1_PASS = 128;                      // positions whose scores a block keeps at once: two tiles of at most 64
constexpr int S1_PAGES = 64;                      // cache pages a block's slice of the context may touch
constexpr int S1_SPINS = 1 << 21;                 // polls before a wait gives up: a second or so
constexpr uint32_t S1_NONE = 0xffffffffu;
// The last S1_OPS bytes of a ring stage hold what the epilogue needs of the tile's rows, fetched with them: scales or gate constants (bf16) at 0, a
// second row of those or the router's bias (fp32) at 64, convolution weights (4 bf16 a row) at 128, taps (3 fp32 a row) at 272. Each
// begins at the 16-byte border before the first row's. (Loaded when the epilogue is near they come behind all the weights that are
// on their way: with a full ring in flight on every SM that is a queue of 4 us.)
constexpr int S1_OPS = 480;
constexpr int S1_LOT = 6;                         // tiles of the head between two barriers
enum Step1Kind : int { S1_IN_DELTA = 0, S1_IN_ATTN = 1, S1_OUT = 2, S1_MOE = 3, S1_SHD = 4, S1_KINDS = 5 };
// segments: in-projections of a DeltaNet layer b, a, qkv, z (of attention q, k, v), out, router | key1 | key2 | shared gate | shared gate-up pairs
__host__ __device__ __forceinline__ bool s1_is_bf(int kind, int seg) { return kind == S1_IN_DELTA ? seg < 2 : kind == S1_MOE && seg < 4; }
// room for a stage's tiles in the block's list, and where they start there
__host__ __device__ __forceinline__ int s1_cap(int kind) { return kind <= S1_IN_ATTN ? S1_MAXT : (kind == S1_OUT ? 3 : (kind == S1_MOE ? 4 : 1)); }
__host__ __device__ __forceinline__ int s1_at(int kind) { return kind <= S1_OUT ? kind * S1_MAXT : (kind == S1_MOE ? 2 * S1_MAXT + 3 : 2 * S1_MAXT + 7); }
constexpr int S1_TILES = 2 * S1_MAXT + 8;
// tile: segment (3 bits) | rows (5) | first row (24)
__host__ __device__ __forceinline__ uint32_t s1_tile(int seg, int n, int row0) { return ((uint32_t)seg << 29) | ((uint32_t)n << 24) | (uint32_t)row0; }
// Rows lie in a stage in two halves, each as dense as in memory (one copy), the second 64 bytes out of step with the first: slot s of a tile is row
// s / 2 of half s & 1, so that the two rows a load of eight lanes takes lie in different banks. A half has room for half of the longest tile.
__host__ __device__ __forceinline__ int s1_half_at(int rows, int rb) { return (rows + 1) / 2 * rb + 64; }
__host__ __device__ __forceinline__ int s1_slot_row(int slot, int n) { const int h = (n + 1) / 2; return (slot & 1) ? ((slot >> 1) < n - h ? h + (slot >> 1) : -1) : ((slot >> 1) < h ? slot >> 1 : -1); }
// a copy of a tile: pointer of the layer (5 bits) | place in the stage / 16 (11) | bytes / 16 (12, 0: none), and its offset / 16 behind the pointer
struct S1Copy { uint32_t what, from; };
constexpr int S1_COPIES = 8;

struct alignas(16) Step1Layer {
    const void* w[12];           // in-projections [0..3] by segment, out [4], router, key1, key2, shared gate vector, gate [5..9], up [10], shared down [11]
    const uint16_t* s[7];        // scales: in-projections [0..2], out [3], gate [4], up [5], shared down [6]
    const uint16_t *norm1, *norm2;
    const uint16_t *n_a, *n_b;   // DeltaNet: gated norm, - ; attention: q norm, k norm
    const uint16_t *conv_w, *a_log, *dt_bias;
    float *conv_state, *state;
    const float* bias;           // router bias or null
    const uint8_t* experts;      // [E][expert_bytes]
    void *kpool, *vpool;
    int* counts;                 // the core engine's tallies, or null
    float* tap;                  // where the hidden state behind this layer is wanted, or null
    int* top_idx;
    float* top_w;
    int attn, pad;
};
// places of its pointers, as 64-bit words
enum Step1Ptr : int { W_OUT = 4, W_ROUTER = 5, W_UP = 10, W_SHD = 11, S_IN = 12, S_OUT = 15, S_GATE = 16, S_UP = 17, S_SHD = 18, Q_CONV_W = 23, Q_A_LOG = 24, Q_DT = 25, Q_CONV_STATE = 26, Q_BIAS = 28, Q_EXPERTS = 29, Q_KPOOL = 30 };
static_assert(offsetof(Step1Layer, s) == 8 * S_IN && offsetof(Step1Layer, conv_w) == 8 * Q_CONV_W && offsetof(Step1Layer, conv_state) == 8 * Q_CONV_STATE && offsetof(Step1Layer, bias) == 8 * Q_BIAS && offsetof(Step1Layer, vpool) == 8 * Q_KPOOL + 8, "Step1Ptr");
static_assert(sizeof(Step1Layer) % 16 == 0, "copied in 16-byte pieces");

struct Step1Args {
    unsigned long long* trace;
    const Step1Layer* layers;
    const uint32_t* tiles;       // [G][S1_TILES]
    const S1Copy* copies;        // [G][S1_TILES][S1_COPIES]
    const uint16_t *embed, *norm;
    const int8_t* head_w;
    const uint16_t* head_s;
    float* logits;
    float* x;                    // [D] hidden state behind the last layer
    uint64_t* ll;                // tagged words: two sets (even and odd layers), the attention partials, the core engine's scores
    uint32_t ll_set, o_xa, o_xb, o_q, o_z, o_bg, o_og, o_rl, o_sa, o_sg, o_act;   // words of a set; offsets of its parts
    uint32_t o_ap, o_cs, cs_words;   // offsets of the attention partials and of the core engine's scores (words per layer)
    uint32_t* epoch;             // tags of this step are epoch + 1 .. epoch + L; the last block moves it on
    const float *rope_cos, *rope_sin;
    const int* page_table;
    float scale, eps;
    uint32_t polls;              // before a wait gives up; at least 1
    int L, V, E, topk, I, SH, HK, HV, DV, H, KV, RD, C, n1, n2, cores_k, kv_f32, kv_tile, head_rows, half_i8, half_bf, half_out, half_pair, half_shd, nst, stage_bytes;
    size_t expert_bytes, off_gu_s, off_gu_m, off_dn_q, off_dn_s, off_dn_m;
    float *cscore, *cselw;
    int* csel;
    float* part_val;
    int *part_idx, *next_tok, *pos, *tok;
    TokHist hist;
    unsigned int* counter;
    int* err;
};

// ---- tagged words ----
__device__ __forceinline__ void ll_store(uint64_t* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((uint64_t)tag << 32) | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ uint64_t ll_load(const uint64_t* p) {
    uint64_t r;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(r) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ void ll_load2(const uint64_t* p, uint64_t& r0, uint64_t& r1) {     // 16-byte aligned; each word whole by itself
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(r0), "=l"(r1) : "l"(p) : "memory");
}
// the same for words whose tag is not there yet
__device__ __forceinline__ void ll_again(const uint64_t* p, uint32_t tag, uint64_t& r) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %1, %2;\n @q ld.relaxed.gpu.global.u64 %0, [%3];\n}" : "+l"(r) : "r"((uint32_t)(r >> 32)), "r"(tag), "l"(p) : "memory");
}
__device__ __forceinline__ void ll_again2(const uint64_t* p, uint32_t tag, uint64_t& r0, uint64_t& r1) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, %4;\n setp.ne.or.u32 q, %3, %4, q;\n @q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%5];\n}"
                 : "+l"(r0), "+l"(r1) : "r"((uint32_t)(r0 >> 32)), "r"((uint32_t)(r1 >> 32)), "r"(tag), "l"(p) : "memory");
}
// Waits are bounded: one that has polled Step1Args::polls times raises the block's flag, all later waits of the block give up at once, and at the
// end the block reports it. (Blocks that wait for this one then get words that mean nothing, and come to their end.)
__device__ __forceinline__ bool s1_given_up(int spin, uint32_t flag) {
    uint32_t f, polls;
    asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(f), "=r"(polls) : "r"(flag) : "memory");
    if ((uint32_t)spin >= polls) { f = 1u; asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(flag), "r"(f) : "memory"); }
    return __any_sync(0xffffffffu, f != 0u);
}
// N neighbouring values per lane, and M more at q, by a whole warp; lanes without need go along. N, M = 1 or even (then 16-byte aligned)
template <int N, int M>
__device__ __forceinline__ void ll_wait2(const uint64_t* p, const uint64_t* q, uint32_t tag, bool need, float (&v)[N], float (&u)[M > 0 ? M : 1], uint32_t flag) {
    // only what is not there yet is asked for again: the polls of many warps are in the way of those who still work
    uint64_t r[N], t[M > 0 ? M : 1];
    const uint64_t not_yet = (uint64_t)(need ? ~tag : tag) << 32;
#pragma unroll
    for (int i = 0; i < N; i++) r[i] = not_yet;
#pragma unroll
    for (int i = 0; i < M; i++) t[i] = not_yet;
#pragma unroll 1
    for (int spin = 0;; spin++) {
        if constexpr (N == 1) ll_again(p, tag, r[0]);
        else {
#pragma unroll
            for (int i = 0; i + 1 < N; i += 2) ll_again2(p + i, tag, r[i], r[i + 1]);
        }
        if constexpr (M == 1) ll_again(q, tag, t[0]);
        else if constexpr (M > 1) {
#pragma unroll
            for (int i = 0; i + 1 < M; i += 2) ll_again2(q + i, tag, t[i], t[i + 1]);
        }
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; i++) ok = ok && (uint32_t)(r[i] >> 32) == tag;
#pragma unroll
        for (int i = 0; i < M; i++) ok = ok && (uint32_t)(t[i] >> 32) == tag;
        if (__all_sync(0xffffffffu, ok) || s1_given_up(spin, flag)) break;
    }
    __syncwarp();                                 // what follows wants the warp together (barriers, matrix instructions)
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = __uint_as_float((uint32_t)r[i]);
#pragma unroll
    for (int i = 0; i < M; i++) u[i] = __uint_as_float((uint32_t)t[i]);
}
template <int N>
__device__ __forceinline__ void ll_wait(const uint64_t* p, uint32_t tag, bool need, float (&v)[N], uint32_t flag) {
    float none[1];
    ll_wait2<N, 0>(p, p, tag, need, v, none, flag);
}
// a phase of an mbarrier of this block, by a whole warp; every lane may look at one of its own
__device__ __forceinline__ void s1_mbar_wait(uint32_t bar, uint32_t parity, uint32_t flag) {
#pragma unroll 1
    for (int spin = 0; !__all_sync(0xffffffffu, mbar_try(bar, parity)); spin += 16)        // (a try may take a while itself)
        if (s1_given_up(spin, flag)) break;
    __syncwarp();
}
__device__ __forceinline__ uint32_t ldg_nc1(const void* p) {
    uint32_t r;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ uint2 ldg_nc2(const void* p) {
    uint2 r;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ uint4 ldg_nc4(const void* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// N scale words (fp16 pairs), as one load
template <int N>
__device__ __forceinline__ void ldg_words(const void* p, uint32_t (&w)[N]) {
    if constexpr (N == 1) w[0] = ldg_nc1(p);
    else if constexpr (N == 2) { const uint2 v = ldg_nc2(p); w[0] = v.x; w[1] = v.y; }
    else { const uint4 v = ldg_nc4(p); w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
}
// a shared-memory store by the threads that say so: one predicated instruction, where an `if` may become a branch and a reconvergence
__device__ __forceinline__ void sts_if(bool yes, void* p, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.u32 [%0], %1;\n\t}" ::"r"(smem_u32(p)), "r"(v), "r"((uint32_t)yes) : "memory");
}
__device__ __forceinline__ void sts_if(bool yes, float* p, float v) { sts_if(yes, (void*)p, __float_as_uint(v)); }
__device__ __forceinline__ float warp_absmax(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7fffffffu)); }
__device__ __forceinline__ void s1_bar() { __syncwarp(); asm volatile("bar.sync 1, 512;" ::: "memory"); }
static_assert(S1_CONS == 512, "s1_bar");

// Eight neighbouring values of every lane, 256 of the warp, as four planes of 256 bytes; in odd planes byte b lies at b ^ 64, so that what a
// lane reads of neighbouring planes lies in different banks. evenodd: within eight the even ones first, as the codes of a word come out
__device__ __forceinline__ void planes8(const float (&v)[8], float inv, bool evenodd, unsigned char* sc, int lane) {
    uint2 w[M1_PLANES];
    digits8(v, inv, evenodd, w);
#pragma unroll
    for (int p = 0; p < M1_PLANES; p++) *reinterpret_cast<uint2*>(sc + p * 256 + ((8 * lane) ^ (64 * (p & 1)))) = w[p];
}

// what a computing warp knows of the ring
struct S1Ring {
    const unsigned char* base;
    uint32_t bars;               // shared-memory address: full[S1_MAXST] | empty[S1_MAXST]
    int stage_bytes, nst, st;
    uint32_t ph;
    uint32_t flag;               // shared-memory address of the block's given-up flag
    __device__ __forceinline__ const unsigned char* stage(int u = 0) const { const int t = st + u; return base + (t >= nst ? t - nst : t) * stage_bytes; }
    // for n neighbouring stages at once: lane u looks at (or hands back) stage u of them
    __device__ __forceinline__ void wait(int n, int lane) {
        const int u = lane < n ? lane : 0, t = st + u;
        s1_mbar_wait(bars + 8 * (t >= nst ? t - nst : t), t >= nst ? ph ^ 1u : ph, flag);
    }
    __device__ __forceinline__ void release(int n, int lane) {
        __syncwarp();
        const int t = st + lane;
        if (lane < n) mbar_arrive(bars + 8 * (S1_MAXST + (t >= nst ? t - nst : t)));
        st += n;
        if (st >= nst) { st -= nst; ph ^= 1u; }
    }
};
// S values from `off` on of a warp's planes as B operand: column gid = plane gid & 3 (nobody looks at the sums of columns 4 .. 7)
template <int S>
__device__ __forceinline__ void load_planes(const unsigned char* sc, int off, int gid, int tid, uint4 (&xb)[S / 64]) {
#pragma unroll
    for (int j = 0; j < S / 64; j++) xb[j] = *reinterpret_cast<const uint4*>(sc + (gid & 3) * 256 + ((off + 64 * j + 16 * tid) ^ (64 * (gid & 1))));
}
// keep(n) is called when n tiles have landed, before they are handed back.
// Slice ks of S values of NT tiles of int8 rows, the first of them tile u0 from the ring's place: partial sums of slots gid (and gid + 8 where TWO:
// `up` bytes behind) into part[16 u + 0 .. 15]. Everything is loaded, then multiplied, so that the tiles hide each other's latencies; slots
// without a row hold what happens to lie there, and nobody reads their sums. |sum| <= S * 128 * 128 <= 2^22 for S <= 256: exact in the
// magic form. The planes are joined as k_tcgemv joins them.
template <int S, int K, bool TWO, int NT>
__device__ __forceinline__ void s1_i8_tiles(const S1Ring& r, int u0, int half, int up, const uint4 (&xb)[S / 64], float pw0, float pw1, float* part, int ks, int lane) {
    constexpr int NJ = S / 64;
    const int gid = lane >> 2, tid = lane & 3;
    const int off = (gid >> 1) * K + (gid & 1 ? half : 0) + ks * S + tid * 16;
    uint4 wa[NT][NJ], wb[NT][NJ];
#pragma unroll
    for (int u = 0; u < NT; u++) {
        const unsigned char* q = r.stage(u0 + u) + off;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            wa[u][j] = *reinterpret_cast<const uint4*>(q + 64 * j);
            wb[u][j] = make_uint4(0u, 0u, 0u, 0u);
            if (TWO) wb[u][j] = *reinterpret_cast<const uint4*>(q + up + 64 * j);
        }
    }
    int c[NT][4];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
#pragma unroll
        for (int u = 0; u < NT; u++) {
            if (j == 0) imma16832_c(c[u], wa[u][j].x, wb[u][j].x, wa[u][j].y, wb[u][j].y, xb[j].x, xb[j].y, F32_MAGIC);
            else imma16832(c[u], wa[u][j].x, wb[u][j].x, wa[u][j].y, wb[u][j].y, xb[j].x, xb[j].y);
        }
#pragma unroll
        for (int u = 0; u < NT; u++) imma16832(c[u], wa[u][j].z, wb[u][j].z, wa[u][j].w, wb[u][j].w, xb[j].z, xb[j].w);
    }
#pragma unroll
    for (int u = 0; u < NT; u++) {
        float v0 = fmaf(magic_sum(c[u][0]), pw0, __fmul_rn(magic_sum(c[u][1]), pw1));
        v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
        sts_if(tid == 0, part + 16 * (u0 + u) + gid, v0);
        if (TWO) {
            float v1 = fmaf(magic_sum(c[u][2]), pw0, __fmul_rn(magic_sum(c[u][3]), pw1));
            v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
            sts_if(tid == 0, part + 16 * (u0 + u) + gid + 8, v1);
        }
    }
}
// n tiles. par < 0: a warp multiplies its slice of all of them; else there are half as many slices as warps, and a warp takes every other tile
template <int S, int K, bool TWO, typename F>
__device__ __forceinline__ void s1_i8_run(S1Ring& r, int n, int half, int up, const uint4 (&xb)[S / 64], float pw0, float pw1, float* part, int ks, int par, int lane, F keep) {
#pragma unroll 1
    for (; n > 0; n -= 2, part += 32) {
        const int m = min(n, 2);
        r.wait(m, lane);
        keep(m);
        if (par < 0) {
            if (m == 2) s1_i8_tiles<S, K, TWO, TWO ? 1 : 2>(r, 0, half, up, xb, pw0, pw1, part, ks, lane);
            if (TWO || m == 1) s1_i8_tiles<S, K, TWO, 1>(r, TWO && m == 2 ? 1 : 0, half, up, xb, pw0, pw1, part, ks, lane);
        } else if (par < m) s1_i8_tiles<S, K, TWO, 1>(r, par, half, up, xb, pw0, pw1, part, ks, lane);
        r.release(m, lane);
    }
}
// n tiles of bf16 rows (8 at most) against fp32 values, slice ks of S; a warp takes every other tile. One chain of sums, as in k_tcgemv
template <int S, int K, typename F>
__device__ __forceinline__ void s1_bf_run(S1Ring& r, int n, int half, const float* xf, float* part, int ks, int par, int lane, F keep) {
    const int gid = lane >> 2, tid = lane & 3;
#pragma unroll 1
    for (int u = 0; u < n; u++, part += 16) {
        const unsigned char* pa = r.stage() + (gid >> 1) * (2 * K) + (gid & 1 ? half : 0) + 2 * ks * S + tid * 16;
        r.wait(1, lane);
        keep(1);
        if ((u & 1) == par) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < S / 32; j++) {
                const uint4 wv = *reinterpret_cast<const uint4*>(pa + 64 * j);
                const float4 x0 = *reinterpret_cast<const float4*>(xf + 32 * j + 8 * tid), x1 = *reinterpret_cast<const float4*>(xf + 32 * j + 8 * tid + 4);
                float p = x0.x * bflo(wv.x);
                p = fmaf(x0.y, bfhi(wv.x), p); p = fmaf(x0.z, bflo(wv.y), p); p = fmaf(x0.w, bfhi(wv.y), p);
                p = fmaf(x1.x, bflo(wv.z), p); p = fmaf(x1.y, bfhi(wv.z), p); p = fmaf(x1.z, bflo(wv.w), p);
                p = fmaf(x1.w, bfhi(wv.w), p);
                acc += p;
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            sts_if(tid == 0, part + gid, acc);
        }
        r.release(1, lane);
    }
}
// the sum of 32 neighbouring values, eight to a lane, added as warp_sum adds them with one to a lane; in all four lanes
__device__ __forceinline__ float sum32(const float (&v)[8]) {
    float b[8];
#pragma unroll
    for (int j = 0; j < 8; j++) b[j] = v[j] + __shfl_xor_sync(0xffffffffu, v[j], 2);
#pragma unroll
    for (int j = 0; j < 8; j++) b[j] += __shfl_xor_sync(0xffffffffu, b[j], 1);
    return ((b[0] + b[4]) + (b[2] + b[6])) + ((b[1] + b[5]) + (b[3] + b[7]));
}

// Softmax over up to 256 logits (eight neighbouring ones in each lane that `has` some) and the topk <= 8 largest in descending order, ties to the lower
// index (aegist/hybrid.py:641-645); picks and probabilities into top and topv. A positive float's bits order like an integer's. A lane
// sorts its own exponentials and a round is one reduction over the lanes' first ones. The division keeps their order, but for what it
// rounds to one value: so only the picks and the best one left are divided, a lane each (256 divisions in one warp cost 0.6 us a layer),
// and where two of those, or two exponentials (which the number of lanes that won a round shows), are equal, all are divided and the
// rounds are made again by index.
__device__ __forceinline__ void s1_route(float (&lg)[8], bool has, int topk, int lane, int* top, float* topv) {
    uint32_t key[8];
    int ex[8];
    float mx = lg[0], sum = 0.f;
#pragma unroll
    for (int i = 1; i < 8; i++) mx = fmaxf(mx, lg[i]);
    {
        const uint32_t b = __float_as_uint(has ? mx : -INFINITY), o = __reduce_max_sync(0xffffffffu, (int)b < 0 ? ~b : b | 0x80000000u);
        mx = __uint_as_float((int)o < 0 ? o & 0x7fffffffu : ~o);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) { const float e = expf(lg[i] - mx); lg[i] = has ? e : 0.f; ex[i] = i; }
    const float s32 = sum32(lg);                  // of experts 32 w .. 32 w + 31, w = lane / 4
#pragma unroll
    for (int w = 0; w < 8; w++) sum += __shfl_sync(0xffffffffu, s32, 4 * w);
#pragma unroll
    for (int i = 0; i < 8; i++) key[i] = has ? __float_as_uint(lg[i]) + 1u : 0u;
    // a network of 19 exchanges; the order of equal ones is left open
#define S1_CX(i, j) { const bool w = key[j] > key[i]; const uint32_t k = w ? key[i] : key[j]; key[i] = w ? key[j] : key[i]; key[j] = k; const int e = w ? ex[i] : ex[j]; ex[i] = w ? ex[j] : ex[i]; ex[j] = e; }
    S1_CX(0, 2) S1_CX(1, 3) S1_CX(4, 6) S1_CX(5, 7)
    S1_CX(0, 4) S1_CX(1, 5) S1_CX(2, 6) S1_CX(3, 7)
    S1_CX(0, 1) S1_CX(2, 3) S1_CX(4, 5) S1_CX(6, 7)
    S1_CX(2, 4) S1_CX(3, 5)
    S1_CX(1, 4) S1_CX(3, 6)
    S1_CX(1, 2) S1_CX(3, 4) S1_CX(5, 6)
#undef S1_CX
    uint32_t order = 0u;                          // the lane's indices in the order of their keys, three bits each
#pragma unroll
    for (int i = 0; i < 8; i++) order |= (uint32_t)ex[i] << (3 * i);
    int wins = 0;
    uint32_t mine = 0u;                           // lane r: the key of round r; lane topk: of the best one left
#pragma unroll
    for (int r = 0; r < 8; r++)
        if (r < topk) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, key[0]);
            const bool w = key[0] == m;
            sts_if(w, (void*)(top + r), (uint32_t)lane * 8u + (order & 7u));
            if (lane == r) mine = m;
            wins += w ? 1 : 0;
            order = w ? order >> 3 : order;
#pragma unroll
            for (int i = 0; i < 7 - r; i++) key[i] = w ? key[i + 1] : key[i];
            key[7 - r] = w ? 0u : key[7 - r];
        }
    {
        const uint32_t m = __reduce_max_sync(0xffffffffu, key[0]);
        if (lane == topk) mine = m;
    }
    const uint32_t prob = mine ? __float_as_uint(__uint_as_float(mine - 1u) / sum) + 1u : 0u, next = __shfl_down_sync(0xffffffffu, prob, 1);
    sts_if(lane < topk, (void*)(topv + lane), prob - 1u);
    if (__reduce_add_sync(0xffffffffu, (unsigned)wins) == (unsigned)topk && !__any_sync(0xffffffffu, lane < topk && prob == next)) return;
    __syncwarp();
    uint32_t p[8];
#pragma unroll
    for (int i = 0; i < 8; i++) p[i] = has ? __float_as_uint(lg[i] / sum) + 1u : 0u;
#pragma unroll 1
    for (int r = 0; r < topk; r++) {
        uint32_t bk = p[0];
        int bi = 0;
#pragma unroll
        for (int i = 1; i < 8; i++)
            if (p[i] > bk) { bk = p[i]; bi = i; }                               // '>' keeps the lower index
        const uint32_t m = __reduce_max_sync(0xffffffffu, bk);
        const int win = __ffs(__ballot_sync(0xffffffffu, bk == m)) - 1;         // the lowest lane holds the lowest experts
        if (lane == win) { top[r] = m ? lane * 8 + bi : -1; topv[r] = m ? __uint_as_float(m - 1u) : 0.f; }
#pragma unroll
        for (int i = 0; i < 8; i++) p[i] = lane == win && i == bi ? 0u : p[i];
    }
}

// where the second half of n rows of `rb` bytes starts behind the first: 64 bytes out of step with it; and one pick's place in a tile of down rows
__host__ __device__ __forceinline__ int s1_half(int n, int rb) { return n * rb + 64; }
__host__ __device__ __forceinline__ int s1_dn_stride(int rows, int rb) { return rows * rb + 64; }
// four rows of gate/up scales side by side, in different banks
__host__ __device__ __forceinline__ int s1_gsc_stride(int D) { return 32 * (D / 32) + 16; }
// one pick's scales (or minima) of up to 16 down rows, from the 16-byte border before the first
__host__ __device__ __forceinline__ int s1_dsc_stride(int I) { return 16 * (I / 32) + 16; }

// what a block needs to know of its share, kept in shared memory: registers are short
struct S1Block {
    int r0, r1;                  // rows of the residual stream
    int gp0, gp1;                // (gate, up) row pairs of the picks
    int v0, v1;                  // rows of the head
    int id, pos;                 // the token and its position
    int kvh, slice, p0, p1, nused;   // attention: KV head, slice (of all heads), its positions; slices in use per head
};

// shared memory behind the ring (bytes)
template <int SD, int SO, int HD, int GH>
struct Step1Smem {
    static constexpr int SCR = 4 * 256 + 64;                                          // per warp: planes, and scales and sums of eight groups
    static constexpr int ATT = 8 * HD * 4 + 8 * (S1_PASS + 4) * 4 + 2 * HD * 4 + 64;  // attention's arrays lie over the warps' scratch
    static constexpr int SCRATCH = ((S1_WARPS * SCR > ATT ? S1_WARPS * SCR : ATT) + 127) / 128 * 128;
    static constexpr int XF = SD * 16 * 4;
    static constexpr int PART = 2 * S1_WARPS * S1_ROWS * 4;
    static constexpr int MIX = (2 * 128 + 3 * 32 + 2 * 8 * 32) * 4;                   // the delta rule's arrays; the merge's are shorter
    static constexpr int DELTA = MIX + S1_ROWS * 28;                                  // and what the epilogue needs of its rows
    static constexpr int LAYERS = 2 * (int)sizeof(Step1Layer);
    static constexpr int TOTAL = SCRATCH + XF + PART + DELTA + LAYERS;
};

// time stamps of a stage (see trace_in); every block with work in the stage stamps it
struct S1Trace {
    unsigned long long* base;    // a kernel parameter
    int stage;
    __device__ __forceinline__ void in(int code, int hint, bool work = true) { stage++; if (base && work) trace_in(base + (size_t)16 * stage, code, hint); }
    __device__ __forceinline__ void pt(int i) const { if (base) trace_pt(base + (size_t)16 * stage, i); }
    __device__ __forceinline__ void out(bool work = true) const { if (base && work) trace_out(base + (size_t)16 * stage); }
};

// core_route_warp (kernels.cuh) for one token, in rolled loops: it runs beside the step, with few registers. Scores in a.cscore.
__device__ __forceinline__ void s1_core_route(const Step1Args& a, int* counts, int lane) {
    const int k0 = min(a.cores_k, a.n1), k1 = min(a.cores_k, a.n2), nc = k0 * k1, k = min(a.cores_k, nc);
    float pv = 0.f, qv = 0.f;                     // lane r: the r-th best of the first table, of the second
    int pi = 0, qi = 0;
#pragma unroll 1
    for (int tab = 0; tab < 2; tab++) {
        const int n = tab ? a.n2 : a.n1, kk = tab ? k1 : k0;
        const float* st = a.cscore + (tab ? a.n1 : 0);
        uint32_t taken = 0u;                      // of this lane's entries lane, lane + 32, ..
#pragma unroll 1
        for (int r = 0; r < kk; r++) {
            float bv = -INFINITY;
            int bi = 0x7fffffff;
#pragma unroll 1
            for (int j = 0; lane + 32 * j < n; j++) {
                const float v = __ldcg(st + lane + 32 * j);
                if (!((taken >> j) & 1u) && v > bv) { bv = v; bi = lane + 32 * j; }          // '>' keeps the lower index
            }
#pragma unroll 1
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
            }
            const bool found = bi < n;            // (no score is left that is a number)
            if (lane == r) { if (tab) { qv = bv; qi = found ? bi : 0; } else { pv = bv; pi = found ? bi : 0; } }
            if (found && (bi & 31) == lane) taken |= 1u << (bi >> 5);
        }
    }
    // the sums of all pairs, candidate c = a k1 + b in lane c & 31; the best ones in turn, ties to the earlier one
    uint32_t taken = 0u;
    float myv = 0.f;
    int mycore = -1;
#pragma unroll 1
    for (int j = 0; j < k; j++) {
        float bv = -INFINITY;
        int bc = 0x7fffffff, core = -1;
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            const int c = lane + 32 * h, x = c / k1, y = c - x * k1;
            const float v = __shfl_sync(0xffffffffu, pv, x & 31) + __shfl_sync(0xffffffffu, qv, y & 31);
            const int id = __shfl_sync(0xffffffffu, pi, x & 31) * a.n2 + __shfl_sync(0xffffffffu, qi, y & 31);
            if (c < nc && !((taken >> h) & 1u) && v > bv) { bv = v; bc = c; core = id; }
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oc = __shfl_xor_sync(0xffffffffu, bc, o), od = __shfl_xor_sync(0xffffffffu, core, o);
            if (ov > bv || (ov == bv && oc < bc)) { bv = ov; bc = oc; core = od; }
        }
        if (lane == j) { myv = bv; mycore = core; }
        if (bc < nc && (bc & 31) == lane) taken |= 1u << (bc >> 5);
    }
    const float best = __shfl_sync(0xffffffffu, myv, 0);
    const float ex = lane < k ? expf(myv - best) : 0.f;
    float sum = 0.f;
#pragma unroll 1
    for (int j = 0; j < k; j++) sum += __shfl_sync(0xffffffffu, ex, j);        // in pick order
    if (lane < a.cores_k) {
        a.csel[lane] = mycore;
        a.cselw[lane] = mycore < 0 ? 0.f : ex / sum;
        if (mycore >= 0) atomicAdd(counts + mycore, 1);
    }
}

// Attention of one token for one KV head over one slice of the context; all computing warps. Keys and values come through the ring, up
// to two tiles of each at a time. Partial results (sum, maximum, weight) per query head go out as tagged words. fp32 throughout, on
// keys and values as the cache holds them.
template <int HD>
__device__ __forceinline__ void s1_attend(const Step1Args& a, const Step1Layer& ly, const uint64_t* set, uint32_t tag, const S1Block& blk, const int* s_page, const float* rope, unsigned char* scratch,
                                          S1Ring& rg, const S1Trace& tr, int warp, int lane) {
    constexpr int DL = HD / 32;
    const bool f32 = a.kv_f32 != 0;
    const int rowb = HD * (f32 ? 4 : 2);
    constexpr int SP = S1_PASS + 4;
    float* sq = reinterpret_cast<float*>(scratch);          // [8][HD]
    float* ssc = sq + 8 * HD;                               // [8][SP]
    float* skn = ssc + 8 * SP;                              // [HD] the new key, as the cache gives it back
    float* svn = skn + HD;                                  // [HD]
    float* scorr = svn + HD;                                // [8]
    const uint32_t w = rg.flag;
    const int G = a.H / a.KV, pos = blk.pos, p0 = blk.p0, p1 = blk.p1, kvh = blk.kvh;
    const bool newest = pos >= p0 && pos < p1;
    const uint64_t* lq = set + a.o_q;
    const uint64_t* lk = lq + 2 * a.H * HD;
    const uint64_t* lv = lk + a.KV * HD;
    // prologue: warps 0 .. 7 a query head each, 8 and 9 the new key and value where this slice holds the newest position. A lane has
    // DL neighbouring dims, which it polls in one go; the partner of a rotated dim is RD / 2 away, RD / 2 / DL lanes
    if (warp < 8 || (newest && warp < 10)) {
        const bool isq = warp < 8, isv = warp == 9;
        const int d0 = lane * DL;
        float y[DL];
        if (isq && warp >= G) {
#pragma unroll
            for (int i = 0; i < DL; i++) y[i] = 0.f;
        } else {
            const uint64_t* src = isq ? lq + (size_t)(kvh * G + warp) * 2 * HD : (isv ? lv : lk) + kvh * HD;
            const uint16_t* nw = isq ? ly.n_a : ly.n_b;
            const int hr = a.RD / 2;
            float sgn;
            uint32_t wn[DL / 2];
            if (!isv) {
                if constexpr (DL == 8) { const uint4 t = *reinterpret_cast<const uint4*>(nw + d0); wn[0] = t.x; wn[1] = t.y; wn[2] = t.z; wn[3] = t.w; }
                else { const uint2 t = *reinterpret_cast<const uint2*>(nw + d0); wn[0] = t.x; wn[1] = t.y; }
            }
            ll_wait<DL>(src + d0, tag, true, y, w);
            tr.pt(1);
            if (!isv) {
                float ss = 0.f;
#pragma unroll
                for (int i = 0; i < DL; i++) ss = fmaf(y[i], y[i], ss);
                ss = warp_sum(ss);
                const float r = 1.0f / sqrtf(ss / (float)HD + a.eps);
#pragma unroll
                for (int i = 0; i < DL; i++) y[i] = y[i] * r * (1.0f + ((i & 1) ? bfhi(wn[i / 2]) : bflo(wn[i / 2])));
                // rotate-half on the first RD dims (aegist/hybrid.py:160-166): (x0, x1) -> (x0 c - x1 s, x1 c + x0 s). They end at a lane's edge
                const bool first = d0 < hr;
                const int from = (first ? lane + hr / DL : lane - hr / DL) & 31, j0 = first ? d0 : d0 - hr;
                if (d0 >= a.RD) sgn = 0.f; else sgn = first ? -1.0f : 1.0f;
#pragma unroll
                for (int i = 0; i < DL; i++) {
                    const float other = __shfl_sync(0xffffffffu, y[i], from) * sgn;
                    if (sgn != 0.f) y[i] = y[i] * rope[j0 + i] + other * rope[HD / 2 + j0 + i];
                }
            }
        }
        if (isq) {
            const float qs = a.scale * 1.4426950408889634f;            // scores in the base-2 domain
#pragma unroll
            for (int i = 0; i < DL; i++) sq[warp * HD + d0 + i] = y[i] * qs;
        } else {
            float* keep = isv ? svn : skn;
            void* pool = isv ? ly.vpool : ly.kpool;
            const size_t at = (((size_t)s_page[pos / KV_PAGE - p0 / KV_PAGE] * a.KV + kvh) * KV_PAGE + pos % KV_PAGE) * HD + d0;
#pragma unroll
            for (int i = 0; i < DL; i++) {
                const uint16_t r = f2bf(y[i]);
                keep[d0 + i] = f32 ? y[i] : bf(r);
                if (f32) ((float*)pool)[at + i] = y[i]; else ((uint16_t*)pool)[at + i] = r;
            }
        }
    }
    s1_bar();
    // Q K^T: warp -> (four heads, every 8th position), a lane DL dims; P V: a warp takes HD / 16 dims, four to a lane
    constexpr int DW = HD / 16, LPP = DW / 4, PPI = 32 / LPP;          // P V: lanes per position, positions per turn
    const int hg = (warp & 1) * 4, pl = lane / LPP, dv = warp * DW + (lane % LPP) * 4;
    constexpr int STEPS = LPP == 4 ? 3 : 4, LEFT = 32 >> STEPS;        // value 4 h + d of a lane's 32 ends in the lanes with pl = its upper bits
    const int ho = (pl * LEFT) >> 2, d_out = dv + ((pl * LEFT) & 3);
    float o_run[LEFT];
#pragma unroll
    for (int i = 0; i < LEFT; i++) o_run[i] = 0.f;
    float m_run = -INFINITY, l_run = 0.f;                    // of head `warp` in warps 0 .. 7
    // position i of a pass is row i % kv_tile of tile i / kv_tile, in the stage the ring is at or the one after
    auto row_at = [&](int i) {
        const bool second = i >= a.kv_tile;
        return rg.stage(second ? 1 : 0) + (i - (second ? a.kv_tile : 0)) * rowb;
    };
    auto tiles_landed = [&](int n) {                         // one or two tiles
        rg.wait(n > a.kv_tile ? 2 : 1, lane);
    };
#pragma unroll 1
    for (int pb = p0; pb < p1; pb += 2 * a.kv_tile) {
        const int n = min(2 * a.kv_tile, p1 - pb);
        tiles_landed(n);
        {
            float q[4][DL];
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int d = 0; d < DL; d += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(sq + (hg + h) * HD + lane * DL + d);
                    q[h][d] = t.x; q[h][d + 1] = t.y; q[h][d + 2] = t.z; q[h][d + 3] = t.w;
                }
#pragma unroll 1
            for (int i = warp >> 1; i < n; i += 16) {        // two positions at a time
                float k[2][DL];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int at = min(i + 8 * u, n - 1);
                    const unsigned char* kr = pb + at == pos ? reinterpret_cast<const unsigned char*>(skn + lane * DL) : row_at(at) + lane * (rowb / 32);
                    if (f32 || pb + at == pos) {
#pragma unroll
                        for (int d = 0; d < DL; d += 4) {
                            const float4 t = *reinterpret_cast<const float4*>(kr + 4 * d);
                            k[u][d] = t.x; k[u][d + 1] = t.y; k[u][d + 2] = t.z; k[u][d + 3] = t.w;
                        }
                    } else {
                        uint32_t t[DL / 2];
                        if constexpr (DL == 8) { const uint4 v = *reinterpret_cast<const uint4*>(kr); t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w; }
                        else { const uint2 v = *reinterpret_cast<const uint2*>(kr); t[0] = v.x; t[1] = v.y; }
#pragma unroll
                        for (int d = 0; d < DL / 2; d++) { k[u][2 * d] = bflo(t[d]); k[u][2 * d + 1] = bfhi(t[d]); }
                    }
                }
                float s[8];                                  // heads hg .. hg + 3 of the first position, then of the second
#pragma unroll
                for (int h = 0; h < 8; h++) {
                    s[h] = q[h & 3][0] * k[h >> 2][0];
#pragma unroll
                    for (int d = 1; d < DL; d++) s[h] = fmaf(q[h & 3][d], k[h >> 2][d], s[h]);
                }
                // eight sums over the lanes: half of them part ways each time, lane group lane >> 2 ends with sum lane >> 2
#pragma unroll
                for (int m = 16, c = 4; m >= 4; m >>= 1, c >>= 1) {
                    const bool hi = (lane & m) != 0;
#pragma unroll
                    for (int h = 0; h < 4; h++)
                        if (h < c) {
                            const float keep = hi ? s[h + c] : s[h], send = hi ? s[h] : s[h + c];
                            s[h] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                        }
                }
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
                const int at = i + 8 * (lane >> 4);
                if ((lane & 3) == 0 && at < n) ssc[(hg + ((lane >> 2) & 3)) * SP + at] = s[0];
            }
        }
        rg.release(n > a.kv_tile ? 2 : 1, lane);             // the keys
        s1_bar();
        if (warp < 8) {
            float sv[S1_PASS / 32], mx = m_run;
#pragma unroll
            for (int j = 0; j < S1_PASS / 32; j++) { const int i = lane + 32 * j; sv[j] = i < n ? ssc[warp * SP + i] : -INFINITY; mx = fmaxf(mx, sv[j]); }
            mx = warp_max(mx);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < S1_PASS / 32; j++) {
                const int i = lane + 32 * j;
                const float e = sv[j] == -INFINITY ? 0.f : exp2f(sv[j] - mx);
                if (i < n) ssc[warp * SP + i] = e;
                sum += e;
            }
            sum = warp_sum(sum);
            const float corr = m_run == -INFINITY ? 0.f : exp2f(m_run - mx);
            l_run = l_run * corr + sum;
            m_run = mx;
            if (lane == 0) scorr[warp] = corr;
        }
        s1_bar();
        float acc[8][4];
#pragma unroll
        for (int h = 0; h < 8; h++)
#pragma unroll
            for (int d = 0; d < 4; d++) acc[h][d] = 0.f;
        tiles_landed(n);
#pragma unroll 1
        for (int i = pl; i < n; i += PPI) {
            float4 v;
            if (pb + i == pos) v = *reinterpret_cast<const float4*>(svn + dv);
            else if (f32) v = *reinterpret_cast<const float4*>(row_at(i) + 4 * dv);
            else {
                const uint2 t = *reinterpret_cast<const uint2*>(row_at(i) + 2 * dv);
                v = make_float4(bflo(t.x), bfhi(t.x), bflo(t.y), bfhi(t.y));
            }
#pragma unroll
            for (int h = 0; h < 8; h++) {
                const float e = ssc[h * SP + i];
                acc[h][0] = fmaf(e, v.x, acc[h][0]); acc[h][1] = fmaf(e, v.y, acc[h][1]); acc[h][2] = fmaf(e, v.z, acc[h][2]); acc[h][3] = fmaf(e, v.w, acc[h][3]);
            }
        }
        rg.release(n > a.kv_tile ? 2 : 1, lane);             // the values
        // sum over the lanes of different positions, halving the heads, then the dims each time
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; i++) f[i] = acc[i >> 2][i & 3];
#pragma unroll
        for (int t = 0; t < STEPS; t++) {
            const int m = 16 >> t, c = 16 >> t;
            const bool hi = (lane & m) != 0;
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i < c) {
                    const float keep = hi ? f[i + c] : f[i], send = hi ? f[i] : f[i + c];
                    f[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                }
        }
        const float corr = pb > p0 ? scorr[ho] : 0.f;
#pragma unroll
        for (int i = 0; i < LEFT; i++) o_run[i] = fmaf(o_run[i], corr, f[i]);
        if (pb + 2 * a.kv_tile < p1) s1_bar();              // the scores may be overwritten
    }
    uint64_t* out = a.ll + a.o_ap + (size_t)blk.slice * 8 * (HD + 2);
    if (ho < G) {
#pragma unroll
        for (int i = 0; i < LEFT; i++) ll_store(out + ho * (HD + 2) + d_out + i, o_run[i], tag);
    }
    if (warp < G && lane < 2) ll_store(out + warp * (HD + 2) + HD + lane, lane ? l_run : m_run, tag);
}

template <int SD, int SO, int DK, int HD, int GH>
__global__ void __launch_bounds__(S1_THREADS, 1) k_step1(const __grid_constant__ Step1Args a) {
    using SM = Step1Smem<SD, SO, HD, GH>;
    // vectors of D: eight slices, as k_tcgemv cuts them; a warp and its neighbour share one and take every other tile. The mixers' output: sixteen
    // where it is long. A warp holds the 256 values (a chunk) its slice lies in, eight to a lane
    constexpr int D = SD * 16, KO = SO * 16, S2 = D / 8, OSL = KO > 2048 ? 16 : 8, S3 = KO / OSL, NC = D / 256, NCO = KO / 256;
    constexpr int GE = D / 512;                   // gate/up: 64-code groups of an eighth of a row
    constexpr int XP = D / 512;                   // values of a lane when all warps share a vector of D
    static_assert(NC <= 8 && S1_WARPS % NC == 0 && (XP == 1 || XP % 2 == 0), "named barriers 3 .. 10, ll_wait");
    extern __shared__ __align__(128) unsigned char s1_smem[];
    unsigned char* ring = s1_smem;
    unsigned char* scratch_all = ring + (size_t)a.nst * a.stage_bytes;
    float* xf_all = reinterpret_cast<float*>(scratch_all + SM::SCRATCH);
    float* part_all = xf_all + D;
    float* dl = part_all + 2 * S1_WARPS * S1_ROWS;
    Step1Layer* s_lay = reinterpret_cast<Step1Layer*>(dl + SM::DELTA / 4);
    float* s_sh = dl;                                  // the mixer's arrays, the shared expert's partial sums and the best logits are never alive together
    float* s_bv = dl;
    int* s_bi = reinterpret_cast<int*>(dl + S1_LOT * 16);
    __shared__ __align__(8) uint64_t s_bars[2 * S1_MAXST];
    __shared__ uint32_t s_tiles[S1_TILES];
    __shared__ __align__(8) S1Copy s_copies[S1_TILES * S1_COPIES];
    __shared__ __align__(16) uint4 s_ecopies[48];      // of the picks' rows: pick, place in the stage, bytes, offset in the expert
    __shared__ int s_count[S1_KINDS];                  // tiles of a stage: int8 | bf16 << 8
    __shared__ __align__(16) float s_ss[2][16], s_mx[2][16];      // per chunk, of one round and the next
    __shared__ float s_xg[D / 64], s_x[16], s_topv[8], s_topw[8], s_sg;
    __shared__ __align__(8) uint64_t s_picked;         // the layer's picks are made
    __shared__ float s_omx[16], s_scale;
    __shared__ int s_top[8], s_page[S1_PAGES], s_last;
    __shared__ S1Block s_blk;
    __shared__ float s_rope[HD];                       // cosines | sines of this position
    __shared__ __align__(8) uint32_t s_given_up[2];    // a wait of this block has run out | after so many polls
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tid = lane & 3;
    const int blk = blockIdx.x, G = gridDim.x;

    if (threadIdx.x == 0) {
        s_given_up[0] = 0u;
        s_given_up[1] = a.polls;
        mbar_init(&s_picked, 1);
        for (int s = 0; s < a.nst; s++) { mbar_init(&s_bars[s], 1); mbar_init(&s_bars[S1_MAXST + s], S1_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < S1_TILES * S1_COPIES; i += S1_THREADS) s_copies[i] = a.copies[(size_t)blk * S1_TILES * S1_COPIES + i];
    if (threadIdx.x < S1_TILES) s_tiles[threadIdx.x] = a.tiles[(size_t)blk * S1_TILES + threadIdx.x];
    for (int i = threadIdx.x; i < (int)(sizeof(Step1Layer) / 8); i += S1_THREADS)
        reinterpret_cast<uint64_t*>(s_lay)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
    const uint32_t epoch = *a.epoch;
    const int pos = a.pos[0];
    for (int i = threadIdx.x; i < HD; i += S1_THREADS) {
        const int hr = a.RD / 2, j = i % (HD / 2);
        if (j < hr) s_rope[i] = (i < HD / 2 ? a.rope_cos : a.rope_sin)[(size_t)pos * hr + j];
    }
    int id = a.tok[0];
    if (id < 0 || id >= a.V) {
        if (blk == 0 && threadIdx.x == 0) atomicExch(a.err, 1);
        id = 0;
    }
    if (threadIdx.x >= 32 && threadIdx.x < 32 + S1_KINDS) {
        const int kind = threadIdx.x - 32;
        int n = 0;
        for (int i = 0; i < s1_cap(kind); i++) {
            const uint32_t t = a.tiles[(size_t)blk * S1_TILES + s1_at(kind) + i];
            if (t != S1_NONE) n += s1_is_bf(kind, t >> 29) ? 256 : 1;
        }
        s_count[kind] = n;
    }
    if (threadIdx.x == 0) {
        S1Block& k = s_blk;
        k.r0 = (int)((long)blk * D / G); k.r1 = (int)((long)(blk + 1) * D / G);
        const int np = a.topk * a.I;
        k.gp0 = (int)((long)blk * np / G); k.gp1 = (int)((long)(blk + 1) * np / G);
        k.v0 = (int)((long)blk * a.V / G); k.v1 = (int)((long)(blk + 1) * a.V / G);
        // the slice of the context is the same in every layer: at least 16 positions, as many slices as there are blocks per KV head
        const int ns = G / a.KV, chunk = max(16, (pos + ns) / ns);
        k.id = id; k.pos = pos;
        k.kvh = blk / ns; k.slice = blk; k.nused = pos / chunk + 1;
        k.p0 = k.kvh < a.KV ? (blk - k.kvh * ns) * chunk : 0;
        k.p1 = k.kvh < a.KV ? min(pos + 1, k.p0 + chunk) : 0;
        for (int i = 0; k.p0 < k.p1 && i <= (k.p1 - 1) / KV_PAGE - k.p0 / KV_PAGE && i < S1_PAGES; i++) s_page[i] = a.page_table[k.p0 / KV_PAGE + i];
    }
    __syncthreads();

    const uint32_t bars = held(smem_u32(s_bars)), ring0 = smem_u32(ring), flag = held(smem_u32(s_given_up));
    if (warp >= S1_WARPS) {
        regs_dec<S1_REGS_LOW>();
        if (warp > S1_WARPS) {
            // the core engine's picks: nothing of the step depends on them, so an idle warp of the last block makes them, at its own pace (its
            // words have a place per layer)
            if (blk != G - 1 || warp != S1_WARPS + 1) return;
#pragma unroll 1
            for (int l = 0; l < a.L; l++) {
                int* counts = a.layers[l].counts;
                if (!counts) continue;
#pragma unroll 1
                for (int i = lane * 2; i < ((a.n1 + a.n2 + 63) / 64) * 64; i += 64) {
                    float t[2];
                    ll_wait<2>(a.ll + a.o_cs + l * a.cs_words + i, epoch + (uint32_t)l + 1, i + 1 < a.n1 + a.n2, t, flag);
                    if (i + 1 < a.n1 + a.n2) { a.cscore[i] = t[0]; a.cscore[i + 1] = t[1]; }
                }
                __threadfence();
                __syncwarp();
                s1_core_route(a, counts, lane);
                __syncwarp();
            }
            return;
        }
        // ---- producer: what the block reads of weights and cache, in the order of use. Every tile is up to 32 copies, a lane each ----
        int st = 0;
        uint32_t ph = 1, cnt = 0;
        bool out = false;                         // a wait has run out: a stage may still be being written, so nothing more is asked for
        // waits for the next stage, announces the bytes and has every lane start its copy: bytes at src to `to` of the stage
        auto issue = [&](const char* src, uint32_t bytes, uint32_t to) {
            s1_mbar_wait(bars + 8 * (S1_MAXST + st), ph, flag);
            out = s1_given_up(0, flag);
            if (out) return;
            const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
            if (lane == 0) mbar_expect_tx(bars + 8 * st, total);
            __syncwarp();
            if (bytes) bulk_load(ring0 + (uint32_t)(st * a.stage_bytes) + to, src, bytes, bars + 8 * st);
            cnt++;
            if (++st == a.nst) { st = 0; ph ^= 1u; }
        };
        // The copies of the picks' rows: lanes 0 .. 3 gate and 4 .. 7 up (half, and on which side of the border between two picks), 8 .. 15 their
        // scales and minima, 16 .. 31 down halves; then the down rows' scales and minima, from the 16-byte border before the first row's
        uint32_t e_total;
        {
            const int gp0 = s_blk.gp0, np = s_blk.gp1 - gp0, r0 = s_blk.r0, nr = s_blk.r1 - r0, nh = (np + 1) / 2, rh = (nr + 1) / 2;
            const uint32_t db = (uint32_t)(r0 * (a.I / 32)) & ~15u, de = ((uint32_t)((r0 + nr) * (a.I / 32)) + 15u) & ~15u;
            uint4 c = make_uint4(0u, 0u, 0u, 0u);
            if (lane < 16) {
                const bool rows = lane < 8, second = rows && (lane & 1), beyond = rows ? (lane & 2) != 0 : (lane & 4) != 0;
                const int border = (gp0 / a.I + 1) * a.I, x0 = gp0 + (second ? nh : 0), y0 = rows && !second ? gp0 + nh : gp0 + np;
                const int x = beyond ? max(x0, border) : x0, y = beyond ? y0 : min(y0, border), rb = rows ? D / 2 : D / 32;
                if (x < y) {
                    c.x = (uint32_t)(x / a.I);
                    c.y = (uint32_t)((x - x0) * rb + (rows ? (second ? s1_half(nh, D / 2) : 0) : (lane & 3) * s1_gsc_stride(D)));
                    c.z = (uint32_t)((y - x) * rb);
                    c.w = (uint32_t)(rows ? 0 : ((lane & 1) ? a.off_gu_m : a.off_gu_s)) + (uint32_t)((((rows ? lane & 4 : lane & 2) ? a.I : 0) + x - (int)c.x * a.I) * rb);
                }
            } else if ((lane - 16) >> 1 < a.topk) {
                const int o = lane & 1 ? rh : 0, n = lane & 1 ? nr - rh : rh;
                c = make_uint4((uint32_t)((lane - 16) >> 1), (uint32_t)(((lane - 16) >> 1) * s1_dn_stride(nr, a.I / 2) + (lane & 1 ? s1_half(rh, a.I / 2) : 0)), (uint32_t)(n * (a.I / 2)),
                               (uint32_t)a.off_dn_q + (uint32_t)((r0 + o) * (a.I / 2)));
            }
            s_ecopies[lane] = c;
            if (lane < 16)
                s_ecopies[32 + lane] = lane < 2 * a.topk ? make_uint4((uint32_t)(lane >> 1), (uint32_t)(4 * s1_gsc_stride(D) + lane * s1_dsc_stride(a.I)), de - db, (uint32_t)((lane & 1) ? a.off_dn_m : a.off_dn_s) + db)
                                                         : make_uint4(0u, 0u, 0u, 0u);
            e_total = lane < 8 ? (uint32_t)(np * (D / 2)) : (lane < 16 ? (uint32_t)(4 * np * (D / 32)) + 2u * (uint32_t)a.topk * (de - db) : (uint32_t)(a.topk * nr * (a.I / 2)));
            __syncwarp();
        }
        uint64_t wn = reinterpret_cast<const uint64_t*>(a.layers)[lane];      // lane q: pointer q of the layer to come
#pragma unroll 1
        for (int l = 0; l < a.L && !out; l++) {
            const uint64_t wp = wn;
            if (l + 1 < a.L) wn = reinterpret_cast<const uint64_t*>(a.layers + l + 1)[lane];
            const bool attn = __shfl_sync(0xffffffffu, wp, Q_KPOOL) != 0;
            // rows of weights, and what the epilogue needs of them
#pragma unroll 1
            for (int kind = attn ? S1_IN_ATTN : S1_IN_DELTA; kind < S1_KINDS; kind = kind < S1_OUT ? (int)S1_OUT : kind + 1) {
#pragma unroll 1
                for (int i = s1_at(kind), e = i + s1_cap(kind); i < e && !out; i++) {
                    if (s_tiles[i] == S1_NONE) break;
                    const S1Copy c = s_copies[i * S1_COPIES + (lane & (S1_COPIES - 1))];
                    const char* src = (const char*)__shfl_sync(0xffffffffu, wp, c.what & 31u);
                    issue(src + (size_t)c.from * 16u, lane < S1_COPIES && src ? (c.what >> 16) * 16u : 0u, ((c.what >> 5) & 2047u) * 16u);       // (a layer may have no core keys: nobody reads what its tiles then hold)
                }
                if (kind == S1_IN_ATTN) {
                    // this block's slice of the cache: keys of up to two tiles, then their values, and again. Rows of a page lie one after another; the
                    // newest position's are read as they are and not used
                    const uint32_t rb = HD * (a.kv_f32 ? 4 : 2);
#pragma unroll 1
                    for (int i = 0; !out; i++) {
                        const int p0 = s_blk.p0, p1 = s_blk.p1, first = p0 + (i >> 2) * 2 * a.kv_tile, f = first + (i & 1) * a.kv_tile, n = min(a.kv_tile, p1 - f);
                        if (first >= p1) break;
                        if (n <= 0) continue;
                        const char* pool = (const char*)__shfl_sync(0xffffffffu, wp, Q_KPOOL + ((i >> 1) & 1));
                        const int cut = min(n, KV_PAGE - f % KV_PAGE), o = lane == 1 ? cut : 0, m = lane == 0 ? cut : (lane == 1 ? n - cut : 0);         // rows in the first page
                        issue(m > 0 ? pool + (((size_t)s_page[(f + o) / KV_PAGE - p0 / KV_PAGE] * a.KV + s_blk.kvh) * KV_PAGE + (f + o) % KV_PAGE) * rb : pool, (uint32_t)m * rb, (uint32_t)o * rb);
                    }
                }
            }
            // the picks' rows, four tiles at once: gate, up, scales, down
            // (from the table made above: what comes between the picks and their rows is waited for by everyone)
            const char* experts = (const char*)__shfl_sync(0xffffffffu, wp, Q_EXPERTS);
            const uint4 c = s_ecopies[lane], cd = s_ecopies[32 + (lane & 15)];
            const int u = lane < 8 ? lane >> 2 : (lane < 16 ? 2 : 3), t = st + u, w = t >= a.nst ? t - a.nst : t;
            const uint32_t bar = bars + 8 * w, at = ring0 + (uint32_t)(w * a.stage_bytes);
            s1_mbar_wait(bars + 8 * S1_MAXST + (bar - bars), t >= a.nst ? ph ^ 1u : ph, flag);
            s1_mbar_wait(smem_u32(&s_picked), l & 1, flag);
            out = s1_given_up(0, flag);
            if (out) break;
            const char* src = experts + (size_t)(uint32_t)max(0, s_top[c.x]) * (uint32_t)a.expert_bytes + c.w;
            const char* srcd = experts + (size_t)(uint32_t)max(0, s_top[cd.x]) * (uint32_t)a.expert_bytes + cd.w;
            if (lane == 0 || lane == 4 || lane == 8 || lane == 16) mbar_expect_tx(bar, e_total);
            __syncwarp();
            if (lane < 16 && c.z) bulk_load(at + c.y, src, c.z, bar);
            {
                const int ts = st + 2, ws = ts >= a.nst ? ts - a.nst : ts;
                if (lane < 16 && cd.z) bulk_load(ring0 + (uint32_t)(ws * a.stage_bytes) + cd.y, srcd, cd.z, bars + 8 * ws);
            }
            // (the down rows, needed a stage later, only when the up rows are here: together they would arrive together)
            {
                const int tu = st + 1;
                s1_mbar_wait(bars + 8 * (tu >= a.nst ? tu - a.nst : tu), tu >= a.nst ? ph : ph ^ 1u, flag);
            }
            if (lane >= 16 && c.z) bulk_load(at + c.y, src, c.z, bar);
            cnt += 4;
            st += 4;
            if (st >= a.nst) { st -= a.nst; ph ^= 1u; }
        }
#pragma unroll 1
        for (int i = s_blk.v0; i < s_blk.v1 && !out; i += a.head_rows) {
            const int n = min(a.head_rows, s_blk.v1 - i), h = (n + 1) / 2;
            const uint32_t from = (uint32_t)(i * 2) & ~15u;
            const char* src = lane < 2 ? (const char*)a.head_w + (size_t)(i + (lane ? h : 0)) * D : (const char*)a.head_s + from;
            issue(src, lane < 2 ? (uint32_t)((lane ? n - h : h) * D) : (lane == 2 ? (((uint32_t)(i + n) * 2 + 15) & ~15u) - from : 0u), lane == 0 ? 0u : (lane == 1 ? (uint32_t)a.half_i8 : (uint32_t)(a.stage_bytes - S1_OPS)));
        }
        // no copy may be in flight when the block leaves
        for (int s = 0; s < a.nst; s++)
            if (cnt > (uint32_t)s) mbar_wait(bars + 8 * s, ((cnt - s + a.nst - 1) / a.nst - 1) & 1, a.err);
        return;
    }

    // ---- computing warps ----
    regs_inc<S1_REGS_HIGH>();
    S1Ring rg{ring, bars, a.stage_bytes, a.nst, 0, 0u, flag};
    int pb = 0;                                   // which half of part and s_ss this stage uses
    S1Trace tr{a.trace, -1};
    int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;               // epilogue: tile and slot of this thread
    unsigned char* scratch = scratch_all;
    // Every stage starts from thread numbers the compiler knows nothing about. It would otherwise work out the addresses of all stages once,
    // ahead of the layers, and keep them in local memory: behind a ring of this size L1 holds a twentieth of that
    auto fresh = [&]() {
        int t = threadIdx.x;
        asm volatile("" : "+r"(t));
        lane = t & 31; warp = t >> 5; gid = lane >> 2; tid = lane & 3; ti = t >> 4; tj = t & 15;
        int z = a.nst * a.stage_bytes;
        asm volatile("" : "+r"(z));
        scratch_all = s1_smem + z;
        xf_all = reinterpret_cast<float*>(scratch_all + SM::SCRATCH);
        part_all = xf_all + D;
        dl = part_all + 2 * S1_WARPS * S1_ROWS;
        s_lay = reinterpret_cast<Step1Layer*>(dl + SM::DELTA / 4);
        s_sh = dl;
        s_bv = dl;
        s_bi = reinterpret_cast<int*>(dl + S1_LOT * 16);
        scratch = scratch_all + warp * SM::SCR;
    };
    fresh();
    if (threadIdx.x < s_blk.r1 - s_blk.r0) s_x[threadIdx.x] = bf(a.embed[(size_t)s_blk.id * D + s_blk.r0 + threadIdx.x]);

    // the factors of plane 0 and 1 (or 2 and 3) of a lane's sums
    auto weights_of = [&](float scale, float& pw0, float& pw1) {
        pw0 = scale * (tid == 0 ? 1.0f : (tid == 1 ? 1.0f / 65536.0f : 0.f));
        pw1 = pw0 * (1.0f / 256.0f);
    };
    auto out_chunk = [](int w) { return (OSL == 16 ? w : w >> 1) * S3 / 256; };      // of the mixers' output: the one warp w holds
    auto sum_of = [&](const float* p, int n) {    // one row's partial sums of n slices
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 16; w++)
            if (w < n) s += p[w * S1_ROWS];
        return s;
    };

    // Two rounds a layer and one for the head. A round is a norm and the matrices behind it, in one place so that the step's code stays short
    // (a stage's code runs once per layer: what does not fit the instruction caches is fetched again every time): in-projections, then
    // mixer and out projection; router and shared expert, then the experts
#pragma unroll 1
    for (int rd = 0;; rd++) {
        fresh();
        const bool head = rd == 2 * a.L, moe = !head && (rd & 1);
        const int l = rd >> 1;
        const Step1Layer& ly = s_lay[l & 1];
        const uint32_t tag = epoch + (uint32_t)l + 1;
        uint64_t* set = a.ll + (size_t)(l & 1) * a.ll_set;
        asm volatile("" : "+l"(set));
        const bool attn = !head && ly.attn != 0;
        tr.in(1, head ? a.V : (moe ? a.E : (attn ? 2 * a.H * HD : a.C)));
        const int kind = moe ? S1_MOE : (attn ? S1_IN_ATTN : S1_IN_DELTA);
        const int ks = warp >> 1, par = warp & 1, ck = ks * S2 / 256;
        const bool chief = par == 0 && ks * S2 % 256 == 0;      // of the warps that hold a chunk
        float pw0, pw1;
        uint4 xb[S2 / 64];
        {
            // (1 + w) x / rms(x): the chunks' sums of squares and largest |(1 + w) x| meet behind one barrier, and the rms joins there
            float xv[8], ss = 0.f, mx = 0.f;
            uint32_t nw[4];
            const int k = ck * 256 + lane * 8;
            ldg_words<4>((head ? a.norm : (moe ? ly.norm2 : ly.norm1)) + k, nw);
            {
                // a chunk's warps poll a part of it each and share it: 148 blocks' polls are bytes that L2 has to deliver (2.4 MB a look, 0.4 us)
                float xp[XP];
                const int kp = ck * 256 + (warp % (S1_WARPS / NC)) * 32 * XP + lane * XP;
                if (rd == 0) {
#pragma unroll
                    for (int i = 0; i < XP; i++) xp[i] = bf(a.embed[(size_t)s_blk.id * D + kp + i]);
                } else ll_wait<XP>((moe ? set + a.o_xb : a.ll + (size_t)((l & 1) ^ 1) * a.ll_set + a.o_xa) + kp, moe ? tag : tag - 1, true, xp, flag);
                tr.pt(1);
#pragma unroll
                for (int i = 0; i < XP; i++) xf_all[kp + i] = xp[i];
                __syncwarp();
                bar_sync(3 + ck, 32 * (S1_WARPS / NC));
                const float4 x0 = *reinterpret_cast<const float4*>(xf_all + k), x1 = *reinterpret_cast<const float4*>(xf_all + k + 4);
                xv[0] = x0.x; xv[1] = x0.y; xv[2] = x0.z; xv[3] = x0.w; xv[4] = x1.x; xv[5] = x1.y; xv[6] = x1.z; xv[7] = x1.w;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) { ss = fmaf(xv[i], xv[i], ss); xv[i] *= 1.0f + ((i & 1) ? bfhi(nw[i / 2]) : bflo(nw[i / 2])); mx = fmaxf(mx, fabsf(xv[i])); }
            ss = warp_sum(ss);
            mx = warp_absmax(mx);
            if (chief && lane == 0) { s_ss[rd & 1][ck] = ss; s_mx[rd & 1][ck] = mx; }
            s1_bar();
            float t = 0.f;
            mx = 0.f;
#pragma unroll
            for (int w = 0; w < NC; w++) { t += s_ss[rd & 1][w]; mx = fmaxf(mx, s_mx[rd & 1][w]); }
            const float rn = 1.0f / sqrtf(t / (float)D + a.eps);
            mx *= rn;
#pragma unroll
            for (int i = 0; i < 8; i++) xv[i] *= rn;
            planes8(xv, mx > 1e-30f ? M1_QMAX / mx : 0.f, false, scratch, lane);
            weights_of(mx / M1_QMAX, pw0, pw1);
            if (!head) {
                // for the bf16 rows; warps that share a chunk write the same values
                *reinterpret_cast<float4*>(xf_all + k) = make_float4(xv[0], xv[1], xv[2], xv[3]);
                *reinterpret_cast<float4*>(xf_all + k + 4) = make_float4(xv[4], xv[5], xv[6], xv[7]);
            }
            __syncwarp();
            load_planes<S2>(scratch, ks * S2 % 256, gid, tid, xb);
        }
        if (!head && !moe && !attn && threadIdx.x < DK && blk < a.HV * (a.DV / 32)) {
            // the state's slab of this block's DeltaNet task, towards L2
            const int nslab = a.DV / 32;
            l2_prefetch(ly.state + ((size_t)(blk / nslab) * DK + threadIdx.x) * a.DV + (blk % nslab) * 32);
        }
        // one lot of tiles; the head takes many, the epilogue of one under the products of the next
        int row_h = s_blk.v0;
#pragma unroll 1
        for (bool first = true;; first = false) {
            int n8, nb = 0, seg = 0, row0, n;
            if (head) {
                n8 = min(S1_LOT, (s_blk.v1 - row_h + a.head_rows - 1) / a.head_rows);
                row0 = row_h + ti * a.head_rows;
                n = ti < S1_LOT ? min(a.head_rows, s_blk.v1 - row0) : 0;
            } else {
                n8 = s_count[kind] & 255; nb = s_count[kind] >> 8;
                const uint32_t td = ti < s1_cap(kind) ? s_tiles[s1_at(kind) + ti] : 0u;
                seg = td >> 29; row0 = td & 0xffffff; n = td == S1_NONE ? 0 : (td >> 24) & 31;
            }
            const int slot_row = s1_slot_row(tj, n), row = row0 + slot_row;
            const bool mine = n > 0 && slot_row >= 0 && (tj < 8 || !(moe && seg == 4));
            // what the epilogue needs of a tile's rows goes from the stage to the threads' own places before the stage is handed back
            float* op = dl + SM::MIX / 4 + 7 * threadIdx.x;
            int tile = 0;                                       // the next one to land
            auto keep = [&](int n) {
                if (mine && ti >= tile && ti < tile + n) {
                    const unsigned char* o = rg.stage(ti - tile) + a.stage_bytes - S1_OPS;
                    op[0] = bf(reinterpret_cast<const uint16_t*>(o)[(row0 & 7) + slot_row]);
                    op[1] = moe && seg == 0 ? reinterpret_cast<const float*>(o + 64)[(row0 & 3) + slot_row] : bf(reinterpret_cast<const uint16_t*>(o + 64)[(row0 & 7) + slot_row]);
                    if (!head && !moe && !attn && seg == 2) {
                        const uint32_t* cw = reinterpret_cast<const uint32_t*>(o + 128 + 8 * ((row0 & 1) + slot_row));
                        const float* ct = reinterpret_cast<const float*>(o + 272 + ((row0 * 12) & 15) + 12 * slot_row);
                        op[2] = __uint_as_float(cw[0]); op[3] = __uint_as_float(cw[1]); op[4] = ct[0]; op[5] = ct[1]; op[6] = ct[2];
                    }
                }
                tile += n;
            };
            float* part = part_all + (pb * S1_WARPS + ks) * S1_ROWS;
            s1_bf_run<S2, D>(rg, nb, a.half_bf, xf_all + ks * S2, part, ks, par, lane, keep);
            s1_i8_run<S2, D, true>(rg, n8, moe ? a.half_pair : a.half_i8, moe ? 2 * a.half_pair : 4 * D, xb, pw0, pw1, part + 16 * nb, ks, par, lane, keep);
            tr.pt(3);
            s1_bar();
            if (head && first && threadIdx.x < S1_LOT * 16) { s_bv[threadIdx.x] = -INFINITY; s_bi[threadIdx.x] = 0x7fffffff; }      // its own only, until the end
            if (mine) {
                const float* pr = part_all + pb * S1_WARPS * S1_ROWS + ti * 16 + tj;
                const float v = sum_of(pr, 8), e0 = op[0], e1 = op[1];
                uint64_t* to = set;
                float y = e0 * v;
                if (head) {
                    a.logits[row] = y;
                    if (y > s_bv[threadIdx.x] || (y == s_bv[threadIdx.x] && row < s_bi[threadIdx.x])) { s_bv[threadIdx.x] = y; s_bi[threadIdx.x] = row; }
                } else {
                    if (moe) {
                        to = seg == 0 ? set + a.o_rl : (seg == 4 ? set + a.o_sa : (seg == 3 ? set + a.o_sg : a.ll + a.o_cs + l * a.cs_words + (seg == 2 ? a.n1 : 0)));
                        if (seg < 3) y = seg == 0 && ly.bias ? v + e1 : v;
                        else if (seg == 3) y = sigmoidf_(v);
                        else y = siluf_(y) * (e1 * sum_of(pr + 8, 8));
                    } else if (attn) to += a.o_q + (seg == 0 ? 0 : (seg == 1 ? 2 * a.H * HD : (2 * a.H + a.KV) * HD));
                    else if (seg == 2) {
                        // hybrid.py:393-398: y = silu(sum_j w[c][j] * taps[j]), taps = 3 previous inputs + the new one
                        float* stt = ly.conv_state + (size_t)row * 3;
                        const uint32_t cw0 = __float_as_uint(op[2]), cw1 = __float_as_uint(op[3]);
                        stt[0] = op[5]; stt[1] = op[6]; stt[2] = y;
                        float c = bflo(cw0) * op[4];
                        c = fmaf(bfhi(cw0), op[5], c);
                        c = fmaf(bflo(cw1), op[6], c);
                        y = siluf_(fmaf(bfhi(cw1), y, c));
                        to += a.o_q;
                    } else if (seg == 3) { y = siluf_(y); to += a.o_z; }
                    else {
                        // beta = sigmoid(b), decay = exp(-exp(A) softplus(a + dt))
                        y = seg == 0 ? sigmoidf_(v) : -expf(e0) * softplusf_(v + e1);
                        to += a.o_bg + seg * a.HV;
                    }
                    ll_store(to + row, y, tag);
                }
            }
            pb ^= 1;
            if (!head) s1_bar();
            row_h += S1_LOT * a.head_rows;
            if (!head || row_h >= s_blk.v1) break;
        }
        tr.out();
        if (head) break;
        if (!moe) {
            // the next layer's pointers: nobody reads the other copy any more
            if (l + 1 < a.L && threadIdx.x < sizeof(Step1Layer) / 16) {
                cp_async16(reinterpret_cast<unsigned char*>(s_lay + ((l + 1) & 1)) + 16 * threadIdx.x, reinterpret_cast<const unsigned char*>(a.layers + l + 1) + 16 * threadIdx.x);
                cp_async_commit();
            }
        }
        fresh();
        if (!moe) {
        // ================= mixer =================
        if (attn) {
            tr.in(7, s_blk.nused, s_blk.p0 < s_blk.p1);
            if (s_blk.p0 < s_blk.p1) {
                s1_attend<HD>(a, ly, set, tag, s_blk, s_page, s_rope, scratch_all, rg, tr, warp, lane);
                tr.out();
            }
            // merge of the slices, x sigmoid(gate) (aegist/hybrid.py:245-262): 32 dims of one head per task, a warp every 16th slice
            fresh();
            float* sm_m = dl;                                   // [16] | [16] | [16][32]
            float* sm_l = dl + 16;
            float* sm_o = dl + 32;
            const int mt = a.H * (HD / 32), ns = G / a.KV, nused = s_blk.nused;
            tr.in(8, nused, blk < mt);
            for (int t = blk; t < mt; t += G) {
                const int h = t / (HD / 32), d = (t % (HD / 32)) * 32 + lane, kv = h / (a.H / a.KV);
                const uint64_t* src = a.ll + a.o_ap + ((size_t)kv * ns * 8 + h % (a.H / a.KV)) * (HD + 2);
                float M = -INFINITY, Ls = 0.f, O = 0.f, g[1] = {0.f};
                if (warp == 0) ll_wait<1>(set + a.o_q + (size_t)h * 2 * HD + HD + d, tag, true, g, flag);
                constexpr int MB = 5;                           // slices whose words are asked for together
                for (int i0 = warp; i0 < nused; i0 += MB * S1_WARPS) {
                    float ml[MB][2], o[MB];
                    uint64_t r[MB][3];
#pragma unroll 1
                    for (int spin = 0;; spin++) {
                        bool ok = true;
#pragma unroll
                        for (int u = 0; u < MB; u++) {
                            const uint64_t* ps = src + (size_t)(i0 + u * S1_WARPS) * 8 * (HD + 2);
                            if (i0 + u * S1_WARPS < nused) { ll_load2(ps + HD, r[u][0], r[u][1]); r[u][2] = ll_load(ps + d); }
                        }
#pragma unroll
                        for (int u = 0; u < MB; u++)
                            if (i0 + u * S1_WARPS < nused) ok = ok && (uint32_t)(r[u][0] >> 32) == tag && (uint32_t)(r[u][1] >> 32) == tag && (uint32_t)(r[u][2] >> 32) == tag;
                        if (__all_sync(0xffffffffu, ok) || s1_given_up(spin, flag)) break;
                    }
                    float mn = M;
#pragma unroll
                    for (int u = 0; u < MB; u++) {
                        const bool on = i0 + u * S1_WARPS < nused;
                        ml[u][0] = on ? __uint_as_float((uint32_t)r[u][0]) : -INFINITY; ml[u][1] = on ? __uint_as_float((uint32_t)r[u][1]) : 0.f;
                        o[u] = on ? __uint_as_float((uint32_t)r[u][2]) : 0.f;
                        mn = fmaxf(mn, ml[u][0]);
                    }
                    const float c0 = M == -INFINITY ? 0.f : exp2f(M - mn);
                    O *= c0; Ls *= c0;
#pragma unroll
                    for (int u = 0; u < MB; u++) {
                        const float c1 = ml[u][0] == -INFINITY ? 0.f : exp2f(ml[u][0] - mn);
                        O = fmaf(o[u], c1, O);
                        Ls = fmaf(ml[u][1], c1, Ls);
                    }
                    M = mn;
                }
                if (lane == 0) { sm_m[warp] = M; sm_l[warp] = Ls; }
                sm_o[warp * 32 + lane] = O;
                s1_bar();
                if (warp == 0) {
                    float mx = -INFINITY;
#pragma unroll
                    for (int w = 0; w < S1_WARPS; w++) mx = fmaxf(mx, sm_m[w]);
                    float o = 0.f, ls = 0.f;
#pragma unroll
                    for (int w = 0; w < S1_WARPS; w++) {
                        const float c = sm_m[w] == -INFINITY ? 0.f : exp2f(sm_m[w] - mx);
                        o = fmaf(sm_o[w * 32 + lane], c, o);
                        ls = fmaf(sm_l[w], c, ls);
                    }
                    ll_store(set + a.o_og + h * HD + d, o / ls * sigmoidf_(g[0]), tag);
                }
                s1_bar();
            }
            if (blk >= mt) s1_bar();                            // the attention's arrays lie over the warps' scratch
            tr.out(blk < mt);
        } else {
            // gated delta rule on a [DK x 32] column slab per task (aegist/hybrid.py:314-324, 409-412); the gated norm is the reader's
            float* qs = dl;
            float* ks = dl + 128;
            float* vs = dl + 256;                               // [32] v
            float* bs = vs + 64;                                // [2] beta, decay
            float* red = bs + 32;                               // [2][8][32]
            constexpr int RPT = DK / 8;                         // state rows of a lane of the eight warps that hold the slab, as in k_delta_step
            const int nslab = a.DV / 32, ntask = a.HV * nslab;
            tr.in(3, ntask, blk < ntask);
            // silu(z) for the out projection, in scratch, slices w and w + 1: warps that do not hold the state fetch them for all, so that the polls for
            // the delta rule's output look at nothing else (9.5 MB a look with both; 0.4 us of a layer)
            auto fetch_z = [&](int w) {
                float z0[8], z1[8];
                ll_wait2<8, 8>(set + a.o_z + out_chunk(w) * 256 + lane * 8, set + a.o_z + out_chunk(w + 1) * 256 + lane * 8, tag, true, z0, z1, flag);
                float4 *t0 = reinterpret_cast<float4*>(scratch_all + w * SM::SCR) + 2 * lane, *t1 = reinterpret_cast<float4*>(scratch_all + (w + 1) * SM::SCR) + 2 * lane;
                t0[0] = make_float4(z0[0], z0[1], z0[2], z0[3]);
                t0[1] = make_float4(z0[4], z0[5], z0[6], z0[7]);
                t1[0] = make_float4(z1[0], z1[1], z1[2], z1[3]);
                t1[1] = make_float4(z1[4], z1[5], z1[6], z1[7]);
            };
            if (blk >= ntask && warp < 8) fetch_z(2 * warp);
            if (blk >= ntask) s1_bar();
            for (int t = blk; t < ntask; t += G) {
                const int col0 = (t % nslab) * 32, h = t / nslab;
                float* S = ly.state + ((size_t)h * DK) * a.DV + col0 + lane;
                float stv[RPT];
                if (warp < 8) {
#pragma unroll
                    for (int r = 0; r < RPT; r++) stv[r] = __ldcg(S + (size_t)(warp + 8 * r) * a.DV);
                }
                const int hk = h / (a.HV / a.HK);
                if (warp == 8 || warp == 9) {                   // q, k: lane + 32 i, as they are normalised there
                    const bool isq = warp == 8;
                    const uint64_t* src = set + a.o_q + (size_t)(isq ? 0 : a.HK * DK) + hk * DK + lane;
                    float v[DK / 32], ss = 0.f;
                    uint64_t w[DK / 32];
#pragma unroll
                    for (int i = 0; i < DK / 32; i++) w[i] = (uint64_t)~tag << 32;
#pragma unroll 1
                    for (int spin = 0;; spin++) {
                        bool ok = true;
#pragma unroll
                        for (int i = 0; i < DK / 32; i++) ll_again(src + 32 * i, tag, w[i]);
#pragma unroll
                        for (int i = 0; i < DK / 32; i++) ok = ok && (uint32_t)(w[i] >> 32) == tag;
                        if (__all_sync(0xffffffffu, ok) || s1_given_up(spin, flag)) break;
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < DK / 32; i++) { v[i] = __uint_as_float((uint32_t)w[i]); ss = fmaf(v[i], v[i], ss); }
                    ss = warp_sum(ss);
                    const float r = 1.0f / sqrtf(ss + 1e-6f);
#pragma unroll
                    for (int i = 0; i < DK / 32; i++) {
                        float y = v[i] * r;
                        if (isq) y *= (DK == 128 ? 0.08838834764831845f : 0.125f);
                        (isq ? qs : ks)[lane + 32 * i] = y;
                    }
                } else if (warp == 10) {
                    float v[1];
                    ll_wait<1>(set + a.o_q + (size_t)2 * a.HK * DK + h * a.DV + col0 + lane, tag, true, v, flag);
                    vs[lane] = v[0];
                } else if (warp == 11) {
                    float v[1];
                    ll_wait<1>(set + a.o_bg + (lane & 1) * a.HV + h, tag, true, v, flag);
                    if (lane < 2) bs[lane] = lane ? expf(v[0]) : v[0];
                }
                s1_bar();
                tr.pt(1);
                if (warp >= 8 && t == blk) fetch_z(2 * (warp - 8));
                if (warp < 8) {
                    const float decay = bs[1];
                    float kv = 0.f;
#pragma unroll
                    for (int r = 0; r < RPT; r++) {
                        stv[r] *= decay;
                        kv = fmaf(stv[r], ks[warp + 8 * r], kv);
                    }
                    red[warp * 32 + lane] = kv;
                    bar_sync(2, 256);
                    kv = 0.f;
#pragma unroll
                    for (int w = 0; w < 8; w++) kv += red[w * 32 + lane];
                    tr.pt(3);
                    const float delta = (vs[lane] - kv) * bs[0];
                    float o = 0.f;
#pragma unroll
                    for (int r = 0; r < RPT; r++) {
                        stv[r] = fmaf(ks[warp + 8 * r], delta, stv[r]);
                        o = fmaf(stv[r], qs[warp + 8 * r], o);
                    }
                    red[(8 + warp) * 32 + lane] = o;
                    bar_sync(2, 256);
                    if (warp == 0) {
                        o = 0.f;
#pragma unroll
                        for (int w = 0; w < 8; w++) o += red[(8 + w) * 32 + lane];
                        ll_store(set + a.o_og + (size_t)h * a.DV + col0 + lane, o, tag);
                    }
#pragma unroll
                    for (int r = 0; r < RPT; r++) S[(size_t)(warp + 8 * r) * a.DV] = stv[r];
                }
                s1_bar();                                       // the arrays may be written again; and who waits for the next stage's input does so when this block's part of it is there
            }
            tr.out(blk < ntask);
        }

        // ================= out projection, into the residual stream =================
        {
            fresh();
            tr.in(1, D);
            const uint32_t td = ti < s1_cap(S1_OUT) ? s_tiles[s1_at(S1_OUT) + ti] : S1_NONE;
            const int row0 = td & 0xffffff, slot_row = s1_slot_row(tj, td == S1_NONE ? 0 : (td >> 24) & 31), row = row0 + slot_row;
            const bool mine = slot_row >= 0;
            float e0 = 0.f;
            int tile = 0;
            auto keep = [&](int n) {
                if (mine && ti >= tile && ti < tile + n) e0 = bf(reinterpret_cast<const uint16_t*>(rg.stage(ti - tile) + a.stage_bytes - S1_OPS)[(row0 & 7) + slot_row]);
                tile += n;
            };
            const int os = OSL == 16 ? warp : warp >> 1, opar = OSL == 16 ? -1 : warp & 1, oc = out_chunk(warp), k0 = oc * 256 + lane * 8;
            float xv[8], mx = 0.f, pw0, pw1;
            if (!attn) {
                // w * rmsnorm_DV(o) * silu(z) per value head (aegist/hybrid.py:133-147); a head is DV / 8 neighbouring lanes
                float zv[8], ss = 0.f;
                uint32_t gw[4];
                ldg_words<4>(ly.n_a + k0 % a.DV, gw);
                ll_wait<8>(set + a.o_og + k0, tag, true, xv, flag);
                {
                    const float4 *from = reinterpret_cast<const float4*>(scratch) + 2 * lane, z0 = from[0], z1 = from[1];
                    zv[0] = z0.x; zv[1] = z0.y; zv[2] = z0.z; zv[3] = z0.w; zv[4] = z1.x; zv[5] = z1.y; zv[6] = z1.z; zv[7] = z1.w;
                }
#pragma unroll
                for (int i = 0; i < 8; i++) ss = fmaf(xv[i], xv[i], ss);
                for (int o = a.DV >> 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float r = 1.0f / sqrtf(ss / (float)a.DV + a.eps);
#pragma unroll
                for (int i = 0; i < 8; i++) xv[i] = (((i & 1) ? bfhi(gw[i / 2]) : bflo(gw[i / 2])) * (xv[i] * r)) * zv[i];
            } else ll_wait<8>(set + a.o_og + k0, tag, true, xv, flag);
            tr.pt(1);
#pragma unroll
            for (int i = 0; i < 8; i++) mx = fmaxf(mx, fabsf(xv[i]));
            mx = warp_absmax(mx);
            if (lane == 0) s_omx[oc] = mx;                      // warps that share a chunk write the same value
            s1_bar();
            mx = 0.f;
#pragma unroll
            for (int w = 0; w < NCO; w++) mx = fmaxf(mx, s_omx[w]);
            planes8(xv, mx > 1e-30f ? M1_QMAX / mx : 0.f, false, scratch, lane);
            weights_of(mx / M1_QMAX, pw0, pw1);
            __syncwarp();
            uint4 xb[S3 / 64];
            load_planes<S3>(scratch, os * S3 % 256, gid, tid, xb);
            float* part = part_all + (pb * S1_WARPS + os) * S1_ROWS;
            s1_i8_run<S3, KO, false>(rg, s_count[S1_OUT] & 255, a.half_out, 0, xb, pw0, pw1, part, os, opar, lane, keep);
            tr.pt(3);
            s1_bar();
            if (mine) {
                const int r0 = s_blk.r0;
                const float v = fmaf(e0, sum_of(part_all + pb * S1_WARPS * S1_ROWS + ti * 16 + tj, OSL), s_x[row - r0]);
                s_x[row - r0] = v;
                ll_store(set + a.o_xb + row, v, tag);
            }
            pb ^= 1;
            s1_bar();
            tr.out();
        }

        continue;
        }

        if (warp % 2 == 0 && (warp >> 1) * S2 % 256 == 0) {
            // for the expert rows: the chunk's planes in nibble order (they lie over its values), and sums of 64 values for the rows' minima
            const int ck = (warp >> 1) * S2 / 256;
            float xv[8], mx = 0.f, t = 0.f, s8 = 0.f;
#pragma unroll
            for (int w = 0; w < NC; w++) { t += s_ss[rd & 1][w]; mx = fmaxf(mx, s_mx[rd & 1][w]); }
            mx *= 1.0f / sqrtf(t / (float)D + a.eps);
#pragma unroll
            for (int i = 0; i < 8; i++) { xv[i] = xf_all[ck * 256 + lane * 8 + i]; s8 += xv[i]; }
            s8 += __shfl_xor_sync(0xffffffffu, s8, 1);
            s8 += __shfl_xor_sync(0xffffffffu, s8, 2);
            s8 += __shfl_xor_sync(0xffffffffu, s8, 4);
            if ((lane & 7) == 0) s_xg[ck * 4 + (lane >> 3)] = s8;
            __syncwarp();
            planes8(xv, mx > 1e-30f ? M1_QMAX / mx : 0.f, true, reinterpret_cast<unsigned char*>(xf_all + ck * 256), lane);
            if (warp == 0 && lane == 0) s_scale = mx / M1_QMAX;
        }

        // ================= experts: picks, gate and up =================
        uint32_t dsl[(GH + 1) / 2], dsh[(GH + 1) / 2], dml[(GH + 1) / 2], dmh[(GH + 1) / 2];
        {
            fresh();
            const int gp0 = s_blk.gp0, np = s_blk.gp1 - gp0;
            tr.in(5, np);
            if (warp == 0) {
                float lg[8];
                const bool has = lane * 8 < a.E;
                ll_wait<8>(set + a.o_rl + lane * 8, tag, has, lg, flag);
                tr.pt(1);
                s1_route(lg, has, a.topk, lane, s_top, s_topv);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_picked));               // the producer fetches their rows
                float ts = 0.f;
                for (int r = 0; r < a.topk; r++) ts += s_topv[r];
                __syncwarp();
                if (lane < a.topk) {
                    const float wt = s_topv[lane] / ts;
                    s_topw[lane] = wt;
                    const int e = s_top[lane];
                    if (e < 0 || e >= a.E) atomicExch(a.err, 2);
                    if (blk == 0) { ly.top_idx[lane] = e; ly.top_w[lane] = wt; }
                }
            }
            // the shared expert's down rows, under the picks and the way of their rows: half of its hidden values to each of two warps
            rg.wait(1, lane);
            if (warp >= S1_WARPS - 2) {
                const int kh = warp - (S1_WARPS - 2), hk = a.SH >> 1;
                float av[8], mx = 0.f;
                ll_wait<8>(set + a.o_sa + kh * hk + lane * 8, tag, lane * 8 < hk, av, flag);
#pragma unroll
                for (int i = 0; i < 8; i++) { av[i] = lane * 8 < hk ? av[i] : 0.f; mx = fmaxf(mx, fabsf(av[i])); }
                mx = warp_absmax(mx);
                planes8(av, mx > 1e-30f ? M1_QMAX / mx : 0.f, false, scratch, lane);
                __syncwarp();
                const unsigned char* stg = rg.stage() + (gid >> 1) * a.SH + (gid & 1 ? a.half_shd : 0) + kh * hk + tid * 16;
                int c[4] = {F32_MAGIC, F32_MAGIC, F32_MAGIC, F32_MAGIC};
#pragma unroll 1
                for (int k = 0; k < hk; k += 64) {
                    const uint4 wl = *reinterpret_cast<const uint4*>(stg + k), wh = *reinterpret_cast<const uint4*>(stg + 4 * a.SH + k);
                    uint4 xb[1];
                    load_planes<64>(scratch, k, gid, tid, xb);
                    imma16832(c, wl.x, wh.x, wl.y, wh.y, xb[0].x, xb[0].y);
                    imma16832(c, wl.z, wh.z, wl.w, wh.w, xb[0].z, xb[0].w);
                }
                float pw0, pw1;
                weights_of(mx / M1_QMAX, pw0, pw1);
                float ylo = fmaf(magic_sum(c[0]), pw0, __fmul_rn(magic_sum(c[1]), pw1)), yhi = fmaf(magic_sum(c[2]), pw0, __fmul_rn(magic_sum(c[3]), pw1));
                ylo += __shfl_xor_sync(0xffffffffu, ylo, 1);
                yhi += __shfl_xor_sync(0xffffffffu, yhi, 1);
                // x the rows' scales
                const uint16_t* sc = reinterpret_cast<const uint16_t*>(rg.stage() + a.stage_bytes - S1_OPS) + (s_blk.r0 & 7);
                const int nr = s_blk.r1 - s_blk.r0, rlo = s1_slot_row(gid, nr), rhi = s1_slot_row(gid + 8, nr);
                sts_if(tid == 0, s_sh + kh * 16 + gid, rlo >= 0 ? ylo * bf(sc[rlo]) : 0.f);
                sts_if(tid == 0, s_sh + kh * 16 + gid + 8, rhi >= 0 ? yhi * bf(sc[rhi]) : 0.f);
            } else if (warp == S1_WARPS - 3) {
                float t[1];
                ll_wait<1>(set + a.o_sg, tag, true, t, flag);
                if (lane == 0) s_sg = t[0];
            }
            rg.release(1, lane);
            s1_bar();                                           // picks, and the planes of every chunk
            const int rb = warp & 3, kq = warp >> 2;            // rows: slots 8 rb + gid; K quarter
            const int h = (np + 1) / 2, sl = rb * 8 + gid, q = sl >> 1;
            const bool gu_on = rb * 8 < 2 * h;
            // even slots are pairs of the first half, odd ones of the second
            const int qi = (sl & 1) ? max(0, min(q, np - h - 1)) : min(q, h - 1), pi = gp0 + ((sl & 1) && np > h ? h + qi : qi);
            // tiles: gate rows, up rows, scales. The lanes of a quad take one of four scale rows each: gate scales, gate minima, up scales, up minima
            const unsigned char *pg = rg.stage(0), *pu = rg.stage(1);
            rg.wait(3, lane);
            {
                // of the down rows, scales and minima of slots gid (low) and gid + 8
                const int nr = s_blk.r1 - s_blk.r0, hr = (nr + 1) / 2, pk = warp >> 1, kh = warp & 1;
                const bool odd = (gid & 1) && nr > hr;
                const int lo = min(gid >> 1, (odd ? nr - hr : hr) - 1) + (odd ? hr : 0), hi = min((gid >> 1) + 4, (odd ? nr - hr : hr) - 1) + (odd ? hr : 0);
                if (pk < a.topk) {
                    const unsigned char* q = rg.stage(2) + 4 * s1_gsc_stride(D) + 2 * pk * s1_dsc_stride(a.I) + ((s_blk.r0 * (a.I / 32)) & 15) + kh * GH * 2;
                    load_f16s<GH>(reinterpret_cast<const uint16_t*>(q + lo * (a.I / 32)), dsl);
                    load_f16s<GH>(reinterpret_cast<const uint16_t*>(q + hi * (a.I / 32)), dsh);
                    load_f16s<GH>(reinterpret_cast<const uint16_t*>(q + s1_dsc_stride(a.I) + lo * (a.I / 32)), dml);
                    load_f16s<GH>(reinterpret_cast<const uint16_t*>(q + s1_dsc_stride(a.I) + hi * (a.I / 32)), dmh);
                }
            }
            float* gpart = part_all + pb * S1_WARPS * S1_ROWS;   // [8 eighths][32 slots][2]
            if (gu_on) {
                const int off = ((sl & 1) && np > h ? s1_half(h, D / 2) : 0) + qi * (D / 2) + kq * (D / 8) + tid * 8;
                pg += off; pu += off;
                float w0, w1;
                plane_weights(tid, s_scale, w0, w1);
                const unsigned char* ps = rg.stage(2) + (pi - gp0) * (D / 32) + kq * (D / 128);
#pragma unroll 1
                for (int e = 0; e < 2; e++) {                   // an eighth of the row, as k_moe_gu1 adds
                    uint32_t sg[(GE + 1) / 2], mg[(GE + 1) / 2], su[(GE + 1) / 2], mu[(GE + 1) / 2];
                    const uint16_t* se = reinterpret_cast<const uint16_t*>(ps) + e * GE;
                    load_f16s<GE>(se, sg); load_f16s<GE>(se + s1_gsc_stride(D) / 2, mg);
                    load_f16s<GE>(se + s1_gsc_stride(D), su); load_f16s<GE>(se + 3 * (s1_gsc_stride(D) / 2), mu);
                    float accg[2] = {0.f, 0.f}, accu[2] = {0.f, 0.f}, mng = 0.f, mnu = 0.f;
                    const int gf = (2 * kq + e) * GE;
#pragma unroll
                    for (int g = 0; g < GE; g++) {
                        const uint2 wg = *reinterpret_cast<const uint2*>(pg + (e * GE + g) * 32), wu = *reinterpret_cast<const uint2*>(pu + (e * GE + g) * 32);
                        uint4 xb[1];
                        load_planes<64>(reinterpret_cast<const unsigned char*>(xf_all) + ((gf + g) >> 2) * 1024, ((gf + g) & 3) * 64, gid, tid, xb);
                        const float xs = s_xg[gf + g];
                        int t[4];
                        imma16832_c(t, wg.x & 0x0F0F0F0Fu, wu.x & 0x0F0F0F0Fu, (wg.x >> 4) & 0x0F0F0F0Fu, (wu.x >> 4) & 0x0F0F0F0Fu, xb[0].x, xb[0].y, F32_MAGIC);
                        imma16832(t, wg.y & 0x0F0F0F0Fu, wu.y & 0x0F0F0F0Fu, (wg.y >> 4) & 0x0F0F0F0Fu, (wu.y >> 4) & 0x0F0F0F0Fu, xb[0].z, xb[0].w);
                        const float sgv = f16_of(sg[g / 2], g & 1), suv = f16_of(su[g / 2], g & 1);
                        accg[0] = fmaf(sgv, magic_sum(t[0]), accg[0]); accg[1] = fmaf(sgv, magic_sum(t[1]), accg[1]);
                        accu[0] = fmaf(suv, magic_sum(t[2]), accu[0]); accu[1] = fmaf(suv, magic_sum(t[3]), accu[1]);
                        mng = fmaf(f16_of(mg[g / 2], g & 1), xs, mng);
                        mnu = fmaf(f16_of(mu[g / 2], g & 1), xs, mnu);
                    }
                    float vg = fmaf(accg[0], w0, __fmul_rn(accg[1], w1)), vu = fmaf(accu[0], w0, __fmul_rn(accu[1], w1));
                    vg += __shfl_xor_sync(0xffffffffu, vg, 1); vu += __shfl_xor_sync(0xffffffffu, vu, 1);
                    sts_if(tid == 0, gpart + ((2 * kq + e) * 32 + sl) * 2, vg + mng);
                    sts_if(tid == 0, gpart + ((2 * kq + e) * 32 + sl) * 2 + 1, vu + mnu);
                }
            }
            rg.release(3, lane);
            tr.pt(3);
            s1_bar();
            if (threadIdx.x < 32) {
                const int j = (lane & 1) ? h + (lane >> 1) : lane >> 1;
                if (j < ((lane & 1) ? np : h)) {
                    float g = 0.f, u = 0.f;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const float2 t = *reinterpret_cast<const float2*>(gpart + (k * 32 + lane) * 2);
                        g += t.x; u += t.y;
                    }
                    ll_store(set + a.o_act + gp0 + j, siluf_(g) * u, tag);
                }
            }
            pb ^= 1;
            s1_bar();
            tr.out();
        }

        // ================= experts: down, into the residual stream =================
        {
            fresh();
            const int r0 = s_blk.r0, nr = s_blk.r1 - r0, h = (nr + 1) / 2;
            tr.in(6, nr);
            const int pk = warp >> 1, kh = warp & 1;            // this warp's pick and half of the hidden width
            const bool on = pk < a.topk;
            float* fpart = part_all + pb * S1_WARPS * S1_ROWS;   // [16][16 slots]
            const int shalf = lane & 1, sj = lane >> 1, my_row = shalf ? h + sj : sj;      // epilogue: slot -> row, as for the pairs above
            const bool mine = warp == 0 && lane < 16 && my_row < (shalf ? nr : h);
            float vlo = 0.f, vhi = 0.f;
            if (on) {
                // slots gid and gid + 8: even ones are rows of the first half, odd ones of the second
                const bool odd = (gid & 1) && nr > h, has = lane * 8 < 64 * GH;
                const int qlo = odd ? min(gid >> 1, nr - h - 1) : min(gid >> 1, h - 1), qhi = odd ? min((gid >> 1) + 4, nr - h - 1) : min((gid >> 1) + 4, h - 1);
                float av[8], mx = 0.f;
                ll_wait<8>(set + a.o_act + pk * a.I + kh * 64 * GH + lane * 8, tag, has, av, flag);
                tr.pt(1);
                // planes with a scale for every 32 values, and their sums, as k_moe_gu1 makes them
#pragma unroll
                for (int i = 0; i < 8; i++) { av[i] = has ? av[i] : 0.f; mx = fmaxf(mx, fabsf(av[i])); }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                planes8(av, mx > 1e-30f ? M1_QMAX / mx : 0.f, true, scratch, lane);
                float* as = reinterpret_cast<float*>(scratch + 1024);
                const float sm = sum32(av);
                if ((lane & 3) == 0) { as[lane >> 2] = mx / M1_QMAX; as[8 + (lane >> 2)] = sm; }
                __syncwarp();
                rg.wait(1, lane);
                const unsigned char* pw = rg.stage() + pk * s1_dn_stride(nr, a.I / 2) + (odd ? s1_half(h, a.I / 2) : 0) + kh * 32 * GH + tid * 8;
                float pw0, pw1, mlo = 0.f, mhi = 0.f;
                plane_weights(tid & 1, 1.0f, pw0, pw1);
                // columns 0-3: the planes of a group's first 32 values, held by lanes tid 0 and 1; columns 4-7: of the other 32, tid 2 and 3. A product then
                // sums both apart; the second ones come over to lanes 0 and 1
                const bool act = (gid >> 2) == (tid >> 1);
#pragma unroll
                for (int g = 0; g < GH; g++) {
                    const uint2 wl = *reinterpret_cast<const uint2*>(pw + qlo * (a.I / 2) + 32 * g), wh = *reinterpret_cast<const uint2*>(pw + qhi * (a.I / 2) + 32 * g);
                    uint4 xb[1];
                    load_planes<64>(scratch, 64 * g, gid, tid, xb);
                    if (!act) xb[0] = make_uint4(0u, 0u, 0u, 0u);
                    int t[4];
                    imma16832_c(t, wl.x & 0x0F0F0F0Fu, wh.x & 0x0F0F0F0Fu, (wl.x >> 4) & 0x0F0F0F0Fu, (wh.x >> 4) & 0x0F0F0F0Fu, xb[0].x, xb[0].y, F32_MAGIC);
                    imma16832(t, wl.y & 0x0F0F0F0Fu, wh.y & 0x0F0F0F0Fu, (wl.y >> 4) & 0x0F0F0F0Fu, (wh.y >> 4) & 0x0F0F0F0Fu, xb[0].z, xb[0].w);
                    const float ulo = fmaf(magic_sum(t[0]), pw0, __fmul_rn(magic_sum(t[1]), pw1)), uhi = fmaf(magic_sum(t[2]), pw0, __fmul_rn(magic_sum(t[3]), pw1));
                    const float ulo1 = __shfl_xor_sync(0xffffffffu, ulo, 2), uhi1 = __shfl_xor_sync(0xffffffffu, uhi, 2);
                    const float c0 = as[2 * g], c1 = as[2 * g + 1], xs = as[8 + 2 * g] + as[8 + 2 * g + 1];
                    vlo = fmaf(f16_of(dsl[g / 2], g & 1), fmaf(c0, ulo, __fmul_rn(c1, ulo1)), vlo);
                    vhi = fmaf(f16_of(dsh[g / 2], g & 1), fmaf(c0, uhi, __fmul_rn(c1, uhi1)), vhi);
                    mlo = fmaf(f16_of(dml[g / 2], g & 1), xs, mlo);
                    mhi = fmaf(f16_of(dmh[g / 2], g & 1), xs, mhi);
                }
                vlo += __shfl_xor_sync(0xffffffffu, vlo, 1); vhi += __shfl_xor_sync(0xffffffffu, vhi, 1);
                vlo += mlo; vhi += mhi;
            } else rg.wait(1, lane);
            rg.release(1, lane);
            sts_if(tid == 0, fpart + warp * 16 + gid, vlo);
            sts_if(tid == 0, fpart + warp * 16 + gid + 8, vhi);
            tr.pt(3);
            cp_async_wait<0>();                                 // the next layer's pointers
            s1_bar();
            if (mine) {
                // x += sum_r w_r y_r + sigmoid(shared gate) y_shared, picks in rank order
                float y = 0.f;
#pragma unroll
                for (int r = 0; r < 8; r++)
                    if (r < a.topk) y = fmaf(s_topw[r], fpart[2 * r * 16 + lane] + fpart[(2 * r + 1) * 16 + lane], y);
                y = fmaf(s_sg, s_sh[lane] + s_sh[16 + lane], y);
                const float v = s_x[my_row] + y;
                s_x[my_row] = v;
                ll_store(set + a.o_xa + r0 + my_row, v, tag);
                if (l + 1 == a.L) a.x[r0 + my_row] = v;
                if (ly.tap) ly.tap[r0 + my_row] = v;
            }
            pb ^= 1;
            s1_bar();
            tr.out();
        }
    }


    // arg-max: of the block, then of all blocks by the one that comes last
    s1_bar();
    if (warp == 0) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
#pragma unroll
        for (int w = 0; w < S1_LOT * 16; w += 32) {
            const float pv = s_bv[w + lane];
            const int pi = s_bi[w + lane];
            if (pv > v || (pv == v && pi < ix)) { v = pv; ix = pi; }
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        if (lane == 0) {
            a.part_val[blk] = v;
            a.part_idx[blk] = ix;
            if (s_given_up[0]) atomicExch(a.err, 4);
            __threadfence();
            s_last = atomicAdd(a.counter, 1u) == (unsigned)G - 1;
            __threadfence();
        }
    }
    s1_bar();
    if (s_last && warp == 0) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
        for (int g = lane; g < G; g += 32) {
            const float pv = __ldcg(a.part_val + g);
            const int pi = __ldcg(a.part_idx + g);
            if (pv > v || (pv == v && pi < ix)) { v = pv; ix = pi; }
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        if (lane == 0) {
            a.next_tok[0] = ix;
            step_done(0, ix, a.pos, a.hist, a.tok);
            *a.counter = 0;
            *a.epoch = epoch + (uint32_t)a.L;
        }
    }
    tr.out();
}

}  // namespace b2
