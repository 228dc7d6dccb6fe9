// k_umma_q4: the 4-bit experts of a step (6 or more tokens) or prompt chunk as a grouped Blackwell tensor-core GEMM
// (the reference's expert GEMMs for more than 8 tokens, aegist_rs/kernels/hybrid.cu:461-549).
//
// k_group_picks has sorted the step's picks by expert, every expert's list starting at a multiple of eight, and cut the lists into
// chunks of at most 32 picks. A unit of work is (chunk, two blocks of 128 weight rows): out[pick][row] = sum_k w[row][k] x[pick][k]
// for the chunk's picks, with w = code * scale_g + min_g per 64-value group g (aegist/hybrid.py ExpertBank), so
//     sum_k w x = sum_g ( scale_g * sum_{k in g} code x  +  min_g * sum_{k in g} x ).
// The sums of a group must not mix with another group's, so every group gets its own accumulator columns in tensor memory and the
// epilogue folds them with the group's fp16 scale. The two row blocks are a unit's gate and up rows (or two neighbouring blocks of
// down rows), and the K loop is outside them.
//
// Arithmetic. An activation is s q / 2^14 with q a whole number below 2^21 in magnitude (22 bits of the pick's largest value), and q is
// two whole numbers of 11 bits, q = 2048 h + l, which fp16 holds exactly. A code (0..15) is an fp16 as it lies in its nibble: the bits
// 0x000c are the subnormal c 2^-24 and 0x00c0 is c 2^-20, so two masks and a shift turn a nibble pair into operands; the planes of
// the values that meet the second kind carry 2^-4. Products and the sums of 64 of them are below 2^20 units: exact in the tensor
// core's fp32 accumulators, whatever its order. One fma joins the planes (rounding once, as a conversion of the whole number would).
// With int8 planes (three digits, half as many products) the epilogue bound the kernel: three columns per pick instead of two, and two
// integer products and a conversion instead of half an fma: 2700 clocks per row block and K step of up to 20 picks.
//
//   producer warp     per K step (256 codes = 4 groups): one bulk copy with the planes of the chunk's picks (8 KB per eight picks,
//                     consecutive in memory and laid out as the operand wants them; a ring slot holds one, two or four K steps), then
//                     per row block the packed codes of 128 rows (128 bytes each, through a 3-D tensor map [expert][row][byte],
//                     128-byte swizzle). Rings: 2 x 2 x 16 KB of codes, 3 x 32 KB of planes (3 and 2 slots: 77 instead of 70 us for
//                     the gate/up rows of 204 experts, one to eight picks each)
//   table warp        the picks' scales, group sums and output rows of the next unit, and per two K steps the scales and minima of
//                     the 256 rows (16 bytes each, cp.async) into a third ring
//   8 converter warps four to a row block; thread = weight row = TMEM lane: the codes of half a K step -> fp16 straight into tensor memory
//                     (tcgen05.st, one of the row block's two buffers of 64 columns), where tcgen05.mma takes its A operand from
//   2 MMA warps       one to a row block, so that one's waits lie under the other's products: per half step two groups of four tcgen05.mma
//                     (kind::f16, M 128, N 16, 32 or 64, K 16) into columns of their own, and commits, which tell the converters that
//                     the code buffer is free and the epilogue that a buffer of sums is full
//   8 epilogue warps  four to a row block; thread = weight row = TMEM lane: a buffer is 64 columns, the four groups of up to 8 picks, two of
//                     up to 16 or one of up to 32: one tcgen05.ld, then four folds of a group of eight picks: planes joined, times the
//                     row's group scale, plus the group minimum times the picks' group sums. A pick's sum takes its groups in order, in
//                     chunks of every size (k_delta_prompt's note says why that matters). Then activation scale and
//                     silu(gate) * up, or the picks' output rows
//
// What bounds it, per row block and K step (16 KB of codes, 2 KB of scales: 780 clocks of HBM at the SM's share): sixteen products,
// whose issue takes 44 to 50 clocks each for any N up to 80, whichever warp issues them, and two and a half to five commits, which take one
// product's time: 810 to 1050 clocks; measured 1170 (45 tokens: up to 8 picks, 3.6 TB/s of codes), 1450 (333: 10 picks on average) and 1660
// (1024: 22), gate/up rows, in the block with the most units. The rest is hand-over: a wait for a phase that is already over takes 100 clocks
// and more when the SM is busy, a wake-up 130, and there are eleven to fourteen to a row block and K step. So a chunk of 32 picks costs
// little more than one pick does. us per layer (gate/up + down, 256 experts, 8 picks a token) with int8 planes and now: 1024 tokens 468 and
// 235, 333 tokens 213 and 131, 45 tokens 120 and 87 (prompts); 7 sequences 43 and 34, 64 of Zipf popularity 62 and 45 (in the step's graph).
//
// Every wait is a bounded mbarrier wait of a whole warp; a warp whose wait gave up skips its later waits, the producer stops issuing
// copies and drains those in flight, and the kernel ends normally with the error word set. setmaxnreg, the one wait that knows no bound, is
// launched only where it cannot wait for good (uq_regs_suffice).
#pragma once

namespace b2 {

constexpr int UQ_G = 8;                          // picks whose planes lie together: 16 accumulator columns per group
constexpr int UQ_FEW = 8;                         // a chunk of at most this many picks has 16 accumulator columns per group, a buffer of 64 for a whole K step;
constexpr int UQ_SMALL = 16;                     // picks of a small chunk: 32 columns per group, a buffer for half a K step
constexpr int UQ_TT = 32;                        // most picks per unit (a chunk of the pick list): 64 columns per group, a buffer for each. Two buffers to a row block
constexpr int UQ_KB = 256;                       // codes per K step: four groups
constexpr int UQ_RAW = UM_M * UQ_KB / 2;         // 16 KB: packed codes of a row block and K step
constexpr int UQ_PL = 2;                         // fp16 planes
constexpr int UQ_GBYTES = UQ_G * UQ_PL * UQ_KB * 2;      // 8 KB: the planes of eight picks and a K step, [plane][group][pick][64 values]
constexpr int UQ_SBO = UQ_KB / 64 * 1024;        // bytes between the eight rows of plane h, those of plane l, those of the next eight picks
constexpr int UQ_PSLOT = UQ_TT / UQ_G * UQ_GBYTES;       // 32 KB: a K step of a large chunk, two or four of smaller ones
__device__ __forceinline__ int uq_ksteps(int picks) { return picks <= UQ_G ? 4 : (picks <= 2 * UQ_G ? 2 : 1); }
constexpr int UQ_NW = 2, UQ_NP = 3, UQ_NS = 3;   // ring slots: codes of each row block, planes, row scales
constexpr int UQ_SSLOT = 4 * UM_M * 16;          // 8 KB: [row block][scale | min][128 rows][8 groups] fp16 of two K steps
constexpr int UQ_MAXG = 32;                      // groups of a row (K <= 2048)
constexpr int UQ_XS = UQ_TT * UQ_MAXG * 4;       // 4 KB: a unit's group sums, [eight picks][group][pick]
constexpr int UQ_RED = UQ_TT * UM_M * 4;         // 16 KB: the gate or up values that a warp hands to the one that finishes the pick, [pick][row]
constexpr int UQ_NA = 4;                         // code buffers in tensor memory, 64 columns each (128 codes)
constexpr int UQ_ACOL = 256;                     // where they start; the accumulators lie before them. A group's columns start at a multiple of N: a
                                                 // tcgen05.mma whose accumulator does not start on the next power of two above N takes about three times as long
constexpr int UQ_UNITS = 32;                     // units of a block whose places in the lists are looked up once
constexpr int UQ_EPI = 8, UQ_CONV = 8;           // epilogue warps, converter warps
constexpr int UQ_THREADS = (4 + UQ_CONV + UQ_EPI) * 32;  // producer, 2 MMA issuers, tables, converters, epilogue
// Registers: producer, issuers, tables and converters (three warpgroups) keep 64 a thread of the 96 that the block is launched with, and the
// epilogue's two get 144: a buffer of 64 columns, the sums of 32 picks and what a fold needs. 3 x 64 + 2 x 144 = 5 x 96
constexpr int UQ_REGS_LOW = 64, UQ_REGS_EPI = 144;
// Whether a launch with `regs` registers a thread, which the compiler decides, has that much to hand over. With fewer the epilogue's
// setmaxnreg would wait for registers that nobody gives back, the one wait without a bound: such a build must not launch the kernel.
constexpr bool uq_regs_suffice(int regs) {
    return regs >= UQ_REGS_LOW && regs <= UQ_REGS_EPI && regs * (4 + UQ_CONV + UQ_EPI) >= UQ_REGS_LOW * (4 + UQ_CONV) + UQ_REGS_EPI * UQ_EPI;
}
constexpr size_t UQ_SMEM = (size_t)2 * UQ_NW * UQ_RAW + (size_t)UQ_NP * UQ_PSLOT + (size_t)UQ_NS * UQ_SSLOT + 2 * UQ_XS + UQ_RED + 1024;

struct UmmaQ4Args {
    CUtensorMap wmap;         // this matrix's packed codes of the layer's experts: [expert][row][K / 2 bytes], box 128 B x 128 rows
    unsigned long long* trace;
    const uint8_t* planes;    // [K step][slots / 8][UQ_GBYTES], the 16-byte pieces of a row where the 128-byte swizzle wants them
    const uint8_t* const* eptr;   // [E] expert blobs (for the scale and min rows)
    const int* list;          // pick ids sorted by expert (k_group_picks)
    ChunkTable small, big;    // chunks of at most UQ_SMALL picks, and of more
    int topk, pair, rows, K;  // pair: rows = pairs (expert_hidden), gate row i and up row up_row0 + i; else rows = output rows
    int up_row0;
    int e0;                   // first expert that lives on this GPU (its blob is index 0 of the tensor map)
    size_t off_s, off_m;      // the matrix's scale and min sections inside an expert blob
    int wide;                 // 16 bytes of a scale row (two K steps) may be copied at once
    int slots;                // capacity of the planes
    const float* xscale;      // [slots] scale of each slot's planes
    const float* xsum;        // [slots / 8][K / 64][8] sum of each 64-value group of the slots' activations, in units of their scale
    float* out;               // pair: act [picks][rows]; else ypart [tokens][topk + 1][rows]
    int* err;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t atmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(atmem),
                 "l"(bdesc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
// 16 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(addr)
                 : "memory");
}
// 16 bytes of packed codes -> 16 cells. Eight codes of a word: 0 and 4, 1 and 5, 2 and 6, 3 and 7 to a cell; the planes hold their values in the same order
__device__ __forceinline__ void uq_cells(const uint4& pk, uint32_t (&o)[16]) {
    const uint32_t pw[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        o[4 * i] = pw[i] & 0x000F000Fu; o[4 * i + 1] = pw[i] & 0x00F000F0u;
        o[4 * i + 2] = (pw[i] >> 8) & 0x000F000Fu; o[4 * i + 3] = (pw[i] >> 8) & 0x00F000F0u;
    }
}
// one arrival when this thread's cp.async copies so far have landed
__device__ __forceinline__ void mbar_arrive_copies(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
// 64 consecutive columns of this thread's TMEM lane, landed
__device__ __forceinline__ void tmem_ld64(uint32_t addr, uint32_t (&r)[64]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x64.b32 {"
                 "%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
                 "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
                 "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
                   "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]),
                   "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]),
                   "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
                   "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
                 : "r"(addr)
                 : "memory");
}
// One group of eight picks into their fp32 sums: columns AT .. AT + 7 hold plane h of the picks, the next eight plane l, both in units of 2^-24; 2^-14 and
// 2^24 are in the scale.
template <int AT>
__device__ __forceinline__ void uq_fold(const uint32_t (&c)[64], float sc, float mn, const float* xs, uint64_t (&acc)[4]) {
    const uint64_t sc2 = f2_pack(sc, sc), mn2 = f2_pack(mn, mn), up = f2_pack(2048.0f, 2048.0f);
    const ulonglong2 x0 = reinterpret_cast<const ulonglong2*>(xs)[0], x1 = reinterpret_cast<const ulonglong2*>(xs)[1];
    const uint64_t x[4] = {x0.x, x0.y, x1.x, x1.y};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint64_t h = f2_pack(__uint_as_float(c[AT + 2 * i]), __uint_as_float(c[AT + 2 * i + 1])),
                       l = f2_pack(__uint_as_float(c[AT + 8 + 2 * i]), __uint_as_float(c[AT + 9 + 2 * i]));
        acc[i] = f2_fma(sc2, f2_fma(h, up, l), f2_fma(mn2, x[i], acc[i]));
    }
}

// The products of a group of 64 codes, N columns. Everything but the bases is a constant: with the groups, their column stride and N as
// run-time values the issuing thread spent 160 to 200 clocks on each instruction.
template <int N>
__device__ __forceinline__ void uq_issue(uint32_t d, uint32_t at, uint64_t bd) {
    constexpr uint32_t idesc = umma_idesc(1, 0, UM_M, N);
#pragma unroll
    for (int k = 0; k < 4; k++) umma_f16_ts(d, at + 8 * k, bd + (uint64_t)(2 * k), idesc, (uint32_t)(k != 0));
}

__global__ void __launch_bounds__(UQ_THREADS, 1) k_umma_q4(const __grid_constant__ UmmaQ4Args a) {
    extern __shared__ unsigned char uq_raw[];
    // Code buffer and accumulator buffer 2 rb + h belong to row block rb. done[b]: the products that read code buffer b are over
    // (first[b]: those of its first group); few[b]: accumulator buffer b holds a K step of few picks. A barrier never runs two phases ahead of
    // a waiting warp: the products of its next phase need a code or accumulator buffer that the warp gives back only after this one (a K step
    // of few picks, which needs one for both halves, sees to it itself)
    enum { W_FULL = 0, W_EMPTY = W_FULL + 2 * UQ_NW, P_FULL = W_EMPTY + 2 * UQ_NW, P_EMPTY = P_FULL + UQ_NP, S_FULL = P_EMPTY + UQ_NP, S_EMPTY = S_FULL + UQ_NS, T_FULL = S_EMPTY + UQ_NS,
           T_EMPTY = T_FULL + 2, CONV = T_EMPTY + 2, FIRST = CONV + UQ_NA, DONE = FIRST + UQ_NA, FEW = DONE + UQ_NA, ACC_EMPTY = FEW + UQ_NA, DRAINED = ACC_EMPTY + UQ_NA, NBAR };
    __shared__ __align__(8) uint64_t s_bar[NBAR];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float s_xscale[2][UQ_TT];
    __shared__ __align__(16) int s_dst[2][UQ_TT];                  // where the output row of each pick of the chunk starts
    __shared__ int4 s_unit[UQ_UNITS];                // the block's first units: expert, start, picks, first row
    const int warp = threadIdx.x >> 5, lane = (int)held(threadIdx.x & 31);
    unsigned char* wring = uq_raw + ((1024u - (smem_u32(uq_raw) & 1023u)) & 1023u);
    unsigned char* pring = wring + (size_t)2 * UQ_NW * UQ_RAW;
    unsigned char* sring = pring + (size_t)UQ_NP * UQ_PSLOT;
    unsigned char* xsums = sring + (size_t)UQ_NS * UQ_SSLOT;
    float* red = reinterpret_cast<float*>(xsums + 2 * UQ_XS);
    grid_dep_launch();
    trace_in(a.trace, 16, gridDim.x);
    if (threadIdx.x == 0) {
        auto init = [&](int first, int n, int count) { for (int i = 0; i < n; i++) mbar_init(&s_bar[first + i], count); };
        init(W_FULL, 2 * UQ_NW, 1); init(W_EMPTY, 2 * UQ_NW, 4);
        init(P_FULL, UQ_NP, 1); init(P_EMPTY, UQ_NP, 2);
        init(S_FULL, UQ_NS, 32); init(S_EMPTY, UQ_NS, UQ_EPI);
        init(T_FULL, 2, 32); init(T_EMPTY, 2, UQ_EPI);
        init(CONV, UQ_NA, 4); init(FIRST, UQ_NA, 1); init(DONE, UQ_NA, 1); init(FEW, UQ_NA, 1); init(ACC_EMPTY, UQ_NA, 4);
        init(DRAINED, 1, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = held(tmem_slot);
    const uint32_t bars = held(smem_u32(s_bar)), ring0 = held(smem_u32(wring));       // shared-memory addresses of the barriers and the rings
    auto bar = [&](int kind, int i) { return bars + 8u * (uint32_t)(kind + i); };
    grid_dep_wait();                                 // the chunk tables, the planes and the activations are earlier launches' results

    const int nbig = *a.big.count, nsmall = *a.small.count;
    const int RG = a.pair ? a.rows / UM_M : a.rows / (2 * UM_M);      // units per chunk
    const int nwork = (nbig + nsmall) * RG;          // big chunks first
    const int nk = a.K / UQ_KB;                      // K steps per unit
    const int ngroup = a.K >> 6;
    auto find = [&](int w) {
        const int c = w / RG;
        const ChunkTable& t = c < nbig ? a.big : a.small;
        const int i = c < nbig ? c : c - nbig;
        return make_int4(t.expert[i], t.start[i], t.n[i], (w - c * RG) * (a.pair ? UM_M : 2 * UM_M));
    };
    for (int i = threadIdx.x; i < UQ_UNITS && (int)(blockIdx.x + i * gridDim.x) < nwork; i += UQ_THREADS) s_unit[i] = find(blockIdx.x + i * gridDim.x);
    __syncthreads();
    // r0: the first weight row of the unit's first block. Every role asks once a unit; a table read costs a trip to L2 each time
    auto chunk_of = [&](int w, int u, int& e, int& start, int& n, int& r0) {
        const int4 v = u < UQ_UNITS ? s_unit[u] : find(w);
        e = v.x; start = v.y; n = v.z; r0 = v.w;
    };
    const int rstep = a.pair ? a.up_row0 : UM_M;     // from the first row block to the second
    auto wait = [&](uint32_t at, uint32_t parity, bool& dead) { warp_wait(at, parity, a.err, dead); };

    if (warp < 4) regs_dec<UQ_REGS_LOW>();
    if (warp == 0) {
        // ---- producer ----
        int ws = 0, wph = 0, ps = 0, pph = 0;
        bool dead = false;
        uint32_t w_armed = 0, w_par = 0, p_armed = 0, p_par = 0;
        for (int w = blockIdx.x, u = 0; w < nwork && !dead; w += gridDim.x, u++) {
            int e, start, n, r0;
            chunk_of(w, u, e, start, n, r0);
            const uint32_t bytes = (uint32_t)((n + UQ_G - 1) / UQ_G) * UQ_GBYTES;
            const int ks = uq_ksteps(n);
            for (int kc = 0; kc < nk && !dead; kc++) {
                if (kc % ks == 0) {
                    wait(bar(P_EMPTY, ps), pph ^ 1, dead);
                    if (dead) break;
                    const int steps = min(ks, nk - kc);
                    if (lane == 0) mbar_expect_tx(bar(P_FULL, ps), bytes * steps);
                    __syncwarp();
                    if (lane < steps)
                        bulk_load(ring0 + (uint32_t)(2 * UQ_NW * UQ_RAW + ps * UQ_PSLOT) + lane * bytes, a.planes + ((size_t)(kc + lane) * a.slots + start) * (UQ_GBYTES / UQ_G), bytes, bar(P_FULL, ps));
                    p_armed |= 1u << ps;
                    p_par = (p_par & ~(1u << ps)) | ((uint32_t)pph << ps);
                    if (++ps == UQ_NP) { ps = 0; pph ^= 1; }
                }
                for (int rb = 0; rb < 2; rb++) {
                    const int slot = rb * UQ_NW + ws;
                    wait(bar(W_EMPTY, slot), wph ^ 1, dead);
                    if (dead) break;
                    if (lane == 0) {
                        mbar_expect_tx(bar(W_FULL, slot), UQ_RAW);
                        tma_load_3d(ring0 + (uint32_t)(slot * UQ_RAW), &a.wmap, kc * (UQ_KB / 2), r0 + rb * rstep, e - a.e0, bar(W_FULL, slot));
                    }
                    w_armed |= 1u << slot;
                    w_par = (w_par & ~(1u << slot)) | ((uint32_t)wph << slot);
                }
                if (++ws == UQ_NW) { ws = 0; wph ^= 1; }
            }
        }
        if (dead && lane == 0) {                     // copies still in flight must land before the block may leave
            for (int i = 0; i < 2 * UQ_NW; i++)
                if (w_armed >> i & 1) mbar_wait(bar(W_FULL, i), (w_par >> i) & 1u, nullptr, 1 << 16);
            for (int i = 0; i < UQ_NP; i++)
                if (p_armed >> i & 1) mbar_wait(bar(P_FULL, i), (p_par >> i) & 1u, nullptr, 1 << 16);
        }
        __syncwarp();
    } else if (warp < 3) {
        // ---- MMA issuers, one for each row block: a warp waits, its elected lane issues ----
        const int rb = warp - 1;
        int ps = 0, pph = 0;
        uint32_t kg = 0, turn = 0, dk = 0;           // K steps and uses of an accumulator buffer so far
        const uint32_t d0 = tmem + 128u * rb;
        bool dead = false, was_few = false;
        const bool lead = elect_one();
        for (int w = blockIdx.x, u = 0; w < nwork; w += gridDim.x, u++) {
            int e, start, cn, r0;
            chunk_of(w, u, e, start, cn, r0);
            const bool big = cn > UQ_SMALL, few = cn <= UQ_FEW;
            bool catch_up = few && !was_few;         // see below
            was_few = few;
            const int ks = uq_ksteps(cn);
            const uint32_t bytes = (uint32_t)((cn + UQ_G - 1) / UQ_G) * UQ_GBYTES;
            for (int kc = 0; kc < nk; kc++, kg++) {
                const int kp = kc % ks;
                if (kp == 0) wait(bar(P_FULL, ps), pph, dead);
                const uint64_t bd = (umma_desc_sw128(ring0 + (uint32_t)(2 * UQ_NW * UQ_RAW + ps * UQ_PSLOT) + kp * bytes) & ~(0x3FFFull << 32)) | ((uint64_t)(UQ_SBO >> 4) << 32);
#pragma unroll 1
                for (int h = 0; h < 2; h++) {
                    const int b = 2 * rb + h;
                    const uint32_t at = tmem + UQ_ACOL + 64u * b;
                    const uint64_t bh = bd + (uint64_t)(h * (2048 >> 4));
                    wait(bar(CONV, b), kg & 1, dead);
                    // the next accumulator buffer: for both groups of this half, for each, or (few picks) for the whole K step
                    auto buffer = [&]() {
                        const uint32_t i = turn & 1;
                        wait(bar(ACC_EMPTY, 2 * rb + (int)i), ((turn >> 1) & 1) ^ 1, dead);
                        tc_fence_after();
                        turn++;
                        return d0 + 64u * i;
                    };
                    if (big) {
                        uint32_t d = buffer();
                        if (lead) { uq_issue<64>(d, at, bh); umma_commit(bar(FIRST, b)); }
                        __syncwarp();
                        d = buffer();
                        if (lead) { uq_issue<64>(d, at + 32, bh + (1024 >> 4)); umma_commit(bar(DONE, b)); }
                    } else if (few) {
                        // With one buffer for both halves these products could end a second phase of done[b] while the epilogue still waits for
                        // the first, that of a larger chunk before this one: behind such a chunk its last buffer must have been read first
                        if (h == 0) dk = buffer();
                        else if (catch_up) { wait(bar(ACC_EMPTY, 2 * rb + (int)(turn & 1)), ((turn >> 1) & 1) ^ 1, dead); catch_up = false; }
                        tc_fence_after();
                        if (lead) {
                            uq_issue<16>(dk + 32u * h, at, bh);
                            uq_issue<16>(dk + 32u * h + 16, at + 32, bh + (1024 >> 4));
                            umma_commit(bar(DONE, b));
                            if (h) umma_commit(bar(FEW, 2 * rb + (int)((turn - 1) & 1)));
                        }
                    } else {
                        const uint32_t d = buffer();
                        if (lead) {
                            uq_issue<32>(d, at, bh);
                            uq_issue<32>(d + 32, at + 32, bh + (1024 >> 4));
                            umma_commit(bar(DONE, b));
                        }
                    }
                    __syncwarp();
                }
                if (kp + 1 == ks || kc + 1 == nk) {
                    if (lead) umma_commit(bar(P_EMPTY, ps));
                    __syncwarp();
                    if (++ps == UQ_NP) { ps = 0; pph ^= 1; }
                }
            }
        }
        if (lead) umma_commit(bar(DRAINED, 0));             // no product may be under way when the block gives its tensor memory back
        __syncwarp();
        mbar_wait(bar(DRAINED, 0), 0, a.err, 1 << 21);
    } else if (warp == 3) {
        // ---- tables ----
        int u = 0, st = 0, ph = 0;
        bool dead = false;
        const size_t step = (size_t)32 * ngroup * 2, rbs = (size_t)rstep * ngroup * 2;
        for (int w = blockIdx.x; w < nwork && !dead; w += gridDim.x, u++) {
            const int ub = u & 1;
            int e, start, cn, r0;
            chunk_of(w, u, e, start, cn, r0);
            wait(bar(T_EMPTY, ub), ((u >> 1) & 1) ^ 1, dead);
            if (dead) break;
            if (lane < cn) {
                const int p = a.list[start + lane];
                s_xscale[ub][lane] = a.xscale[start + lane];
                s_dst[ub][lane] = (a.pair ? p : (p / a.topk) * (a.topk + 1) + p % a.topk) * a.rows;
            }
            if (lane == 0) {
                const uint32_t bytes = (uint32_t)((cn + UQ_G - 1) / UQ_G * UQ_G * ngroup * 4);
                mbar_expect_tx(bar(T_FULL, ub), bytes);
                bulk_load(xsums + (size_t)ub * UQ_XS, a.xsum + (size_t)start * ngroup, bytes, bar(T_FULL, ub));
            } else {
                mbar_arrive(bar(T_FULL, ub));
            }
            const uint8_t* blob = a.eptr[e];
            const size_t row_off = (size_t)(r0 + lane) * ngroup * 2;
            for (int kc = 0; kc < nk; kc += 2) {
                wait(bar(S_EMPTY, st), ph ^ 1, dead);
                if (dead) break;
                const uint32_t dst = ring0 + (uint32_t)(2 * UQ_NW * UQ_RAW + UQ_NP * UQ_PSLOT + st * UQ_SSLOT + lane * 16);
#pragma unroll
                for (int i = 0; i < 16; i++) {       // rows lane, + 32, .. of (row block, scale | min)
                    const uint8_t* src = blob + (i & 4 ? a.off_m : a.off_s) + row_off + (i & 3) * step + (i & 8 ? rbs : 0) + 8 * kc;
                    const uint32_t d = dst + ((i >> 2) * UM_M + 32 * (i & 3)) * 16;
                    if (a.wide) {
                        cp_async_16(d, src);
                    } else {
                        cp_async_8(d, src);
                        if (kc + 1 < nk) cp_async_8(d + 8, src + 8);
                    }
                }
                mbar_arrive_copies(bar(S_FULL, st));
                if (++st == UQ_NS) { st = 0; ph ^= 1; }
            }
        }
        // copies still in flight must land before the block may leave
        cp_async_commit();
        cp_async_wait<0>();
        if (lane == 0)
            for (int i = u > 2 ? u - 2 : 0; i < u; i++) mbar_wait(bar(T_FULL, i & 1), (i >> 1) & 1, nullptr, 1 << 16);
        __syncwarp();
    } else if (warp < 4 + UQ_CONV) {
        // ---- converters, four warps to a row block: this thread's row of 128 packed bytes -> 2 x 64 cells of two fp16 codes in its TMEM lane ----
        regs_dec<UQ_REGS_LOW>();
        const int q = warp & 3, rb = (warp >> 2) - 1, r = q * 32 + lane;
        const uint32_t col0 = held(tmem + ((uint32_t)(q * 32) << 16) + UQ_ACOL + 128u * rb);
        // the copy's 128-byte swizzle puts 16-byte piece c of row r at c ^ (r & 7), so the same piece of eight neighbouring rows covers all banks
        const unsigned char* row0 = wring + (size_t)rb * UQ_NW * UQ_RAW + r * 128;
        int st = 0, ph = 0;                          // a ring for each row block: shared, one's converters would pass a barrier by that the other's wait for
        uint32_t kg = 0;
        bool dead = false;
        for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
#pragma unroll 1
            for (int kc = 0; kc < nk; kc++, kg++) {
                wait(bar(W_FULL, rb * UQ_NW + st), ph, dead);
                const unsigned char* row = row0 + (size_t)st * UQ_RAW;
#pragma unroll 1
                for (int h = 0; h < 2; h++) {
                    uint4 pk[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) pk[c] = *reinterpret_cast<const uint4*>(row + (((4 * h + c) ^ (r & 7)) << 4));
                    wait(bar(DONE, 2 * rb + h), (kg & 1) ^ 1, dead);                 // the products that read this code buffer are over
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint32_t o[16];
                        uq_cells(pk[c], o);
                        tmem_st16(col0 + 64u * h + 16u * c, o);
                    }
                    // the stores have taken the codes out of the registers, so their loads have left the ring slot
                    if (h) mbar_arrive_if(lane == 0, bar(W_EMPTY, rb * UQ_NW + st));
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    mbar_arrive_if(lane == 0, bar(CONV, 2 * rb + h));
                }
                if (++st == UQ_NW) { st = 0; ph ^= 1; }
            }
        }
    } else {
        // ---- epilogue: warp w may touch TMEM lanes 32 (w % 4) .. + 31; four warps to a row block ----
        regs_inc<UQ_REGS_EPI>();
        const int q = warp & 3, rb = (warp - 4 - UQ_CONV) >> 2;
        const int vrow = q * 32 + lane;
        const uint32_t col0 = held(tmem + ((uint32_t)(q * 32) << 16) + 128u * rb);
        int st = 0, ph = 0;
        uint32_t kg = 0, turn = 0, few_par = 0, first_par = 0;       // few_par: bit i, the parity of few[2 rb + i]'s next phase; first_par: of first's
        bool dead = false;
        uint32_t c[64];
        // the next accumulator buffer into registers, once the products that `full` stands for are over; then they may overwrite it
        auto load = [&](uint32_t full, uint32_t parity) {
            wait(full, parity, dead);
            tc_fence_after();
            tmem_ld64(col0 + 64u * (turn & 1), c);
            tc_fence_before();
            __syncwarp();
            mbar_arrive_if(lane == 0, bar(ACC_EMPTY, 2 * rb + (int)(turn & 1)));
            turn++;
        };
        for (int w = blockIdx.x, u = 0; w < nwork; w += gridDim.x, u++) {
            int e, start, cn, r0;
            chunk_of(w, u, e, start, cn, r0);
            const int ub = u & 1;
            wait(bar(T_FULL, ub), (u >> 1) & 1, dead);
            const float* xs = reinterpret_cast<const float*>(xsums + (size_t)ub * UQ_XS);
            const int xg = ngroup * UQ_G;            // to the sums of the next eight picks
            uint64_t acc[UQ_TT / UQ_G][4];
#pragma unroll
            for (int s = 0; s < UQ_TT / UQ_G; s++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[s][i] = 0ull;
#pragma unroll 1
            for (int kc = 0; kc < nk; kc++, kg++, xs += 4 * UQ_G) {
                if (!(kc & 1)) wait(bar(S_FULL, st), ph, dead);
                const unsigned char* sc4 = sring + (size_t)st * UQ_SSLOT + (2 * rb * UM_M + vrow) * 16 + (kc & 1) * 8;
                const uint2 s4 = *reinterpret_cast<const uint2*>(sc4), m4 = *reinterpret_cast<const uint2*>(sc4 + UM_M * 16);
                if (cn <= UQ_FEW) {                  // a buffer holds the four groups of eight picks
                    const uint32_t i = turn & 1;
                    load(bar(FEW, 2 * rb + (int)i), (few_par >> i) & 1);
                    few_par ^= 1u << i;
                    uq_fold<0>(c, f16_of(s4.x, 0) * 1024.0f, f16_of(m4.x, 0), xs, acc[0]);
                    uq_fold<16>(c, f16_of(s4.x, 1) * 1024.0f, f16_of(m4.x, 1), xs + UQ_G, acc[0]);
                    uq_fold<32>(c, f16_of(s4.y, 0) * 1024.0f, f16_of(m4.y, 0), xs + 2 * UQ_G, acc[0]);
                    uq_fold<48>(c, f16_of(s4.y, 1) * 1024.0f, f16_of(m4.y, 1), xs + 3 * UQ_G, acc[0]);
                } else {
                    const float* x = xs;
#pragma unroll 1
                    for (int h = 0; h < 2; h++, x += 2 * UQ_G) {
                        const uint32_t sw = h ? s4.y : s4.x, mw = h ? m4.y : m4.x;
                        const float sca = f16_of(sw, 0) * 1024.0f, scb = f16_of(sw, 1) * 1024.0f, mna = f16_of(mw, 0), mnb = f16_of(mw, 1);
                        if (cn <= UQ_SMALL) {        // two groups of sixteen
                            load(bar(DONE, 2 * rb + h), kg & 1);
                            uq_fold<0>(c, sca, mna, x, acc[0]);
                            uq_fold<16>(c, sca, mna, x + xg, acc[1]);
                            uq_fold<32>(c, scb, mnb, x + UQ_G, acc[0]);
                            uq_fold<48>(c, scb, mnb, x + xg + UQ_G, acc[1]);
                        } else {                     // one group of 32
#pragma unroll
                            for (int g = 0; g < 2; g++) {
                                load(g ? bar(DONE, 2 * rb + h) : bar(FIRST, 2 * rb + h), g ? kg & 1 : first_par);
                                const float sc = g ? scb : sca, mn = g ? mnb : mna;
                                const float* xx = x + g * UQ_G;
                                uq_fold<0>(c, sc, mn, xx, acc[0]);
                                uq_fold<16>(c, sc, mn, xx + xg, acc[1]);
                                uq_fold<32>(c, sc, mn, xx + 2 * xg, acc[2]);
                                uq_fold<48>(c, sc, mn, xx + 3 * xg, acc[3]);
                            }
                        }
                    }
                }
                if (cn > UQ_SMALL) first_par ^= 1;
                if ((kc & 1) || kc + 1 == nk) {
                    __syncwarp();
                    mbar_arrive_if(lane == 0, bar(S_EMPTY, st));
                    if (++st == UQ_NS) { st = 0; ph ^= 1; }
                }
            }
            // act = silu(gate) * up per pick (pairs): of every eight picks the gate rows' warp finishes the first four and the up rows' warp the
            // others; or the picks' rows of ypart (nothing after a wait that gave up: the tables may be stale)
            const int np = dead ? 0 : cn;
            float* out = a.out + r0 + vrow;
            if (a.pair) {
                float* rd = red + (size_t)(rb ? 0 : 4) * UM_M + vrow;
                asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");        // the unit before has read its values
#pragma unroll
                for (int s = 0; s < UQ_TT / UQ_G; s++) {
                    if (UQ_G * s >= cn) break;
                    f2_unpack(rb ? acc[s][0] : acc[s][2], rd[UQ_G * s * UM_M], rd[(UQ_G * s + 1) * UM_M]);
                    f2_unpack(rb ? acc[s][1] : acc[s][3], rd[(UQ_G * s + 2) * UM_M], rd[(UQ_G * s + 3) * UM_M]);
                }
                asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");        // the quarter's two warps
#pragma unroll
                for (int s = 0; s < UQ_TT / UQ_G; s++) {
                    const int t = UQ_G * s + 4 * rb;
                    if (t >= np) break;
                    const float4 x4 = *reinterpret_cast<const float4*>(&s_xscale[ub][t]);
                    const int4 d4 = *reinterpret_cast<const int4*>(&s_dst[ub][t]);
                    const float xsc[4] = {x4.x, x4.y, x4.z, x4.w};
                    const int dst[4] = {d4.x, d4.y, d4.z, d4.w};
                    float own[4];
                    f2_unpack(rb ? acc[s][2] : acc[s][0], own[0], own[1]);
                    f2_unpack(rb ? acc[s][3] : acc[s][1], own[2], own[3]);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float o = red[(size_t)(t + i) * UM_M + vrow];
                        const float y = siluf_((rb ? o : own[i]) * xsc[i]) * ((rb ? own[i] : o) * xsc[i]);
                        if (t + i < np) out[dst[i]] = y;
                    }
                }
            } else {
                out += rb * UM_M;
#pragma unroll
                for (int t = 0; t < UQ_TT; t += 4) {
                    if (t >= np) break;
                    const float4 x4 = *reinterpret_cast<const float4*>(&s_xscale[ub][t]);
                    const int4 d4 = *reinterpret_cast<const int4*>(&s_dst[ub][t]);
                    const float xsc[4] = {x4.x, x4.y, x4.z, x4.w};
                    const int dst[4] = {d4.x, d4.y, d4.z, d4.w};
                    float v[4];
                    f2_unpack(acc[t / UQ_G][(t & 4) / 2], v[0], v[1]);
                    f2_unpack(acc[t / UQ_G][(t & 4) / 2 + 1], v[2], v[3]);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (t + i < np) out[dst[i]] = v[i] * xsc[i];
                }
            }
            __syncwarp();
            mbar_arrive_if(lane == 0, bar(T_EMPTY, ub));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { __syncwarp(); tmem_dealloc(tmem, 512); }
    trace_out(a.trace);
}

// ---- the activations of the sorted picks as planes -----------------------------------------------------------
struct PrepSlotsArgs {
    unsigned long long* trace;
    const float* src;         // [rows][stride]: by_pick ? one row per pick : one row per token
    int stride, by_pick, topk;
    const uint16_t* norm_w;   // ZNorm weight [K] or null
    float eps;
    int K, rows;              // rows = tokens, or picks (by_pick)
    const int* slot;          // [picks] a pick's place in the sorted list, or -1 (its expert lives elsewhere)
    uint8_t* planes;          // [K / 256][slots / 8][plane][group][8 slots][64 values] fp16, the 16-byte pieces of a row of 64 swizzled
    int slots;
    float* xscale;            // [slots]
    float* xsum;              // [slots / 8][K / 64][8] in units of the slot's scale, which multiplies once at the end of the product
};

// A row is normalised and split once and written to the slots of all its picks (a block per pick normalised every token
// topk times: 47 us for 8192 picks). NW warps per row: 8 for token rows of up to 2048 values, 2 for the expert activations
// (K <= 512), whose rows go one to a pick; 256 threads, 8 / NW rows per block.
template <int NW>
__global__ void __launch_bounds__(256) k_prep_q_slots(const PrepSlotsArgs a) {
    __shared__ float red[2][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp / NW, wi = warp % NW;
    const int row = blockIdx.x * (8 / NW) + sub;
    grid_dep_launch();
    trace_in(a.trace, 17, gridDim.x);
    grid_dep_wait();
    const int k = (wi * 32 + lane) * 8;
    const bool ok = row < a.rows && k < a.K;
    const float* x = a.src + (size_t)row * a.stride;
    float xv[8];
    float ss = 0.f;
    {
        float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
        if (ok) { v0 = *reinterpret_cast<const float4*>(x + k); v1 = *reinterpret_cast<const float4*>(x + k + 4); }
        xv[0] = v0.x; xv[1] = v0.y; xv[2] = v0.z; xv[3] = v0.w; xv[4] = v1.x; xv[5] = v1.y; xv[6] = v1.z; xv[7] = v1.w;
        if (a.norm_w) {
            uint4 wv = make_uint4(0u, 0u, 0u, 0u);
            if (k < a.K) wv = *reinterpret_cast<const uint4*>(a.norm_w + k);
            const float nw[8] = {1.0f + bflo(wv.x), 1.0f + bfhi(wv.x), 1.0f + bflo(wv.y), 1.0f + bfhi(wv.y),
                                 1.0f + bflo(wv.z), 1.0f + bfhi(wv.z), 1.0f + bflo(wv.w), 1.0f + bfhi(wv.w)};
#pragma unroll
            for (int i = 0; i < 8; i++) { ss = fmaf(xv[i], xv[i], ss); xv[i] *= nw[i]; }
        }
    }
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) mx = fmaxf(mx, fabsf(xv[i]));
    ss = warp_sum(ss);
    mx = warp_max(mx);
    if (lane == 0) { red[0][warp] = ss; red[1][warp] = mx; }
    __syncthreads();
    ss = 0.f; mx = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) { ss += red[0][sub * NW + w]; mx = fmaxf(mx, red[1][sub * NW + w]); }
    if (a.norm_w) {
        const float rn = 1.0f / sqrtf(ss / (float)a.K + a.eps);
#pragma unroll
        for (int i = 0; i < 8; i++) xv[i] *= rn;
        mx *= rn;
    }
    const float inv = mx > 1e-30f ? 127.0f / mx : 0.f;
    // the sum of a 64-value group: 8 neighbouring lanes, values in index order within a lane
    float s8 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) s8 += xv[i];
    s8 += __shfl_xor_sync(0xffffffffu, s8, 1);
    s8 += __shfl_xor_sync(0xffffffffu, s8, 2);
    s8 += __shfl_xor_sync(0xffffffffu, s8, 4);
    if (ok) {
        // q = 2048 h + l in the order of the codes' cells (0, 4, 1, 5, 2, 6, 3, 7); values 1, 3, 5, 7 meet codes in units of 2^-20: times 2^-4
        uint32_t w[UQ_PL][4] = {{0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int qv = __float2int_rn(xv[i] * inv * 16384.0f);
            const int hi = (qv + 1024) >> 11, lo = qv - (hi << 11);
            const float f = i & 1 ? 0.0625f : 1.0f;
            w[0][i & 3] |= (uint32_t)__half_as_ushort(__float2half_rn((float)hi * f)) << (i & 4 ? 16 : 0);
            w[1][i & 3] |= (uint32_t)__half_as_ushort(__float2half_rn((float)lo * f)) << (i & 4 ? 16 : 0);
        }
        const int np = a.by_pick ? 1 : a.topk;
        for (int r = 0; r < np; r++) {
            const int s = a.slot[row * np + r];
            if (s < 0) continue;
            if (k == 0) a.xscale[s] = mx / 127.0f;
            if ((lane & 7) == 0) a.xsum[((size_t)(s >> 3) * (a.K >> 6) + (k >> 6)) * UQ_G + (s & 7)] = mx > 0.f ? s8 / (mx / 127.0f) : 0.f;
            uint8_t* dst = a.planes + ((size_t)(k >> 8) * (a.slots / UQ_G) + (s >> 3)) * UQ_GBYTES + ((k >> 6) & 3) * 1024 + (s & 7) * 128 + ((((k >> 3) & 7) ^ (s & 7)) << 4);
#pragma unroll
            for (int pl = 0; pl < UQ_PL; pl++) *reinterpret_cast<uint4*>(dst + pl * UQ_SBO) = make_uint4(w[pl][0], w[pl][1], w[pl][2], w[pl][3]);
        }
    }
    trace_out(a.trace);
}

}  // namespace b2
