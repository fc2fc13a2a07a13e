// K2, small batches: y[M,N] = x[M,K] . deq(W)[N,K]^T for a few activation rows (M <= 16 in one launch), on the
// 5th-generation tensor cores with the weights' exact codes as the A operand in tensor memory.
//
// Bound: expanding the packed codes, about 0.3 us per SM for 128 rows x 64 codes; the tensor pipe has slack (N = 16 of 256
// columns) and HBM waits.  Measured (B200, us, kernels it replaces -> this one): 16 rows, 14336x4096 4-bit 52 -> 26;
// 16 rows, 4096x4096 6-bit 26 -> 14 (two launches of eight rows before); 8 rows, 14336x4096 8-bit 30 -> 23.
//
// A weight row is a TMEM lane: a dequantizer thread expands the codes of its row and k-block (exact integers times a
// power of two, jq_ts.cuh) and stores them with tcgen05.st; four MMAs (M = 128, N = 16, K = 16) sum the k-block into a
// slot of its own in tensor memory, and the same thread reads that slot one k-block later and adds
//     acc[m] += s * D[m] + b * X[m],      X[m] = sum of the block's activations of row m
// in float32.  So scales and biases stay unrounded, as in the mat-vec kernels for one row.  Warp roles:
//   warp 0        TMA: 16 activation rows x 64 per k-block;        warp 1   tensor memory, MMAs;
//   warps 2, 3    coalesced cp.async of the packed rows;            warp 4   the sums X of every k-block;
//   warps 5..12   dequantizers: two groups of four take alternate k-blocks; afterwards the epilogue.
// CTAs of a cluster split K; their sums and those of the two groups meet in shared memory and are added in rank order.
// Every mbarrier wait is bounded; a wait that runs out sets the status word and the CTA leaves through the common exit.
#include <cuda.h>

#include <atomic>

#include "jq_qgemv.cuh"
#include "jq_ts.cuh"

namespace jq {
namespace tsv {

constexpr int ROWS = 128;      // weight rows per CTA
constexpr int MC = 16;         // activation rows per launch = MMA N
constexpr int NKG = 2;         // groups of four dequantizer warps
constexpr int RA = 4;          // A slots: 32 columns each
constexpr int RD = 4;          // D slots: 16 columns each (k-block i is added before k-block i + 4 is stored)
constexpr int NCOLS = 256;     // of which 192 are used: two CTAs per SM
constexpr int RS = 16;         // slots of the activation sums: twice the activation stages (see the drain)
constexpr int SX = 8;          // activation stages of 2 KB
constexpr int X_STAGE = MC * 128;
constexpr int NDW = 4 * NKG;
constexpr int THREADS = 32 * (5 + NDW);
constexpr int DCOL = RA * 32;
static_assert(DCOL + RD * MC <= NCOLS, "A and D slots fit");

template <int BITS> struct Cfg {
    using CS = CodeStage<BITS>;
    static constexpr int CD = 6;                                   // code stages
    static constexpr int C_STAGE = ROWS * CS::RB;
    static constexpr int NBAR = 2 * SX + RA + RD + RS + 2 * CD;
    static constexpr int SIDE_OFF = SX * X_STAGE + CD * C_STAGE;
    static constexpr int XS_OFF = SIDE_OFF + CD * SIDE_SLOT;       // float X[RS][MC]
    static constexpr int BAR_OFF = XS_OFF + RS * MC * 4;
    static constexpr size_t SMEM = 1024 + BAR_OFF + NBAR * 8 + 16;
};

template <typename AT, int BITS, int MU>      // MU: activation rows computed (8 or 16)
__global__ void __launch_bounds__(THREADS, 2)
qgemv_ts_kernel(const __grid_constant__ CUtensorMap xmap, const GemvArgs a, const GemvBatch bt) {
    using A = Act<AT>;
    using C = Cfg<BITS>;
    constexpr int CKB = C::CS::CKB, RB = C::CS::RB, CPR = RB / 16, CD = C::CD;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sX = smem;
    uint8_t* sC = smem + SX * X_STAGE;
    float* sSum = reinterpret_cast<float*>(smem + C::XS_OFF);
    uint64_t* xfull = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF);
    uint64_t* xempty = xfull + SX;
    uint64_t* afull = xempty + SX;
    uint64_t* dfull = afull + RA;
    uint64_t* sfull = dfull + RD;
    uint64_t* cfull = sfull + RS;
    uint64_t* cempty = cfull + CD;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cempty + CD);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = a.ksplit;                                  // cluster size along K
    const int rank = S > 1 ? (int)(blockIdx.x % (unsigned)S) : 0;
    const int blk = (int)(blockIdx.x / (unsigned)S);
    int mi = 0, blk0 = 0;
    while (mi + 1 < bt.count && blk >= bt.blk_end[mi]) { blk0 = bt.blk_end[mi]; ++mi; }
    const int64_t N = bt.N[mi];
    const int64_t n0 = (int64_t)(blk - blk0) * ROWS;
    const int nkb_all = (int)(a.K / 64);
    const int kb0 = (rank * nkb_all / S) / 4 * 4;            // whole code stages and scale chunks
    const int kb1 = rank == S - 1 ? nkb_all : ((rank + 1) * nkb_all / S) / 4 * 4;
    const int nkb = kb1 - kb0, nst = (nkb + CKB - 1) / CKB;

    if (threadIdx.x == 0) {
        for (int i = 0; i < SX; ++i) { mbar_init(xfull + i, 1); mbar_init(xempty + i, 2); }
        for (int i = 0; i < RA; ++i) mbar_init(afull + i, 4);
        for (int i = 0; i < RD; ++i) mbar_init(dfull + i, 1);
        for (int i = 0; i < RS; ++i) mbar_init(sfull + i, 1);
        // the groups that have k-blocks in a stage: both, or one when a stage is one k-block
        for (int i = 0; i < CD; ++i) { mbar_init(cfull + i, 64); mbar_init(cempty + i, CKB == 1 ? 4 : NDW); }
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, NCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // under programmatic dependent launch the weights may be requested while the predecessor still runs; the
    // activations only after griddepcontrol.wait
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    bool ok = true;
    float acc[MU];
#pragma unroll
    for (int j = 0; j < MU; ++j) acc[j] = 0.f;

    if (warp == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int i = 0; i < nkb; ++i) {
            const int s = i % SX;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(xempty + s, ((uint32_t)(i / SX) & 1u) ^ 1u));
            if (!ok) break;
            if (elect_one()) {
                mbar_expect_tx(xfull + s, X_STAGE);
                tma_load_2d(sX + s * X_STAGE, &xmap, (kb0 + i) * 64, 0, xfull + s);     // rows past M read as zeros
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc_ts<AT>(MC);
        const uint32_t x_lo = umma_desc_sw128_lo(smem_u32(sX));
        for (int i = 0; i < nkb; ++i) {
            const int s = i % SX, t = i % RA;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(xfull + s, (uint32_t)(i / SX) & 1u) && ts_wait(afull + t, (uint32_t)(i / RA) & 1u));
            if (!ok) break;
            tc_fence_after();
            const uint32_t xd = x_lo + (uint32_t)s * (X_STAGE >> 4), ac = tmem_base + (uint32_t)(t * 32);
            const uint32_t dc = tmem_base + (uint32_t)(DCOL + t * MC);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_f16_ts(dc, ac + k * 8, umma_desc_join(xd + k * 2), idesc, k > 0 ? 1u : 0u);
                umma_commit(dfull + t);
                umma_commit(xempty + s);
            }
            __syncwarp();
        }
    } else if (warp < 4) {
        int buf = 0, slot = 0;
        uint32_t phase = 1u;
        const SideSrc side = {bt.scales[mi], bt.biases[mi], nullptr, nullptr, a.G, a.gs_shift ? 3 : 1};
        ok = load_codes<BITS, CD>(bt.codes[mi], n0, N, a.K, kb0 / CKB, nst, sC, cfull, cempty, threadIdx.x - 64, buf,
                                     phase, side, smem + C::SIDE_OFF, slot);
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp == 4) {
        // X of every k-block: lane = (row, half of the 64 activations), read through the stage's swizzle
        const int row = lane & 15, half = lane >> 4;
        for (int i = 0; i < nkb && ok; ++i) {
            const int s = i % SX, d = i % RS;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(xfull + s, (uint32_t)(i / SX) & 1u));
            if (!ok) break;
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint4 v = *reinterpret_cast<const uint4*>(sX + s * X_STAGE + row * 128 + (((half * 4 + c) ^ (row & 7)) << 4));
                sum += ((A::lo_f32(v.x) + A::hi_f32(v.x)) + (A::lo_f32(v.y) + A::hi_f32(v.y))) +
                       ((A::lo_f32(v.z) + A::hi_f32(v.z)) + (A::lo_f32(v.w) + A::hi_f32(v.w)));
            }
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 16);
            if (lane < 16) sSum[d * MC + row] = sum;
            __syncwarp();
            if (lane == 0) { mbar_arrive(sfull + d); mbar_arrive(xempty + s); }
        }
    } else {
        const int dw = warp - 5;
        const int quarter = warp & 3, kg = dw >> 2;              // four consecutive warps cover the four TMEM quarters
        const int r = quarter * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        float ps = 0.f, pb = 0.f;                                // scale and bias of the k-block whose sum is pending
        int pend = -1;
        // Adds the pending k-block's sum.  It also frees what later k-blocks reuse: a group adds k-block i - 4 before it
        // stores k-block i, so A slot and D slot i % 4 need no barrier of their own; and a sum slot is written again 16
        // k-blocks later, when the MMAs of 8 k-blocks later are done (the stage of the activations was free).
        auto drain = [&]() {
            const int d = pend % RD, x = pend % RS;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(dfull + d, (uint32_t)(pend / RD) & 1u) &&
                                             ts_wait(sfull + x, (uint32_t)(pend / RS) & 1u));
            if (!ok) return;
            tc_fence_after();
            uint32_t v[MU];
            tmem_ldn<MU>(lane_base + (uint32_t)(DCOL + d * MC), v);
            const float4* xs = reinterpret_cast<const float4*>(sSum + x * MC);
#pragma unroll
            for (int j = 0; j < MU / 4; ++j) {
                const float4 x4 = xs[j];
                acc[4 * j] = fmaf(ps, __uint_as_float(v[4 * j]), fmaf(pb, x4.x, acc[4 * j]));
                acc[4 * j + 1] = fmaf(ps, __uint_as_float(v[4 * j + 1]), fmaf(pb, x4.y, acc[4 * j + 1]));
                acc[4 * j + 2] = fmaf(ps, __uint_as_float(v[4 * j + 2]), fmaf(pb, x4.z, acc[4 * j + 2]));
                acc[4 * j + 3] = fmaf(ps, __uint_as_float(v[4 * j + 3]), fmaf(pb, x4.w, acc[4 * j + 3]));
            }
            tc_fence_before();
        };
        int buf = CKB == 1 ? kg : 0;                             // code ring position, with the parity of the pass on top
        for (int st = CKB == 1 ? kg : 0; st < nst && ok; st += CKB == 1 ? 2 : 1) {
            const bool odd = buf >= CD;
            const int cb = odd ? buf - CD : buf;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(cfull + cb, odd ? 1u : 0u));
            if (!ok) break;
            buf += CKB == 1 ? 2 : 1;
            if (buf >= 2 * CD) buf -= 2 * CD;
            const uint8_t* crow = sC + cb * C::C_STAGE + r * RB;
#pragma unroll 1
            for (int kbi = CKB == 1 ? 0 : kg; kbi < CKB; kbi += 2) {
                const int i = st * CKB + kbi;
                if (i >= nkb) break;
                const int t = i % RA;
#pragma unroll
                for (int h = 0; h < 2; ++h) {                    // 32 codes at a time keep the registers for two CTAs per SM
                    uint32_t cur[BITS], out[16];
                    load_codes32<BITS, CPR>(crow, r, kbi, h, cur);
                    dequant_fast<AT, BITS, 1, true>(cur, TsExact<AT>::C, 0u, out);
                    tmem_st16(lane_base + (uint32_t)(t * 32 + h * 16), out);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(afull + t);
                const uint16_t* side = reinterpret_cast<const uint16_t*>(smem + C::SIDE_OFF + (i >> 2) % CD * SIDE_SLOT) + r * 4 +
                                       (a.gs_shift ? (i & 3) >> 1 : i & 3);
                const float ns = A::to_f32(side[0]) * TsExact<AT>::POST, nb = A::to_f32(side[128 * 4]);
                if (pend >= 0) {
                    drain();
                    if (!ok) break;
                }
                ps = ns; pb = nb;
                pend = i;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(cempty + cb);
        }
        if (ok && pend >= 0) drain();
    }
    // sums of the two groups (and of the cluster's CTAs) meet as float [group][m][row] in the idle code stages
    __syncthreads();
    float* part = reinterpret_cast<float*>(sC);
    static_assert(NKG * MC * ROWS * 4 <= C::CD * C::C_STAGE, "partial sums fit the code stages");
    if (warp >= 5) {
        const int kg = (warp - 5) >> 2, r = (warp & 3) * 32 + lane;
#pragma unroll
        for (int j = 0; j < MU; ++j) part[(kg * MC + j) * ROWS + r] = acc[j];
    }
    if (S > 1) ts_cluster_sync(); else __syncthreads();
    {
        // this CTA stores the activation rows m = rank, rank + S, ..; a thread adds four neighbouring weight rows
        uint16_t* y16 = reinterpret_cast<uint16_t*>(bt.y[mi]);
        const int64_t ldy = bt.ldy[mi];
        for (int q = threadIdx.x; q < MU * (ROWS / 4); q += THREADS) {
            const int m = q / (ROWS / 4), nl = (q % (ROWS / 4)) * 4;
            if (m >= a.M || m % S != rank) continue;
            float f[4] = {0.f, 0.f, 0.f, 0.f};
            for (int rk = 0; rk < S; ++rk)
#pragma unroll
                for (int kg = 0; kg < NKG; ++kg) {
                    const float* src = part + (kg * MC + m) * ROWS + nl;
                    const float4 g = S > 1 ? ld_cluster_f32x4(src, (uint32_t)rk) : *reinterpret_cast<const float4*>(src);
                    f[0] += g.x; f[1] += g.y; f[2] += g.z; f[3] += g.w;
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n0 + nl + j < N) y16[m * ldy + n0 + nl + j] = A::from_f32(f[j]);
        }
    }
    if (S > 1) ts_cluster_sync();                           // every CTA keeps its shared memory until all have read it
    if (!ok) atomicOr(a.status, JQ_STATUS_LOCAL_WAIT);
    tc_fence_before();
    const int gave_up = __syncthreads_or(ok ? 0 : 1);
    if (warp == 1) {
        if (gave_up)                                        // copies and MMAs may still be in flight
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
        tc_fence_after();
        tmem_dealloc(tmem_base, NCOLS);
    }
}

template <typename AT, int BITS, int MU>
static int launch(const CUtensorMap& xmap, GemvArgs a, GemvBatch bt, int S, cudaStream_t st, bool* launched) {
    using C = Cfg<BITS>;
    static_assert(C::SMEM <= 113 * 1024, "two CTAs per SM");
    auto kernel = qgemv_ts_kernel<AT, BITS, MU>;
    static bool attr_done[64] = {};        // per device; benign race: the attribute call is idempotent
    int dev = 0;
    JQ_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        JQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    a.ksplit = S;
    a.status = status_word();
    JQ_REQUIRE(a.status != nullptr, JQ_ECUDA, "could not locate the device status word");
    int64_t row_blocks = 0;
    for (int i = 0; i < bt.count; ++i) {
        row_blocks += (bt.N[i] + ROWS - 1) / ROWS;
        bt.blk_end[i] = (int)row_blocks;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)row_blocks * (unsigned)S);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (S > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)S;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (a.pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    JQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, xmap, a, bt));
    *launched = true;
    return JQ_OK;
}

}  // namespace tsv

// Stands for a kernel whose shared memory decides how many CTAs an SM holds; never launched.  (Asked about the mat-vec kernel
// itself, whose thirteen warps of 72 registers fit an SM twice, the query says once.)
static __global__ void residency_kernel() {}

// Clusters of S CTAs that the GPU holds at once with per_sm (1 or 2) CTAs on an SM.  Fewer than sms * per_sm / S: a cluster
// stays inside a processing cluster whose SMs S need not divide (of 148 SMs: 45 threes, 33 fours, 15 eights; 93, 71, 33).
int resident_clusters(int S, int per_sm) {
    static std::atomic<int> cached[64][9][3];              // 0: not asked yet; host threads may ask twice
    const int even = sm_count() * per_sm / S;
    int dev = 0;
    if (S <= 1 || S > 8 || per_sm < 1 || per_sm > 2 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return even;
    int n = cached[dev][S][per_sm].load(std::memory_order_relaxed);
    if (n > 0) return n;
    constexpr int MOST = 200 * 1024;                       // over half of an SM's shared memory: one CTA each
    auto kernel = residency_kernel;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S * 1024u);               // the answer is no larger than the grid
    cfg.blockDim = dim3(tsv::THREADS);
    cfg.dynamicSmemBytes = per_sm == 1 ? MOST : MOST / 2;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = even;
    }
    cached[dev][S][per_sm].store(n, std::memory_order_relaxed);
    return n;
}

// Cluster size along K with the shortest estimated time (us): of two CTAs on an SM each walks a k-block in 0.52 us and
// a round of them starts and ends in 3.6 us (4.2 where four or more split K), one alone takes 0.33 (and 4.4), and a split
// adds the exchange of the sums, more with every round.  Measured on B200 over 4 to 460 row blocks, 2- to 8-bit codes, 6
// to 16 rows (all scale alike).  The largest split that one round holds, as before, left half of the chip idle between
// one and 1.4 row blocks per SM (9 rows, 22016x4096 2-bit, group 128: 40.5 us unsplit, 36.5 by 3; 16 rows, 9600x11264
// 6-bit: 66.5 by 2, 48.7 by 3).
TsSplit ts_split(int64_t row_blocks, int64_t K) {
    TsSplit best = {1, 1e30f};
    const int64_t chunks = K / 256;                        // of four k-blocks: what a split deals out
    for (int S : {1, 2, 3, 4, 8}) {
        if (chunks < S) break;
        const int64_t one = resident_clusters(S, 1), two = resident_clusters(S, 2), rest = row_blocks % two;
        const float pairs = (float)(row_blocks / two + (rest > one ? 1 : 0)), single = rest > 0 && rest <= one ? 1.f : 0.f;
        const float k = (float)((chunks + S - 1) / S) * 4.f;
        const float exchange = S == 1 ? 0.f : S == 2 ? 1.0f : S == 3 ? 2.5f : S == 4 ? 1.3f : 2.0f;
        const float us = pairs * (0.52f * k + (S < 4 ? 3.6f : 4.2f)) + single * (0.33f * k + (S < 4 ? 3.6f : 4.4f)) +
                         exchange * (0.4f + 0.6f * (pairs + single));
        if (us < best.us) best = {S, us};
    }
    return best;
}

// Dense mat-vecs of up to 16 activation rows (a.M may exceed the 8 rows of the other kernels), one launch for all
// matrices of `bt`; *launched stays false when the shape does not fit it.
int launch_ts_kernel(const GemvArgs& a0, const GemvBatch& bt, int act_dtype, int bits, int gs, cudaStream_t st,
                     bool* launched) {
    *launched = false;
    GemvArgs a = a0;
    if (a.M < 1 || a.M > tsv::MC || a.K % 256 != 0 || a.G % 4 != 0 || !(gs == 64 || gs == 128)) return JQ_OK;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return JQ_OK;
    CUtensorMap xmap;
    const cuuint64_t gdim[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M};
    const cuuint64_t gstride[1] = {(cuuint64_t)a.ldx * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)tsv::MC};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&xmap, act_dtype == JQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                      const_cast<void*>(a.x), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    JQ_REQUIRE(cr == CUDA_SUCCESS, JQ_ECUDA, "cuTensorMapEncodeTiled failed with code %d", (int)cr);
    a.gs_shift = gs == 128 ? 1 : 0;
    int64_t row_blocks = 0;
    for (int i = 0; i < bt.count; ++i) row_blocks += (bt.N[i] + tsv::ROWS - 1) / tsv::ROWS;
    const int S = ts_split(row_blocks, a.K).S;
    int rc = JQ_OK;
#define JQ_TS_CASE(B)                                                                                     \
    if (bits == B) {                                                                                      \
        if (act_dtype == JQ_BF16)                                                                         \
            rc = a.M <= 8 ? tsv::launch<__nv_bfloat16, B, 8>(xmap, a, bt, S, st, launched)                \
                          : tsv::launch<__nv_bfloat16, B, 16>(xmap, a, bt, S, st, launched);              \
        else                                                                                              \
            rc = a.M <= 8 ? tsv::launch<__half, B, 8>(xmap, a, bt, S, st, launched)                       \
                          : tsv::launch<__half, B, 16>(xmap, a, bt, S, st, launched);                     \
    }
    JQ_TS_CASE(2) JQ_TS_CASE(3) JQ_TS_CASE(4) JQ_TS_CASE(6) JQ_TS_CASE(8)
#undef JQ_TS_CASE
    return rc;
}

}  // namespace jq
