// K3: prefill-shaped quantized GEMM  Y[M,N] = X[M,K] . deq(W)[N,K]^T  on the 5th-generation
// tensor cores (tcgen05.mma), weights as the A operand in tensor memory.
//
// Bound: dense bf16/f16 tensor throughput for large M (2*M*N*K flops); for few rows the rate at which the
// packed codes are expanded.
//
// The dequantized weight is the A operand: a weight row is a TMEM lane, so a dequantizer thread expands the 64 codes of
// its row and k-block in registers and stores them with one tcgen05.st -- no shared-memory tile, no proxy fence, and the
// MMAs read only the activations from shared memory.  The activations are the B operand, so the MMA's N is the number
// of activation rows rounded up to 16: a short batch or a short expert costs no padded work, and one 128-row weight
// tile feeds up to 256 of them.  Warp roles:
//   warp 0        TMA producer: copies the activation tile of every k-block into a 128-byte-swizzled stage;
//   warp 1        allocates the tensor memory; one elected lane issues the MMAs (M = 128, N <= 256, K = 16) and commits
//                 their completion to the mbarriers that free the stages and the A slots;
//   warps 2, 3    code loaders: coalesced 16-byte cp.async of the packed rows and small copies of their scales and
//                 biases, six stages deep, completion counted on mbarriers (no barrier between warps);
//   dequantizers  four groups of four warps, one weight row per thread: group g takes k-blocks g, g + 4, ... and owns
//                 A slot g.
// Two forms: one tile per CTA with an optional split of K over a cluster (dense products), and a persistent one that
// walks the tiles of the routed experts.
// Every mbarrier wait is bounded; a wait that runs out sets the library's status word and the
// CTA leaves through the common exit (tensor memory is always released).
//
// Measured (B200, N x K): 4096 rows, 14336x4096 4-bit 492 -> 364 us (978 -> 1322 TFLOP/s); 512 rows, 11008x4096 2-bit
// 68 -> 50 us; 333 rows, 4096x4096 8-bit f16 55 -> 20 us; 61 rows, 4096x4096 6-bit 34 -> 12 us (before: the dequantized
// tile as the B operand in shared memory, one thread per weight row, one group of dequantizer warps).
//
// Numerics: the A operand is the dequantized weight rounded once to the activation type (what
// MLX's qmm feeds its matrix units), products are accumulated in f32 in ascending k order.  8-bit codes with bf16 round
// to f32 first in the general form of the expansion (groups of 32, or a scale of the warp's rows at 2^-5 or above).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "jq_ts.cuh"

namespace jq {


constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_SMEM = 227 * 1024;   // dynamic shared memory of one CTA

struct GemmArgs {
    const uint32_t* codes;
    const void* scales;
    const void* biases;
    void* y;
    int64_t M, N, K, ldy;
    int gs, G;
    int tn;          // activation rows per tile (multiple of 16, <= TNMAX)
    int box_rows;    // activation rows per TMA box: tn, or 32 when the rows of a tile vary (grouped mode)
    int y_pair_ok;   // rows of y are 4-byte aligned
    int y_vec_ok;    // rows of y are 8-byte aligned
    int* status;     // device status word, set to 1 when a bounded wait ran out
    // grouped mode (routed experts): CTAs walk a tile list built by jq_moe_sort; rows are the expert-sorted
    // (token, slot) pairs, weights come from per-expert pointer tables
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* num_tiles;
    int max_tiles;                 // entries the caller stated the list to have: no more are read, whatever *num_tiles says
    const int32_t* expert_offsets;
    const uint32_t* const* codes_tab;
    const void* const* scales_tab;
    const void* const* biases_tab;
    const int32_t* bits_tab;       // optional per-expert bit width: tiles of other widths exit
    // gate/up mode (GU): the tables above are the gate's, these the up projection's; y = h of
    // h[p, n] = silu(min(g, lim)) * clip(u, -lim, lim) * wts[order[p]]  (dsv41/model.py:1216-1226)
    const uint32_t* const* codes_tab2;
    const void* const* scales_tab2;
    const void* const* biases_tab2;
    const float* wts;
    const int32_t* order;
    float lim;
};

// Scales and biases of one weight row: from the staged chunk (jq_ts.cuh), or, where rows are not staged, loaded one
// k-block of this thread ahead (both scales of a k-block with groups of 32).
struct Sidecars {
    const uint16_t *srow, *brow;
    int gs, mode;
    uint32_t ns, nb;              // not staged: the next k-block's, one per half
    __device__ __forceinline__ void row(const void* scales, const void* biases, int64_t n, int64_t G) {
        srow = reinterpret_cast<const uint16_t*>(scales) + n * G;
        brow = reinterpret_cast<const uint16_t*>(biases) + n * G;
    }
    __device__ __forceinline__ void fetch(int kb) {
        const int g = gs == 32 ? 2 * kb : gs == 64 ? kb : kb >> 1;
        ns = __ldg(srow + g);
        nb = __ldg(brow + g);
        if (gs == 32) {
            ns |= (uint32_t)__ldg(srow + g + 1) << 16;
            nb |= (uint32_t)__ldg(brow + g + 1) << 16;
        }
    }
};

// The 64 codes of row r and k-block kb (block kbi of the staged row at crow) -> 32 registers of dequantized weights.
// side: this row's staged chunk; kb_next: the thread's next k-block, or -1.
template <typename AT, int BITS>
__device__ __forceinline__ void expand_block(const uint8_t* crow, int r, int kbi, int kb, int kb_next, const uint16_t* side,
                                             Sidecars& sc, uint32_t (&out)[32]) {
    using A = Act<AT>;
    constexpr int UW = 2 * BITS, CPR = CodeStage<BITS>::RB / 16;
    uint32_t cur[UW];
    if constexpr (UW % 4 == 0) {
        const uint4* cp = reinterpret_cast<const uint4*>(crow);
#pragma unroll
        for (int w = 0; w < UW / 4; ++w) {
            const uint4 v = cp[code_chunk<CPR>(kbi * (UW / 4) + w, r)];
            cur[4 * w] = v.x; cur[4 * w + 1] = v.y; cur[4 * w + 2] = v.z; cur[4 * w + 3] = v.w;
        }
    } else {
        const uint2* cp = reinterpret_cast<const uint2*>(crow + kbi * 8 * BITS);
#pragma unroll
        for (int w = 0; w < UW / 2; ++w) {
            const uint2 v = cp[w];
            cur[2 * w] = v.x; cur[2 * w + 1] = v.y;
        }
    }
    uint16_t s0h, b0h, s1h, b1h;
    if (sc.mode != 0) {
        const int i = sc.mode == 3 ? (kb & 3) >> 1 : kb & 3;
        s0h = s1h = side[i];
        b0h = b1h = side[128 * 4 + i];
    } else {
        s0h = (uint16_t)sc.ns; b0h = (uint16_t)sc.nb;
        s1h = sc.gs == 32 ? (uint16_t)(sc.ns >> 16) : s0h;
        b1h = sc.gs == 32 ? (uint16_t)(sc.nb >> 16) : b0h;
        if (kb_next >= 0) sc.fetch(kb_next);
    }
    const float s0 = A::to_f32(s0h), s1 = A::to_f32(s1h);
    const uint32_t bb0 = (uint32_t)b0h * 0x00010001u, bb1 = (uint32_t)b1h * 0x00010001u;
    // scales too large for the fast form (or not finite) send the warp's k-block through the general one
    const bool fast = sc.gs >= 64 && __all_sync(0xFFFFFFFFu, fabsf(s0) < fast_limit<AT, BITS>());
    if (fast) {
        dequant_fast<AT, BITS, 2>(cur, s0, bb0, out);
    } else {
        const uint32_t sp0 = A::pack_hi(s0, s0), sp1 = A::pack_hi(s1, s1);
        dequant_general<AT, BITS, 0, 0>(cur, sp0, bb0, s0, A::to_f32(b0h), out);
        dequant_general<AT, BITS, 16, 0>(cur, sp1, bb1, s1, A::to_f32(b1h), out);
    }
}

// 32 accumulator columns (activation rows row0 .. row0 + 31 of y, `rows` of them valid) of one weight row per lane
template <typename AT>
__device__ __forceinline__ void store_columns(const GemmArgs& a, const uint32_t (&v)[32], int64_t row0, int rows, int64_t nn,
                                              bool whole, int lane) {
    using A = Act<AT>;
    uint16_t* yb = reinterpret_cast<uint16_t*>(a.y) + row0 * a.ldy;
    if (a.y_pair_ok && whole) {
        // neighbouring lanes swap halves: an even lane stores rows (n, n+1) of the even columns, an
        // odd lane (n-1, n) of the odd ones, 4 bytes each
        const bool odd = lane & 1;
        uint16_t* yl = yb + (odd ? a.ldy : 0) + (nn & ~1ll);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            const float keep = __uint_as_float(odd ? v[j + 1] : v[j]);
            const float got = __uint_as_float(__shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[j + 1], 1));
            const uint32_t pk = odd ? A::pack_hi(got, keep) : A::pack_hi(keep, got);
            if (j + (odd ? 1 : 0) < rows) *reinterpret_cast<uint32_t*>(yl + j * a.ldy) = pk;
        }
    } else if (nn < a.N) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < rows) yb[j * a.ldy + nn] = A::from_f32(__uint_as_float(v[j]));
    }
}

// four neighbouring outputs of the gate/up mode: g4 and u4 are the sums, wt the routing weight
template <typename AT>
__device__ __forceinline__ void store_swiglu(const GemmArgs& a, const float4& g4, const float4& u4, float wt, int64_t row,
                                             int64_t n) {
    using A = Act<AT>;
    const float gv[4] = {g4.x, g4.y, g4.z, g4.w}, uv[4] = {u4.x, u4.y, u4.z, u4.w};
    float f[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float g = gv[j], u = uv[j];
        if (a.lim > 0.f) {
            g = fminf(g, a.lim);
            u = fminf(fmaxf(u, -a.lim), a.lim);
        }
        f[j] = g / (1.0f + __expf(-g)) * u * wt;
    }
    uint16_t* yp = reinterpret_cast<uint16_t*>(a.y) + row * a.ldy + n;
    if (a.y_vec_ok && n + 4 <= a.N) {
        *reinterpret_cast<uint2*>(yp) = make_uint2(A::pack_hi(f[0], f[1]), A::pack_hi(f[2], f[3]));
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n + j < a.N) yp[j] = A::from_f32(f[j]);
    }
}

// Shape of one CTA of the one-tile form: up to 256 activation rows, four A slots (32 columns = one k-block each).
template <int BITS> struct GemmCfg {
    static constexpr int TNMAX = 256, RA = 4, NKG = RA, ACOL = TNMAX, NCOLS = 512;
    static constexpr int CKB = CodeStage<BITS>::CKB, RB = CodeStage<BITS>::RB, CD = 6;
    static constexpr int C_STAGE = 128 * RB, X_STAGE = TNMAX * GEMM_BK * 2;
    static constexpr int NDW = 4 * NKG, THREADS = 128 + 32 * NDW;
    static constexpr int NBAR = 2 * RA + 2 * CD + 1;
    static constexpr size_t SMEM = 1024 + (size_t)RA * X_STAGE + (size_t)CD * (C_STAGE + SIDE_SLOT) + NBAR * 8 + 16;
};

// KS: CTAs of a cluster (along blockIdx.z) that split K, for grids that would leave most SMs idle: every CTA
// accumulates its share of the k-blocks in its own tensor memory and leaves the sums as float32 in its (by then
// idle) shared memory; after a cluster barrier CTA r adds and stores the activation rows of its share, in rank order.
// Both cluster barriers are reached by every thread on every path.
template <typename AT, int BITS, int KS>
__global__ void __launch_bounds__(GemmCfg<BITS>::THREADS, 1)
qgemm_ts_kernel(const __grid_constant__ CUtensorMap xmap, const GemmArgs a) {
    using A = Act<AT>;
    using C = GemmCfg<BITS>;
    constexpr int CKB = C::CKB, RB = C::RB, CD = C::CD, RA = C::RA, NKG = C::NKG;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // the dynamic shared-memory base is only guaranteed 16-byte aligned: realign to 1024
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sX = smem;
    uint8_t* sC = sX + RA * C::X_STAGE;
    uint8_t* sSide = sC + CD * C::C_STAGE;
    uint64_t* full = reinterpret_cast<uint64_t*>(sSide + CD * SIDE_SLOT);     // both operands of a k-block
    uint64_t* empty = full + RA;
    uint64_t* cfull = empty + RA;
    uint64_t* cempty = cfull + CD;
    uint64_t* accfull = cempty + CD;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfull + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n0 = (int64_t)blockIdx.x * 128;
    const int64_t m0 = (int64_t)blockIdx.y * a.tn;
    // activation rows of this tile, and the MMA's N
    const int rows = (int)min((int64_t)a.tn, a.M - m0);
    const int n_mma = (rows + 15) & ~15;
    // this CTA's k-blocks [kb0, kb1): all of them, or its share (whole code stages and sidecar chunks) of a split K
    const int nkb_all = (int)(a.K / GEMM_BK);
    int kb0 = 0, kb1 = nkb_all;
    const int ks_rank = KS > 1 ? (int)blockIdx.z : 0;
    if constexpr (KS > 1) {
        kb0 = (ks_rank * nkb_all / KS) / 4 * 4;
        kb1 = ks_rank == KS - 1 ? nkb_all : ((ks_rank + 1) * nkb_all / KS) / 4 * 4;
    }
    const int nkb = kb1 - kb0, nst = (nkb + CKB - 1) / CKB;

    if (threadIdx.x == 0) {
        for (int i = 0; i < RA; ++i) { mbar_init(full + i, 5); mbar_init(empty + i, 1); }      // 4 dequantizer warps + TMA
        for (int i = 0; i < CD; ++i) { mbar_init(cfull + i, 64); mbar_init(cempty + i, 4 * CKB); }
        mbar_init(accfull, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::NCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        int s = 0;
        uint32_t ph = 1u;
        const uint32_t bytes = (uint32_t)(a.tn * GEMM_BK * 2);
        for (int i = 0; i < nkb; ++i) {
            ok = __all_sync(0xFFFFFFFFu, ts_wait(empty + s, ph));
            if (!ok) break;
            if (elect_one()) {
                mbar_expect_tx(full + s, bytes);
                tma_load_2d(sX + s * C::X_STAGE, &xmap, (kb0 + i) * GEMM_BK, (int)m0, full + s);   // rows past M read as zeros
            }
            __syncwarp();
            if (++s == RA) { s = 0; ph ^= 1u; }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t idesc = umma_idesc_ts<AT>(n_mma);
        const uint32_t x_lo = umma_desc_sw128_lo(smem_u32(sX));
        int s = 0;
        uint32_t ph = 0u;
        for (int i = 0; i < nkb; ++i) {
            ok = __all_sync(0xFFFFFFFFu, ts_wait(full + s, ph));
            if (!ok) break;
            tc_fence_after();
            const uint32_t xd = x_lo + (uint32_t)s * (uint32_t)(C::X_STAGE >> 4);
            const uint32_t ac = tmem_base + (uint32_t)(C::ACOL + s * 32);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < GEMM_BK / 16; ++k)
                    umma_f16_ts(tmem_base, ac + k * 8, umma_desc_join(xd + k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(empty + s);
                if (i == nkb - 1) umma_commit(accfull);
            }
            __syncwarp();
            if (++s == RA) { s = 0; ph ^= 1u; }
        }
    } else if (warp < 4) {
        // ---------------- code loaders ----------------
        int buf = 0, slot = 0;
        uint32_t phase = 1u;
        const SideSrc side = {a.scales, a.biases, nullptr, nullptr, a.G, side_mode(a.scales, a.biases, a.G, a.gs)};
        ok = load_codes<BITS, CD>(a.codes, n0, a.N, a.K, kb0 / CKB, nst, sC, cfull, cempty, threadIdx.x - 64, buf, phase, side,
                                     sSide, slot);
        cp_async_commit();
        cp_async_wait<0>();
    } else {
        // ---------------- dequantizers: one weight row per thread; group kg takes every fourth k-block, A slot kg --------
        const int quarter = warp & 3, kg = (warp - 4) >> 2;
        const int r = quarter * 32 + lane;
        const int64_t n = min(n0 + r, a.N - 1);               // rows past N are computed but never stored
        const uint32_t a_dst = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(C::ACOL + kg * 32);
        Sidecars sc;
        sc.gs = a.gs;
        sc.mode = side_mode(a.scales, a.biases, a.G, a.gs);
        sc.row(a.scales, a.biases, n, a.G);
        if (sc.mode == 0 && kg < nkb) sc.fetch(kb0 + kg);
        int slot = 0;                                         // chunk ring: this group's k-blocks are in successive chunks
        uint32_t ph = 1u;
        int buf = kg / CKB;                                   // ring position, with the parity of the pass on top of it
        for (int i = kg; i < nst * CKB; i += RA) {
            const bool odd = buf >= CD;
            const int cb = odd ? buf - CD : buf;
            ok = __all_sync(0xFFFFFFFFu, ts_wait(cfull + cb, odd ? 1u : 0u));
            if (!ok) break;
            buf += RA / CKB;
            if (buf >= 2 * CD) buf -= 2 * CD;
            if (i < nkb) {
                const int kb = kb0 + i;                        // absolute k-block
                uint32_t out[32];
                expand_block<AT, BITS>(sC + cb * C::C_STAGE + r * RB, r, i % CKB, kb, i + RA < nkb ? kb + RA : -1,
                                       reinterpret_cast<const uint16_t*>(sSide + slot * SIDE_SLOT) + r * 4, sc, out);
                if (++slot == CD) slot = 0;
                __syncwarp();
                if (lane == 0) mbar_arrive(cempty + cb);
                ok = __all_sync(0xFFFFFFFFu, ts_wait(empty + kg, ph));
                if (!ok) break;
                ph ^= 1u;
                tc_fence_after();
                tmem_st32(a_dst, out);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full + kg);
            } else if (lane == 0) {                            // the last stage is not always whole
                mbar_arrive(cempty + cb);
            }
        }

        // ---------------- epilogue: lane = weight row, TMEM column = activation row ----------------
        if (ok) ok = __all_sync(0xFFFFFFFFu, ts_wait(accfull, 0));
        if (ok) {
            tc_fence_after();
            const uint32_t d_src = tmem_base + ((uint32_t)(quarter * 32) << 16);
            const int64_t nn = n0 + r;
#pragma unroll 1
            for (int c0 = kg * 32; c0 < rows; c0 += NKG * 32) {
                uint32_t v[32];
                tmem_ld32(d_src + (uint32_t)c0, v);
                if constexpr (KS > 1) {
                    float* part = reinterpret_cast<float*>(smem) + (size_t)c0 * 128 + r;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c0 + j < rows) part[j * 128] = __uint_as_float(v[j]);
                } else {
                    store_columns<AT>(a, v, m0 + c0, rows - c0, nn, n0 + 128 <= a.N, lane);
                }
            }
        }
    }
    if constexpr (KS > 1) {
        static_assert((size_t)C::TNMAX * 128 * 4 <= (size_t)RA * C::X_STAGE + CD * C::C_STAGE, "staged sums fit");
        ts_cluster_sync();                               // the staged sums are complete
        if (warp >= 4 && ok) {
            // CTA r stores activation rows [r, r+1) * rows / KS; a thread adds four neighbouring weight rows
            const int t0 = ks_rank * rows / KS, t1 = (ks_rank + 1) * rows / KS;
            constexpr int QPR = 128 / 4;
            for (int q = threadIdx.x - 128 + t0 * QPR; q < t1 * QPR; q += C::NDW * 32) {
                const int tok = q / QPR, nl = (q % QPR) * 4;
                const float* src = reinterpret_cast<const float*>(smem) + (size_t)tok * 128 + nl;
                float4 f = ld_cluster_f32x4(src, 0);
#pragma unroll
                for (int rk = 1; rk < KS; ++rk) {           // rank order: the same sum whatever the timing
                    const float4 g = ld_cluster_f32x4(src, (uint32_t)rk);
                    f.x += g.x; f.y += g.y; f.z += g.z; f.w += g.w;
                }
                uint16_t* yp = reinterpret_cast<uint16_t*>(a.y) + (m0 + tok) * a.ldy + n0 + nl;
                if (a.y_vec_ok && n0 + nl + 4 <= a.N) {
                    *reinterpret_cast<uint2*>(yp) = make_uint2(A::pack_hi(f.x, f.y), A::pack_hi(f.z, f.w));
                } else {
                    const float fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (n0 + nl + j < a.N) yp[j] = A::from_f32(fv[j]);
                }
            }
        }
        ts_cluster_sync();                               // every CTA keeps its shared memory until all have read it
    }
    if (!ok) atomicOr(a.status, JQ_STATUS_LOCAL_WAIT);
    tc_fence_before();
    const int gave_up = __syncthreads_or(ok ? 0 : 1);
    if (warp == 1) {
        // after a wait that gave up, copies and MMAs of this CTA may still be in flight: give them a millisecond
        // to land before the tensor memory goes back and the CTA's shared memory is reused
        if (gave_up)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
        tc_fence_after();
        tmem_dealloc(tmem_base, C::NCOLS);
    }
}

// ---- persistent form --------------------------------------------------------------------------------------
// One CTA per SM walks tiles of 128 weight rows x up to TN activation rows (blockIdx.x, + gridDim.x, ...).  TN = 192: two
// accumulators and four A slots fill the tensor memory; while the epilogue warps store one tile, the MMAs fill the other
// accumulator, and copies and expansion of the next tile start before this one's MMAs are done.  TN = 256 (tile lists of
// 256 rows): one accumulator, so the next tile's MMAs wait until this one is read, but its four A slots are full by then;
// one expansion of a weight tile serves 256 rows (as two tiles of 128 they were expanded twice: 8192 rows over 8
// experts, 2048x4096 2-bit 185 us, now 134).
// Without it every 128-row tile of an expert paid 5.5 us of start and epilogue for 12 to 64 k-blocks of 0.3 us, and a
// grid sized for the largest possible tile list started thousands of CTAs that had nothing to do.
// GU (grouped mode): the tile's 128 weight rows are 64 rows of the gate projection and the same 64 rows of the up
// projection, so both sums of an output meet in one CTA: the epilogue exchanges them through shared memory in f32 and
// stores h.  Gate and up results never go through memory, and one launch replaces three.
template <int BITS, int TN> struct PersCfg {
    static constexpr int TNMAX = TN, ND = TN == 192 ? 2 : 1, RA = 4, NCOLS = 512, NKG = RA;
    static constexpr int ACOL = ND * TNMAX;
    static constexpr int CKB = CodeStage<BITS>::CKB, RB = CodeStage<BITS>::RB, CD = 6;
    static constexpr int C_STAGE = 128 * RB, X_STAGE = TNMAX * GEMM_BK * 2;
    static constexpr int NDW = 4 * NKG, THREADS = 32 * (8 + NDW);
    static constexpr int NBAR = 2 * RA + 2 * CD + 2 * ND;
    static constexpr int SIDE_OFF = RA * X_STAGE + CD * C_STAGE;
    static constexpr int SW_OFF = SIDE_OFF + CD * SIDE_SLOT;             // float[32][128]: gate/up exchange
    static constexpr int WT_OFF = SW_OFF + 32 * 128 * 4;                 // float[TN]: routing weights of the tile's rows
    static constexpr int BAR_OFF = WT_OFF + TNMAX * 4;
    static constexpr size_t SMEM = 1024 + BAR_OFF + NBAR * 8 + 16;
    static_assert(ACOL + RA * 32 <= NCOLS, "accumulators and A slots fit the tensor memory");
};

struct PersTile {
    int64_t n0, m0;
    int rows;                     // <= 0: nothing to do
    const uint32_t *codes, *codes2;
    const void *scales, *biases, *scales2, *biases2;
};

template <int BITS, bool GU>
__device__ __forceinline__ PersTile pers_tile(const GemmArgs& a, int tile, int nx) {
    PersTile t;
    const int bx = tile % nx, by = tile / nx;
    t.n0 = (int64_t)bx * (GU ? 64 : 128);
    const int e = a.tile_expert[by];
    t.m0 = a.tile_row0[by];
    int64_t m_end = a.expert_offsets[e + 1];
    t.codes = a.codes_tab[e]; t.scales = a.scales_tab[e]; t.biases = a.biases_tab[e];
    t.codes2 = nullptr; t.scales2 = nullptr; t.biases2 = nullptr;
    if constexpr (GU) { t.codes2 = a.codes_tab2[e]; t.scales2 = a.scales_tab2[e]; t.biases2 = a.biases_tab2[e]; }
    if (a.bits_tab && a.bits_tab[e] != BITS) m_end = t.m0;             // a launch of its own width takes it
    t.rows = (int)min((int64_t)a.tn, m_end - t.m0);
    return t;
}

template <bool GU> __device__ __forceinline__ int pers_side_mode(const GemmArgs& a, const PersTile& t) {
    const int m = side_mode(t.scales, t.biases, a.G, a.gs);
    if constexpr (!GU) return m;
    const int m2 = side_mode(t.scales2, t.biases2, a.G, a.gs);
    return m == 0 || m2 == 0 ? 0 : max(m, m2);               // the copy that both matrices are aligned for
}

template <typename AT, int BITS, bool GU, int TN>
__global__ void __launch_bounds__(PersCfg<BITS, TN>::THREADS, 1)
qgemm_pers_kernel(const __grid_constant__ CUtensorMap xmap, const GemmArgs a) {
    using C = PersCfg<BITS, TN>;
    constexpr int CKB = C::CKB, RB = C::RB, CD = C::CD, RA = C::RA, NKG = C::NKG;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sX = smem;
    uint8_t* sC = sX + RA * C::X_STAGE;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF);      // both operands of a k-block
    uint64_t* empty = full + RA;
    uint64_t* cfull = empty + RA;
    uint64_t* cempty = cfull + CD;
    uint64_t* accfull = cempty + CD;
    uint64_t* accempty = accfull + C::ND;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accempty + C::ND);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nkb = (int)(a.K / GEMM_BK), nst = (nkb + CKB - 1) / CKB;
    const int nx = (int)((a.N + (GU ? 63 : 127)) / (GU ? 64 : 128));
    const int total = nx * min(*a.num_tiles, a.max_tiles);
    const int first = blockIdx.x, step = gridDim.x;
    if (first >= total) return;              // uniform for the CTA, before any barrier or tensor-memory allocation

    if (threadIdx.x == 0) {
        for (int i = 0; i < RA; ++i) { mbar_init(full + i, 5); mbar_init(empty + i, 1); }      // 4 dequantizer warps + TMA
        for (int i = 0; i < CD; ++i) { mbar_init(cfull + i, 64); mbar_init(cempty + i, 4 * CKB); }      // every k-block of a stage has its group
        for (int i = 0; i < C::ND; ++i) { mbar_init(accfull + i, 1); mbar_init(accempty + i, 4); }
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::NCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    // every wait on an "empty" barrier starts at parity 1: a fresh barrier counts as released.  Each role looks the next
    // tile up while it works on this one (in grouped mode that is a chain of dependent loads).
    PersTile next = pers_tile<BITS, GU>(a, first, nx);
    auto take = [&](int tile) {
        const PersTile cur = next;
        if (tile + step < total) next = pers_tile<BITS, GU>(a, tile + step, nx);
        return cur;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        int s = 0;
        uint32_t ph = 1u;
        for (int tile = first; tile < total && ok; tile += step) {
            const PersTile t = take(tile);
            if (t.rows <= 0) continue;
            const int boxes = (((t.rows + 15) & ~15) + a.box_rows - 1) / a.box_rows;
            const uint32_t box_bytes = (uint32_t)(a.box_rows * GEMM_BK * 2), bytes = (uint32_t)boxes * box_bytes;
            for (int i = 0; i < nkb; ++i) {
                ok = __all_sync(0xFFFFFFFFu, ts_wait(empty + s, ph));
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(full + s, bytes);
                    for (int b = 0; b < boxes; ++b)          // rows past M read as zeros
                        tma_load_2d(sX + s * C::X_STAGE + b * box_bytes, &xmap, i * GEMM_BK, (int)t.m0 + b * a.box_rows,
                                    full + s);
                }
                __syncwarp();
                if (++s == RA) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t x_lo = umma_desc_sw128_lo(smem_u32(sX));
        int s = 0, d = 0;
        uint32_t ph = 0u, dph = 1u;
        for (int tile = first; tile < total && ok; tile += step) {
            const PersTile t = take(tile);
            if (t.rows <= 0) continue;
            const uint32_t idesc = umma_idesc_ts<AT>((t.rows + 15) & ~15);
            const uint32_t dcol = tmem_base + (uint32_t)(d * C::TNMAX);
            ok = __all_sync(0xFFFFFFFFu, ts_wait(accempty + d, dph));
            for (int i = 0; i < nkb && ok; ++i) {
                ok = __all_sync(0xFFFFFFFFu, ts_wait(full + s, ph));
                if (!ok) break;
                tc_fence_after();
                const uint32_t xd = x_lo + (uint32_t)s * (uint32_t)(C::X_STAGE >> 4);
                const uint32_t ac = tmem_base + (uint32_t)(C::ACOL + s * 32);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k)
                        umma_f16_ts(dcol, ac + k * 8, umma_desc_join(xd + k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit(empty + s);
                    if (i == nkb - 1) umma_commit(accfull + d);
                }
                __syncwarp();
                if (++s == RA) { s = 0; ph ^= 1u; }
            }
            if (++d == C::ND) { d = 0; dph ^= 1u; }
        }
    } else if (warp < 4) {
        // ---------------- code loaders ----------------
        int buf = 0, slot = 0;
        uint32_t ph = 1u;
        for (int tile = first; tile < total && ok; tile += step) {
            const PersTile t = take(tile);
            if (t.rows <= 0) continue;
            const SideSrc side = {t.scales, t.biases, t.scales2, t.biases2, a.G, pers_side_mode<GU>(a, t)};
            ok = load_codes<BITS, CD, GU>(t.codes, t.n0, a.N, a.K, 0, nst, sC, cfull, cempty, threadIdx.x - 64, buf, ph, side,
                                             smem + C::SIDE_OFF, slot, t.codes2);
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp < 8) {
        // ---------------- epilogue: lane = weight row, TMEM column = activation row ----------------
        const int quarter = warp & 3, r = quarter * 32 + lane;
        int d = 0;
        uint32_t dph = 0u;
        for (int tile = first; tile < total && ok; tile += step) {
            const PersTile t = take(tile);
            if (t.rows <= 0) continue;
            if constexpr (GU) {
                // the rows' routing weights while the MMAs run: fetched in the loop below they are two dependent loads per
                // step and made the epilogue as long as the k-loop (2048 tokens, 128 experts: 161 us for the launch).
                // The last barrier of the previous tile has released the buffer.
                float* wt = reinterpret_cast<float*>(smem + C::WT_OFF);
                for (int q = r; q < t.rows; q += 128) wt[q] = a.wts ? a.wts[a.order[t.m0 + q]] : 1.0f;
            }
            ok = __all_sync(0xFFFFFFFFu, ts_wait(accfull + d, dph));
            if constexpr (GU) {      // the four warps meet in barriers below: they go on or leave together
                int all;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
                             "barrier.cta.red.and.aligned.pred q, 1, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                             : "=r"(all) : "r"(ok ? 1 : 0) : "memory");
                ok = all != 0;
            }
            if (!ok) break;
            tc_fence_after();
            const uint32_t src = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(d * C::TNMAX);
#pragma unroll 1
            for (int c0 = 0; c0 < t.rows; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(src + (uint32_t)c0, v);
                if (c0 + 32 >= t.rows) {                     // the accumulator is read: the MMAs may have it back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty + d);
                }
                if constexpr (GU) {
                    float* sw = reinterpret_cast<float*>(smem + C::SW_OFF);
#pragma unroll
                    for (int j = 0; j < 32; ++j) sw[j * 128 + r] = __uint_as_float(v[j]);
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    const int nrow = min(32, t.rows - c0);
                    for (int q = r; q < nrow * 16; q += 128) {
                        const int tok = q >> 4, nl = (q & 15) * 4;
                        const float4 g4 = *reinterpret_cast<const float4*>(sw + tok * 128 + nl);
                        const float4 u4 = *reinterpret_cast<const float4*>(sw + tok * 128 + 64 + nl);
                        const int64_t row = t.m0 + c0 + tok;
                        store_swiglu<AT>(a, g4, u4, reinterpret_cast<const float*>(smem + C::WT_OFF)[c0 + tok], row, t.n0 + nl);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                } else {
                    store_columns<AT>(a, v, t.m0 + c0, t.rows - c0, t.n0 + r, t.n0 + 128 <= a.N, lane);
                }
            }
            if (++d == C::ND) { d = 0; dph ^= 1u; }
        }
    } else {
        // ---------------- dequantizers: one weight row per thread, alternate k-blocks per group ----------------
        const int quarter = warp & 3, kg = (warp - 8) >> 2, r = quarter * 32 + lane;
        const uint32_t a_dst = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)C::ACOL;
        const bool up = GU && r >= 64;                        // warp-uniform
        auto row_of = [&](const PersTile& t) { return min(t.n0 + (GU ? r & 63 : r), a.N - 1); };   // past N: computed, never stored
        Sidecars sc;
        sc.gs = a.gs;
        int slot0 = 0;                                        // sidecar ring: slot of the tile's first chunk
        // k-block g of this CTA (counted over all its tiles) belongs to group g % 4 and to A slot g % 4; the codes are in
        // stages of CKB k-blocks, each of another group, counted over all tiles as well
        uint32_t ph = 1u;
        int base = 0, sbase = 0;                              // k-blocks (mod 4) and stages (mod 2 CD) before this tile
        for (int tile = first; tile < total && ok; tile += step) {
            const PersTile t = take(tile);
            if (t.rows <= 0) continue;
            int kb = (kg - base) & 3;
            int buf = sbase + kb / CKB;                       // ring position, with the parity of the pass on top of it
            if (buf >= 2 * CD) buf -= 2 * CD;
            int slot = slot0;                                 // this group's k-blocks are in successive chunks
            sc.mode = pers_side_mode<GU>(a, t);
            sc.row(up ? t.scales2 : t.scales, up ? t.biases2 : t.biases, row_of(t), a.G);
            if (sc.mode == 0 && kb < nkb) sc.fetch(kb);
            for (; kb < nst * CKB; kb += RA) {
                const bool odd = buf >= CD;
                const int cb = odd ? buf - CD : buf;
                ok = __all_sync(0xFFFFFFFFu, ts_wait(cfull + cb, odd ? 1u : 0u));
                if (!ok) break;
                buf += RA / CKB;
                if (buf >= 2 * CD) buf -= 2 * CD;
                if (kb < nkb) {
                    uint32_t out[32];
                    expand_block<AT, BITS>(sC + cb * C::C_STAGE + r * RB, r, kb % CKB, kb, kb + RA < nkb ? kb + RA : -1,
                                           reinterpret_cast<const uint16_t*>(smem + C::SIDE_OFF + slot * SIDE_SLOT) + r * 4, sc,
                                           out);
                    if (++slot == CD) slot = 0;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(cempty + cb);
                    ok = __all_sync(0xFFFFFFFFu, ts_wait(empty + kg, ph));
                    if (!ok) break;
                    ph ^= 1u;
                    tc_fence_after();
                    tmem_st32(a_dst + (uint32_t)(kg * 32), out);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full + kg);
                } else if (lane == 0) {                       // the last stage of a tile is not always whole
                    mbar_arrive(cempty + cb);
                }
            }
            base = (base + nkb) & 3;
            sbase = (sbase + nst) % (2 * CD);
            slot0 = (slot0 + (nkb + 3) / 4) % CD;
        }
    }
    if (!ok) atomicOr(a.status, JQ_STATUS_LOCAL_WAIT);
    tc_fence_before();
    const int gave_up = __syncthreads_or(ok ? 0 : 1);
    if (warp == 1) {
        // after a wait that gave up, copies and MMAs of this CTA may still be in flight: give them a millisecond
        // to land before the tensor memory goes back and the CTA's shared memory is reused
        if (gave_up)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
        tc_fence_after();
        tmem_dealloc(tmem_base, C::NCOLS);
    }
}

// ---- host side ------------------------------------------------------------------------------------------
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

template <typename AT, int BITS, int KS>
static int launch_gemm(const CUtensorMap& xmap, const GemmArgs& a, int64_t m_tiles, cudaStream_t st) {
    using C = GemmCfg<BITS>;
    constexpr size_t smem = C::SMEM;
    static_assert(smem <= GEMM_SMEM, "shared memory of one CTA");
    auto kernel = qgemm_ts_kernel<AT, BITS, KS>;
    static bool attr_done[64] = {};
    int dev = 0;
    JQ_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        JQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    dim3 grid((unsigned)((a.N + 127) / 128), (unsigned)m_tiles, KS);
    if constexpr (KS > 1) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(C::THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = KS;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        JQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, xmap, a));
        return JQ_OK;
    }
    kernel<<<grid, C::THREADS, smem, st>>>(xmap, a);
    return check_launch("qgemm");
}

template <typename AT, int BITS, bool GU, int TN>
static int launch_pers(const CUtensorMap& xmap, const GemmArgs& a, int64_t m_tiles, cudaStream_t st) {
    using C = PersCfg<BITS, TN>;
    static_assert(C::SMEM <= GEMM_SMEM, "shared memory of one CTA");
    auto kernel = qgemm_pers_kernel<AT, BITS, GU, TN>;
    static bool attr_done[64] = {};
    int dev = 0;
    JQ_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        JQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    const int64_t nx = (a.N + (GU ? 63 : 127)) / (GU ? 64 : 128), tiles = nx * m_tiles;
    JQ_REQUIRE(tiles < (1ll << 31), JQ_EUNSUPPORTED, "too many tiles for one launch (%lld)", (long long)tiles);
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, sm_count());
    kernel<<<grid, C::THREADS, C::SMEM, st>>>(xmap, a);
    return check_launch("qgemm");
}

struct GroupedArgs {
    const int32_t *tile_expert, *tile_row0, *num_tiles, *expert_offsets, *bits_tab;
    const uint32_t* const* codes_tab;
    const void* const* scales_tab;
    const void* const* biases_tab;
    int64_t max_tiles;
    int tile_m;       // rows per entry of the tile list: 128, 192 or 256
    // gate/up mode: the up projection's tables and what the epilogue needs (GemmArgs)
    const uint32_t* const* codes_tab2 = nullptr;
    const void* const* scales_tab2 = nullptr;
    const void* const* biases_tab2 = nullptr;
    const float* wts = nullptr;
    const int32_t* order = nullptr;
    float lim = 0.f;
};

// Dense when grp == nullptr (codes/scales/biases of one matrix); grouped otherwise (x holds the M
// expert-sorted rows, the weight pointers come from the tables).
int qgemm_dispatch(const void* x, int x_dtype, int64_t M, int64_t ldx, const uint32_t* codes, const void* scales,
                   const void* biases, int sidecar_dtype, int64_t N, int64_t K, int bits, int gs, void* y,
                   int y_dtype, int64_t ldy, const GroupedArgs* grp, cudaStream_t st) {
    int rc = check_quant_shape(N, K, bits, gs);
    if (rc != JQ_OK) return rc;
    JQ_REQUIRE(M >= 0, JQ_EINVAL, "negative M");
    if (M == 0 || N == 0) return JQ_OK;
    JQ_REQUIRE(K > 0, JQ_EINVAL, "K must be positive");
    JQ_REQUIRE(x && y && (grp || (codes && scales && biases)), JQ_EINVAL, "null pointer");
    JQ_REQUIRE(x_dtype == JQ_BF16 || x_dtype == JQ_F16, JQ_EINVAL, "qgemm activations must be bf16 or f16");
    JQ_REQUIRE(sidecar_dtype == x_dtype && y_dtype == x_dtype, JQ_EUNSUPPORTED,
               "qgemm needs scales/biases and the output in the activation dtype");
    JQ_REQUIRE(K % GEMM_BK == 0, JQ_EUNSUPPORTED, "qgemm needs K to be a multiple of 64, got %lld", (long long)K);
    JQ_REQUIRE((K * bits / 8) % 16 == 0, JQ_EUNSUPPORTED,
               "qgemm needs packed rows of a multiple of 16 bytes (K %% 128 == 0 for odd widths), got K=%lld bits=%d",
               (long long)K, bits);
    JQ_REQUIRE(grp || aligned(codes, 16), JQ_EINVAL, "codes must be 16-byte aligned");
    JQ_REQUIRE(aligned(x, 16) && ldx % 8 == 0 && ldx >= K, JQ_EINVAL, "x must be 16-byte aligned with ldx %% 8 == 0");
    JQ_REQUIRE(ldy >= N, JQ_EINVAL, "ldy too small");
    JQ_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), JQ_EUNSUPPORTED, "dimension too large");
    EncodeTiledFn enc = encode_tiled_fn();
    JQ_REQUIRE(enc != nullptr, JQ_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");

    GemmArgs a;
    a.codes = codes; a.scales = scales; a.biases = biases; a.y = y;
    a.M = M; a.N = N; a.K = K; a.ldy = ldy; a.gs = gs; a.G = (int)(K / gs);
    a.y_pair_ok = (aligned(y, 4) && ldy % 2 == 0) ? 1 : 0;
    a.y_vec_ok = (aligned(y, 8) && ldy % 4 == 0) ? 1 : 0;
    a.status = status_word();
    JQ_REQUIRE(a.status != nullptr, JQ_ECUDA, "could not locate the device status word");
    a.tile_expert = grp ? grp->tile_expert : nullptr;
    a.tile_row0 = grp ? grp->tile_row0 : nullptr;
    a.num_tiles = grp ? grp->num_tiles : nullptr;
    a.max_tiles = grp ? (int)std::min<int64_t>(grp->max_tiles, INT32_MAX) : 0;       // 65535 at most, checked below
    a.expert_offsets = grp ? grp->expert_offsets : nullptr;
    a.codes_tab = grp ? grp->codes_tab : nullptr;
    a.scales_tab = grp ? grp->scales_tab : nullptr;
    a.biases_tab = grp ? grp->biases_tab : nullptr;
    a.bits_tab = grp ? grp->bits_tab : nullptr;
    const bool gu = grp && grp->codes_tab2;
    a.codes_tab2 = gu ? grp->codes_tab2 : nullptr;
    a.scales_tab2 = gu ? grp->scales_tab2 : nullptr;
    a.biases_tab2 = gu ? grp->biases_tab2 : nullptr;
    a.wts = gu ? grp->wts : nullptr;
    a.order = gu ? grp->order : nullptr;
    a.lim = gu ? grp->lim : 0.f;
    int ks = 1;
    int64_t m_tiles;
    if (grp) {
        JQ_REQUIRE(grp->tile_m == 128 || grp->tile_m == 192 || (grp->tile_m == 256 && N >= 256 && x_dtype == JQ_BF16),
                   JQ_EUNSUPPORTED, "tile lists of 256 rows need bf16 activations and N >= 256 (128 or 192 otherwise)");
        a.tn = grp->tile_m;
        a.box_rows = 32;
        m_tiles = grp->max_tiles;
    } else {
        // The number of row tiles (nt, of tn rows each) and the K split with the shortest estimated time.  Measured on
        // B200 over M = 17 .. 4096: a CTA walks a k-block in 0.20 + 0.0006 tn us (the expansion of the codes sets the
        // pace below some 150 rows, the MMAs above) and spends 5.5 us on its start, first copies and epilogue; a split
        // adds 1.5 us + 8 ns per row for the exchange of the sums.  One CTA per SM, so what counts is the number of waves.
        // Examples (us): 61 rows, 4096x4096 6-bit: 12.2 split by 4, 15.9 by 2, 27 unsplit; 512 rows, 11008x4096 2-bit:
        // 50.1 with three tiles of 176, 53.3 with two of 256, 66.6 with four of 128.
        const int64_t sms = sm_count(), ncol = (N + 127) / 128, nkb_all = K / GEMM_BK;
        const int64_t least = (M + 255) / 256;
        m_tiles = least;
        a.tn = 256;
        double best = 1e30;
        for (int64_t nt = least; nt <= least + 3; ++nt) {
            const int64_t tn = ((M + nt - 1) / nt + 15) / 16 * 16, tiles = (M + tn - 1) / tn;
            for (int S : {1, 2, 4}) {
                if (S > 1 && nkb_all / S < 8) continue;
                const int64_t slots = sms / S * S, ctas = ncol * tiles * S;
                const double t = (double)((ctas + slots - 1) / slots) *
                                 ((double)nkb_all / S * (0.20 + 0.0006 * tn) + 5.5 + (S > 1 ? 1.5 + 0.008 * tn : 0.0));
                if (t < best) { best = t; m_tiles = tiles; a.tn = (int)tn; ks = S; }
            }
        }
        a.box_rows = a.tn;
    }
    if (m_tiles == 0) return JQ_OK;
    JQ_REQUIRE((grp ? grp->max_tiles : (M + GEMM_BM - 1) / GEMM_BM) < 65536, JQ_EUNSUPPORTED,
               "too many row tiles for one launch (%lld)", (long long)(grp ? grp->max_tiles : (M + GEMM_BM - 1) / GEMM_BM));
    CUtensorMap xmap;
    const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t gstride[1] = {(cuuint64_t)ldx * 2};
    const cuuint32_t box[2] = {GEMM_BK, (cuuint32_t)a.box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&xmap, x_dtype == JQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                      const_cast<void*>(x), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    JQ_REQUIRE(cr == CUDA_SUCCESS, JQ_ECUDA, "cuTensorMapEncodeTiled failed with code %d", (int)cr);

#define JQ_GEMM_T(T, B)                                                                                   \
    {                                                                                                     \
        if (gu) return launch_pers<T, B, true, 192>(xmap, a, m_tiles, st);                                \
        if (grp) return launch_pers<T, B, false, 192>(xmap, a, m_tiles, st);                              \
        if (ks == 4) return launch_gemm<T, B, 4>(xmap, a, m_tiles, st);                                   \
        if (ks == 2) return launch_gemm<T, B, 2>(xmap, a, m_tiles, st);                                   \
        return launch_gemm<T, B, 1>(xmap, a, m_tiles, st);                                                \
    }
#define JQ_GEMM_CASE(B)                                                                                   \
    if (bits == B) {                                                                                      \
        if (grp && grp->tile_m == 256)                         /* bf16 only, see above */                 \
            return gu ? launch_pers<__nv_bfloat16, B, true, 256>(xmap, a, m_tiles, st)                    \
                      : launch_pers<__nv_bfloat16, B, false, 256>(xmap, a, m_tiles, st);                  \
        if (x_dtype == JQ_BF16) JQ_GEMM_T(__nv_bfloat16, B)                                               \
        JQ_GEMM_T(__half, B)                                                                              \
    }
    JQ_GEMM_CASE(2) JQ_GEMM_CASE(3) JQ_GEMM_CASE(4) JQ_GEMM_CASE(5) JQ_GEMM_CASE(6) JQ_GEMM_CASE(8)
#undef JQ_GEMM_CASE
#undef JQ_GEMM_T
    return fail(JQ_EUNSUPPORTED, "bits=%d", bits);
}

// ---- allocation-free grouped GEMM ------------------------------------------------------------------
// The grouped GEMM walks a tile list (expert id and first row of every 128-row tile, plus their
// count).  jq_moe_gemm gets that list from buffers the caller allocated for jq_moe_sort; the variant
// below rebuilds it from expert_offsets into this fixed array instead, so the call needs no
// workspace at all.  Every device that loads the library holds the array (about 12 KB) until exit.
constexpr int STATIC_MAX_EXPERTS = 1024;
constexpr int64_t STATIC_MAX_ROWS = 65536;
constexpr int STATIC_MAX_TILES = (int)(STATIC_MAX_ROWS / GEMM_BM) + STATIC_MAX_EXPERTS;
constexpr int STATIC_HDR = 64;     // word 0 = number of tiles; the lists start 256 bytes in
static __device__ __align__(256) int32_t g_static_tiles[STATIC_HDR + 2 * STATIC_MAX_TILES];

// One CTA of STATIC_MAX_EXPERTS threads rewrites the whole list on every call, so nothing of an earlier
// call survives into this one: thread e counts the tiles of expert e, a block-wide exclusive scan gives
// the position of its first tile, and it writes its own tiles (experts ascending, rows ascending: the
// order jq_moe_sort emits).  Tiles past STATIC_MAX_TILES are dropped (offsets beyond the stated rows).
__global__ void __launch_bounds__(STATIC_MAX_EXPERTS)
build_tiles_kernel(const int32_t* __restrict__ offsets, int E, int tile_m, int32_t* __restrict__ out) {
    __shared__ int warp_sum[32];
    int32_t* tile_expert = out + STATIC_HDR;
    int32_t* tile_row0 = out + STATIC_HDR + STATIC_MAX_TILES;
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    int lo = 0, hi = 0;
    if (e < E) { lo = offsets[e]; hi = offsets[e + 1]; }
    const int mine = hi > lo ? (hi - lo + tile_m - 1) / tile_m : 0;
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sum[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= d) w += v;
        }
        warp_sum[lane] = w;            // inclusive sums of the warps
    }
    __syncthreads();
    int pos = incl - mine + (warp > 0 ? warp_sum[warp - 1] : 0);
    for (int r = lo; r < hi && pos < STATIC_MAX_TILES; r += tile_m, ++pos) {
        tile_expert[pos] = e;
        tile_row0[pos] = r;
    }
    if (e == 0) out[0] = min(warp_sum[31], STATIC_MAX_TILES);
}

// Device address of the array on the current device.  In host code the array's name is only a
// host-side handle, never a device address, so it is resolved with cudaGetSymbolAddress once per
// device (with that device current) and the pointer is what the kernels receive.
static int static_tiles_ptr(int32_t** out) {
    static std::atomic<int32_t*> cached[64];      // zero-initialised; host threads may race on the first call
    int dev = 0;
    JQ_CUDA_OK(cudaGetDevice(&dev));
    JQ_REQUIRE(dev >= 0 && dev < 64, JQ_EUNSUPPORTED, "device ordinal %d out of range", dev);
    int32_t* p = cached[dev].load(std::memory_order_acquire);
    if (!p) {
        JQ_CUDA_OK(cudaGetSymbolAddress((void**)&p, g_static_tiles));
        JQ_REQUIRE(p != nullptr, JQ_ECUDA, "cudaGetSymbolAddress returned a null address");
        cached[dev].store(p, std::memory_order_release);
    }
    *out = p;
    return JQ_OK;
}

}  // namespace jq

extern "C" {

int jq_moe_gemm_static(const void* x_sorted, int act_dtype, int64_t max_rows, int64_t ldx,
                       const int32_t* expert_offsets, int num_experts, const uint32_t* const* codes_tab,
                       const void* const* scales_tab, const void* const* biases_tab, const int32_t* bits_tab,
                       int sidecar_dtype, int64_t N, int64_t K, int bits, int group_size, void* y_sorted, int64_t ldy,
                       jq_stream_t stream) {
    using namespace jq;
    JQ_REQUIRE(expert_offsets && codes_tab && scales_tab && biases_tab, JQ_EINVAL, "null pointer");
    JQ_REQUIRE(num_experts > 0 && num_experts <= STATIC_MAX_EXPERTS, JQ_EUNSUPPORTED,
               "jq_moe_gemm_static holds tile lists for at most %d experts, got %d", STATIC_MAX_EXPERTS, num_experts);
    JQ_REQUIRE(max_rows >= 0 && max_rows <= STATIC_MAX_ROWS, JQ_EUNSUPPORTED,
               "jq_moe_gemm_static holds tile lists for at most %lld rows, got %lld", (long long)STATIC_MAX_ROWS,
               (long long)max_rows);
    if (max_rows == 0 || N == 0) return JQ_OK;
    int32_t* tiles = nullptr;
    int rc = static_tiles_ptr(&tiles);
    if (rc != JQ_OK) return rc;
    build_tiles_kernel<<<1, STATIC_MAX_EXPERTS, 0, (cudaStream_t)stream>>>(expert_offsets, num_experts, GEMM_BM, tiles);
    rc = check_launch("build_tiles");
    if (rc != JQ_OK) return rc;
    GroupedArgs g;
    g.tile_expert = tiles + STATIC_HDR;
    g.tile_row0 = tiles + STATIC_HDR + STATIC_MAX_TILES;
    g.num_tiles = tiles;
    g.expert_offsets = expert_offsets;
    g.bits_tab = bits_tab; g.codes_tab = codes_tab; g.scales_tab = scales_tab; g.biases_tab = biases_tab;
    g.max_tiles = max_rows / GEMM_BM + num_experts;
    g.tile_m = 128;
    return qgemm_dispatch(x_sorted, act_dtype, max_rows, ldx, nullptr, nullptr, nullptr, sidecar_dtype, N, K, bits,
                          group_size, y_sorted, act_dtype, ldy, &g, (cudaStream_t)stream);
}

int jq_qgemm(const void* x, int x_dtype, int64_t M, int64_t ldx, const uint32_t* codes, const void* scales,
             const void* biases, int sidecar_dtype, int64_t N, int64_t K, int bits, int group_size, void* y,
             int y_dtype, int64_t ldy, jq_stream_t stream) {
    return jq::qgemm_dispatch(x, x_dtype, M, ldx, codes, scales, biases, sidecar_dtype, N, K, bits, group_size, y,
                              y_dtype, ldy, nullptr, (cudaStream_t)stream);
}

int jq_moe_gemm(const void* x_sorted, int act_dtype, int64_t max_rows, int64_t ldx, const int32_t* expert_offsets,
                const int32_t* tile_expert, const int32_t* tile_row0, const int32_t* num_tiles, int64_t max_tiles,
                const uint32_t* const* codes_tab, const void* const* scales_tab, const void* const* biases_tab,
                const int32_t* bits_tab, int sidecar_dtype, int64_t N, int64_t K, int bits, int group_size,
                void* y_sorted, int64_t ldy, jq_stream_t stream) {
    return jq_moe_gemm_tiled(x_sorted, act_dtype, max_rows, ldx, expert_offsets, tile_expert, tile_row0, num_tiles,
                             max_tiles, 128, codes_tab, scales_tab, biases_tab, bits_tab, sidecar_dtype, N, K, bits,
                             group_size, y_sorted, ldy, stream);
}

int jq_moe_gemm_tiled(const void* x_sorted, int act_dtype, int64_t max_rows, int64_t ldx, const int32_t* expert_offsets,
                      const int32_t* tile_expert, const int32_t* tile_row0, const int32_t* num_tiles, int64_t max_tiles,
                      int tile_m, const uint32_t* const* codes_tab, const void* const* scales_tab,
                      const void* const* biases_tab, const int32_t* bits_tab, int sidecar_dtype, int64_t N, int64_t K,
                      int bits, int group_size, void* y_sorted, int64_t ldy, jq_stream_t stream) {
    using namespace jq;
    JQ_REQUIRE(tile_m == 128 || tile_m == 192 || tile_m == 256, JQ_EINVAL, "tile_m must be 128, 192 or 256");
    JQ_REQUIRE(expert_offsets && tile_expert && tile_row0 && num_tiles && codes_tab && scales_tab && biases_tab,
               JQ_EINVAL, "null pointer");
    JQ_REQUIRE(max_tiles >= 0, JQ_EINVAL, "negative max_tiles");
    GroupedArgs g;
    g.tile_expert = tile_expert; g.tile_row0 = tile_row0; g.num_tiles = num_tiles; g.expert_offsets = expert_offsets;
    g.bits_tab = bits_tab; g.codes_tab = codes_tab; g.scales_tab = scales_tab; g.biases_tab = biases_tab;
    g.max_tiles = max_tiles;
    g.tile_m = tile_m;
    return qgemm_dispatch(x_sorted, act_dtype, max_rows, ldx, nullptr, nullptr, nullptr, sidecar_dtype, N, K, bits,
                          group_size, y_sorted, act_dtype, ldy, &g, (cudaStream_t)stream);
}

int jq_moe_gate_up_swiglu(const void* x_sorted, int act_dtype, int64_t max_rows, int64_t ldx,
                          const int32_t* expert_offsets, const int32_t* tile_expert, const int32_t* tile_row0,
                          const int32_t* num_tiles, int64_t max_tiles, int tile_m, const uint32_t* const* gate_codes,
                          const void* const* gate_scales, const void* const* gate_biases,
                          const uint32_t* const* up_codes, const void* const* up_scales, const void* const* up_biases,
                          int sidecar_dtype, int64_t N, int64_t K, int bits, int group_size, const float* weights,
                          const int32_t* order, float limit, void* h, int64_t ldh, jq_stream_t stream) {
    using namespace jq;
    JQ_REQUIRE(tile_m == 128 || tile_m == 192 || tile_m == 256, JQ_EINVAL, "tile_m must be 128, 192 or 256");
    JQ_REQUIRE(expert_offsets && tile_expert && tile_row0 && num_tiles && gate_codes && gate_scales && gate_biases &&
               up_codes && up_scales && up_biases, JQ_EINVAL, "null pointer");
    JQ_REQUIRE(weights == nullptr || order != nullptr, JQ_EINVAL, "routing weights need the sort order");
    JQ_REQUIRE(max_tiles >= 0, JQ_EINVAL, "negative max_tiles");
    GroupedArgs g;
    g.tile_expert = tile_expert; g.tile_row0 = tile_row0; g.num_tiles = num_tiles; g.expert_offsets = expert_offsets;
    g.bits_tab = nullptr; g.codes_tab = gate_codes; g.scales_tab = gate_scales; g.biases_tab = gate_biases;
    g.max_tiles = max_tiles;
    g.tile_m = tile_m;
    g.codes_tab2 = up_codes; g.scales_tab2 = up_scales; g.biases_tab2 = up_biases;
    g.wts = weights; g.order = order; g.lim = limit;
    return qgemm_dispatch(x_sorted, act_dtype, max_rows, ldx, nullptr, nullptr, nullptr, sidecar_dtype, N, K, bits,
                          group_size, h, act_dtype, ldh, &g, (cudaStream_t)stream);
}

}  // extern "C"
