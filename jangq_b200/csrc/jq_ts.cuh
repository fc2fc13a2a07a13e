// Weights as the A operand of tcgen05.mma in tensor memory: the pieces shared by the prefill GEMM (jq_qgemm.cu) and
// the small-batch mat-vec (jq_qgemv_ts.cu) -- register expansion of packed codes into 16-bit floats, the code loaders,
// MMA and cluster wrappers.
#pragma once

#include <cmath>

#include "jq_mma.cuh"
#include "jq_tc.cuh"

namespace jq {

template <typename AT> __host__ __device__ constexpr uint32_t umma_fmt();
template <> __host__ __device__ constexpr uint32_t umma_fmt<__nv_bfloat16>() { return 1u; }
template <> __host__ __device__ constexpr uint32_t umma_fmt<__half>() { return 0u; }

// A (tensor memory) and B both K-major, no negate, dense, D = f32, M = 128; N is added at run time
template <typename AT>
__device__ __forceinline__ uint32_t umma_idesc_ts(int n) {
    return (1u << 4) | (umma_fmt<AT>() << 7) | (umma_fmt<AT>() << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}

// ---- packed 16-bit float helpers --------------------------------------------------------------------
// An integer v < 2^(MANT+1) read as the bits of a 16-bit float is v * 2^-DEN: subnormals and the first normal
// binade share one spacing.  So a masked code field IS the code times a power of two, and
// fma(field, s * 2^(DEN-p), bias) = rn(q*s + bias) for a code at bit p -- one AND and one FMA per two weights, no
// exponent to insert and subtract.  It holds while s * 2^(DEN-p) is finite (|s| < LIM * 2^p).
template <typename AT> struct P2;
template <> struct P2<__nv_bfloat16> {
    static constexpr int TOP = 8;            // bits of v
    static constexpr float LIM = 0x1p-5f;    // |s| * 2^133 < 2^128
    // s * 2^(133-p), exact
    template <int P> __device__ static __forceinline__ float lift(float s) { return s * 0x1p100f * (0x1p33f / (float)(1 << P)); }
    __device__ static __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
        uint32_t r;
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
        return r;
    }
    __device__ static __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
        uint32_t r;
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
        return r;
    }
};
template <> struct P2<__half> {
    static constexpr int TOP = 11;
    static constexpr float LIM = 0x1.ff8p-9f;     // |s| * 2^24 <= 65504
    template <int P> __device__ static __forceinline__ float lift(float s) { return s * (0x1p24f / (float)(1 << P)); }
    __device__ static __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
        uint32_t r;
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
        return r;
    }
    __device__ static __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
        uint32_t r;
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
        return r;
    }
};

// 32 bits of a row's code stream starting at bit A (negative A: zero-filled below bit 0)
template <int NWORDS, int A>
__device__ __forceinline__ uint32_t stream_at(const uint32_t (&u)[NWORDS]) {
    if constexpr (A < 0) return u[0] << (-A);
    else if constexpr (A % 32 == 0) return u[A / 32];
    else if constexpr (A / 32 + 1 < NWORDS) return __funnelshift_r(u[A / 32], u[A / 32 + 1], A % 32);
    else return u[A / 32] >> (A % 32);
}

// Weights J and J+1 of a 64-code unit: rn(q*s + bias) in the activation type, packed; any finite or non-finite s.
// s2 = (s, s), b2 = (bias, bias); s/bias are the same values in f32.  The code stands at bit 0 of the mantissa, so the
// scale is used as it is (shifted up to the mantissa's top it needs s * 2^-k, which underflows for small f16 scales).
template <typename AT, int BITS, int J>
__device__ __forceinline__ uint32_t dequant_pair(const uint32_t (&u)[2 * BITS], uint32_t s2, uint32_t b2, float s,
                                                 float bias) {
    if constexpr (BITS <= Act<AT>::MANT) {
        constexpr uint32_t MASK = ((1u << BITS) - 1u) * 0x00010001u;
        const uint32_t lo = stream_at<2 * BITS, J * BITS>(u);
        const uint32_t hi = stream_at<2 * BITS, (J + 1) * BITS>(u);
        const uint32_t v = and_or(prmt(lo, hi, 0x5410), MASK, Act<AT>::MAGIC);   // 2^MANT + q, twice
        const uint32_t q2 = P2<AT>::sub(v, Act<AT>::MAGIC);                       // q, exact
        return P2<AT>::fma(q2, s2, b2);                                           // one rounding
    } else {
        // codes wider than the mantissa (8-bit with bf16): exact q in f32 through the 2^23 trick
        static_assert(BITS == 8, "only 8-bit codes take the f32 route");
        const uint32_t word = u[J / 4];
        const float q0 = __uint_as_float(prmt(word, 0x4B000000u, 0x7540u | (uint32_t)(J % 4))) - 8388608.0f;
        const float q1 = __uint_as_float(prmt(word, 0x4B000000u, 0x7540u | (uint32_t)(J % 4 + 1))) - 8388608.0f;
        return Act<AT>::pack_hi(fmaf(q0, s, bias), fmaf(q1, s, bias));
    }
}

// pairs 2*J.. of half a k-block (32 codes) through dequant_pair
template <typename AT, int BITS, int J0, int J>
__device__ __forceinline__ void dequant_general(const uint32_t (&u)[2 * BITS], uint32_t sp2, uint32_t b2, float s, float bias,
                                                uint32_t (&out)[32]) {
    if constexpr (J < 16) {
        out[J0 + J] = dequant_pair<AT, BITS, 2 * (J0 + J)>(u, sp2, b2, s, bias);
        dequant_general<AT, BITS, J0, J + 1>(u, sp2, b2, s, bias, out);
    }
}

// largest |s| the fast form below takes
template <typename AT, int BITS>
__host__ __device__ constexpr float fast_limit() {
    constexpr bool bf = P2<AT>::TOP == 8;
    if (BITS == 8) return bf ? P2<AT>::LIM : INFINITY;                       // f16: exponent inserted by the byte permute
    if (BITS == 4) return bf ? P2<AT>::LIM : P2<AT>::LIM * 16.f;             // lowest field at bit 0 / bit 4
    if (BITS == 2) return bf ? P2<AT>::LIM * 16.f : P2<AT>::LIM * 64.f;      // bit 4 / bit 6
    return P2<AT>::LIM * (float)(1 << (P2<AT>::TOP - BITS));                 // top-aligned field
}

// pairs J.. of a 3-, 5- or 6-bit row (H halves of a 64-code unit)
template <typename AT, int BITS, int H, int J>
__device__ __forceinline__ void dequant_stream(const uint32_t (&u)[H * BITS], uint32_t sp, uint32_t b2, uint32_t (&out)[16 * H]) {
    if constexpr (J < 16 * H) {
        constexpr int TGT = P2<AT>::TOP - BITS;
        constexpr uint32_t MASK = (((1u << BITS) - 1u) << TGT) * 0x00010001u;
        const uint32_t lo = stream_at<H * BITS, 2 * J * BITS - TGT>(u);
        const uint32_t hi = stream_at<H * BITS, (2 * J + 1) * BITS - TGT>(u);
        out[J] = P2<AT>::fma(prmt(lo, hi, 0x5410) & MASK, sp, b2);
        dequant_stream<AT, BITS, H, J + 1>(u, sp, b2, out);
    }
}

// 32*H codes of one row -> 16*H registers of two weights in k order, every weight rn(q*s + bias).
// Fields of a word are taken two at a time, 16 bits apart, where they stand (or after one shift of the word), and the
// results are put in k order by a byte permute: 13 instructions per 8 codes at 4 bits, 27 per 16 at 2 bits, 4 per 4 at
// 8 bits (24, 48 and 14 with the exponent insert + subtract of dequant_pair).  EXACT: s is a power of two and b2 zero, so
// nothing is rounded, and the 1024 that an 8-bit code of float16 carries leaves in the multiply-add.
template <typename AT, int BITS, int H, bool EXACT = false>
__device__ __forceinline__ void dequant_fast(const uint32_t (&u)[H * BITS], float s, uint32_t b2, uint32_t (&out)[16 * H]) {
    using A = Act<AT>;
    using P = P2<AT>;
    constexpr bool bf = P::TOP == 8;
    if constexpr (BITS == 8) {
        if constexpr (bf) {
            const float l = P::template lift<0>(s);
            const uint32_t sp = A::pack_hi(l, l);
#pragma unroll
            for (int i = 0; i < 8 * H; ++i) {
                out[2 * i] = P::fma(prmt(u[i], 0u, 0x4140), sp, b2);
                out[2 * i + 1] = P::fma(prmt(u[i], 0u, 0x4342), sp, b2);
            }
        } else {
            const uint32_t sp = A::pack_hi(s, s), off = A::pack_hi(-1024.0f * s, -1024.0f * s);
#pragma unroll
            for (int i = 0; i < 8 * H; ++i) {      // 0x64qq = 1024 + q
                const uint32_t v0 = prmt(u[i], 0x64646464u, 0x4140), v1 = prmt(u[i], 0x64646464u, 0x4342);
                out[2 * i] = EXACT ? P::fma(v0, sp, off) : P::fma(P::sub(v0, A::MAGIC), sp, b2);
                out[2 * i + 1] = EXACT ? P::fma(v1, sp, off) : P::fma(P::sub(v1, A::MAGIC), sp, b2);
            }
        }
    } else if constexpr (BITS == 4) {
        const float l0 = P::template lift<0>(s), l4 = P::template lift<4>(s);
        const uint32_t sp0 = A::pack_hi(l0, l0), sp4 = A::pack_hi(l4, l4);
#pragma unroll
        for (int i = 0; i < 4 * H; ++i) {
            const uint32_t w = u[i];
            uint32_t f0, f1, f2, f3;            // codes (j, j + 4)
            if constexpr (bf) {
                const uint32_t w8 = w >> 8;
                f0 = P::fma(w & 0x000F000Fu, sp0, b2); f1 = P::fma(w & 0x00F000F0u, sp4, b2);
                f2 = P::fma(w8 & 0x000F000Fu, sp0, b2); f3 = P::fma(w8 & 0x00F000F0u, sp4, b2);
            } else {
                f0 = P::fma((w << 4) & 0x00F000F0u, sp4, b2); f1 = P::fma(w & 0x00F000F0u, sp4, b2);
                f2 = P::fma((w >> 4) & 0x00F000F0u, sp4, b2); f3 = P::fma((w >> 8) & 0x00F000F0u, sp4, b2);
            }
            out[4 * i] = prmt(f0, f1, 0x5410); out[4 * i + 1] = prmt(f2, f3, 0x5410);
            out[4 * i + 2] = prmt(f0, f1, 0x7632); out[4 * i + 3] = prmt(f2, f3, 0x7632);
        }
    } else if constexpr (BITS == 2) {
        constexpr int PA = bf ? 4 : 6;
        constexpr uint32_t MA = (3u << PA) * 0x00010001u, MB = MA << 2;
        const float la = P::template lift<PA>(s), lb = P::template lift<PA + 2>(s);
        const uint32_t spa = A::pack_hi(la, la), spb = A::pack_hi(lb, lb);
#pragma unroll
        for (int i = 0; i < 2 * H; ++i) {
            const uint32_t w = u[i];
            uint32_t f[8];                      // codes (j, j + 8)
#pragma unroll
            for (int j = 0; j < 4; ++j) {       // codes 2j and 2j+1 to bits PA and PA+2
                const int sh = PA - 4 * j;
                const uint32_t v = sh >= 0 ? w << sh : w >> -sh;
                f[2 * j] = P::fma(v & MA, spa, b2);
                f[2 * j + 1] = P::fma(v & MB, spb, b2);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                out[8 * i + j] = prmt(f[2 * j], f[2 * j + 1], 0x5410);
                out[8 * i + 4 + j] = prmt(f[2 * j], f[2 * j + 1], 0x7632);
            }
        }
    } else {
        const float l = P::template lift<P::TOP - BITS>(s);
        dequant_stream<AT, BITS, H, 0>(u, A::pack_hi(l, l), b2, out);
    }
}

// The exact form: codes times a power of two that both types represent; the power of two goes back into the scale.
template <typename AT> struct TsExact;
template <> struct TsExact<__nv_bfloat16> { static constexpr float C = 0x1p-6f, POST = 0x1p6f; };
template <> struct TsExact<__half> { static constexpr float C = 0x1p-9f, POST = 0x1p9f; };

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One lane of a converged warp, the same one every time.  Unlike `lane == 0` it tells the compiler that a single thread
// runs the block, so descriptors and barrier addresses stay in uniform registers.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// Bounded wait on a phase parity that sleeps in hardware (a suspend-time hint of 20 us): a dozen warps of a CTA wait at
// any time, and polling loops take issue slots and barrier-unit throughput from the warps that work -- with the short
// default hint the loops between two waits ran at 10 to 20 cycles per instruction.  Gives up after a second and at least
// 4096 wake-ups (a poll count alone runs out under a profiler, time alone under time-slicing).
__device__ __forceinline__ bool ts_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    unsigned long long t0 = 0;
    for (uint32_t i = 0;; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(20000u)
            : "memory");
        if (done) return true;
        const unsigned long long now = wall_ns();
        if (t0 == 0) t0 = now;
        else if (i >= 4096u && now - t0 > MBAR_WAIT_NS) return false;
    }
}
// arrives on `bar` when all cp.async copies this thread has issued so far have landed (counts as one of the
// barrier's expected arrivals)
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 16 consecutive columns, this warp's lane quarter
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
template <int W>
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[W]) {
    static_assert(W == 8 || W == 16, "8 or 16 columns");
    if constexpr (W == 8) tmem_ld8(taddr, v); else tmem_ld16(taddr, v);
}

// ---- packed codes through shared memory -------------------------------------------------------------------
// k-blocks (64 codes) per stage and bytes per row and stage: 48, 64 or 80.  Rows of 64 bytes have their 16-byte chunks
// XOR-swizzled by the row so that eight rows read together fall into eight bank groups; rows of 48 and 80 bytes do so
// as they are.
template <int BITS> struct CodeStage {
    static constexpr int CKB = BITS == 2 ? 4 : (BITS == 6 || BITS == 8) ? 1 : 2;
    static constexpr int RB = CKB * 8 * BITS;
};
template <int CPR> __device__ __forceinline__ int code_chunk(int chunk, int row) {
    return CPR == 4 ? (chunk ^ ((row >> 1) & 3)) : chunk;
}

// Scales and biases travel with the codes: a chunk of four k-blocks (8 bytes per row at group size 64, 4 at 128) is
// copied with the first code stage of the chunk into a ring of as many chunks as there are code stages, so a slot is
// free again when its code stage is (every chunk has at least one).  Read straight from global memory by the
// dequantizers they cost more than the codes: every load touched 32 lines for 8 bytes of each, once per group of warps.
//   mode 0: not staged (rows not aligned for a copy, groups of 32): the dequantizers load them;
//   1: one 8-byte copy per row, 2: two 4-byte copies (group size 64);  3: one 4-byte copy (group size 128)
struct SideSrc {
    const void *scales, *biases, *scales2, *biases2;      // ..2: the second matrix of a pair tile
    int64_t G;
    int mode;
};
__host__ __device__ inline int side_mode(const void* scales, const void* biases, int64_t G, int gs) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(biases);
    if (gs == 64) return G % 4 == 0 && at % 8 == 0 ? 1 : (G % 2 == 0 && at % 4 == 0 ? 2 : 0);
    return gs == 128 && G % 2 == 0 && at % 4 == 0 ? 3 : 0;
}
constexpr int SIDE_SLOT = 2 * 128 * 8;                    // bytes of a chunk: scales [128][4], then biases
// base + row * pitch with a 64-bit product (rows of 2^31 bytes are taken, so 128 of them do not fit 32 bits), where it
// stands: computed ahead, the addresses would take two registers each for the length of a loop
__device__ __forceinline__ const uint8_t* row_at(const uint8_t* base, uint32_t row, uint32_t pitch) {
    uint64_t p;
    asm volatile("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p) : "r"(row), "r"(pitch), "l"(base));
    return reinterpret_cast<const uint8_t*>(p);
}
template <int N> __device__ __forceinline__ void cp_async_small(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}

// The loader warps' loop: 64 lanes (l) copy nst stages of 128 rows, starting at stage st0 of the rows, into a ring
// of CD stages; consecutive lanes take consecutive 16-byte chunks of a row, completion is counted on cfull (64
// arrivals).  A lane's chunks keep their rows and columns from stage to stage, so only one multiply-add and one copy per
// chunk are left in the loop (a warp alone on its scheduler issues an instruction every ~6 cycles;
// with the addresses computed per stage the loaders set the pace of the whole CTA).  (buf, phase) is the ring position,
// (0, 1) at the start: the first pass finds every stage empty.  Returns false when a wait ran out; the caller waits for
// the copies in flight.
//   codes2 (PAIR): the tile is rows [n0, n0 + 64) of two matrices, the second one's behind the first one's
template <int BITS, int CD, bool PAIR = false>
__device__ __forceinline__ bool load_codes(const uint32_t* codes, int64_t n0, int64_t N, int64_t K, int st0, int nst,
                                           uint8_t* sC, uint64_t* cfull, uint64_t* cempty, int l, int& buf,
                                           uint32_t& phase, const SideSrc& side, uint8_t* sSide, int& slot,
                                           const uint32_t* codes2 = nullptr) {
    constexpr int RB = CodeStage<BITS>::RB, CPR = RB / 16;
    constexpr int NCH = 128 * CPR / 64;                               // chunks per lane and stage
    const uint32_t rowbytes = (uint32_t)(K * BITS / 8);
    const int last = (int)min((int64_t)((PAIR ? 64 : 128) - 1), N - 1 - n0);       // rows past N repeat the last one
    const uint8_t* src = reinterpret_cast<const uint8_t*>(codes) + n0 * (int64_t)rowbytes + (int64_t)st0 * RB;
    const int64_t second = PAIR ? reinterpret_cast<const uint8_t*>(codes2) - reinterpret_cast<const uint8_t*>(codes) : 0;
    uint32_t row[NCH];
#pragma unroll
    for (int j = 0; j < NCH; ++j) row[j] = (uint32_t)min(PAIR ? (l + 64 * j) / CPR & 63 : (l + 64 * j) / CPR, last);
    // CPR == 4: the chunks of a lane are 16 rows apart and keep their (swizzled) column; otherwise the columns of chunk j
    // and j + CPR are the same, and the stage holds the chunks in order
    constexpr int NCOL = CPR == 4 ? 1 : CPR;
    const uint8_t* srcc[NCOL];
#pragma unroll
    for (int j = 0; j < NCOL; ++j) srcc[j] = src + (l + 64 * j) % CPR * 16;
    const uint32_t dst0 = smem_u32(sC) + (uint32_t)(CPR == 4 ? l / 4 * RB + code_chunk<CPR>(l & 3, l / 4) * 16 : l * 16);
    // sidecars: this lane's rows l and l + 64 (of the second matrix in a pair tile)
    constexpr int CKB = CodeStage<BITS>::CKB;
    const int64_t r0 = n0 + min(l, last), r1 = PAIR ? r0 : n0 + min(l + 64, last);
    const int chunk_bytes = side.mode == 3 ? 4 : 8;
    const char* sp[4];
    sp[0] = reinterpret_cast<const char*>(side.scales) + r0 * side.G * 2;
    sp[1] = reinterpret_cast<const char*>(PAIR ? side.scales2 : side.scales) + r1 * side.G * 2;
    sp[2] = reinterpret_cast<const char*>(side.biases) + r0 * side.G * 2;
    sp[3] = reinterpret_cast<const char*>(PAIR ? side.biases2 : side.biases) + r1 * side.G * 2;
    int soffb = st0 * CKB / 4 * chunk_bytes;                                 // byte offset of the chunk in a row
    int rem = (int)rowbytes - st0 * RB;                                     // bytes of a row left from this stage on
    bool ok = true;
    for (int st = 0; st < nst; ++st) {
        ok = __all_sync(0xFFFFFFFFu, ts_wait(cempty + buf, phase));
        if (!ok) break;
        const uint32_t d = dst0 + (uint32_t)(buf * (128 * RB));
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
            const uint32_t dj = d + (uint32_t)(j * 1024);
            const uint8_t* s = row_at(srcc[j % NCOL], row[j], rowbytes);
            if (PAIR && j >= NCH / 2) s += second;
            const int col = CPR == 4 ? (l & 3) : (l + 64 * j) % CPR;
            if (col * 16 < rem) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dj), "l"(s) : "memory");
        }
        if (((st0 + st) * CKB) % 4 == 0) {             // a chunk has its slot whether it is staged or not: the mode may
            if (side.mode != 0) {                      // change from tile to tile, and the dequantizers count every chunk
                const uint32_t sd = smem_u32(sSide) + (uint32_t)(slot * SIDE_SLOT + l * 8);
#pragma unroll
                for (int i = 0; i < 4; ++i) {                              // scales of both rows, then biases
                    const uint32_t di = sd + (uint32_t)(i * 64 * 8);
                    if (side.mode == 1) {
                        cp_async_small<8>(di, sp[i] + soffb);
                    } else {
                        cp_async_small<4>(di, sp[i] + soffb);
                        if (side.mode == 2 && soffb + 4 < (int)side.G * 2) cp_async_small<4>(di + 4, sp[i] + soffb + 4);
                    }
                }
            }
            soffb += chunk_bytes;
            if (++slot == CD) slot = 0;
        }
        cp_async_arrive(cfull + buf);
#pragma unroll
        for (int j = 0; j < NCOL; ++j) srcc[j] += RB;
        rem -= RB;
        if (++buf == CD) { buf = 0; phase ^= 1u; }
    }
    return ok;
}

// 32 codes (half h of k-block kbi of a stage) of row r, whose staged bytes start at crow
template <int BITS, int CPR>
__device__ __forceinline__ void load_codes32(const uint8_t* crow, int r, int kbi, int h, uint32_t (&cur)[BITS]) {
    const int off = kbi * 8 * BITS + h * 4 * BITS;
    if constexpr (BITS % 4 == 0) {
#pragma unroll
        for (int w = 0; w < BITS / 4; ++w) {
            const uint4 v = reinterpret_cast<const uint4*>(crow)[code_chunk<CPR>((off >> 4) + w, r)];
            cur[4 * w] = v.x; cur[4 * w + 1] = v.y; cur[4 * w + 2] = v.z; cur[4 * w + 3] = v.w;
        }
    } else if constexpr (BITS % 2 == 0) {
#pragma unroll
        for (int w = 0; w < BITS / 2; ++w) {
            const int o = off + 8 * w;
            const uint2 v = *reinterpret_cast<const uint2*>(crow + code_chunk<CPR>(o >> 4, r) * 16 + (o & 8));
            cur[2 * w] = v.x; cur[2 * w + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int w = 0; w < BITS; ++w) cur[w] = *reinterpret_cast<const uint32_t*>(crow + off + 4 * w);
    }
}

__device__ __forceinline__ void ts_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f32x4(const float* own, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(own)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

}  // namespace jq
