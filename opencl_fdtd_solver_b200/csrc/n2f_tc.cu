// Near-to-far contraction on the tensor cores (tcgen05, TMEM accumulators).
//
// The far-field integrals of the reference (farfield_accumulate_nl,
// dft_farfield.cl:372-556) are, per direction r̂_o, frequency f and face,
//   NL_face(o, c) = Σ_{p,q} e^{jk r̂_o·r'_{pq}} cur[p][q][c],
// with k = 2πf/c0, c over the face's four tangential currents (J_b, J_c, M_b,
// M_c; b, c the in-face axes) and r'_{pq} = x_n n̂ + (o_p + p·h) b̂ + (o_q + q·h) ĉ.
// The phase separates: e^{jk r̂·r'} = C(o)·u_p(o)·v_q(o) with
//   u_p = e^{j2π γ_p p}, v_q = e^{j2π γ_q q}, γ = f·h·r̂/c0 (turns per sample),
//   C   = e^{j2π f (r̂_n x_n + r̂_b o_p + r̂_c o_q)/c0}.
// So T[o][q][c] = Σ_p u_p(o)·cur[p][q][c] is a complex GEMM (M = directions,
// K = p, N = (q, c)), and NL_face(o, c) = C(o)·Σ_q v_q(o)·T[o][q][c] is a
// row-wise reduction of its output.  In real form K interleaves (Re, Im) of u_p and N
// those of T, with B = [[Br, Bi], [−Bi, Br]] per (p, (q, c)).
//
// Split-BF16 folds both sums about the middle of the face: with θ = 2πγ(i + s) the
// offset from it of the i-th pair of samples (s = 0 for an odd count, whose middle
// sample is a pair with itself, 1/2 for an even one),
//   Σ_p u_p x_p = Σ_i cos θ_i (x⁺_i + x⁻_i) + j sin θ_i (x⁺_i − x⁻_i),
// a real matrix of directions × (cos, sin) against the sums and differences of the
// currents: half the products of the complex GEMM (the phases of the other half of
// the face are conjugates), half its operand bytes and half its phases.  K is then
// (i, cos | sin), N (q pair, even | odd, c, Re | Im), and the reduction
// Σ_q cos·T_even + j sin·T_odd.  The sums and differences are formed in float64 and
// rounded once to float32 before the split.  TF32 stays unfolded: its 2^-11 rounding
// of the operands is its result's error, and folding would round other operands.
//
// Kernel k_n2f_tc: one CTA per (128-direction tile, face_group faces, frequency),
// 6 + 4·NGRP warps.
//   * warp 0: B producer.  B (currents, N × K) is pre-packed by k_n2f_pack in
//     the K-major core-matrix layout, one contiguous 32 KB block per
//     (n tile, K step) in both modes, and moved with one cp.async.bulk per
//     stage (no tensor map, no multicast).
//   * warp 1: issues tcgen05.mma (kind::f16 BF16: hi·hi + hi·lo + lo·hi, or
//     kind::tf32), MPS K groups per stage (2 BF16, 4 TF32), into the two 128 × 128
//     halves of a 128 × 256 FP32 accumulator in TMEM: BATCH stages for the one half,
//     then the same stages for the other, so that one half is read while the other
//     is written and the MMAs never wait for the epilogue.
//   * warps 2-5 and 10 onwards: A (phases, 128 × K), generated per K step, one
//     direction per thread, NGRP groups on interleaved stages: a float64 rotation
//     times PS (16) precomputed float phases, split into bf16 hi + lo (or rounded
//     to tf32).
//   * warps 6-9: epilogue.  Each thread owns one TMEM lane (one direction),
//     reads it with tcgen05.ld and folds Σ_q into four complex sums.
//
// What bounds it.  6 faces of 320 × 320 samples, 8 frequencies, 65,341 directions:
// split-BF16 23.3 -> 11.7 ms, 1.54e13 operations at 1.32 PFLOP/s of the 1.65 that a plain
// BF16 GEMM reaches, so the tensor cores and their power (the fold saved 6.2 ms, the
// converged issue 5.2 ms).  TF32 18.0 -> 16.2 ms, with the stream of B from L2 at about
// 9 TB/s.  89 × 89 samples, 16,471 directions: split-BF16 0.92 -> 0.53 ms, of which
// several faces per CTA 0.1; TF32 0.83 -> 0.68 ms.
//
// Every mbarrier wait is bounded in wall time (Params::wait_ns, 0.2 s by
// default; fdtd_set_wait_budget lowers it); on timeout the kernel raises bit 1
// of the device error flag, stops issuing, drains its own copies and MMAs (with
// the default bound), frees TMEM and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "launch_count.cuh"
#include "n2f.cuh"

namespace fdtd {
namespace n2f {

__device__ int g_n2f_error;

constexpr int NGRP = 2;  // phase-generator groups of four warps, on stages g % NGRP
constexpr int NTHREADS = (6 + 4 * NGRP) * 32;  // B loader, MMA issuer, epilogue, phase groups
constexpr int MAX_STAGE = 16;
constexpr int HN = BN / 2;          // columns of an accumulator half
constexpr int BATCH = 3;            // stages issued for one half before the other
constexpr int ATM_NST = 6;          // stages when A is in tensor memory (6 x 32 KB of B)
constexpr uint32_t ATM_ACOL = 256;  // first TMEM column of the A ring (32 per stage)
constexpr double C0 = 299792458.0;

constexpr bool folded(int mode) { return mode == FDTD_N2F_BF16X3; }

template <int MODE>
struct Cfg;
// A stage holds KR real K values: NCH 16-byte K chunks per operand row, MPS
// MMAs of two chunks each (K = 16 BF16 or 8 TF32 per MMA).  Wider stages
// amortise the per-stage barrier round trips over more MMAs.
template <>
struct Cfg<FDTD_N2F_BF16X3> {
    static constexpr int KR = 32;                 // real K per stage
    static constexpr int PS = KR / 2;             // complex samples p per stage
    static constexpr int NCH = KR / 8;            // 16-byte chunks per row
    static constexpr int MPS = NCH / 2;           // MMA K groups per stage
    static constexpr int A_BYTES = BM * KR * 2;   // one of hi / lo
    static constexpr int B_BYTES = BN * KR * 2;   // one of hi / lo
    static constexpr int STAGE = 2 * A_BYTES + 2 * B_BYTES;
    static constexpr int B_COPY = 2 * B_BYTES;
    static constexpr int NST = (192 * 1024) / STAGE;  // 192 KB of stages: one CTA per SM
    static constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(HN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};
template <>
struct Cfg<FDTD_N2F_TF32> {
    static constexpr int KR = 32;
    static constexpr int PS = KR / 2;
    static constexpr int NCH = KR / 4;
    static constexpr int MPS = NCH / 2;
    static constexpr int A_BYTES = BM * KR * 4;
    static constexpr int B_BYTES = BN * KR * 4;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int B_COPY = B_BYTES;
    static constexpr int NST = (192 * 1024) / STAGE;
    static constexpr uint32_t IDESC =
        (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(HN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};
static_assert(ATM_NST <= MAX_STAGE && ATM_ACOL + 32 * ATM_NST <= 512 && ATM_ACOL >= BN,
              "the tensor-memory A ring must fit beside one accumulator in 512 columns");
static_assert(Cfg<FDTD_N2F_BF16X3>::NST <= MAX_STAGE && Cfg<FDTD_N2F_TF32>::NST <= MAX_STAGE,
              "stage ring larger than the barrier arrays");

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Non-blocking probe of a phase (no suspension), used by a zero wait budget.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
// Issued by the lane with `one` set.  The instruction is predicated and not branched
// around, so that the warp stays converged and the operands in uniform registers: from
// inside a one-lane branch each MMA took 136-185 cycles, against the 64 it needs.
template <int MODE>
__device__ __forceinline__ void mma(bool one, uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
    if (MODE == FDTD_N2F_BF16X3) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "setp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
            "l"(a), "l"(b), "r"(Cfg<MODE>::IDESC), "r"(acc), "r"((uint32_t)one)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "setp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
            "l"(a), "l"(b), "r"(Cfg<MODE>::IDESC), "r"(acc), "r"((uint32_t)one)
            : "memory");
    }
}
// The same MMA with A (M x K, one row per TMEM lane, K packed along columns)
// read from tensor memory instead of shared memory.
template <int MODE>
__device__ __forceinline__ void mma_ts(bool one, uint32_t d, uint32_t a, uint64_t b, uint32_t acc) {
    if (MODE == FDTD_N2F_BF16X3) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "setp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
            "r"(a), "l"(b), "r"(Cfg<MODE>::IDESC), "r"(acc), "r"((uint32_t)one)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "setp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
            "r"(a), "l"(b), "r"(Cfg<MODE>::IDESC), "r"(acc), "r"((uint32_t)one)
            : "memory");
    }
}

// Each thread of the warp writes 16 consecutive 32-bit columns of its own lane.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void mma_commit(bool one, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar), "r"((uint32_t)one)
        : "memory");
}
// 64 consecutive columns of the thread's lane, complete on return.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&v)[64]) {
    uint32_t r[64];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {"
        "%0, %1, %2, %3, %4, %5, %6, %7, "
        "%8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, "
        "%24, %25, %26, %27, %28, %29, %30, %31, "
        "%32, %33, %34, %35, %36, %37, %38, %39, "
        "%40, %41, %42, %43, %44, %45, %46, %47, "
        "%48, %49, %50, %51, %52, %53, %54, %55, "
        "%56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]),
          "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]),
          "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]),
          "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
          "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]),
          "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
          "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]),
          "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}

// K-major, no-swizzle shared-memory matrix descriptor: core matrices of 8 rows
// x 16 bytes, SBO between 8-row groups, LBO between the two 16-byte K chunks.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version for tcgen05
    return d;
}

__device__ __forceinline__ float tf32_rna(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// e^{j2π t} for t = g·n, reduced to [-1/2, 1/2] turns in float64 first.
__device__ __forceinline__ float2 phase_turns(double g, double n) {
    double t = g * n;
    t = t - rint(t);
    float s, c;
    sincospif(2.0f * (float)t, &s, &c);
    return make_float2(c, s);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// e^{j2π t} for t = g·n in float64 (reduction in turns, then sincospi).
__device__ __forceinline__ double2 zphase_turns(double g, double n) {
    double t = g * n;
    t = t - rint(t);
    double s, c;
    sincospi(2.0 * t, &s, &c);
    return make_double2(c, s);
}

__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait shared by all roles: gives up after `budget_ns` of wall time
// (the launch's Params::wait_ns, 0.2 s unless a caller lowered it), when another
// role of this CTA aborted, or when another CTA raised the error flag.  Returns
// false in all three cases (and raises the flags on a timeout).  A zero budget
// gives up at once unless the phase has already completed (non-blocking probe).
constexpr uint64_t WAIT_NS = 200000000ull;  // 0.2 s; a normal wait is microseconds
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                         uint64_t budget_ns) {
    if (budget_ns == 0) {
        if (mbar_test_wait(bar, parity)) return true;
        *abort_flag = 1;
        atomicOr(&g_n2f_error, 1);
        return false;
    }
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gtimer();
    uint32_t it = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++it & 255u) == 0) {
            if (*abort_flag || *(volatile int *)&g_n2f_error) {
                *abort_flag = 1;
                return false;
            }
            if (gtimer() - t0 > budget_ns) {
                *abort_flag = 1;
                atomicOr(&g_n2f_error, 1);
                return false;
            }
        }
    }
    return true;
}

// Drain wait: bounded by time only (used before the CTA exits).
__device__ __forceinline__ void drain_bar(uint32_t bar, uint32_t parity) {
    const uint64_t t0 = gtimer();
    while (!mbar_try_wait(bar, parity) && gtimer() - t0 < WAIT_NS) {
    }
}

struct Smem {
    uint64_t full_b[MAX_STAGE], full_a[MAX_STAGE], empty[MAX_STAGE];
    uint64_t acc_full[2], acc_empty[2];  // per accumulator half
    uint64_t drain;
    uint32_t tmem;
    int abort_flag;
};

// ATM: the A operand (phases) lives in tensor memory: the generators write it
// with tcgen05.st, one row (direction) per TMEM lane, and the MMAs read it from
// there, so shared memory carries only B (its copies and the MMAs' B reads).
// TMEM holds the two halves of a 128 x 256 accumulator (columns 0-255) and, with
// ATM, the A ring (columns 256-511, 32 per stage); without it A is in the
// shared-memory stages.
template <int MODE, bool ATM>
__global__ void __launch_bounds__(NTHREADS, 1) k_n2f_tc(Params P) {
    using C = Cfg<MODE>;
    constexpr bool FOLD = folded(MODE);
    constexpr int NSTAGE = ATM ? ATM_NST : C::NST;
    constexpr int SSTAGE = ATM ? C::B_COPY : C::STAGE;  // shared-memory bytes per stage
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *stages = smem_raw;
    Smem *sm = reinterpret_cast<Smem *>(smem_raw + NSTAGE * SSTAGE);
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform
    const int mt = blockIdx.x, fr = blockIdx.z;
    // the faces of this CTA, one after the other through the same pipeline
    const int f0 = blockIdx.y * P.face_group, f1 = min(f0 + P.face_group, P.nfaces);
    const double freq = P.freqs[fr];
    volatile int *abort_flag = &sm->abort_flag;

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(smem_u32(&sm->full_b[s]), 1);
            mbar_init(smem_u32(&sm->full_a[s]), BM);
            mbar_init(smem_u32(&sm->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&sm->acc_full[b]), 1);
            mbar_init(smem_u32(&sm->acc_empty[b]), 128);
        }
        mbar_init(smem_u32(&sm->drain), 1);
        sm->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&sm->tmem), 2 * BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm->tmem, 0);  // warp-uniform

    if (warp == 0) {
        // ---- B producer: one bulk copy per stage
        if (lane == 0) {
            int issued = 0;
            bool ok = true;
            for (int fi = f0; fi < f1 && ok; ++fi) {
                const Face &F = P.face[fi];
                const unsigned char *src = P.btiles + F.b_off + (int64_t)fr * F.b_freq_stride;
                const int total = F.nt * F.ks;
                for (int q = 0; q < total; ++q) {
                    const int g = issued, s = g % NSTAGE;
                    if (g >= NSTAGE && !wait_bar(smem_u32(&sm->empty[s]), ((g / NSTAGE) - 1) & 1,
                                                 abort_flag, P.wait_ns)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&sm->full_b[s]);
                    mbar_arrive_tx(bar, C::B_COPY);
                    const int boff = ATM ? 0 : (MODE == FDTD_N2F_BF16X3 ? 2 : 1) * C::A_BYTES;
                    bulk_load(smem_u32(stages + s * SSTAGE + boff), src + (int64_t)q * C::B_COPY,
                              C::B_COPY, bar);
                    issued = g + 1;
                }
            }
            // every issued copy has landed before the CTA may exit
            for (int g = (issued > NSTAGE ? issued - NSTAGE : 0); g < issued; ++g)
                drain_bar(smem_u32(&sm->full_b[g % NSTAGE]), (g / NSTAGE) & 1);
        }
    } else if (warp == 1) {
        // ---- MMA issuer.  The whole warp walks the loop, so that descriptors and
        // TMEM addresses stay in uniform registers; one elected lane issues.
        const bool one = elect_one();
        const uint64_t a0 = make_desc(smem_u32(stages), BM * 16, 128);
        const uint32_t boff = ATM ? 0 : (MODE == FDTD_N2F_BF16X3 ? 2 : 1) * C::A_BYTES;
        const uint64_t b0 = make_desc(smem_u32(stages) + boff, BN * 16, 128);
        bool ok = true;
        int s0 = 0;           // stage of the batch's first K step
        uint32_t par0 = 0;    // and its phase
        int tile = 0;         // n tiles so far, over the faces
        for (int fi = f0; fi < f1 && ok; ++fi) {
            const int KS = P.face[fi].ks, NT = P.face[fi].nt;
            for (int nt = 0; nt < NT && ok; ++nt, ++tile) {
                for (int k0 = 0; k0 < KS && ok; k0 += BATCH) {
                    const int k1 = min(k0 + BATCH, KS);
#pragma unroll 1
                    for (int h = 0; h < 2 && ok; ++h) {
                        // half h is free once the epilogue read it for the tile before
                        if (k0 == 0 && tile > 0)
                            ok = __all_sync(0xffffffffu,
                                            wait_bar(smem_u32(&sm->acc_empty[h]), (tile - 1) & 1,
                                                     abort_flag, P.wait_ns));
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t d = tmem + (uint32_t)(h * HN);
                        int s = s0;
                        uint32_t par = par0;
#pragma unroll 1
                        for (int ks = k0; ks < k1; ++ks) {
                            if (h == 0) {
                                const uint32_t fb = smem_u32(&sm->full_b[s]);
                                const uint32_t fa = smem_u32(&sm->full_a[s]);
                                ok = __all_sync(0xffffffffu,
                                                wait_bar(fb, par, abort_flag, P.wait_ns) &&
                                                    wait_bar(fa, par, abort_flag, P.wait_ns));
                                if (!ok) break;
                                tc_fence_after();
                            }
                            // descriptors count 16-byte units; half h starts 16 row groups on
                            const uint64_t bd =
                                b0 + (uint32_t)(s * (SSTAGE / 16) + h * (HN / 8) * 8);
                            const uint64_t ad = a0 + (uint32_t)(s * (SSTAGE / 16));
                            const uint32_t at = tmem + ATM_ACOL + (uint32_t)(s * 32);
#pragma unroll
                            for (int m = 0; m < C::MPS; ++m) {
                                // MMA m reads K chunks 2m and 2m+1 of the stage
                                constexpr uint32_t BLO = C::B_BYTES / 16, ALO = C::A_BYTES / 16;
                                const uint64_t bm = bd + (uint32_t)(m * 2 * (BN / 8) * 8);
                                const uint64_t am = ad + (uint32_t)(m * 2 * (BM / 8) * 8);
                                const uint32_t acc0 = m > 0 ? 1u : (uint32_t)(ks > 0);
                                if (ATM) {
                                    // A of MMA m: 8 TMEM columns (16 BF16 or 8 TF32 of K) per row
                                    mma_ts<MODE>(one, d, at + m * 8, bm, acc0);
                                    if (MODE == FDTD_N2F_BF16X3) {
                                        mma_ts<MODE>(one, d, at + m * 8, bm + BLO, 1u);
                                        mma_ts<MODE>(one, d, at + m * 8 + 16, bm, 1u);
                                    }
                                } else {
                                    mma<MODE>(one, d, am, bm, acc0);
                                    if (MODE == FDTD_N2F_BF16X3) {
                                        mma<MODE>(one, d, am, bm + BLO, 1u);
                                        mma<MODE>(one, d, am + ALO, bm, 1u);
                                    }
                                }
                            }
                            if (h == 1) mma_commit(one, smem_u32(&sm->empty[s]));
                            if (++s == NSTAGE) {
                                s = 0;
                                par ^= 1u;
                            }
                        }
                        if (ok && k1 == KS) mma_commit(one, smem_u32(&sm->acc_full[h]));
                        if (h == 1) {
                            s0 = s;
                            par0 = par;
                        }
                    }
                }
            }
        }
        // every MMA issued has completed before the CTA may exit
        mma_commit(one, smem_u32(&sm->drain));
        drain_bar(smem_u32(&sm->drain), 0);
    } else if ((warp >= 2 && warp < 6) || warp >= 10) {
        // group 0: warps 2-5; group h >= 1: warps 10 + 4(h-1) .. 13 + 4(h-1)
        // ---- A producers: phases u_p(o), or (cos θ, sin θ) of a pair, one row
        // (direction) per thread; NGRP groups of four warps take the stages g with
        // g % NGRP == group.
        // Sample or pair ks*PS + i has e^{jθ} = U_ks * w_i with w_i = e^{j2π γ i} (float,
        // exact to an ulp) and U_ks = e^{j2π γ (ks PS + s)}, evaluated in float64 at the
        // group's first stage of each n tile and advanced by a float64 rotation of NGRP
        // K steps after that, so each value carries one float rounding.
        const int grp = warp >= 10 ? 1 + (warp - 10) / 4 : 0;
        // ATM: the row is the TMEM lane this warp may write (lanes 32*(warp%4) ..)
        const int r = ATM ? 32 * (warp & 3) + lane
                          : (grp ? tid - (320 + 128 * (grp - 1)) : tid - 64);  // 0..127
        const int o = mt * BM + r;
        const bool valid = o < P.n_obs;
        // core-matrix offset of (row r, chunk c): (c*BM/8 + r/8)*128 + (r%8)*16
        const int roff = (r >> 3) * 128 + (r & 7) * 16;
        float2 w[C::PS];
        double2 W2 = make_double2(1.0, 0.0), U = make_double2(1.0, 0.0);
        double gp_w = 0.0;  // γ of w and W2: opposite faces share them
        int g0 = 0;         // stages before this face
        bool ok = true;
        for (int fi = f0; fi < f1 && ok; g0 += P.face[fi].nt * P.face[fi].ks, ++fi) {
            const Face &F = P.face[fi];
            const int KS = F.ks, total = F.nt * F.ks;
            const double gp = valid ? freq * F.pitch * P.dirs[3 * o + F.axis_p] / C0 : 0.0;
            const double s_p = FOLD && !(F.np & 1) ? 0.5 : 0.0;
            if (fi == f0 || __any_sync(0xffffffffu, gp != gp_w)) {
#pragma unroll
                for (int i = 0; i < C::PS; ++i) w[i] = phase_turns(gp, (double)i);
                W2 = zphase_turns(gp, (double)(NGRP * C::PS));
                gp_w = gp;
            }
            int prev_ks = -1;
            for (int q = (grp + NGRP - g0 % NGRP) % NGRP; q < total; q += NGRP) {
                const int g = g0 + q, s = g % NSTAGE, ks = q % KS;
                if (ks <= prev_ks || prev_ks < 0) U = zphase_turns(gp, (double)(ks * C::PS) + s_p);
                prev_ks = ks;
                if (g >= NSTAGE) {
                    // the warp leaves together: its tcgen05.st and votes are collective
                    ok = __all_sync(0xffffffffu, wait_bar(smem_u32(&sm->empty[s]),
                                                          ((g / NSTAGE) - 1) & 1, abort_flag,
                                                          P.wait_ns));
                    if (!ok) break;
                    if (ATM) tc_fence_after();
                }
                unsigned char *st = stages + s * SSTAGE;
                const float2 uf = make_float2((float)U.x, (float)U.y);
                U = zmul(U, W2);
                float vals[2 * C::PS];
#pragma unroll
                for (int i = 0; i < C::PS; ++i) {
                    const float2 u = cmul(uf, w[i]);
                    vals[2 * i] = valid ? u.x : 0.f;
                    vals[2 * i + 1] = valid ? u.y : 0.f;
                }
                if (ATM) {
                    // one TMEM row: column c holds K = 2c, 2c+1 (BF16, hi then lo
                    // 16 columns later) or K = c (TF32), the order of the smem rows
                    const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + ATM_ACOL +
                                        (uint32_t)(s * 32);
                    if (MODE == FDTD_N2F_BF16X3) {
                        uint32_t hr[16], lr[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const __nv_bfloat162 h = __floats2bfloat162_rn(vals[2 * e], vals[2 * e + 1]);
                            const float2 hf = __bfloat1622float2(h);
                            const __nv_bfloat162 l =
                                __floats2bfloat162_rn(vals[2 * e] - hf.x, vals[2 * e + 1] - hf.y);
                            hr[e] = *reinterpret_cast<const uint32_t *>(&h);
                            lr[e] = *reinterpret_cast<const uint32_t *>(&l);
                        }
                        tmem_st16(ta, hr);
                        tmem_st16(ta + 16, lr);
                    } else {
                        uint32_t t0[16], t1[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            t0[e] = __float_as_uint(tf32_rna(vals[e]));
                            t1[e] = __float_as_uint(tf32_rna(vals[16 + e]));
                        }
                        tmem_st16(ta, t0);
                        tmem_st16(ta + 16, t1);
                    }
                    tmem_st_wait();
                    tc_fence_before();
                } else if (MODE == FDTD_N2F_BF16X3) {
#pragma unroll
                    for (int c = 0; c < C::NCH; ++c) {
                        // packed conversions: two values per cvt.rn.bf16x2.f32
                        __align__(16) __nv_bfloat162 hi[4], lo[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float x0 = vals[8 * c + 2 * e], x1 = vals[8 * c + 2 * e + 1];
                            hi[e] = __floats2bfloat162_rn(x0, x1);
                            const float2 hf = __bfloat1622float2(hi[e]);
                            lo[e] = __floats2bfloat162_rn(x0 - hf.x, x1 - hf.y);
                        }
                        const int off = c * (BM / 8) * 128 + roff;
                        *reinterpret_cast<uint4 *>(st + off) = *reinterpret_cast<const uint4 *>(hi);
                        *reinterpret_cast<uint4 *>(st + C::A_BYTES + off) =
                            *reinterpret_cast<const uint4 *>(lo);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < C::NCH; ++c) {
                        float4 v4 = make_float4(tf32_rna(vals[4 * c]), tf32_rna(vals[4 * c + 1]),
                                                tf32_rna(vals[4 * c + 2]), tf32_rna(vals[4 * c + 3]));
                        *reinterpret_cast<float4 *>(st + c * (BM / 8) * 128 + roff) = v4;
                    }
                }
                if (!ATM) fence_proxy_async();
                mbar_arrive(smem_u32(&sm->full_a[s]));
            }
        }
    } else {
        // ---- epilogue: warps 6..9, one direction (TMEM lane) per thread; a warp
        // may read TMEM lanes 32*(warp % 4) .. +31 only
        const int q4 = warp & 3;
        const int row = q4 * 32 + lane;
        const int o = mt * BM + row;
        const bool valid = o < P.n_obs;
        int tile = 0;  // n tiles before this face
        bool ok = true;
        for (int fi = f0; fi < f1 && ok; tile += P.face[fi].nt, ++fi) {
            const Face &F = P.face[fi];
            double gq = 0.0, gc = 0.0;
            if (valid) {
                const double rn = P.dirs[3 * o + F.axis_n], rp = P.dirs[3 * o + F.axis_p],
                             rq = P.dirs[3 * o + F.axis_q];
                gq = freq * F.pitch * rq / C0;
                // the face's first sample, or its middle
                const double mid = FOLD ? 0.5 * F.pitch : 0.0;
                gc = freq * (rn * F.x_n + rp * (F.o_p + mid * (F.np - 1)) +
                             rq * (F.o_q + mid * (F.nq - 1))) / C0;
            }
            // the phase of sample or pair q = 4j + i is V_j * wq_i, V advanced by a
            // float64 rotation per 4 of them
            float2 wq[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) wq[i] = phase_turns(gq, (double)i);
            const double2 WQ = zphase_turns(gq, 4.0);
            double2 V = zphase_turns(gq, FOLD && !(F.nq & 1) ? 0.5 : 0.0);
            float2 S[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f),
                           make_float2(0.f, 0.f)};
            for (int hh = 2 * tile; hh < 2 * (tile + F.nt); ++hh) {
                const int h = hh & 1;
                // tcgen05.ld is warp-collective: the warp leaves together on a timeout
                if (!__all_sync(0xffffffffu, wait_bar(smem_u32(&sm->acc_full[h]), (hh >> 1) & 1,
                                                      abort_flag, P.wait_ns))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t base = tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(h * HN);
#pragma unroll 1
                for (int j = 0; j < HN / 64; ++j) {
                    float v[64];
                    tmem_ld64(base + 64 * j, v);
#pragma unroll
                    for (int u = 0; u < (FOLD ? 1 : 2); ++u) {
                        const float2 vf = make_float2((float)V.x, (float)V.y);
                        V = zmul(V, WQ);
#pragma unroll
                        for (int qq = 0; qq < 4; ++qq) {
                            const float2 w = cmul(vf, wq[qq]);
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                // FOLD: even part t[0], t[1]; odd part t[8], t[9]
                                const float *t = &v[(u * 4 + qq) * (FOLD ? 16 : 8) + 2 * c];
                                S[c].x += w.x * t[0] - w.y * t[FOLD ? 9 : 1];
                                S[c].y += w.x * t[1] + w.y * t[FOLD ? 8 : 0];
                            }
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(smem_u32(&sm->acc_empty[h]));
            }
            if (valid) {
                const float2 cph = phase_turns(gc, 1.0);
                float2 *out = P.partial + (((int64_t)fr * P.nfaces + fi) * P.n_obs + o) * 4;
#pragma unroll
                for (int c = 0; c < 4; ++c) out[c] = cmul(S[c], cph);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 2 * BN);
    }
}

// Pack the faces' currents (face blockIdx.y) into the tiled B operand: for every
// (frequency, n tile, K step) a contiguous block [hi|lo][chunk NCH][256 rows][16 bytes]
// (BF16) or [chunk NCH][256 rows][16 bytes] (TF32).
// Folded: rows n = ((q pair of the tile * 2 + odd) * 4 + c) * 2 + ri_n, K index
// k = 2 * (p pair) + ri_k.  With x±± the samples at the pair's two ends in p and q, the
// q-even and q-odd sums X = x.+ ± x.-, and the p-even E = X+ + X- and p-odd O = X+ - X-
// of those, the value is Re E, -Im O, Im E, Re O by (ri_n, ri_k); zero beyond the last
// pair.  The middle sample of an odd count pairs with zero.
// Not folded: rows n = (q of the tile * 4 + c) * 2 + ri_n, k = 2p + ri_k, value Re, -Im,
// Im, Re of cur[p][q][c]; zero beyond the samples.
// A thread takes one q pair (two neighbours when not folded), one c and one 16-byte
// chunk of K: four rows, whose loads are shared.
template <int MODE, typename CT>
__global__ void k_n2f_pack(Params P, int nfreq, unsigned char *ws) {
    using C = Cfg<MODE>;
    constexpr int EPC = MODE == FDTD_N2F_BF16X3 ? 8 : 4;  // elements per 16-byte chunk
    constexpr int NP = EPC / 2;                           // p pairs per chunk
    const Face &F = P.face[blockIdx.y];
    const CT *cur = reinterpret_cast<const CT *>(P.cur[blockIdx.y]);
    unsigned char *dst = ws + F.b_off;
    const int np = F.np, nq = F.nq, KS = F.ks, NT = F.nt;
    const int64_t n = (int64_t)nfreq * NT * KS * C::NCH * (BN / 4);
    for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t0 < n;
         t0 += (int64_t)gridDim.x * blockDim.x) {
        int64_t t = t0;
        const int c = (int)(t % 4);
        t /= 4;
        const int ql = (int)(t % (BN / 16));
        t /= BN / 16;
        const int chunk = (int)(t % C::NCH);
        t /= C::NCH;
        const int ks = (int)(t % KS);
        t /= KS;
        const int nt = (int)(t % NT);
        const int fr = (int)(t / NT);
        float val[2][2][EPC];  // [odd in q, or second q][ri_n][k]
        if (folded(MODE)) {
            const int qi = nt * (QT / 2) + ql;
            // the pair's ends, or both the middle
            const int q1 = nq / 2 + qi, q0 = (nq - 1) / 2 - qi;
#pragma unroll
            for (int e = 0; e < NP; ++e) {
                const int pi = ks * C::PS + chunk * NP + e;
                const int p1 = np / 2 + pi, p0 = (np - 1) / 2 - pi;
                double2 x[2][2];  // [p end][q end]
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int p = a ? p1 : p0, q = b ? q1 : q0;
                        x[a][b] = make_double2(0.0, 0.0);
                        if (p0 >= 0 && q0 >= 0 && (a || p0 != p1) && (b || q0 != q1)) {
                            const CT z = cur[(((int64_t)fr * np + p) * nq + q) * 4 + c];
                            x[a][b] = make_double2((double)z.x, (double)z.y);
                        }
                    }
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const double s = o ? -1.0 : 1.0;
                    const double ar = x[1][1].x + s * x[1][0].x, ai = x[1][1].y + s * x[1][0].y;
                    const double br = x[0][1].x + s * x[0][0].x, bi = x[0][1].y + s * x[0][0].y;
                    // no odd part at a middle sample
                    const bool mq = o && q0 == q1, mp = p0 == p1;
                    val[o][0][2 * e] = mq ? 0.f : (float)(ar + br);
                    val[o][0][2 * e + 1] = mq || mp ? 0.f : (float)(bi - ai);
                    val[o][1][2 * e] = mq ? 0.f : (float)(ai + bi);
                    val[o][1][2 * e + 1] = mq || mp ? 0.f : (float)(ar - br);
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < NP; ++e) {
                const int p = ks * C::PS + chunk * NP + e;
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const int q = nt * QT + ql * 2 + o;
                    float2 x = make_float2(0.f, 0.f);
                    if (p < np && q < nq) {
                        const CT z = cur[(((int64_t)fr * np + p) * nq + q) * 4 + c];
                        x = make_float2((float)z.x, (float)z.y);
                    }
                    val[o][0][2 * e] = x.x;
                    val[o][0][2 * e + 1] = -x.y;
                    val[o][1][2 * e] = x.y;
                    val[o][1][2 * e + 1] = x.x;
                }
            }
        }
        unsigned char *blk = dst + (((int64_t)fr * NT + nt) * KS + ks) * C::B_COPY;
#pragma unroll
        for (int o = 0; o < 2; ++o)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = ((ql * 2 + o) * 4 + c) * 2 + r;
                const int off = chunk * (BN / 8) * 128 + (row >> 3) * 128 + (row & 7) * 16;
                const float(&vals)[EPC] = val[o][r];
                if (MODE == FDTD_N2F_BF16X3) {
                    __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
                    for (int e = 0; e < EPC; ++e) {
                        hi[e] = __float2bfloat16_rn(vals[e]);
                        lo[e] = __float2bfloat16_rn(vals[e] - __bfloat162float(hi[e]));
                    }
                    *reinterpret_cast<uint4 *>(blk + off) = *reinterpret_cast<const uint4 *>(hi);
                    *reinterpret_cast<uint4 *>(blk + C::B_BYTES + off) =
                        *reinterpret_cast<const uint4 *>(lo);
                } else {
                    *reinterpret_cast<float4 *>(blk + off) = make_float4(
                        tf32_rna(vals[0]), tf32_rna(vals[1]), tf32_rna(vals[2]), tf32_rna(vals[3]));
                }
            }
    }
}

// NL[o][6] of one frequency: Σ_faces partial[face][o][c] mapped to (J_b, J_c, M_b, M_c);
// false if one of them is not finite.
__device__ __forceinline__ bool combine_faces(const Params &P, int fr, int o, float2 *nl) {
    float2 acc[6];
    for (int c = 0; c < 6; ++c) acc[c] = make_float2(0.f, 0.f);
    for (int fi = 0; fi < P.nfaces; ++fi) {
        const float2 *p = P.partial + (((int64_t)fr * P.nfaces + fi) * P.n_obs + o) * 4;
        for (int c = 0; c < 4; ++c) {
            const int m = P.comp_map[fi * 4 + c];
            acc[m].x += p[c].x;
            acc[m].y += p[c].y;
        }
    }
    bool ok = true;
    for (int c = 0; c < 6; ++c) {
        nl[c] = acc[c];
        ok = ok && isfinite(acc[c].x) && isfinite(acc[c].y);
    }
    return ok;
}

// The same with the faces whose sums are not finite summed again in float64, straight
// from the currents and with the phases rotated along a row.  A face with a current that
// is not finite keeps its sums.
template <typename CT>
__device__ __noinline__ void combine_again(const Params &P, int fr, int o, float2 *nl) {
    const double freq = P.freqs[fr];
    for (int fi = 0; fi < P.nfaces; ++fi) {
        float2 *out = P.partial + (((int64_t)fr * P.nfaces + fi) * P.n_obs + o) * 4;
        bool ok = true;
        for (int c = 0; c < 4; ++c) ok = ok && isfinite(out[c].x) && isfinite(out[c].y);
        if (ok) continue;
        const Face &F = P.face[fi];
        const CT *cur = reinterpret_cast<const CT *>(P.cur[fi]) + (int64_t)fr * F.np * F.nq * 4;
        const double rn = P.dirs[3 * o + F.axis_n], rp = P.dirs[3 * o + F.axis_p],
                     rq = P.dirs[3 * o + F.axis_q];
        const double base = rn * F.x_n + rp * F.o_p + rq * F.o_q;
        const double2 W = zphase_turns(freq * F.pitch * rq / C0, 1.0);
        double2 S[4] = {};
        ok = true;
        for (int p = 0; p < F.np && ok; ++p) {
            double2 u = zphase_turns(freq * (base + rp * F.pitch * p) / C0, 1.0);
            for (int q = 0; q < F.nq && ok; ++q, cur += 4) {
                for (int c = 0; c < 4; ++c) {
                    const double2 z = make_double2((double)cur[c].x, (double)cur[c].y);
                    ok = ok && isfinite(z.x) && isfinite(z.y);
                    S[c].x += u.x * z.x - u.y * z.y;
                    S[c].y += u.x * z.y + u.y * z.x;
                }
                u = zmul(u, W);
            }
        }
        for (int c = 0; c < 4 && ok; ++c) out[c] = make_float2((float)S[c].x, (float)S[c].y);
    }
    combine_faces(P, fr, o, nl);
}

// AGAIN (the folded sums): the sums of up to four currents leave float32 (and bfloat16)
// where the currents themselves, from 8.5e37 on, and their far field do not.  A direction
// that comes out infinite or NaN is therefore summed again directly; the check of the
// results costs the others nothing measurable.
template <typename CT, bool AGAIN>
__global__ void k_n2f_combine(const __grid_constant__ Params P, int nfreq, float2 *nl) {
    const int64_t n = (int64_t)nfreq * P.n_obs;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int fr = (int)(q / P.n_obs), o = (int)(q % P.n_obs);
        const bool ok = combine_faces(P, fr, o, nl + q * 6);
        if (AGAIN && !ok) combine_again<CT>(P, fr, o, nl + q * 6);
    }
}

// FP64 direct sum (no separation, no tensor cores): one block per (direction,
// frequency), exact phases e^{j2π f r̂·r'/c0} with the reduction in turns.
template <typename CT>
__global__ void k_n2f_fp64(Params P, double2 *nl) {
    const int o = blockIdx.x, fr = blockIdx.y;
    const double freq = P.freqs[fr];
    const double rv[3] = {P.dirs[3 * o], P.dirs[3 * o + 1], P.dirs[3 * o + 2]};
    double ar[6] = {0, 0, 0, 0, 0, 0}, ai[6] = {0, 0, 0, 0, 0, 0};
    for (int fi = 0; fi < P.nfaces; ++fi) {
        const Face &F = P.face[fi];
        const CT *cur = reinterpret_cast<const CT *>(P.cur[fi]) + (int64_t)fr * F.np * F.nq * 4;
        const double base = rv[F.axis_n] * F.x_n + rv[F.axis_p] * F.o_p + rv[F.axis_q] * F.o_q;
        const int64_t ns = (int64_t)F.np * F.nq;
        for (int64_t s = threadIdx.x; s < ns; s += blockDim.x) {
            const int p = (int)(s / F.nq), q = (int)(s % F.nq);
            double t = freq * (base + rv[F.axis_p] * F.pitch * p + rv[F.axis_q] * F.pitch * q) / C0;
            t = t - rint(t);
            double sn, cs;
            sincospi(2.0 * t, &sn, &cs);
            for (int c = 0; c < 4; ++c) {
                const CT z = cur[s * 4 + c];
                const int m = P.comp_map[fi * 4 + c];
                ar[m] += cs * (double)z.x - sn * (double)z.y;
                ai[m] += cs * (double)z.y + sn * (double)z.x;
            }
        }
    }
    __shared__ double red[2][6][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c = 0; c < 6; ++c) {
        double x = ar[c], y = ai[c];
        for (int sh = 16; sh > 0; sh >>= 1) {
            x += __shfl_down_sync(0xffffffffu, x, sh);
            y += __shfl_down_sync(0xffffffffu, y, sh);
        }
        if (lane == 0) {
            red[0][c][w] = x;
            red[1][c][w] = y;
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int c = threadIdx.x;
        double x = 0.0, y = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            x += red[0][c][i];
            y += red[1][c][i];
        }
        nl[((int64_t)fr * P.n_obs + o) * 6 + c] = make_double2(x, y);
    }
}

// ------------------------------------------------------------------- launchers
size_t stage_smem(int mode, bool atm) {
    size_t st;
    if (atm)
        st = (size_t)ATM_NST * (mode == FDTD_N2F_BF16X3 ? Cfg<FDTD_N2F_BF16X3>::B_COPY
                                                        : Cfg<FDTD_N2F_TF32>::B_COPY);
    else
        st = mode == FDTD_N2F_BF16X3
                 ? (size_t)Cfg<FDTD_N2F_BF16X3>::NST * Cfg<FDTD_N2F_BF16X3>::STAGE
                 : (size_t)Cfg<FDTD_N2F_TF32>::NST * Cfg<FDTD_N2F_TF32>::STAGE;
    return st + sizeof(Smem) + 64;
}

// Where the A operand lives: tensor memory by default; FDTD_B200_N2F_A=smem
// (read at each call) selects the shared-memory form, with the same MMAs in
// the same order.
bool a_in_tmem() {
    const char *e = getenv("FDTD_B200_N2F_A");
    return !(e && strcmp(e, "smem") == 0);
}

int b_copy_bytes(int mode) {
    return mode == FDTD_N2F_BF16X3 ? Cfg<FDTD_N2F_BF16X3>::B_COPY : Cfg<FDTD_N2F_TF32>::B_COPY;
}

static int k_real_per_step(int mode) {
    return mode == FDTD_N2F_BF16X3 ? Cfg<FDTD_N2F_BF16X3>::KR : Cfg<FDTD_N2F_TF32>::KR;
}

void operand_steps(int mode, int np, int nq, int &ks, int &nt) {
    // samples, or pairs of samples about the middle of the face, per K step and n tile
    const bool f = folded(mode);
    const int p = f ? np / 2 + np % 2 : np, q = f ? nq / 2 + nq % 2 : nq, qt = f ? QT / 2 : QT;
    const int kr = k_real_per_step(mode);
    ks = (2 * p + kr - 1) / kr;
    nt = (q + qt - 1) / qt;
}

template <typename CT>
cudaError_t launch_pack(int mode, const Params &P, int nfreq, unsigned char *dst,
                        cudaStream_t st) {
    const int nch = mode == FDTD_N2F_BF16X3 ? Cfg<FDTD_N2F_BF16X3>::NCH : Cfg<FDTD_N2F_TF32>::NCH;
    int64_t blocks = 1;
    for (int f = 0; f < P.nfaces; ++f) {
        const int64_t n = (int64_t)nfreq * P.face[f].nt * P.face[f].ks * nch * (BN / 4);
        if (blocks < (n + 255) / 256) blocks = (n + 255) / 256;
    }
    if (blocks > 148 * 16) blocks = 148 * 16;
    const dim3 grid((unsigned)blocks, P.nfaces);
    if (mode == FDTD_N2F_BF16X3)
        k_n2f_pack<FDTD_N2F_BF16X3, CT><<<grid, 256, 0, st>>>(P, nfreq, dst);
    else
        k_n2f_pack<FDTD_N2F_TF32, CT><<<grid, 256, 0, st>>>(P, nfreq, dst);
    count_launches(1);
    return cudaGetLastError();
}

namespace {
std::atomic<long long> g_wait_ns{(long long)WAIT_NS};
}

void set_wait_ns(int64_t ns) { g_wait_ns.store(ns < 0 ? (long long)WAIT_NS : ns); }

// Faces per CTA.  A CTA's start (barriers, TMEM, first phases and copies) and its last
// epilogue take about 4,500 cycles with the tensor pipe idle, which more faces per CTA
// save; fewer fill the last wave.  A stage's MMAs take 768 cycles (BF16) or 512 (TF32).
static int face_group(int mode, const Params &P, int nfreq) {
    double stages = 0.0;
    for (int f = 0; f < P.nfaces; ++f) stages += (double)P.face[f].ks * P.face[f].nt;
    const double t_face = stages / P.nfaces * (mode == FDTD_N2F_BF16X3 ? 768.0 : 512.0);
    const int64_t mt = (P.n_obs + BM - 1) / BM;
    int best = 1;
    double t_best = 0.0;
    for (int g = 1; g <= P.nfaces; ++g) {
        const int64_t ctas = mt * nfreq * ((P.nfaces + g - 1) / g);
        const double t = (double)((ctas + 147) / 148) * (g * t_face + 4500.0);
        if (g == 1 || t < t_best) {
            best = g;
            t_best = t;
        }
    }
    return best;
}

template <int MODE, bool ATM>
static cudaError_t launch_tc(const Params &P, int nfreq, cudaStream_t st) {
    const size_t smem = stage_smem(MODE, ATM);
    const int mt = (P.n_obs + BM - 1) / BM;
    dim3 grid(mt, (P.nfaces + P.face_group - 1) / P.face_group, nfreq);
    cudaError_t e =
        cudaFuncSetAttribute(k_n2f_tc<MODE, ATM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    k_n2f_tc<MODE, ATM><<<grid, NTHREADS, smem, st>>>(P);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_contract(int mode, const Params &Pin, int nfreq, cudaStream_t st) {
    Params P = Pin;
    P.wait_ns = (uint64_t)g_wait_ns.load();
    P.face_group = face_group(mode, P, nfreq);
    const bool atm = a_in_tmem();
    if (mode == FDTD_N2F_BF16X3)
        return atm ? launch_tc<FDTD_N2F_BF16X3, true>(P, nfreq, st)
                   : launch_tc<FDTD_N2F_BF16X3, false>(P, nfreq, st);
    return atm ? launch_tc<FDTD_N2F_TF32, true>(P, nfreq, st)
               : launch_tc<FDTD_N2F_TF32, false>(P, nfreq, st);
}

template <typename CT>
cudaError_t launch_combine(int mode, const Params &P, int nfreq, float2 *nl, cudaStream_t st) {
    const int64_t n = (int64_t)nfreq * P.n_obs;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (folded(mode))
        k_n2f_combine<CT, true><<<(unsigned)blocks, 256, 0, st>>>(P, nfreq, nl);
    else
        k_n2f_combine<CT, false><<<(unsigned)blocks, 256, 0, st>>>(P, nfreq, nl);
    count_launches(1);
    return cudaGetLastError();
}

template <typename CT>
cudaError_t launch_fp64(const Params &P, int nfreq, double2 *nl, cudaStream_t st) {
    dim3 grid(P.n_obs, nfreq);
    k_n2f_fp64<CT><<<grid, 256, 0, st>>>(P, nl);
    count_launches(1);
    return cudaGetLastError();
}

int read_error(int reset) {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_n2f_error, sizeof(int));
    if (reset) {
        int z = 0;
        cudaMemcpyToSymbol(g_n2f_error, &z, sizeof(int));
    }
    return v;
}

template cudaError_t launch_pack<float2>(int, const Params &, int, unsigned char *, cudaStream_t);
template cudaError_t launch_pack<double2>(int, const Params &, int, unsigned char *, cudaStream_t);
template cudaError_t launch_combine<float2>(int, const Params &, int, float2 *, cudaStream_t);
template cudaError_t launch_combine<double2>(int, const Params &, int, float2 *, cudaStream_t);
template cudaError_t launch_fp64<float2>(const Params &, int, double2 *, cudaStream_t);
template cudaError_t launch_fp64<double2>(const Params &, int, double2 *, cudaStream_t);

}  // namespace n2f
}  // namespace fdtd
