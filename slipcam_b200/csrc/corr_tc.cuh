// corr_tc.cuh -- the tensor-core form: the 2-D DFTs of the correlation as dense DFT-matrix GEMMs
// on tcgen05 (FP16 operands, FP32 accumulation in TMEM), (window, frame) pairs streaming through a
// persistent CTA per SM. With C = [cos(2 pi r c / N)] and S = [-sin(2 pi r c / N)], FP16, resident in
// shared memory, a pair is
//
//   S1  Yr^T = C X^T, Yi^T = S X^T       rows kappa (frequency across), columns i   X = chip - round(mean)
//   S2  [P1|P3] = Yr [C|S]^T,            rows kappa, columns r = 0 .. N/2 - 1 (frequency down) of each:
//       [P4|P2] = Yi [C|S]^T             the spectrum at ky = r is (P1 - P2, P3 + P4), at N - r (P1 + P2, P4 - P3)
//   S3  P = Z conj(R) 2^-s               per thread (one kappa row), R the resident reference spectrum
//   S4  [Pr C|Pr S], [Pi C|Pi S]         rows kappa, columns u = 0 .. N/2 - 1, as S2: Q at u and at N - u
//   S5  c^T = [C|S] (w Q)                rows v, columns u < M, w the Hermitian weights
//
// then the normalization by the variance denominators, the argmax and the peak's values. C at N - r is
// C at r and S changes sign, so columns r < N/2 give the whole of S2's and S4's results in half the
// products, and one table serves every stage: its rows are C 0 .. N/2 - 1, then the Nyquist row (-1)^c,
// then S 1 .. N/2. The Nyquist row is C's row N/2 and stands where S's row 0 (zero) would: S1 and S5 zero
// what it touches as S's, and as a column of P2 and P3 it is the spectrum at ky = N/2 that r < N/2 lacks
// (the same for u = N/2). As A the table is read K-major in S1 and MN-major in S5, as B (its first N rows,
// C and S at once, so that an MMA is N columns wide and the tensor core, not the operands' 128 bytes of
// shared memory a cycle, bounds it: 80 cycles at N = 160) K-major in S2 and S4.
//
// Seven roles, linked by mbarriers (one completion per pair and barrier):
//   control   issues every MMA; the order S4(p), S1(p + 1) Yr, S5(p), S1(p + 1) Yi, S2(p + 1) keeps the
//             tensor core busy while the drains run
//   drain     12 warps, four per TMEM quadrant 0-2 (kappa < 96): Y to the FP16 operand of S2, S3, Q to
//             the FP16 operand of S5
//   epilogue  8 warps: c of the last pair from TMEM, normalized, its argmax and patch sums
//   gather    8 warps: the next chip
//   setup     works out the pairs ahead, 32 at a time, one per lane
//   relay     waits for the MMAs of each stage and wakes the warps that go on with them at a hardware
//             barrier (28 warps polling mbarriers took most of the load-store unit's cycles)
//   spectrum  brings R in by bulk copies, a ring of 5 x 8 frequencies, four of them in S5's operand's
//             bytes, which are free from S5(p) to S4(p + 1): loads to registers would pass through the
//             few KB of L1 that this much shared memory leaves
// An MMA here takes nine tenths of the SM's shared-memory bandwidth, so whatever else goes through it
// (stores of operands, copies, loads through L1) all but waits while MMAs run: S2 starts when both halves
// of its operand are in.
//
// Measured at 720p, window 64, search 48 (N = 160, 39,200 pairs a launch): 2.20 ms, 16,300 cycles a pair
// and SM, where one role after the other in the same 12 warps took 3.96 ms; N = 96 (window 48, search 24)
// 10,600 cycles. The MMAs are 5,500 of them. No unit is full: ncu of such a launch has the tensor pipe 37 % busy, the
// issue slots 50 %, the L1 and shared memory 49 %. Of 15.9 stalled warps per issue 5.2 wait at a barrier and 4.4 for TMEM
// or L2 loads: what bounds a pair is the chain S4, Q's drain, S5, Yi, its drain, S2, S3 with the
// epilogue's hold on c beside it. The code has to stay small: unrolled to 179 KB the same design took 2.39 ms
// against 2.16 in 68 KB, and in the latter only 0.3 of those stalls are for instructions.
//
// TMEM columns: Q [0, 2N), then c [0, NO) and Yi [NO, NO + N) once it is drained; Yr [2N, 3N); S2's
// products replace Y where it was.
//
// Power-of-two scales keep every FP16 operand in range: |X| <= 255, |Y| <= 255 N, the reference
// spectrum is scaled by 2^-e with 2^e > W * norm >= max |R|, P by 2^-8 (|P| <= N^2 255 2^-8 < 2^15
// for N <= 160) and w Q by 2^-9. Fixed-size tensor-core tiles: rows beyond the data (kappa rows >= KP,
// output rows >= M) read whatever follows in shared memory and their results are ignored.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "corr_fft.cuh"
#include "tc.cuh"

namespace b200 {

constexpr uint32_t cmax(uint32_t a, uint32_t b) { return a > b ? a : b; }

// the frequency rows kappa of a real N-point row transform (N / 2 + 1), padded to 16
__host__ __device__ constexpr int tc_kp(int N) { return (N / 2 + 1 + 15) / 16 * 16; }
// the rows of the table: C 0 .. N/2 - 1, the Nyquist row, S 1 .. N/2, zeros up to S's row KP - 1
__host__ __device__ constexpr int tc_rt(int N) { return N / 2 + tc_kp(N); }
// element (r, c) of the table, bytes: column groups of 8, rows of 16 bytes
B200_HD uint32_t tc_table_offset(int N, int r, int c)
{
    return uint32_t(c / 8) * uint32_t(tc_rt(N)) * 16u + uint32_t(r) * 16u + uint32_t(c % 8) * 2u;
}

template <int N>
struct TcGeo {
    static constexpr int NH = N / 2 + 1;                            // frequencies of a real row
    static constexpr int KP = tc_kp(N);                             // kappa rows, padded
    static constexpr int RT = tc_rt(N);
    static constexpr uint32_t SBO_T = uint32_t(RT) * 16u;           // the table's column groups
    static constexpr uint32_t T_BYTES = uint32_t(N / 8) * SBO_T;
    static constexpr uint32_t SBO_X = uint32_t(N / 8) * 128u;       // X: K-major rows of N
    static constexpr uint32_t SBO_A = uint32_t(2 * N / 8) * 128u;   // Y, P: K-major rows (Re | Im, i or ky)
    static constexpr uint32_t SBO_B5 = uint32_t(2 * KP / 8) * 128u; // w Q (MN-major): K = 2 KP
    static constexpr uint32_t A_BYTES = uint32_t(KP / 8) * SBO_A;
    static constexpr uint32_t X_BYTES = uint32_t(N / 8) * SBO_X;
    static constexpr uint32_t B5_BYTES = 16u * SBO_B5;              // = 4 slots of R_BYTES
    static constexpr uint32_t R_BYTES = 8u * uint32_t(KP) * 16u;    // 8 frequencies (and their mirrors) of R
    static constexpr uint32_t OFF_A = T_BYTES, OFF_X = OFF_A + A_BYTES, OFF_B5 = OFF_X + X_BYTES;
    static constexpr uint32_t END = OFF_B5 + 5u * R_BYTES;           // the ring: B5 and one slot more
    // the furthest byte a full 128-row tile reads: rows of A, table rows (S1), table columns (S5)
    static constexpr uint32_t READ_END =
        cmax(cmax(END, OFF_A + 16u * SBO_A), cmax(uint32_t(N / 8 - 1) * SBO_T + uint32_t(N / 2 + 128) * 16u, 16u * SBO_T + uint32_t(N / 2) * 16u));
    static constexpr size_t smem_bytes = READ_END;
    static constexpr uint32_t TMEM_COLS = 512;
    static constexpr int NR = N / 16;   // chunks of 8 frequencies (S3) or rows u (S5's operand) and their mirrors
    static_assert(KP <= 96 && 3 * N <= 512, "TMEM or tile bounds");
    static_assert(READ_END <= 225 * 1024 + 512 && 4 * R_BYTES == B5_BYTES, "shared memory");
};

#ifdef __CUDACC__

__device__ __forceinline__ uint4 pack8(const float *v)
{
    uint4 r;
    __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
    __half2 h2 = __floats2half2_rn(v[4], v[5]), h3 = __floats2half2_rn(v[6], v[7]);
    r.x = *reinterpret_cast<uint32_t *>(&h0);
    r.y = *reinterpret_cast<uint32_t *>(&h1);
    r.z = *reinterpret_cast<uint32_t *>(&h2);
    r.w = *reinterpret_cast<uint32_t *>(&h3);
    return r;
}

// two floats in one register pair: one instruction works on both, each rounded as the scalar one rounds
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { f32x2 d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ f32x2 both(float x) { const uint32_t b = __float_as_uint(x); return (f32x2(b) << 32) | b; }
// the j-th pair of registers read from TMEM
template <int R>
__device__ __forceinline__ f32x2 pair2(const uint32_t (&r)[R], int j) { return (f32x2(r[2 * j + 1]) << 32) | r[2 * j]; }
// the two rounded to FP16, in order and exchanged
__device__ __forceinline__ uint32_t half2_bits(f32x2 a)
{
    const __half2 h = __floats2half2_rn(__uint_as_float(uint32_t(a)), __uint_as_float(uint32_t(a >> 32)));
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t half2_swapped(f32x2 a)
{
    const __half2 h = __floats2half2_rn(__uint_as_float(uint32_t(a >> 32)), __uint_as_float(uint32_t(a)));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// read-only loads that stay where they are written, so that what is fetched ahead of a wait is in
// flight during it (the compiler moves a plain __ldg down to its first use)
__device__ __forceinline__ float ldg_here(const float *p)
{
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 ldg_here(const uint4 *p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// the warps of each role, 32 in all (eight per SM partition, which is also the TMEM quadrant a warp
// reads): of 0-15 the first three of each four drain; the others, whose quadrant has nothing to drain,
// are control (3), the spectrum's copies (7), the pairs' setup (11) and the relay (15); 16-23 epilogue,
// 24-31 gather
constexpr int kTcParts = 4;                 // drain warps per quadrant
constexpr int kTcDrain = 3 * kTcParts;
constexpr int kTcControl = 3, kTcFetch = 7, kTcSetup = 11, kTcRelay = 15;
constexpr int kTcEpi = 8, kTcGather = 8;
constexpr int kTcThreads = 1024;
constexpr int kTcSlots = 5;                 // of the spectrum's ring: 8 frequencies each
// the hardware barriers on which the relay wakes the drain warps and (C) the epilogue warps
constexpr int kTcWake = 2, kTcWakeQ = 2, kTcWakeYr = 3, kTcWakeC = 4, kTcWakeYi = 5, kTcWakeZ = 6;

// 4 pixels (a little-endian word) minus the same offset, as two exact FP16 pairs: a byte b placed
// under the exponent byte 0x64 reads as the half 1024 + b, and 1024 + b - (1024 + m) is exact
__device__ __forceinline__ void bytes_to_half(uint32_t word, __half2 off, uint32_t &lo, uint32_t &hi)
{
    uint32_t a = __byte_perm(word, 0x64646464u, 0x4140);   // (1024 + b0, 1024 + b1)
    uint32_t b = __byte_perm(word, 0x64646464u, 0x4342);   // (1024 + b2, 1024 + b3)
    __half2 ha = __hsub2(*reinterpret_cast<__half2 *>(&a), off);
    __half2 hb = __hsub2(*reinterpret_cast<__half2 *>(&b), off);
    lo = *reinterpret_cast<uint32_t *>(&ha);
    hi = *reinterpret_cast<uint32_t *>(&hb);
}

// one (window, frame) pair of the tensor-core kernel, as the setup warp works it out ahead of time
struct PairSetup {
    int64_t q;              // the output index f * nwin + k
    int k, f, gy, gx;       // window, frame, gross offset
    int sy, sx, mean;       // the chip's top-left corner and its rounded mean
    float scale;            // of c: undoes the power-of-two scales, the transform's N^2 and the norm
    bool end;               // no pair: the roles leave
    uint32_t seq;           // which pair of the CTA, from 1 (entries are read before a barrier says so)
};

// the mbarriers of the tensor-core kernel, one completion of each per pair
struct TcBars {
    uint64_t xfull, xfree;          // the chip is in X; S1 has read it
    uint64_t afull;                 // S2's operand is in shared memory
    uint64_t pfull, b5full;         // S4's, S5's
    uint64_t cfree;                 // the correlation is read
    uint64_t stage[5];              // in TMEM: Q (S4), Yr (S1), c (S5), Yi (S1), Z (S2)
    uint64_t rfull[kTcSlots], rfree[kTcSlots];   // a slot of the reference spectrum's ring, per use of the slot
};

// wait for the phase `parity` of the mbarrier; false if another role gave up or two seconds went by
// (the abort flag is then set for the others). The polling is one function for all roles, for the size of the
// code.
__device__ __noinline__ bool tc_wait_poll(uint64_t *bar, uint32_t parity, volatile int *abort)
{
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (;;) {
        if (tc::mbar_wait(bar, parity, 16)) return true;
        if (*abort) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 2000000000ull) {
            *abort = 1;
            return false;
        }
    }
}

__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile int *abort)
{
    return tc::mbar_wait(bar, parity, 1) || tc_wait_poll(bar, parity, abort);
}

// the same for a whole warp, the answer uniform
__device__ __forceinline__ bool tc_wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort)
{
    const bool ok = __all_sync(0xffffffffu, tc_wait(bar, parity, abort));
    tc::fence_after_sync();
    return ok;
}

// The relay's wake-up and its other side: `threads` threads at hardware barrier id, 32 of them the
// relay's. good holds how many of the barrier's events have come about: the relay counts one before the
// wake-up or, once a wait gave up, never again, so all who are woken for event n take the same decision
// (and all leave before they would meet at another barrier).
__device__ __forceinline__ void wake(int id, int threads, volatile uint32_t *good, uint32_t n, bool ok, int lane)
{
    if (ok && lane == 0) *good = n + 1;
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
template <int ID>
__device__ __forceinline__ bool woken(int threads, const volatile uint32_t *good, uint32_t n)
{
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(threads) : "memory");
    tc::fence_after_sync();
    return __all_sync(0xffffffffu, *good > n);
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// this warp's shared-memory operands (and TMEM reads) are done: one arrival for the warp
__device__ __forceinline__ void warp_publish(uint64_t *bar, int lane)
{
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// the outputs of a pair without a peak, and of one whose peak is not refined, out of the kernel's way
__device__ __noinline__ void tc_invalid(const CorrArgs *a, int64_t q)
{
    invalid_outputs(q, a->offset, a->peak, a->snr, a->cov);
    if (a->peaks) a->peaks[q].valid = 0;
}
__device__ __noinline__ void tc_outputs(const CorrArgs *a, const float *fit, int u, int v, int gy, int gx, double sum, int count, int64_t q)
{
    peak_outputs(fit + 4, 3, a->M, u, v, a->R, gy, gx, a->W * a->W, sum, count, q, a->offset, a->peak, a->snr, a->cov);
}

// the chip of pair c into X by the gather warps (gw). rows16: a warp takes groups of 8 chip rows, lane
// (r, c) = (lane & 7, lane >> 3) loads the aligned 16-byte chunks c, c + 4, c + 8 of row r (the chip's first
// byte is byte o of chunk 0, the same o on every row), two steps ahead, and writes chip columns 16 q ..
// 16 q + 15 (q = c + 4 k) from chunks q and q + 1 as two 16-byte FP16 pieces: the 8 lanes of one c fill
// 128 contiguous bytes of a core matrix. Chunk q + 1 comes from its lane, not from memory again: lanes down
// the rows cost the L1 a line's lookup each. Else a warp takes 8 rows x 4 pieces of 8 pixels as 4-byte
// words (bytes where the rows are not word-aligned).
template <int N>
__device__ __forceinline__ void tc_gather(const CorrArgs &a, const PairSetup &c, unsigned char *X, bool rows16, int gw,
                                          int lane)
{
    using G = TcGeo<N>;
    const int L = a.L;
    const __half2 off = __float2half2_rn(1024.0f + float(c.mean));
    const uint8_t *chip = a.frames + c.f * a.fstride + int64_t(c.sy) * a.pitch + c.sx;
    if (rows16) {
        const int o = c.sx & 15, sw = o >> 2, sb = 8 * (o & 3);
        const int r = lane & 7, cg = lane >> 3;
        const int nq = (o + L + 15) >> 4;   // chunks holding chip bytes (they end inside the row)
        const uint4 *rb = reinterpret_cast<const uint4 *>(chip - o);
        const int pq = a.pitch >> 4;        // chunks per frame row
        constexpr int NG = N / 8, NQ = N / 16, NK = (NQ + 4) / 4;    // groups, pieces, rounds of a row
        auto load = [&](int g, int k) {
            const int i = 8 * g + r, q = 4 * k + cg;
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (i < L && q < nq) w = ldg_here(rb + (i * pq + q));
            return w;
        };
        auto next = [](int &g, int &k) {
            if (++k == NK) {
                k = 0;
                g += kTcGather;
            }
        };
        int g = gw, k = 0, g2 = gw, k2 = 0;   // this step, the step whose chunks are loaded
        uint4 raw = load(g2, k2);
        next(g2, k2);
        uint4 then = load(g2, k2);
        {
#pragma unroll 1
            for (; g < NG; next(g, k)) {
                next(g2, k2);
                const uint4 later = load(g2, k2);
                // lane (r, 0) gives its next chunk to lane (r, 3), the others this one to their left
                const bool give = cg == 0;
                const int from = (lane + 8) & 31;
                uint4 nx;
                nx.x = __shfl_sync(0xffffffffu, give ? then.x : raw.x, from);
                nx.y = __shfl_sync(0xffffffffu, give ? then.y : raw.y, from);
                nx.z = __shfl_sync(0xffffffffu, give ? then.z : raw.z, from);
                nx.w = __shfl_sync(0xffffffffu, give ? then.w : raw.w, from);
                const int i = 8 * g + r, q = 4 * k + cg;
                if (q < NQ) {
                    // bytes 4 sw .. 4 sw + 19 of the 32 (sw is the same on every lane)
                    const bool s2 = sw & 2, s1 = sw & 1;
                    const uint32_t a0 = s2 ? raw.z : raw.x, a1 = s2 ? raw.w : raw.y, a2 = s2 ? nx.x : raw.z;
                    const uint32_t a3 = s2 ? nx.y : raw.w, a4 = s2 ? nx.z : nx.x, a5 = s2 ? nx.w : nx.y;
                    const uint32_t b[5] = {s1 ? a1 : a0, s1 ? a2 : a1, s1 ? a3 : a2, s1 ? a4 : a3, s1 ? a5 : a4};
                    uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = make_uint4(0u, 0u, 0u, 0u);
                    const int keep = i < L ? L - 16 * q : 0;   // chip columns from 16 q on
                    if (keep > 0) {
                        bytes_to_half(__funnelshift_r(b[0], b[1], sb), off, lo.x, lo.y);
                        bytes_to_half(__funnelshift_r(b[1], b[2], sb), off, lo.z, lo.w);
                        bytes_to_half(__funnelshift_r(b[2], b[3], sb), off, hi.x, hi.y);
                        bytes_to_half(__funnelshift_r(b[3], b[4], sb), off, hi.z, hi.w);
                    }
                    if (keep < 16) {   // the 8 words of the 16 halves: zero past the chip
                        uint32_t hv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            if (2 * e >= keep) hv[e] = 0u;
                            else if (2 * e + 1 >= keep) hv[e] &= 0xFFFFu;
                        }
                        lo = make_uint4(hv[0], hv[1], hv[2], hv[3]);
                        hi = make_uint4(hv[4], hv[5], hv[6], hv[7]);
                    }
                    unsigned char *d = X + tc::k_major_offset(i, 16 * q, G::SBO_X, 128);
                    *reinterpret_cast<uint4 *>(d) = lo;
                    *reinterpret_cast<uint4 *>(d + 128) = hi;
                }
                raw = then;
                then = later;
            }
        }
        return;
    }
    const bool words = ((a.pitch | reinterpret_cast<uintptr_t>(a.frames) | int(a.fstride)) & 3) == 0;
    constexpr int NCG = (N / 8 + 3) / 4;               // groups of 4 pieces per row
    constexpr int NB = (N / 8) * NCG;                   // blocks of 8 rows x 4 pieces
    constexpr int AHEAD = 2;                            // blocks loaded before they are used
    for (int b0 = gw; b0 < NB; b0 += AHEAD * kTcGather) {
        uint32_t w0[AHEAD], w1[AHEAD], w2[AHEAD];
#pragma unroll
        for (int t = 0; t < AHEAD; ++t) {
            const int b = b0 + kTcGather * t;
            const int i = 8 * (b / NCG) + (lane & 7), j0 = 8 * (4 * (b % NCG) + (lane >> 3));
            w0[t] = w1[t] = w2[t] = 0u;
            if (b < NB && i < L && j0 < L) {
                const uint8_t *src = chip + int64_t(i) * a.pitch + j0;
                const int left = L - j0;   // chip bytes from src on
                if (words) {
                    // the aligned words holding the chip bytes among src[0 .. 8)
                    const uintptr_t addr = reinterpret_cast<uintptr_t>(src);
                    const uint32_t *wp = reinterpret_cast<const uint32_t *>(addr & ~uintptr_t(3));
                    const int sh = int(addr & 3);
                    w0[t] = __ldg(wp);
                    if (4 - sh < left) w1[t] = __ldg(wp + 1);
                    if (sh > 0 && 8 - sh < left) w2[t] = __ldg(wp + 2);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const uint32_t bt = e < left ? uint32_t(__ldg(src + e)) : 0u;
                        if (e < 4) w0[t] |= bt << (8 * e);
                        else w1[t] |= bt << (8 * (e - 4));
                    }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < AHEAD; ++t) {
            const int b = b0 + kTcGather * t;
            const int i = 8 * (b / NCG) + (lane & 7), j0 = 8 * (4 * (b % NCG) + (lane >> 3));
            if (b < NB && j0 < N) {
                uint4 out = make_uint4(0u, 0u, 0u, 0u);
                if (i < L && j0 < L) {
                    uint32_t lo = w0[t], hi = w1[t];
                    if (words) {
                        const int sh = int(reinterpret_cast<uintptr_t>(chip + int64_t(i) * a.pitch + j0) & 3);
                        lo = __funnelshift_r(w0[t], w1[t], 8 * sh);
                        hi = __funnelshift_r(w1[t], w2[t], 8 * sh);
                    }
                    bytes_to_half(lo, off, out.x, out.y);
                    bytes_to_half(hi, off, out.z, out.w);
                    if (j0 + 8 > L) {   // the last piece of a row: zero past the chip
                        const int keep = L - j0;   // 1 .. 7 pixels
                        uint32_t hv[4] = {out.x, out.y, out.z, out.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (2 * e >= keep) hv[e] = 0u;
                            else if (2 * e + 1 >= keep) hv[e] &= 0xFFFFu;
                        }
                        out = make_uint4(hv[0], hv[1], hv[2], hv[3]);
                    }
                }
                *reinterpret_cast<uint4 *>(X + tc::k_major_offset(i, j0, G::SBO_X, 128)) = out;
            }
        }
    }
}

// The entry of the CTA's pair n, as soon as it is written; false if a role gave up. Called by whole warps, whose
// lanes vote at each poll: all leave at the same one with the same answer, also when an abort and the entry
// come about between the lanes' reads. (Bounded by the abort flag: a kernel that comes to a stop has a wait in the control
// warp, and that one gives up.)
__device__ __forceinline__ bool tc_entry(const PairSetup &e, uint32_t n, const volatile int *abort)
{
    for (;;) {
        const bool there = *const_cast<const volatile uint32_t *>(&e.seq) == n + 1;
        const bool stop = !there && *abort;
        if (__all_sync(0xffffffffu, there)) break;
        if (__any_sync(0xffffffffu, stop)) return false;
        __nanosleep(64);
    }
    asm volatile("" ::: "memory");   // shared-memory reads stay in order
    return true;
}

// the same for a thread by itself
__device__ __forceinline__ bool tc_entry_one(const PairSetup &e, uint32_t n, const volatile int *abort)
{
    while (*const_cast<const volatile uint32_t *>(&e.seq) != n + 1) {
        if (*abort) return false;
        __nanosleep(64);
    }
    asm volatile("" ::: "memory");
    return true;
}

template <int N>
__global__ void __launch_bounds__(kTcThreads, 1) corr_tc_kernel(const __grid_constant__ CorrArgs a, const uint4 *dtab, int *status)
{
    using G = TcGeo<N>;
    constexpr int NH = G::NH, KP = G::KP, NT = kTcThreads;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint32_t tmem_base;
    __shared__ __align__(8) TcBars bar;
    __shared__ __align__(8) uint64_t bar_last;
    __shared__ int s_abort;
    __shared__ PairSetup ring[4];      // the pairs in flight: gathered, drained, in the epilogue
    __shared__ uint32_t s_good[5];     // the events the relay has told of (wake)
    __shared__ uint32_t s_taken;       // the pairs whose entries the epilogue has read to the end
    __shared__ int s_key[kTcEpi], s_peak;   // the warps' largest values (as ints), the peak u M + v
    __shared__ double s_sq[kTcEpi];
    __shared__ float s_fit[9];
    constexpr int kRowWarps = (KP + 31) / 32;   // drain warps with rows, of each part
    // the same on every lane, and known to be: the roles' branches are uniform
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int quad = warp & 3;
    const int row = 32 * quad + lane;   // the TMEM lane of an epilogue or drain thread
    unsigned char *A = smem + G::OFF_A, *X = smem + G::OFF_X, *B5 = smem + G::OFF_B5;
    volatile int *ab = &s_abort;

    // the DFT table (already in its layout), once per CTA
    for (int i = tid; i < int(G::T_BYTES / 16); i += NT) reinterpret_cast<uint4 *>(smem)[i] = __ldg(dtab + i);
    if (warp == 0) tc::tmem_alloc(&tmem_base, G::TMEM_COLS);
    if (tid < 4) ring[tid].seq = 0;
    if (tid == 0) {
        s_abort = 0;
        s_taken = 0;
        for (int i = 0; i < 5; ++i) s_good[i] = 0;
        s_peak = INT_MAX;
        tc::mbar_init(&bar.xfull, kTcGather);
        tc::mbar_init(&bar.xfree, 1);
        tc::mbar_init(&bar.stage[1], 1);
        tc::mbar_init(&bar.stage[3], 1);
        tc::mbar_init(&bar.afull, kTcDrain);
        tc::mbar_init(&bar.stage[4], 1);
        tc::mbar_init(&bar.pfull, kTcDrain);
        tc::mbar_init(&bar.stage[0], 1);
        tc::mbar_init(&bar.b5full, kTcDrain);
        tc::mbar_init(&bar.stage[2], 1);
        tc::mbar_init(&bar.cfree, kTcEpi);
        tc::mbar_init(&bar_last, 1);
        for (int i = 0; i < kTcSlots; ++i) {
            tc::mbar_init(&bar.rfull[i], 1);
            tc::mbar_init(&bar.rfree[i], kRowWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t lane_base = uint32_t(32 * quad) << 16;
    const int L = a.L, M = a.M, R = a.R, W = a.W;
    const int NO = (M + 15) / 16 * 16;
    // TMEM columns of Yr (then [P1|P3]), of Yi (then [P4|P2]); Q and c start at 0
    const uint32_t CR = 2 * N, CI = uint32_t(NO);

    if (warp == kTcControl) {
        // ---- control: the MMAs, issued by one thread of the warp
        const uint32_t one = tc::elect_one();
        const uint32_t sT = tc::smem_u32(smem), sA = tc::smem_u32(A), sX = tc::smem_u32(X), sB5 = tc::smem_u32(B5);
        // the table's rows along M or N, contraction over its columns (k-step s: + KT s) ...
        const uint64_t c_rows = tc::smem_desc(sT, G::SBO_T, 128);
        // ... and its columns along M, contraction over its rows (k-step s: + 16 s); S starts N/2 rows on
        const uint64_t c_cols = tc::smem_desc(sT, 128, G::SBO_T);
        const uint64_t dX = tc::smem_desc(sX, 128, G::SBO_X), dA = tc::smem_desc(sA, 128, G::SBO_A);
        const uint64_t dB5 = tc::smem_desc(sB5, 128, G::SBO_B5);
        constexpr uint32_t KT = 2u * uint32_t(G::RT);
        const uint32_t idn = tc::instr_desc(128, N, false, false, false, false);
        const uint32_t id5 = tc::instr_desc(128, NO, true, true, false, false);
        auto wait = [&](uint64_t *b, uint32_t par) { return tc_wait_warp(b, par, ab); };
        // one pair per turn: the back of pair n - 1 (S4, S5) woven into the front of pair n (S1, S2), as
        // eight runs of MMAs through one loop
        bool ok = true, end = false;
        for (uint32_t n = 0; ok && !end; ++n) {
            const uint32_t par = n & 1u, prv = par ^ 1u;
#pragma unroll 1
            for (int step = n ? 0 : 2; step < 8 && ok; ++step) {
                if (step == 3 && !n) step = 5;        // no pair before
                if (step == 5 && end) break;
                uint32_t d = 0, acc = 0;                 // columns d: A from da (and, S5, B from db)
                uint64_t da = dA, db = dB5, *done = nullptr;
                if (step == 0) {          // S4: c of pair n - 2 is read (its columns are Q's), and S2's products (theirs too)
                    ok = (n < 2 || wait(&bar.cfree, par)) && wait(&bar.pfull, prv);
                } else if (step == 1) {
                    d = N;
                    da += N;
                    done = &bar.stage[0];
                } else if (step == 2) {   // S1, Yr
                    ok = wait(&bar.xfull, par);
                    end = ok && __any_sync(0xffffffffu, ring[n & 3].end);
                    d = CR;
                    da = c_rows;
                    done = &bar.stage[1];
                } else if (step == 3) {   // S5, C then S
                    ok = wait(&bar.b5full, prv);
                    da = c_cols;
                } else if (step == 4) {
                    da = c_cols + N / 2;
                    db += KP;
                    acc = 1;
                    done = &bar.stage[2];
                } else if (step == 5) {   // S1, Yi
                    d = CI;
                    da = c_rows + N / 2;
                    done = &bar.stage[3];
                } else if (step == 6) {   // S2
                    ok = wait(&bar.afull, par);
                    d = CR;
                } else {
                    d = CI;
                    da += N;
                    done = &bar.stage[4];
                }
                if (!ok) break;
                // (unrolled by kind, the steps constant: 55 cycles an MMA to issue)
                if (step == 3 || step == 4) {
#pragma unroll
                    for (int s = 0; s < KP / 16; ++s) tc::mma_f16_warp(tmem, da + 16u * s, db + 16u * s, id5, s ? 1u : acc, one);
                } else if (step == 2 || step == 5) {
                    if (!end)
#pragma unroll
                        for (int s = 0; s < N / 16; ++s) tc::mma_f16_warp(tmem + d, da + KT * s, dX + 16u * s, idn, s > 0, one);
                } else {
#pragma unroll
                    for (int s = 0; s < N / 16; ++s) tc::mma_f16_warp(tmem + d, da + 16u * s, c_rows + KT * s, idn, s > 0, one);
                }
                if (done && one) {
                    if (step == 2 && end) mbar_arrive(done);   // no pair: the drain warps leave
                    else tc::mma_commit(done);
                    if (step == 5) tc::mma_commit(&bar.xfree);
                }
            }
        }
        if (!ok) *ab = 1;
    } else if (warp == kTcRelay) {
        // ---- relay: the MMAs complete in the order they are issued in. After a wait gives up, the turn's
        // wake-ups (and the epilogue's next) go on without waiting, uncounted, and who is woken leaves.
        constexpr int DW = 32 * (kTcDrain + 1), EW = 32 * (kTcEpi + 1);
        bool ok = true, end = false;
        for (uint32_t n = 0; ok && !end; ++n) {
            int told = 0;   // C of the pair before: 1 come about, 2 not
#pragma unroll 1
            for (int ev = n ? 0 : 1; ev < 5; ++ev) {   // Q, Yr, C, Yi, Z: Q and C of the pair before
                if (ev == 2 && !n) continue;
                const uint32_t m = ev == 0 || ev == 2 ? n - 1 : n;
                ok = ok && tc_wait_warp(&bar.stage[ev], m & 1u, ab);
                if (ev == 1) end = ok && __any_sync(0xffffffffu, ring[n & 3].end);
                wake(kTcWake + ev, ev == 2 ? EW : DW, &s_good[ev], m, ok, lane);
                if (ev == 2) told = ok ? 1 : 2;
                if (end && ev == (n ? 2 : 1)) break;
            }
            if (!ok && told < 2) wake(kTcWakeC, EW, &s_good[2], told || !n ? n : n - 1, false, lane);
        }
    } else if (warp == kTcSetup) {
        // ---- the pairs ahead: lane l works out the CTA's next pair but l, then they are published in
        // order, each when its entry of the ring is free; invalid pairs are written here and passed over
        const int npairs = a.nwin * a.nf;
        const size_t ss = size_t(a.w) + 1;
        uint32_t n = 0;
        bool ok = true;
        auto publish = [&](PairSetup &c, bool mine) -> bool {   // entry n, by the lane whose it is
            while (n >= 4 && *const_cast<volatile uint32_t *>(&s_taken) < n - 3) {
                if (*ab) return false;
                __nanosleep(100);
            }
            __threadfence_block();
            if (mine) {
                c.seq = n;   // not a pair's yet
                ring[n & 3] = c;
                __threadfence_block();
                *const_cast<volatile uint32_t *>(&ring[n & 3].seq) = n + 1;
            }
            ++n;
            return true;
        };
        for (int p0 = blockIdx.x; p0 < npairs && ok; p0 += 32 * gridDim.x) {
            const int p = p0 + lane * gridDim.x;
            PairSetup c{};
            bool valid = false;
            if (p < npairs) {
                c.k = p / a.nf;
                c.f = p % a.nf;
                c.q = int64_t(c.f) * a.nwin + c.k;
                if (a.gross_mode == 1) {
                    c.gy = a.gross[2 * c.f];
                    c.gx = a.gross[2 * c.f + 1];
                } else if (a.gross_mode == 2) {
                    c.gy = a.gross[2 * c.q];
                    c.gx = a.gross[2 * c.q + 1];
                }
                c.sy = a.down[c.k / a.nx] + c.gy - R;
                c.sx = a.across[c.k % a.nx] + c.gx - R;
                const float norm = a.norm[c.k];
                valid = norm > 0 && c.sy >= 0 && c.sx >= 0 && c.sy + L <= a.h && c.sx + L <= a.w;
                if (valid) {
                    const uint32_t *sat = a.sat + size_t(c.f) * a.sat_fstride;
                    const size_t t0 = c.sy * ss + c.sx, t1 = t0 + L * ss;
                    const uint32_t box = sat[t1 + L] - sat[t0 + L] - sat[t1] + sat[t0];
                    const uint32_t LL = uint32_t(L) * uint32_t(L);
                    c.mean = int((box + LL / 2) / LL);
                    int eR = 0;
                    frexpf(float(W) * norm, &eR);   // the reference spectrum is scaled by 2^-(eR + 8)
                    c.scale = ldexpf(1.0f, eR + 17) / (float(N) * float(N) * norm);
                } else {
                    tc_invalid(&a, c.q);
                }
            }
            const uint32_t todo = __ballot_sync(0xffffffffu, valid), bad = __ballot_sync(0xffffffffu, p < npairs && !valid);
            if (a.surface)
                for (uint32_t b = bad; b; b &= b - 1) {
                    const int64_t q = __shfl_sync(0xffffffffu, c.q, __ffs(int(b)) - 1);
                    for (int i = lane; i < M * M; i += 32) a.surface[q * M * M + i] = 0.0f;
                }
            for (uint32_t b = todo; b && ok; b &= b - 1) {
                const int src = __ffs(int(b)) - 1;
                ok = __all_sync(0xffffffffu, publish(c, lane == src));
                // the window's spectrum into L2 before its pairs (on the CTAs around, at the same time) want it,
                // by one of them
                const int k = __shfl_sync(0xffffffffu, c.k, src), f = __shfl_sync(0xffffffffu, c.f, src);
                const char *r = reinterpret_cast<const char *>(a.spec_tc + size_t(k) * (N / 2) * KP);
                if (f == 0)
#pragma unroll 1
                    for (int i = lane; i < (N / 2) * KP * 16 / 128; i += 32)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(r + 128 * size_t(i)));
            }
        }
        PairSetup c{};
        c.end = true;
        if (ok) publish(c, lane == 0);
    } else if (warp == kTcFetch) {
        // ---- the reference spectrum of the pairs, chunk after chunk
        if (lane == 0) {
            uint32_t g = 0;   // chunks so far: slot g % kTcSlots, its use g / kTcSlots
            for (uint32_t n = 0;; ++n) {
                const PairSetup &e = ring[n & 3];
                if (!tc_entry_one(e, n, ab) || e.end) break;
                const float4 *r = a.spec_tc + size_t(e.k) * (N / 2) * KP;
                if (n && !tc_wait(&bar.stage[2], (n - 1) & 1u, ab)) break;   // S5 has read what the ring overwrites
                bool ok = true;
#pragma unroll 1
                for (int j = 0; j < G::NR; ++j, ++g) {
                    const uint32_t slot = g % kTcSlots, use = g / kTcSlots;
                    if (use && !(ok = tc_wait(&bar.rfree[slot], (use - 1) & 1u, ab))) break;
                    tc::mbar_expect_tx(&bar.rfull[slot], G::R_BYTES);
                    tc::bulk_load(B5 + slot * G::R_BYTES, r + size_t(8 * j) * KP, G::R_BYTES, &bar.rfull[slot]);
                }
                if (!ok) break;
            }
            // no copy into this CTA's memory may outlive it
            int none = 0;
            for (uint32_t u = g > kTcSlots ? g - kTcSlots : 0; u < g; ++u)
                tc_wait(&bar.rfull[u % kTcSlots], (u / kTcSlots) & 1u, &none);
        }
    } else if (warp < 16 && quad < 3) {
        // ---- drain: thread kappa holds row kappa of every stage's accumulator
        const int part = warp >> 2;   // of the quadrant's four warps
        const int kap = row;
        const bool has = 32 * quad < KP, in = kap < KP;   // rows of this warp (warp-uniform), of this thread
        constexpr int DW = 32 * (kTcDrain + 1);
        const uint32_t tl = tmem + lane_base;
        const float wgt = kap >= NH ? 0.0f : ((kap == 0 || 2 * kap == N) ? 1.0f : 2.0f) * (1.0f / 512.0f);
        for (uint32_t n = 0;; ++n) {
            // S1 -> S2's operand (row kappa, k = (Re | Im) N + i), 16 columns at a time
            auto drain1 = [&](uint32_t col, int im) {
                if (!has) return;
#pragma unroll 1
                for (int c = 16 * part; c < N; c += 16 * kTcParts) {
                    float y[16];
                    tc::tmem_ld16(tl + col + uint32_t(c), y);
                    if (im && kap == 0) {   // the Nyquist row is not S's row 0
#pragma unroll
                        for (int t = 0; t < 16; ++t) y[t] = 0.0f;
                    }
                    if (in) {
                        unsigned char *o = A + tc::k_major_offset(kap, im * N + c, G::SBO_A, 128);
                        *reinterpret_cast<uint4 *>(o) = pack8(y);
                        *reinterpret_cast<uint4 *>(o + 128) = pack8(y + 8);
                    }
                }
            };
            if (!woken<kTcWakeYr>(DW, &s_good[1], n)) break;
            if (__any_sync(0xffffffffu, ring[n & 3].end)) break;
            drain1(CR, 0);
            if (!woken<kTcWakeYi>(DW, &s_good[3], n)) break;
            drain1(CI, 1);
            warp_publish(&bar.afull, lane);

            // S3: chunk t, dealt to the quadrant's warps, gives P at ky = r, r = 8 t .. 8 t + 7, and at
            // N - r, r = 8 t + 1 .. 8 t + 8 (whole 16-byte pieces of the operand both), two frequencies per
            // instruction. R's ring holds them in pairs: (x, x', y, y') of two ky, then of their mirrors.
            if (!woken<kTcWakeZ>(DW, &s_good[4], n)) break;
#pragma unroll 1
            for (int t = part; t < G::NR && has; t += kTcParts) {
                const uint32_t g = n * uint32_t(G::NR) + uint32_t(t), slot = g % kTcSlots;
                tc_wait_warp(&bar.rfull[slot], (g / kTcSlots) & 1u, ab);   // if it gives up, the next wake-up says so
                const ulonglong2 *rs = reinterpret_cast<const ulonglong2 *>(B5 + slot * G::R_BYTES) + (in ? kap : 0);
                uint32_t o1[4], o2[4], o3[4], o4[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // columns r of the four products, and columns r + 1 for the mirrors
                    uint32_t a[4][4], m[4][4];
                    const uint32_t z = tl + uint32_t(8 * t + 4 * h);
                    tc::tmem_ld4_nowait(z + CR, a[0]);
                    tc::tmem_ld4_nowait(z + CI + N / 2, a[1]);
                    tc::tmem_ld4_nowait(z + CR + N / 2, a[2]);
                    tc::tmem_ld4_nowait(z + CI, a[3]);
                    tc::tmem_ld4_nowait(z + CR + 1, m[0]);
                    tc::tmem_ld4_nowait(z + CI + N / 2 + 1, m[1]);
                    tc::tmem_ld4_nowait(z + CR + N / 2 + 1, m[2]);
                    tc::tmem_ld4_nowait(z + CI + 1, m[3]);
                    tc::tmem_wait();
                    // column 0 of P2 and P3 is ky = N/2: column N/2 of P1 and P4, which lie before them
                    if (h == 0 && t == 0) a[1][0] = a[2][0] = 0u;
                    if (h == 1 && t == G::NR - 1) m[1][3] = m[2][3] = 0u;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const ulonglong2 rd = rs[(4 * h + 2 * j) * KP], rm = rs[(4 * h + 2 * j + 1) * KP];
                        const f32x2 a1 = pair2(a[0], j), a2 = pair2(a[1], j), m1 = pair2(m[0], j), m3 = pair2(m[2], j);
                        const f32x2 ar = sub2(a1, a2), na = sub2(a2, a1), ai = add2(pair2(a[2], j), pair2(a[3], j));
                        const f32x2 br = add2(m1, pair2(m[1], j)), bi = sub2(pair2(m[3], j), m3), nb = neg2(br);
                        o1[2 * h + j] = half2_bits(fma2(ar, rd.x, mul2(ai, rd.y)));
                        o2[2 * h + j] = half2_bits(fma2(ai, rd.x, mul2(na, rd.y)));
                        o3[3 - 2 * h - j] = half2_swapped(fma2(br, rm.x, mul2(bi, rm.y)));
                        o4[3 - 2 * h - j] = half2_swapped(fma2(bi, rm.x, mul2(nb, rm.y)));
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.rfree[slot]);
                if (in) {
                    unsigned char *o = A + tc::k_major_offset(kap, 8 * t, G::SBO_A, 128);
                    unsigned char *m = A + tc::k_major_offset(kap, N - 8 * t - 8, G::SBO_A, 128);
                    *reinterpret_cast<uint4 *>(o) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
                    *reinterpret_cast<uint4 *>(o + 16 * N) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
                    *reinterpret_cast<uint4 *>(m) = make_uint4(o3[0], o3[1], o3[2], o3[3]);
                    *reinterpret_cast<uint4 *>(m + 16 * N) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
                }
            }
            warp_publish(&bar.pfull, lane);

            // S4 -> S5's operand (MN-major: n = u, k = (Re | Im) KP + kappa) with the Hermitian weights and
            // 2^-9: chunk t gives u = 8 t .. 8 t + 7, and N - u for 8 t + 1 .. 8 t + 8 where the surface
            // reaches
            if (!woken<kTcWakeQ>(DW, &s_good[0], n)) break;
            const f32x2 wr = both(wgt), wi = both(kap == 0 ? 0.0f : wgt);   // S5 reads the Nyquist row as S's row 0
            auto load = [&](int u, uint32_t (&q)[4][8]) {   // Pr C, Pi S, Pi C, Pr S
                tc::tmem_ld8_nowait(tl + uint32_t(u), q[0]);
                tc::tmem_ld8_nowait(tl + uint32_t(3 * N / 2 + u), q[1]);
                tc::tmem_ld8_nowait(tl + uint32_t(N + u), q[2]);
                tc::tmem_ld8_nowait(tl + uint32_t(N / 2 + u), q[3]);
                tc::tmem_wait();
            };
            auto put = [&](int u, const uint32_t (&r)[4], const uint32_t (&m)[4]) {
                if (!in) return;
                unsigned char *o = B5 + tc::mn_major_offset(u, kap, G::SBO_B5, 128);
                *reinterpret_cast<uint4 *>(o) = make_uint4(r[0], r[1], r[2], r[3]);
                *reinterpret_cast<uint4 *>(o + 16 * KP) = make_uint4(m[0], m[1], m[2], m[3]);
            };
#pragma unroll 1
            for (int t = part; t < G::NR && has; t += kTcParts) {
                uint32_t q[4][8], r[4], m[4];
                if (8 * t < M) {
                    load(8 * t, q);
                    if (t == 0) q[1][0] = q[3][0] = 0u;   // column 0 of the S products is u = N/2
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        r[j] = half2_bits(mul2(add2(pair2(q[0], j), pair2(q[1], j)), wr));
                        m[j] = half2_bits(mul2(sub2(pair2(q[2], j), pair2(q[3], j)), wi));
                    }
                    put(8 * t, r, m);
                }
                if (N - 8 * t - 8 < M) {
                    load(8 * t + 1, q);
                    if (t == G::NR - 1) q[1][7] = q[3][7] = 0u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        r[3 - j] = half2_swapped(mul2(sub2(pair2(q[0], j), pair2(q[1], j)), wr));
                        m[3 - j] = half2_swapped(mul2(add2(pair2(q[2], j), pair2(q[3], j)), wi));
                    }
                    put(N - 8 * t - 8, r, m);
                }
            }
            warp_publish(&bar.b5full, lane);
        }
    } else if (warp < 24) {
        // ---- epilogue: thread v holds column v of the surface, the two warps of a quadrant alternate
        // groups of 8 rows u
        const int ew = warp - 16, part = ew >> 2, v = row, dw = a.dpitch;
        const bool mine = 32 * quad < M, vin = v < M;   // of this warp, of this thread
        for (uint32_t n = 0;; ++n) {
            const PairSetup &e = ring[n & 3];
            const bool known = tc_entry(e, n, ab);      // if not, the wake-up says to leave
            if (known && __any_sync(0xffffffffu, e.end)) break;
            const float *dcol = a.dinv + (vin ? v : 0);
            if (known) dcol += size_t(e.f) * a.dinv_fstride + size_t(e.sy) * dw + e.sx;
            const float scale = e.scale;
            // 8 rows' denominators (rows past the surface lie in the table or its padding, unused); the first
            // 24 are on their way while the tensor core works on the pair
            auto fetch = [&](float (&d)[8], int u0) {
                if (!mine || !known || u0 >= M) return;
                const float *p = dcol + u0 * dw;
#pragma unroll
                for (int t = 0; t < 8; ++t, p += dw) d[t] = ldg_here(p);
            };
            auto rows = [&](int u0, float (&x)[8]) {   // denominators to surface
                uint32_t cr[8];
                tc::tmem_ld8_nowait(tmem + lane_base + uint32_t(u0), cr);
                tc::tmem_wait();
#pragma unroll
                for (int t = 0; t < 8; ++t) x[t] *= __uint_as_float(cr[t]) * scale;
            };
            float d0[8], d1[8], d2[8];
            fetch(d0, 8 * part);
            fetch(d1, 8 * part + 16);
            fetch(d2, 8 * part + 32);
            if (!woken<kTcWakeC>(32 * (kTcEpi + 1), &s_good[2], n)) break;
            // this thread's largest value and its row (NaN never wins, ties keep the first)
            float best = -2.0f;
            int bu = 0;
            if (mine) {
#pragma unroll 1
                for (int u0 = 8 * part; u0 < M; u0 += 16) {
                    rows(u0, d0);
                    if (a.surface && vin) {
                        float *sv = a.surface + (e.q * M + u0) * M + v;
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            if (u0 + t < M) sv[t * M] = d0[t];
                    }
                    float m = -2.0f;
                    int first = 0;
#pragma unroll
                    for (int t = 7; t >= 0; --t) {
                        const bool up = d0[t] >= m && u0 + t < M;
                        m = up ? d0[t] : m;
                        first = up ? u0 + t : first;
                    }
                    bu = m > best ? first : bu;
                    best = m > best ? m : best;
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        d0[t] = d1[t];
                        d1[t] = d2[t];
                    }
                    fetch(d2, u0 + 48);
                }
            }
            // positive floats order as their bits do; a surface without a positive value has no peak
            const int mykey = __reduce_max_sync(0xffffffffu, vin ? __float_as_int(best) : INT_MIN);
            if (lane == 0) s_key[ew] = mykey;
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kTcEpi) : "memory");
            const int key = __reduce_max_sync(0xffffffffu, s_key[lane & 7]);
            const bool valid = key > 0;
            if (valid && mykey == key) {   // warp-uniform: where, the first in raster order if equal
                const int at = __reduce_min_sync(0xffffffffu, vin && __float_as_int(best) == key ? bu * M + v : INT_MAX);
                if (lane == 0) atomicMin(&s_peak, at);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kTcEpi) : "memory");
            const int at = valid ? s_peak : 0, pu = at / M, pv = at - pu * M;
            int i0 = 0, i1 = 0, j0 = 0, j1 = 0;
            // the SNR patch's sum of squares (of the FP32 values, in FP64) and the 3 x 3 values, with the same
            // arithmetic
            double sq = 0.0;
            auto release = [&] {   // this warp reads c's columns no more
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.cfree);
            };
            if (valid) snr_patch(M, a.stat, pu, pv, i0, i1, j0, j1);
            // the warp's first group with a row of the patch, if it holds columns of it (warp-uniform)
            const bool cols = valid && 32 * quad < j1 && 32 * quad + 32 > j0;
            int u0 = 8 * part + (max(i0 - 7 - 8 * part, 0) + 15) / 16 * 16;
            if (!cols || u0 >= i1) {
                release();
            } else {
                const bool col = v >= j0 && v < j1;
                const uint32_t fv = uint32_t(v - pv + 1);
#pragma unroll 1
                for (; u0 < i1; u0 += 32) {   // two groups at a time
                    fetch(d0, u0);
                    fetch(d1, u0 + 16);
                    rows(u0, d0);
                    if (u0 + 16 < M) rows(u0 + 16, d1);
                    if (u0 + 32 >= i1) release();
#pragma unroll 1
                    for (int ub = u0; ub < u0 + 32; ub += 16) {
                        // two chains of FP64 (one: 2507 us for 16 720p frames against 2498; four: the same as two)
                        double even = 0.0, odd = 0.0;
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            const uint32_t fu = uint32_t(ub + t - pu + 1);
                            float x = d0[t];
                            if (fu < 3u && fv < 3u) s_fit[fu * 3 + fv] = x;
                            if (!col || ub + t < i0 || ub + t >= i1) x = 0.0f;
                            (t & 1 ? odd : even) += double(x) * double(x);
                        }
                        sq += even + odd;
#pragma unroll
                        for (int t = 0; t < 8; ++t) d0[t] = d1[t];
                    }
                }
                for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            }
            if (lane == 0) s_sq[ew] = sq;
            // the last reads of the entry: the barrier is between them and the store below, which lets the setup warp
            // overwrite it (without one the compiler may move these plain loads past the store)
            const int64_t q = e.q;
            const int gy = e.gy, gx = e.gx;
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kTcEpi) : "memory");
            if (ew == 0 && lane == 0) {
                *const_cast<volatile uint32_t *>(&s_taken) = n + 1;
                s_peak = INT_MAX;
                if (!valid) {
                    tc_invalid(&a, q);
                } else {
                    double sum = 0.0;
#pragma unroll 1
                    for (int w = 0; w < kTcEpi; ++w) sum += s_sq[w];
                    const int count = (i1 - i0) * (j1 - j0);
                    if (a.peaks) {   // for the exact refinement of the peak, which writes the pair's outputs
                        PeakInfo &pi = a.peaks[q];
                        pi.valid = 1;
                        pi.u = pu;
                        pi.v = pv;
                        pi.count = count;
                        pi.sum = sum;
                        for (int t = 0; t < 9; ++t) pi.fit[t] = s_fit[t];
                    } else {
                        tc_outputs(&a, s_fit, pu, pv, gy, gx, sum, count, q);
                    }
                }
            }
        }
    } else {
        // ---- gather: the chip of the next pair, S1's operand (K-major rows i, columns j, zero outside L x L)
        // aligned 16-byte chunks when the frame rows start on 16-byte boundaries and hold whole chunks
        const bool rows16 = ((reinterpret_cast<uintptr_t>(a.frames) | uintptr_t(a.pitch) | uintptr_t(a.fstride)) & 15) == 0 &&
                            (a.w & 15) == 0;
        for (uint32_t n = 0;; ++n) {
            const PairSetup &c = ring[n & 3];
            if (!tc_entry(c, n, ab)) break;
            // S1 of the pair before has read X
            if (n && !tc_wait_warp(&bar.xfree, (n - 1) & 1u, ab)) break;
            const bool end = __any_sync(0xffffffffu, c.end);
            if (!end) tc_gather<N>(a, c, X, rows16, warp - 24, lane);
            warp_publish(&bar.xfull, lane);
            if (end) break;
        }
    }
    // every role has left its loop; after a wait gave up, what was issued is waited out (with the same
    // bound) before the tensor memory goes back
    __syncthreads();
    if (s_abort && warp == kTcControl) {
        if (tc::elect_one()) tc::mma_commit(&bar_last);
        int none = 0;
        tc_wait(&bar_last, 0, &none);
        if (status && lane == 0) atomicExch(status, 3);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem, G::TMEM_COLS);
}

// the reference spectra as S3 of the tensor-core form reads them: for window k and chunk t of 8
// frequencies, the rows kappa < KP side by side, 8 float4 each: for the pairs j, j + 1 (j = 0, 2, 4, 6)
// (x, x', y, y') of R[kappa][8 t + j], R[kappa][8 t + j + 1], then of R[kappa][N - 8 t - 1 - j] and
// R[kappa][N - 8 t - 2 - j]; scaled by 2^-(e + 8), 2^e > W norm (exact); rows NH .. KP - 1 zero. spec
// holds nwin x NH x N.
__global__ void spec_tc_kernel(const float2 *__restrict__ spec, const float *__restrict__ norm, int W, float4 *__restrict__ out,
                               int N, int nwin)
{
    const int NH = N / 2 + 1, KP = tc_kp(N);
    const int64_t total = int64_t(nwin) * (N / 2) * KP;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
        const int kap = int(i % KP);
        const int64_t ks = i / KP;
        const int slot = int(ks % (N / 2)), t = slot / 8, j = slot & 6;
        const int64_t k = ks / (N / 2);
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kap < NH) {
            int eR = 0;
            frexpf(float(W) * norm[k], &eR);
            const float sc = ldexpf(1.0f, -(eR + 8));
            const float2 *row = spec + (k * NH + kap) * N;
            const bool mirror = slot & 1;
            const float2 x = row[mirror ? N - 8 * t - 1 - j : 8 * t + j], y = row[mirror ? N - 8 * t - 2 - j : 8 * t + j + 1];
            o = make_float4(x.x * sc, y.x * sc, x.y * sc, y.y * sc);
        }
        out[i] = o;
    }
}

#endif   // __CUDACC__

// the DFT table of the tensor-core form as the kernel keeps it in shared memory (tc_table_offset), FP16
// bits; out holds tc_rt(N) * N halves
void tc_dft_table(int N, uint16_t *out);

}   // namespace b200
