// sat.cuh -- the exact summed-area tables of the frames and the per-shift variance denominators.
//
// For each frame (h x w uint8) the tables are (h + 1) x (w + 1) with a first row and column of
// zeros, as the reference's (slipcam cxx/cpu.cpp:24-42, cxx/cuda.cu:72-110):
//   sat  = sum of x   as uint32, exact modulo 2^32 (every box sum below 2^32 -- all boxes up to
//          16.8 M pixels -- comes out exact from the 4-corner difference in wrapping arithmetic;
//          the table itself is exact outright for frames below 16.8 M pixels)
//   sat2 = sum of x^2, as uint32 modulo 2^32 for the correlation, whose windows hold at most 256 x 256
//          pixels (256^2 255^2 < 2^32, so every box sum comes out exact in the same way), and as int64,
//          exact outright, for callers that ask for the table itself
// Two passes, both bound by the tables' bytes: a warp scans each row, four pixels per lane; then a
// block takes 32 columns, holding a chunk of rows in registers so that each entry is read once and
// written once. Measured for 16 frames of 1280 x 720 (the 64-bit table, a scan per pixel and two reads
// of every entry before): rows 54.8 to 29.3 us, columns 117.7 to 66.1,
// the denominators (four boxes per thread, a reciprocal root for a division, a root and a division) 84.0 to 61.5.
//
// dinv_kernel then gives, for every W x W box of a frame, 1 / sqrt(v / n) with v = n S2 - S^2 from
// the integer box sums in int64 and the root in FP64 (0 where v <= 0, the reference's
// "not normalizable" case, cxx/surface.h:30-35).
#pragma once

#include "common.cuh"

namespace b200 {

#ifdef __CUDACC__

// one warp per row: rows y + 1 of the tables, and row 0 (zeros) by the warp of row 0. Lane l scans pixels
// x0 + 4 l .. x0 + 4 l + 3 (one word where the rows start on words); the sums pass through shared memory, so
// that the stores, whose rows of w + 1 entries start anywhere, are contiguous over the lanes
template <class T2>
__global__ void __launch_bounds__(256) sat_rows_kernel(const uint8_t *frames, int64_t fstride, int pitch,
                                                       int h, int w, uint32_t *sat, T2 *sat2, int64_t sfs)
{
    __shared__ __align__(16) uint32_t sums[8][2][128];
    const int f = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = blockIdx.x * 8 + warp;
    if (y >= h) return;
    const size_t ss = size_t(w) + 1;
    uint32_t *s = sat + f * sfs;
    T2 *s2 = sat2 + f * sfs;
    if (y == 0)
        for (int x = lane; x <= w; x += 32) {
            s[x] = 0;
            s2[x] = 0;
        }
    const uint8_t *row = frames + f * fstride + int64_t(y) * pitch;
    const bool words = (reinterpret_cast<uintptr_t>(row) & 3) == 0;
    auto load = [&](int x) -> uint32_t {   // pixels x .. x + 3, zeros past the row
        if (words && x + 4 <= w) return __ldg(reinterpret_cast<const uint32_t *>(row + x));
        uint32_t v = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (x + i < w) v |= uint32_t(__ldg(row + x + i)) << (8 * i);
        return v;
    };
    uint32_t *o = s + (y + 1) * ss;
    T2 *o2 = s2 + (y + 1) * ss;
    if (lane == 0) {
        o[0] = 0;
        o2[0] = 0;
    }
    uint32_t (*b)[128] = sums[warp];
    uint32_t carry = 0;
    T2 carry2 = 0;
    uint32_t next = load(4 * lane);
    for (int x0 = 0; x0 < w; x0 += 128) {
        const uint32_t v = next;
        if (x0 + 128 < w) next = load(x0 + 128 + 4 * lane);
        const uint32_t p0 = v & 255, p1 = (v >> 8) & 255, p2 = (v >> 16) & 255, p3 = v >> 24;
        // the sums within 128 pixels fit 32 bits: 128 x 255^2 < 2^23
        uint32_t sa = p0 + p1 + p2 + p3, sb = p0 * p0 + p1 * p1 + p2 * p2 + p3 * p3;
        const uint32_t ta = sa, tb = sb;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t na = __shfl_up_sync(0xffffffffu, sa, d), nb = __shfl_up_sync(0xffffffffu, sb, d);
            if (lane >= d) {
                sa += na;
                sb += nb;
            }
        }
        uint4 a, q;
        a.x = sa - ta + p0;
        a.y = a.x + p1;
        a.z = a.y + p2;
        a.w = sa;
        q.x = sb - tb + p0 * p0;
        q.y = q.x + p1 * p1;
        q.z = q.y + p2 * p2;
        q.w = sb;
        __syncwarp();   // the last step's reads
        *reinterpret_cast<uint4 *>(&b[0][4 * lane]) = a;
        *reinterpret_cast<uint4 *>(&b[1][4 * lane]) = q;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = x0 + 32 * i + lane;
            if (x < w) {
                o[1 + x] = carry + b[0][32 * i + lane];
                o2[1 + x] = carry2 + b[1][32 * i + lane];
            }
        }
        carry += __shfl_sync(0xffffffffu, sa, 31);
        carry2 += __shfl_sync(0xffffffffu, sb, 31);
    }
}

constexpr int kSatSegs = 16, kSatRows = 12;   // segments of a chunk, rows of a segment

// the column sums of the row prefix sums; block (32, kSatSegs): 32 columns, chunks of kSatSegs segments of
// kSatRows rows, each row of a segment in a register of its thread
template <class T2>
__global__ void __launch_bounds__(32 * kSatSegs) sat_cols_kernel(int h, int w, uint32_t *sat, T2 *sat2, int64_t sfs)
{
    __shared__ uint32_t c32[kSatSegs][32];
    __shared__ T2 c64[kSatSegs][32];
    const int f = blockIdx.y, tx = threadIdx.x, ty = threadIdx.y;
    const int x = blockIdx.x * 32 + tx;
    const size_t ss = size_t(w) + 1;
    uint32_t *s = sat + f * sfs + x;
    T2 *s2 = sat2 + f * sfs + x;
    uint32_t base = 0;
    T2 base2 = 0;
    for (int r0 = 1; r0 <= h; r0 += kSatSegs * kSatRows) {
        const int r = r0 + ty * kSatRows;
        uint32_t v[kSatRows];
        T2 v2[kSatRows];
#pragma unroll
        for (int j = 0; j < kSatRows; ++j) {
            const bool in = x <= w && r + j <= h;
            v[j] = in ? s[(r + j) * ss] : 0u;
            v2[j] = in ? s2[(r + j) * ss] : T2(0);
        }
#pragma unroll
        for (int j = 1; j < kSatRows; ++j) {
            v[j] += v[j - 1];
            v2[j] += v2[j - 1];
        }
        c32[ty][tx] = v[kSatRows - 1];
        c64[ty][tx] = v2[kSatRows - 1];
        __syncthreads();
        uint32_t ca = base;
        T2 cb = base2;
#pragma unroll
        for (int t = 0; t < kSatSegs; ++t) {
            const uint32_t a = c32[t][tx];
            const T2 b = c64[t][tx];
            if (t < ty) {
                ca += a;
                cb += b;
            }
            base += a;
            base2 += b;
        }
#pragma unroll
        for (int j = 0; j < kSatRows; ++j)
            if (x <= w && r + j <= h) {
                s[(r + j) * ss] = ca + v[j];
                s2[(r + j) * ss] = cb + v2[j];
            }
        __syncthreads();   // the segments' sums are the next chunk's
    }
}

constexpr int kDinvCols = 4;   // boxes per thread, 128 columns apart: their 32 loads are in flight together

// dinv[y][x] (row pitch dpitch floats) for the W x W boxes at (y, x), y <= h - W, x <= w - W; and,
// when bstat is given, {the box's pixel sum, the bits of its dinv} in the same layout
__global__ void __launch_bounds__(128) dinv_kernel(const uint32_t *sat, const uint32_t *sat2, int64_t sfs,
                                                   int h, int w, int W, float *dinv, int64_t dfs, int dpitch,
                                                   int2 *bstat = nullptr)
{
    const int x0 = blockIdx.x * 128 * kDinvCols + threadIdx.x, y = blockIdx.y, f = blockIdx.z;
    const size_t ss = size_t(w) + 1;
    const uint32_t *s = sat + f * sfs + y * ss, *s2 = sat2 + f * sfs + y * ss;
    const int64_t n = int64_t(W) * W;
    const double rn = 1.0 / double(n);
    uint32_t bs[kDinvCols], bs2[kDinvCols];
#pragma unroll
    for (int i = 0; i < kDinvCols; ++i) {
        const int x = x0 + 128 * i;
        if (x > w - W) continue;
        const size_t a = x, b = a + W, c = a + W * ss, d = c + W;
        bs[i] = s[d] - s[b] - s[c] + s[a];
        bs2[i] = s2[d] - s2[b] - s2[c] + s2[a];
    }
#pragma unroll
    for (int i = 0; i < kDinvCols; ++i) {
        const int x = x0 + 128 * i;
        if (x > w - W) continue;
        const int64_t v = n * int64_t(bs2[i]) - int64_t(bs[i]) * int64_t(bs[i]);
        const float di = v > 0 ? float(rsqrt(double(v) * rn)) : 0.0f;
        dinv[f * dfs + size_t(y) * dpitch + x] = di;
        if (bstat) bstat[f * dfs + size_t(y) * dpitch + x] = make_int2(int(bs[i]), __float_as_int(di));
    }
}

#endif   // __CUDACC__

}   // namespace b200
