// diff.cuh -- the kernels of the differentiable correlation (the math is in diff.h)
#pragma once

#include "corr_fft.cuh"
#include "diff.h"

namespace b200 {

#ifdef __CUDACC__

// the mean of a pair's L x L chip, in double, every thread of the block receives it
template <int NT>
__device__ double chip_mean(const float *x, int L)
{
    __shared__ double red[NT / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < L * L; i += NT) s += x[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < NT / 32; ++i) t += red[i];
    __syncthreads();
    return t / (double(L) * L);
}

// a frame index clamped to [0, n): the edge pixel repeats beyond the frame
__device__ __forceinline__ int clamp_index(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

// The interpolation is separable, and so is its transpose: in the kernels below a thread takes a column of a
// chip and a segment of its rows, applies the six taps along each row as it comes and keeps the last six rows'
// results in registers for the taps down the column: 12 multiply-adds and 6 loads per pixel instead of 36 and
// 36 (the gather, bound by its instructions: 91.6 to 29.0 us), and one atomic per frame pixel that a segment touches
// instead of 36 per chip pixel (the scatter: 234 to 67.9 us; both for 1,025 pairs of 80 x 80 chips). The segments fill
// the block: blockDim / columns of them.
__device__ __forceinline__ int column_rows(int cols, int rows)
{
    const int segs = max(1, int(blockDim.x) / cols);
    return (rows + segs - 1) / segs;
}

// for each row i of [i0, i1): out(i, ring), ring(d) the result of row(i + d), d < kTaps, for the rows
// row(i0) .. row(i1 + kTaps - 2) in turn
template <class T, class Row, class Out>
__device__ __forceinline__ void slide_rows(int i0, int i1, Row &&row, Out &&out)
{
    T r[kTaps];
#pragma unroll
    for (int d = 0; d < kTaps - 1; ++d) r[d] = row(i0 + d);
    for (int i = i0; i < i1; i += kTaps) {
#pragma unroll
        for (int t = 0; t < kTaps; ++t) {
            if (i + t >= i1) break;
            r[(t + kTaps - 1) % kTaps] = row(i + t + kTaps - 1);
            out(i + t, [&](int d) { return r[(t + d) % kTaps]; });
        }
    }
}

// the chips: one CTA per pair
__global__ void __launch_bounds__(256) diff_gather_kernel(DiffArgs a)
{
    const int64_t q = blockIdx.x;
    const DiffPair p = diff_pair(a, q);
    const int L = a.L;
    float *x = a.chips + q * L * L;
    if (!p.ok) {
        for (int i = threadIdx.x; i < L * L; i += blockDim.x) x[i] = 0.0f;
        return;
    }
    float wy[kTaps], wx[kTaps], dw[kTaps];
    interp_weights(p.ay, wy, dw);
    interp_weights(p.ax, wx, dw);
    const float *F = a.frames + p.f * a.fstride;
    const int rows = column_rows(L, L), segs = (L + rows - 1) / rows;
    for (int idx = threadIdx.x; idx < segs * L; idx += blockDim.x) {
        const int j = idx % L, i0 = idx / L * rows;
        int cx[kTaps];
#pragma unroll
        for (int e = 0; e < kTaps; ++e) cx[e] = clamp_index(p.x0 + kTap0 + j + e, a.w);
        slide_rows<float>(
            i0, min(L, i0 + rows),
            [&](int i) {
                const float *r = F + int64_t(clamp_index(p.y0 + kTap0 + i, a.h)) * a.pitch;
                float s = 0.0f;
#pragma unroll
                for (int e = 0; e < kTaps; ++e) s += wx[e] * r[cx[e]];
                return s;
            },
            [&](int i, auto ring) {
                float v = 0.0f;
#pragma unroll
                for (int d = 0; d < kTaps; ++d) v += wy[d] * ring(d);
                x[i * L + j] = v;
            });
    }
}

// the box statistics of each pair: (mu, 1 / s) for every (u, v), sums in FP64 over strips of up to kStatStrip
// grid rows: a thread takes a column of the chip and a segment of the strip, then kStatSlide neighbours along a
// grid row (an odd number: the lanes' 8-byte reads are then conflict-free). The boxes of a segment share the rows
// (columns) that are in all of them; a box adds those of the ones before that only it and its predecessors
// hold and those after. Nothing is subtracted: a sum that slides by what enters and leaves keeps the rounding of
// pixels that have left, and a black box beside texture is then not flat (its 1 / s about 1e5 instead of 0). It
// reads as few pixels as sliding does. Summing along the rows first, W loads and conversions per box and row:
// 65.5 us for 1,025 pairs of 80 x 80 chips, this way 33.3 us.
// A box is flat, 1 / s = 0, where n var is within its own rounding: each sum is a chain of at most 2 W + 4
// additions of non-negative (or, for S1, bounded by those) terms, so with u = 2^-53 S2 is off by at most
// (2 W + 4) u S2, S1^2 / n by twice that and its own two roundings, by Cauchy-Schwarz.
constexpr int kStatStrip = 16, kStatSlide = 3;
__global__ void __launch_bounds__(256) diff_stats_kernel(DiffArgs a)
{
    extern __shared__ double rs[];   // 2 x kStatStrip x L: column sums of x and x^2 over W rows
    const int64_t q = blockIdx.x;
    const DiffPair p = diff_pair(a, q);
    const int L = a.L, M = a.M, W = a.W;
    float *st = a.stats + q * M * M * 2;
    if (!p.ok) {
        for (int i = threadIdx.x; i < 2 * M * M; i += blockDim.x) st[i] = 0.0f;
        return;
    }
    const float *x = a.chips + q * L * L;
    const double n = double(W) * W, flat = (6 * W + 16) * 0x1p-53;
    const int strips = (M + kStatStrip - 1) / kStatStrip, su = (M + strips - 1) / strips;
    double *r1 = rs, *r2 = rs + L * kStatStrip;
    for (int u0 = 0; u0 < M; u0 += su) {
        const int nu = min(su, M - u0), rows = min(W, column_rows(L, nu)), segs = (nu + rows - 1) / rows;
        for (int idx = threadIdx.x; idx < segs * L; idx += blockDim.x) {
            const int j = idx % L, t0 = idx / L * rows, t1 = min(nu, t0 + rows);
            const float *c = x + (u0 + t0) * L + j;
            double s1 = 0.0, s2 = 0.0;
            for (int t = t1 - 2; t >= t0; --t) {   // the rows before the shared ones, from box t on
                const double e = c[(t - t0) * L];
                s1 += e;
                s2 += e * e;
                r1[t * L + j] = s1;
                r2[t * L + j] = s2;
            }
            s1 = s2 = 0.0;
#pragma unroll 8
            for (int i = t1 - t0 - 1; i < W; ++i) {
                const double e = c[i * L];
                s1 += e;
                s2 += e * e;
            }
            for (int t = t0; t < t1; ++t) {
                if (t > t0) {   // the row after, box t's last
                    const double e = c[(t - t0 - 1 + W) * L];
                    s1 += e;
                    s2 += e * e;
                }
                const bool more = t < t1 - 1;
                r1[t * L + j] = s1 + (more ? r1[t * L + j] : 0.0);
                r2[t * L + j] = s2 + (more ? r2[t * L + j] : 0.0);
            }
        }
        __syncthreads();
        const int ng = (M + kStatSlide - 1) / kStatSlide;
        for (int idx = threadIdx.x; idx < nu * ng; idx += blockDim.x) {
            const int t = idx / ng, v0 = idx % ng * kStatSlide;
            const double *c1 = r1 + t * L + v0, *c2 = r2 + t * L + v0;
            double s1 = 0.0, s2 = 0.0;
            for (int j = kStatSlide - 1; j < W; ++j) {
                s1 += c1[j];
                s2 += c2[j];
            }
            double b1[kStatSlide], b2[kStatSlide];   // the columns before the shared ones, from box k on
            b1[kStatSlide - 1] = b2[kStatSlide - 1] = 0.0;
#pragma unroll
            for (int k = kStatSlide - 2; k >= 0; --k) {
                b1[k] = b1[k + 1] + c1[k];
                b2[k] = b2[k + 1] + c2[k];
            }
#pragma unroll
            for (int k = 0; k < kStatSlide; ++k) {
                if (v0 + k >= M) break;
                if (k > 0) {
                    s1 += c1[k - 1 + W];
                    s2 += c2[k - 1 + W];
                }
                const double S1 = s1 + b1[k], S2 = s2 + b2[k];
                const double var_n = S2 - S1 * S1 / n;   // n var
                const int uv = (u0 + t) * M + v0 + k;
                st[2 * uv] = float(S1 / n);
                st[2 * uv + 1] = var_n > flat * S2 ? float(1.0 / sqrt(var_n)) : 0.0f;
            }
        }
        __syncthreads();
    }
}

// the normalized surfaces and the peak outputs: one CTA per pair, the FFT passes of corr_kernel
// on the float chip (minus its mean, which the zero-mean reference window does not see)
template <int N, int NT>
__global__ void __launch_bounds__(NT, corr_blocks(N)) diff_corr_kernel(DiffArgs a)
{
    using G = Geo<N>;
    extern __shared__ float4 smem_raw[];
    float2 *S = reinterpret_cast<float2 *>(smem_raw);
    float2 *TW = S + size_t(N) * G::NHP, *TWI = TW + N;
    float *Sr = reinterpret_cast<float *>(S);
    const int64_t q = blockIdx.x;
    const DiffPair p = diff_pair(a, q);
    const int L = a.L, M = a.M;
    if (!p.ok) {
        if (threadIdx.x == 0) {
            invalid_outputs(q, a.offset, a.peak, a.snr, a.cov);
            a.peak_at[q] = -1;
        }
        for (int i = threadIdx.x; i < M * M; i += NT) a.surface[q * M * M + i] = 0.0f;
        return;
    }
    for (int i = threadIdx.x; i < 2 * N; i += NT) TW[i] = a.twiddles[i];
    const float *x = a.chips + q * L * L;
    const float mean = float(chip_mean<NT>(x, L));
    const int Lr = (L + 1) & ~1;
    for (int idx = threadIdx.x; idx < Lr * N; idx += NT) {
        const int i = idx / N, j = idx % N;
        Sr[size_t(i) * G::RP + j] = (i < L && j < L) ? x[i * L + j] - mean : 0.0f;
    }
    __syncthreads();
    const DevExec ex{int(threadIdx.x >> 5), NT / 32};
    row_forward<N>(ex, S, Lr / 2, TW);
    __syncthreads();
    col_pass<N, true>(ex, S, Lr, M, TW, TWI, a.spec + size_t(p.k) * G::NH * N, nullptr);
    __syncthreads();
    const float inv = 1.0f / (float(N) * float(N) * a.norm[p.k]);
    const float *st = a.stats + q * M * M * 2;
    row_inverse<N>(ex, S, M, TWI, [&](int u, int c, float v) { return v * inv * st[2 * (u * M + c) + 1]; });
    __syncthreads();
    for (int i = threadIdx.x; i < M * M; i += NT) a.surface[q * M * M + i] = Sr[size_t(i / M) * G::RP + i % M];
    surface_peak<NT>(Sr, G::RP, M, a.R, a.stat, p.gy, p.gx, a.W * a.W, q, a.offset, a.peak, a.snr, a.cov, a.peak_at);
}

// the chip cotangents from the surface cotangents: one CTA per pair
template <int N, int NT>
__global__ void __launch_bounds__(NT, corr_blocks(N)) adjoint_kernel(DiffArgs a)
{
    using G = Geo<N>;
    extern __shared__ float4 smem_raw[];
    float2 *S = reinterpret_cast<float2 *>(smem_raw);
    float2 *TW = S + size_t(N) * G::NHP, *TWI = TW + N;
    float *Sr = reinterpret_cast<float *>(S);
    const int64_t q = blockIdx.x;
    const DiffPair p = diff_pair(a, q);
    const int L = a.L, M = a.M, W = a.W;
    float *gx = a.g_chips + q * L * L;
    if (!p.ok) {
        for (int i = threadIdx.x; i < L * L; i += NT) gx[i] = 0.0f;
        return;
    }
    for (int i = threadIdx.x; i < 2 * N; i += NT) TW[i] = a.twiddles[i];
    const float *gs = a.g_surface + q * M * M, *rho = a.surface + q * M * M, *st = a.stats + q * M * M * 2;
    const float *x = a.chips + q * L * L;
    const float rnorm = 1.0f / a.norm[p.k];
    // the reversed A = G / (norm s) at rows and columns [W - 1, L)
    const int Lr = (L + 1) & ~1;
    for (int idx = threadIdx.x; idx < Lr * N; idx += NT) {
        const int i = idx / N, j = idx % N;
        float v = 0.0f;
        if (i >= W - 1 && i < L && j >= W - 1 && j < L) {
            const int uv = (L - 1 - i) * M + (L - 1 - j);
            v = gs[uv] * st[2 * uv + 1] * rnorm;
        }
        Sr[size_t(i) * G::RP + j] = v;
    }
    __syncthreads();
    const DevExec ex{int(threadIdx.x >> 5), NT / 32};
    row_forward<N>(ex, S, Lr / 2, TW);
    __syncthreads();
    col_pass<N, true>(ex, S, Lr, L, TW, TWI, a.spec + size_t(p.k) * G::NH * N, nullptr);
    __syncthreads();
    const float inv = 1.0f / (float(N) * float(N));
    row_inverse<N>(ex, S, L, TWI, [&](int u, int c, float v) {
        gx[(L - 1 - u) * L + (L - 1 - c)] = v * inv;
        return v;
    });
    __syncthreads();

    // minus sum over the boxes holding p of B (x[p] - mu), B = G rho / s^2, as two box filters of
    // B and B mu over the M x M grid (x and mu taken about the chip mean). Along the rows a warp scans a grid
    // row in FP64 and takes differences; down the columns a thread sums the first position of its segment of
    // kAdjointRows rows and slides. The chip's columns go in tiles whose two M x tile sums fit the FFT's tile
    // of shared memory. (One thread per grid row and per column, in two passes, left the block waiting for
    // its serial loops: 234 to 134 us, with the threads of corr_threads for 1,025 pairs of 80 x 80 chips.)
    constexpr int kAdjointRows = 16;
    const float mean = float(chip_mean<NT>(x, L));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = NT / 32;
    double *P = reinterpret_cast<double *>(S) + warp * M;   // the warp's prefix sums
    float2 *cb = S + NW * M;                                // M x tile: the sums along the rows of {B, B mu}
    const int fit = (N * G::NHP - NW * M) / M, tile = min(L, fit >= 32 ? fit & ~31 : fit);
    for (int p0 = 0; p0 < L; p0 += tile) {
        const int np = min(tile, L - p0);
        for (int u = warp; u < M; u += NW)
            for (int pass = 0; pass < 2; ++pass) {
                double carry = 0.0;
                for (int v0 = 0; v0 < M; v0 += 32) {
                    const int v = v0 + lane, uv = u * M + v;
                    double b = 0.0;
                    if (v < M) {
                        const float is = st[2 * uv + 1];
                        float t = gs[uv] * rho[uv] * is * is;
                        if (pass == 1) t *= st[2 * uv] - mean;
                        b = t;
                    }
                    for (int o = 1; o < 32; o <<= 1) {
                        const double t = __shfl_up_sync(0xffffffffu, b, o);
                        if (lane >= o) b += t;
                    }
                    if (v < M) P[v] = carry + b;
                    carry += __shfl_sync(0xffffffffu, b, 31);
                }
                __syncwarp();
                for (int c = lane; c < np; c += 32) {
                    const int px = p0 + c, lo = px - W;
                    const float t = float(P[min(px, M - 1)] - (lo >= 0 ? P[lo] : 0.0));
                    if (pass == 0)
                        cb[u * np + c].x = t;
                    else
                        cb[u * np + c].y = t;
                }
                __syncwarp();
            }
        __syncthreads();
        const int npw = (np + 31) & ~31, segs = (L + kAdjointRows - 1) / kAdjointRows;
        for (int idx = threadIdx.x; idx < segs * npw; idx += NT) {
            const int c = idx % npw, y0 = idx / npw * kAdjointRows, y1 = min(L, y0 + kAdjointRows);
            if (c >= np) continue;
            double s0 = 0.0, s1 = 0.0;
            for (int u = max(0, y0 - W); u < min(y0, M); ++u) {   // the grid rows over row y0 - 1
                const float2 t = cb[u * np + c];
                s0 += t.x;
                s1 += t.y;
            }
            for (int py = y0; py < y1; ++py) {
                if (py < M) {
                    const float2 t = cb[py * np + c];
                    s0 += t.x;
                    s1 += t.y;
                }
                if (py - W >= 0 && py - W < M) {
                    const float2 t = cb[(py - W) * np + c];
                    s0 -= t.x;
                    s1 -= t.y;
                }
                const int i = py * L + p0 + c;
                gx[i] = float(float(gx[i] - (x[i] - mean) * s0) + s1);
            }
        }
        __syncthreads();
    }
}

// the frame and shift cotangents from the chip cotangents (the transposed interpolation): one CTA
// per pair, frame cotangents accumulated atomically (windows overlap)
__global__ void __launch_bounds__(256) diff_scatter_kernel(DiffArgs a)
{
    __shared__ float red[2][8];
    const int64_t q = blockIdx.x;
    const DiffPair p = diff_pair(a, q);
    const int L = a.L;
    if (!p.ok) {
        if (threadIdx.x == 0 && a.g_shift) a.g_shift[2 * q] = a.g_shift[2 * q + 1] = 0.0f;
        return;
    }
    float wy[kTaps], wx[kTaps], dy[kTaps], dx[kTaps];
    interp_weights(p.ay, wy, dy);
    interp_weights(p.ax, wx, dx);
    const int64_t base = p.f * a.fstride;
    const float *F = a.frames + base;
    float *GF = a.g_frames ? a.g_frames + base : nullptr;
    const float *gx = a.g_chips + q * L * L;
    float ty = 0.0f, tx = 0.0f;
    if (a.g_shift) {
        const int rows = column_rows(L, L), segs = (L + rows - 1) / rows;
        for (int idx = threadIdx.x; idx < segs * L; idx += blockDim.x) {
            const int j = idx % L, i0 = idx / L * rows;
            int cx[kTaps];
#pragma unroll
            for (int e = 0; e < kTaps; ++e) cx[e] = clamp_index(p.x0 + kTap0 + j + e, a.w);
            slide_rows<float2>(
                i0, min(L, i0 + rows),
                [&](int i) {   // {F interpolated along the row, its derivative}
                    const float *r = F + int64_t(clamp_index(p.y0 + kTap0 + i, a.h)) * a.pitch;
                    float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int e = 0; e < kTaps; ++e) {
                        const float f = r[cx[e]];
                        s.x += wx[e] * f;
                        s.y += dx[e] * f;
                    }
                    return s;
                },
                [&](int i, auto ring) {
                    const float g = gx[i * L + j];
                    if (g == 0.0f) return;
                    float sy = 0.0f, sx = 0.0f;
#pragma unroll
                    for (int d = 0; d < kTaps; ++d) {
                        const float2 r = ring(d);
                        sy += dy[d] * r.x;
                        sx += wy[d] * r.y;
                    }
                    ty += g * sy;
                    tx += g * sx;
                });
        }
    }
    if (GF) {
        const int T = L + kTaps - 1;   // the chip's frame pixels: T x T from (y0 + kTap0, x0 + kTap0)
        const int rows = column_rows(T, T), segs = (T + rows - 1) / rows;
        for (int idx = threadIdx.x; idx < segs * T; idx += blockDim.x) {
            const int c = idx % T, r0 = idx / T * rows;
            const int col = clamp_index(p.x0 + kTap0 + c, a.w);
            slide_rows<float>(
                r0, min(T, r0 + rows),
                [&](int t) {   // chip row t - 5 spread along the frame's columns
                    const int i = t - (kTaps - 1);
                    float s = 0.0f;
                    if (i >= 0 && i < L)
#pragma unroll
                        for (int e = 0; e < kTaps; ++e)
                            if (unsigned(c - e) < unsigned(L)) s += wx[e] * gx[i * L + c - e];
                    return s;
                },
                [&](int r, auto ring) {
                    float s = 0.0f;
#pragma unroll
                    for (int d = 0; d < kTaps; ++d) s += wy[kTaps - 1 - d] * ring(d);
                    if (s != 0.0f)
                        atomicAdd(GF + int64_t(clamp_index(p.y0 + kTap0 + r, a.h)) * a.pitch + col, s);
                });
        }
    }
    if (!a.g_shift) return;
    for (int o = 16; o > 0; o >>= 1) {
        ty += __shfl_xor_sync(0xffffffffu, ty, o);
        tx += __shfl_xor_sync(0xffffffffu, tx, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = ty;
        red[1][threadIdx.x >> 5] = tx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float sy = 0.0f, sx = 0.0f;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) {
            sy += red[0][w];
            sx += red[1][w];
        }
        a.g_shift[2 * q] = sy;
        a.g_shift[2 * q + 1] = sx;
    }
}

#endif   // __CUDACC__

#ifdef __CUDACC__

// the surface cotangents from the offset cotangents: one thread per pair, into a zeroed g_surface
__global__ void offset_adjoint_kernel(const float *surface, const int *peak_at, const float *g_offset, float *g_surface,
                                      int M, int64_t pairs)
{
    const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= pairs) return;
    const int at = peak_at[q];
    if (at < 0) return;
    const int u = at / M, v = at % M;
    double g[9];
    const float *s = surface + q * M * M;
    offset_adjoint(s + u * M + v, M, M, u, v, g_offset[2 * q], g_offset[2 * q + 1], g);
    if (!(u > 0 && u < M - 1 && v > 0 && v < M - 1)) return;
    float *gs = g_surface + q * M * M;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) gs[(u + i - 1) * M + v + j - 1] += float(g[3 * i + j]);
}

#endif   // __CUDACC__

}   // namespace b200
