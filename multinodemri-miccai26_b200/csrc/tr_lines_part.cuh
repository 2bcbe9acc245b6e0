// FFT pass kernels of tr_lines.cuh, instantiated for the lengths L with L % kLineParts == TR_LINES_PART.
#pragma once

#include <utility>

#include "tr_fft.cuh"
#include "tr_lines.cuh"

namespace tr {

constexpr int kLineParts = 8;        // translation units that share the lengths

// ------------------------------------------------------------------ radix plans
__host__ __device__ constexpr bool lp_is_radix(int r) {
    return (r >= 2 && r <= 10) || r == 12 || r == 14 || r == 15 || r == 16 || r == 18 || r == 20 || r == 21;
}
// The split into two radices with the smallest larger one (larger first: more loads in flight per
// thread), else into three (125, 175, 243, 245, 250).
__host__ __device__ constexpr int lp_radix(int L, int s) {
    int best = 0;
    for (int r = 21; r >= 2; --r)
        if (L % r == 0 && lp_is_radix(r) && lp_is_radix(L / r) && r >= L / r) best = r;
    if (best) return s == 0 ? best : (s == 1 ? L / best : 0);
    int b0 = 0, b1 = 0;
    for (int r = 21; r >= 2; --r)
        for (int q = r; q >= 2; --q)
            if (L % (r * q) == 0 && lp_is_radix(r) && lp_is_radix(q) && lp_is_radix(L / (r * q)) && q >= L / (r * q)) {
                b0 = r;
                b1 = q;
            }
    if (!b0) return 0;
    return s == 0 ? b0 : (s == 1 ? b1 : (s == 2 ? L / (b0 * b1) : 0));
}
__host__ __device__ constexpr int lp_stages(int L) {
    int s = 0;
    while (lp_radix(L, s)) ++s;
    return s;
}
// Oversampled lengths ceil(1.25 n) are never 1 mod 5.
__host__ __device__ constexpr bool lp_supported(int L) {
    if (L < kMinLineLen || L > kMaxLineLen || L % 5 == 1) return false;
    int n = L;
    for (int r : {2, 3, 5, 7})
        while (n % r == 0) n /= r;
    return n == 1 && lp_radix(L, 0) != 0;
}
// Threads, whole warps: one butterfly each per pass, at most 416 (two butterflies at 250 = 10 x 5 x 5;
// 384 threads take three: forward x pass 239 against 197 us at 84 x 117 x 200, 15 columns).
__host__ __device__ constexpr int lp_threads(int L) {
    int most = 0;
    for (int s = 0; s < lp_stages(L); ++s) most = most > L / lp_radix(L, s) ? most : L / lp_radix(L, s);
    const int nt = most * kLineW;
    return nt <= 416 ? (nt + 31) / 32 * 32 : 416;
}
// CTAs per SM the register budget is set for: about 64 registers a thread.
__host__ __device__ constexpr int lp_min_ctas(int L) { return 1024 / lp_threads(L) > 0 ? 1024 / lp_threads(L) : 1; }
// The x passes keep a column's map in registers as well.
__host__ __device__ constexpr int lp_x_min_ctas(int L) { return 768 / lp_threads(L) > 0 ? 768 / lp_threads(L) : 1; }
__host__ __device__ constexpr int lp_smem(int L) { return L * kLineW * 8 + L * 8; }

// Butterflies per thread of pass s.
__host__ __device__ constexpr int lp_iters(int L, int s) {
    return (L / lp_radix(L, s) + lp_threads(L) / kLineW - 1) / (lp_threads(L) / kLineW);
}
// A thread's inputs of the first pass: element j + r NB of its column, from load(m, index).
template <int L>
using LpFirst = float2[lp_iters(L, 0)][lp_radix(L, 0)];
template <int L, class Load>
__device__ __forceinline__ void lp_load(LpFirst<L>& v, const Load& load) {
    constexpr int R = lp_radix(L, 0), NB = L / R, JS = lp_threads(L) / kLineW;
#pragma unroll
    for (int it = 0; it < lp_iters(L, 0); ++it) {
        const int j = threadIdx.x / kLineW + it * JS;
#pragma unroll
        for (int r = 0; r < R; ++r) v[it][r] = j < NB ? load(j + r * NB, it * R + r) : make_float2(0.f, 0.f);
    }
}

// One Stockham pass on the [L][16] tile `buf` (in place: the results of a pass are stored after every
// input was read).  The first pass takes its inputs from v, the last hands its outputs to
// store(k, v, index); kSyncLast: store() writes into buf.
template <int L, bool INV, int s, int Ns, bool kSyncLast, class Store>
__device__ __forceinline__ void lp_pass(float2 (&v)[lp_iters(L, s)][lp_radix(L, s)], float2* buf, const float2* tw,
                                        const Store& store) {
    constexpr int R = lp_radix(L, s), NB = L / R, JS = lp_threads(L) / kLineW, IT = lp_iters(L, s);
    constexpr int STEP = L / (Ns * R);
    constexpr bool last = s == lp_stages(L) - 1;
    const int w = threadIdx.x & (kLineW - 1), j0 = threadIdx.x / kLineW;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = j0 + it * JS;
        if (j < NB) {
            if constexpr (s > 0) {
                const int k = Ns == 1 ? 0 : j % Ns;
#pragma unroll
                for (int r = 0; r < R; ++r) v[it][r] = buf[(j + r * NB) * kLineW + w];
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    float2 t = tw[k * r * STEP];
                    if (INV) t.y = -t.y;
                    v[it][r] = cmul_p(v[it][r], t);
                }
            }
            Dft<R>::run(v[it], INV);
        }
    }
    if constexpr (s > 0 && (!last || kSyncLast)) __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = j0 + it * JS;
        if (j < NB) {
            const int k = Ns == 1 ? 0 : j % Ns, d0 = (j / Ns) * Ns * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if constexpr (last) store(d0 + r * Ns, v[it][r], it * R + r);
                else buf[(d0 + r * Ns) * kLineW + w] = v[it][r];
            }
        }
    }
    if constexpr (!last) {
        __syncthreads();
        float2 next[lp_iters(L, s + 1)][lp_radix(L, s + 1)];
        lp_pass<L, INV, s + 1, Ns * R, kSyncLast>(next, buf, tw, store);
    }
}

// Place of element m of a centred, padded line among the n rows kept: (m + h) mod L - pad; outside
// [0, n) for the padding.
template <int L>
struct LineRow {
    int d, wrap;                             // h - pad; elements from wrap = L - h on lie L lower
    __device__ __forceinline__ LineRow(int h, int pad) : d(h - pad), wrap(L - h) {}
    __device__ __forceinline__ int operator()(int m) const { return m + d - (m >= wrap ? L : 0); }
};

// ------------------------------------------------------------------ line pass
// Loads are predicated, never branched around, so that a thread's loads are all in flight together.
template <int L, bool INV>
__global__ void __launch_bounds__(lp_threads(L), lp_min_ctas(L)) k_lp_line(LineArgs a) {
    extern __shared__ float2 sm[];
    float2* tw = sm + L * kLineW;
    const int64_t q0 = (int64_t)blockIdx.x * kLineW, outer = blockIdx.y;
    if (lines_unoccupied(a, q0, kLineW)) {
        if (a.skip_zero) lines_write_zeros(a, q0, kLineW, outer);
        return;
    }
    for (int i = threadIdx.x; i < L; i += lp_threads(L)) tw[i] = a.tw[i];
    const int64_t q = q0 + (threadIdx.x & (kLineW - 1));
    const bool on = q < a.inner;
    const float2* in = a.in + outer * a.Lin * a.inner + q;
    float2* out = a.out + outer * a.Lout * a.inner + q;
    // lines of unoccupied and occupied columns in one CTA: the former's tiles hold no values (compiled only
    // where it can happen: the check cost the z passes of other lengths 2 %)
    const bool empty = lp_mixed_columns(L) && on && a.colmask && a.mcol % kLineW && lines_unoccupied(a, q, 1);
    const int lin = on && !empty ? a.Lin : 0, lout = on ? a.Lout : 0;
    const LineRow<L> from(a.h, a.p_in), to(a.h, a.p_out);
    LpFirst<L> v;
    lp_load<L>(v, [&](int m, int) -> float2 {
        const int i = from(m);
        return (unsigned)i < (unsigned)lin ? in[i * a.inner] : make_float2(0.f, 0.f);
    });
    lp_pass<L, INV, 0, 1, false>(v, sm, tw, [&](int k, float2 r, int) {
        const int o = to(k);
        if ((unsigned)o < (unsigned)lout) out[o * a.inner] = r;
    });
}

// ------------------------------------------------------------------ x passes
// A CTA takes 16 (row, coil) columns and walks over the images, so that a column's scaled coil map
// stays in registers: the forward pass multiplies a thread's first inputs with it, the adjoint pass its
// last outputs.  Without maps (one image, one column per row) the apodisation takes its place.
// Reading the maps for every column of every image instead (as one flat list of columns, sums by
// shuffles), the two passes took 204 and 239 us at 56 x 134 x 60 (60 columns), now 180 and 218 us, and
// 86 and 142 us at 100 x 56 x 72 (48 columns), now 80 and 113 us.  Bound by instruction issue and the
// latency of the two barriers an image takes; tiles of 8 columns gave 3 % at 200 points with 12 coils
// and lost 40 % with 5 coils.
//
// Forward: 16 consecutive (row, coil) pairs, any coil count fills the tile.  The image rows they share
// come through shared memory, the next image's while this one's is transformed.
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_x_min_ctas(L)) k_lp_fwd_x(FwdXArgs a) {
    extern __shared__ float2 sm[];
    constexpr int NT = lp_threads(L);
    float2* tw = sm + L * kLineW;
    const int pitch = lp_row_pitch(a.X), nrows = lp_rows_per_cta(a.C);
    float2* rowbuf = tw + L;                              // [2 (one image: 1)][nrows][pitch]
    for (int i = threadIdx.x; i < L; i += NT) tw[i] = a.tw[i];
    const int64_t rows = (int64_t)a.Z * a.Y, q0 = (int64_t)blockIdx.x * kLineW, r0 = q0 / a.C;
    const int64_t q = q0 + (threadIdx.x & (kLineW - 1));
    const bool on = q < rows * a.C;
    const int64_t row = on ? q / a.C : r0;
    const int c = on ? (int)(q - row * a.C) : 0;
    const LineRow<L> from(a.h, a.pad);
    auto fetch = [&](int e) {
        const float2* src = a.img + (int64_t)e * a.img_stride + r0 * a.X;
        float2* dst = rowbuf + (e & 1) * nrows * pitch;
        const int n = (int)min((int64_t)nrows, rows - r0) * a.X;
        for (int i = threadIdx.x; i < n; i += NT) {
            const int r = i / a.X;
            cp_async8(dst + r * pitch + (i - r * a.X), src + i, 8);
        }
    };
    fetch(0);
    LpFirst<L> map;
    {
        const int z = (int)(row / a.Y), y = (int)(row - (int64_t)z * a.Y);
        const float sc = a.apz[z] * a.apy[y] * a.scale;
        const float2* mp = a.maps ? a.maps + row * a.X * a.C + c : nullptr;
        lp_load<L>(map, [&](int m, int) -> float2 {
            const int x = from(m);
            const bool in = (unsigned)x < (unsigned)a.X;
            if (mp) return in ? mp[x * a.C] : make_float2(0.f, 0.f);
            return make_float2(in ? sc * a.apx[x] : 0.f, 0.f);
        });
    }
    const float2* mine = rowbuf + (int)(row - r0) * pitch;
    float2* out = a.out + row * a.OSX * a.ncol + c;
    for (int e = 0; e < a.n_img; ++e) {
        cp_async_wait_all();
        __syncthreads();                                  // image e's rows are there; the tile is free
        if (e + 1 < a.n_img) fetch(e + 1);
        const float2* u = mine + (e & 1) * nrows * pitch;
        LpFirst<L> v;
        lp_load<L>(v, [&](int m, int i) -> float2 {
            const int x = from(m);
            return (unsigned)x < (unsigned)a.X ? cmul(u[x], map[i / lp_radix(L, 0)][i % lp_radix(L, 0)])
                                               : make_float2(0.f, 0.f);
        });
        lp_pass<L, false, 0, 1, false>(v, sm, tw, [&](int k, float2 r, int) {
            int g = k + a.h;
            if (g >= L) g -= L;
            if (on) out[g * a.ncol + e * a.C] = r;
        });
    }
}

// Forward, several images of one coil at long lengths: 16 consecutive (row, image) columns, so that a row's images are
// stored beside one another, each column's image row in shared memory.  (The kernel above stores 8 bytes a row apart, and
// its two buffers of 16 rows leave two CTAs a multiprocessor; one coil, 6 images: 64 x 192 x 192 217 us, 105 now,
// 32 x 256 x 256 199 us, 112 now.)
constexpr int kLongLen = 240;
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_x_min_ctas(L)) k_lp_fwd_x_images(FwdXArgs a) {
    extern __shared__ float2 sm[];
    constexpr int NT = lp_threads(L);
    float2* tw = sm + L * kLineW;
    float2* rowbuf = tw + L;                              // [16][pitch]
    const int pitch = lp_row_pitch(a.X);
    for (int i = threadIdx.x; i < L; i += NT) tw[i] = a.tw[i];
    const int64_t q0 = (int64_t)blockIdx.x * kLineW, total = (int64_t)a.Z * a.Y * a.n_img;
    for (int r = threadIdx.x >> 5; r < kLineW; r += NT / 32) {
        if (q0 + r >= total) break;
        const int64_t row = (q0 + r) / a.n_img;
        const float2* src = a.img + (q0 + r - row * a.n_img) * a.img_stride + row * a.X;
        for (int x = threadIdx.x & 31; x < a.X; x += 32) cp_async8(rowbuf + r * pitch + x, src + x, 8);
    }
    const int w = threadIdx.x & (kLineW - 1);
    const bool on = q0 + w < total;
    const int64_t row = on ? (q0 + w) / a.n_img : 0;
    const int e = on ? (int)(q0 + w - row * a.n_img) : 0;
    const LineRow<L> from(a.h, a.pad);
    const float2* mp = a.maps + row * a.X;
    cp_async_wait_all();
    __syncthreads();
    const float2* u = rowbuf + w * pitch;
    LpFirst<L> v;
    lp_load<L>(v, [&](int m, int) -> float2 {
        const int x = from(m);
        return (unsigned)x < (unsigned)a.X ? cmul(u[x], mp[x]) : make_float2(0.f, 0.f);
    });
    float2* out = a.out + row * a.OSX * a.ncol + e;
    lp_pass<L, false, 0, 1, false>(v, sm, tw, [&](int k, float2 r, int) {
        int g = k + a.h;
        if (g >= L) g -= L;
        if (on) out[g * a.ncol] = r;
    });
}

// Adjoint: whole rows of at most 16 coils (several rows where they fit), or 16 coils of a row at a
// time; the products go back into the tile with 17 columns, where the threads along x sum a row's coils
// in order and write the image row (coils past the first 16 are added to it).  The next image's inputs
// are loaded during the sums.
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_x_min_ctas(L)) k_lp_adj_x(AdjXArgs a) {
    extern __shared__ float2 sm[];
    constexpr int NT = lp_threads(L), kLast = lp_stages(L) - 1, kPitch = kLineW + 1;
    constexpr int RL = lp_radix(L, kLast), IL = lp_iters(L, kLast);
    float2* tw = sm + L * kLineW;
    for (int i = threadIdx.x; i < L; i += NT) tw[i] = a.tw[i];
    const int w = threadIdx.x & (kLineW - 1);
    const int64_t rows = (int64_t)a.Z * a.Y;
    const int rpc = a.C >= kLineW ? 1 : kLineW / a.C;
    const int64_t row0 = (int64_t)blockIdx.x * rpc;
    const LineRow<L> to(a.h, a.pad);
    for (int c0 = 0; c0 < a.C; c0 += kLineW) {
        const int nc = min(kLineW, a.C - c0), rl = a.C >= kLineW ? 0 : w / a.C, c = c0 + w - rl * a.C;
        const int64_t row = row0 + rl;
        const bool on = rl < rpc && row < rows && c < a.C;
        const float2* in = a.in + (on ? row * a.OSX * a.ncol + c : 0);
        auto inputs = [&](LpFirst<L>& v, int e) {
            lp_load<L>(v, [&](int m, int) -> float2 {
                int j = m + a.h;
                if (j >= L) j -= L;
                return on ? in[j * a.ncol + e * a.C] : make_float2(0.f, 0.f);
            });
        };
        LpFirst<L> v;
        inputs(v, 0);
        float2 map[IL][RL];                               // of the last pass's outputs
        {
            // the last pass's butterflies j < L / RL hold the outputs j + r (L / RL)
            const int z = on ? (int)(row / a.Y) : 0, y = on ? (int)(row - (int64_t)z * a.Y) : 0;
            const float sc = a.apz[z] * a.apy[y] * a.scale;
            const float2* mp = a.maps ? a.maps + (on ? row * a.X * a.C + c : 0) : nullptr;
#pragma unroll
            for (int it = 0; it < IL; ++it)
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const int j = threadIdx.x / kLineW + it * (NT / kLineW), x = to(j + r * (L / RL));
                    const bool in_x = on && j < L / RL && (unsigned)x < (unsigned)a.X;
                    if (mp) map[it][r] = in_x ? mp[x * a.C] : make_float2(0.f, 0.f);
                    else map[it][r] = make_float2(in_x ? sc * a.apx[x] : 0.f, 0.f);
                }
        }
        for (int e = 0; e < a.n_img; ++e) {
            lp_pass<L, true, 0, 1, true>(v, sm, tw, [&](int k, float2 r, int i) {
                const int x = to(k);
                if ((unsigned)x < (unsigned)a.X) sm[x * kPitch + w] = cmulc(r, map[i / RL][i % RL]);
            });
            if (e + 1 < a.n_img) inputs(v, e + 1);
            __syncthreads();
            for (int i = threadIdx.x; i < rpc * a.X; i += NT) {
                const int r = rpc == 1 ? 0 : i / a.X, x = i - r * a.X;
                if (row0 + r >= rows) break;
                const float2* p = sm + x * kPitch + r * a.C;
                float2 t = p[0];
                for (int k = 1; k < nc; ++k) t = cadd(t, p[k]);
                float2* dst = a.img + (int64_t)e * a.img_stride + (row0 + r) * a.X + x;
                *dst = c0 > 0 ? cadd(*dst, t) : t;
            }
            __syncthreads();
        }
    }
}

// Adjoint of one image at long lengths, where a map held in registers spills (336 to 448 bytes a thread at 240 and
// 320): the map is read where it is used, and a CTA takes a.cta_rows rows in a.tiles tiles of 16 columns, so that
// the coils of several rows fill whole tiles; a row whose coils began in an earlier tile is added to.
// 64 x 192 x 192: 5 coils 171 -> 124 us, 6 coils 214 -> 152, 10 coils 375 -> 230; 32 x 256 x 256: 6 coils 230 -> 153,
// 10 coils 407 -> 236.  At 125 and 200 points the kernel above is a quarter faster.
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_x_min_ctas(L)) k_lp_adj_x_one(AdjXArgs a) {
    extern __shared__ float2 sm[];
    constexpr int NT = lp_threads(L), kPitch = kLineW + 1;
    float2* tw = sm + L * kLineW;
    for (int i = threadIdx.x; i < L; i += NT) tw[i] = a.tw[i];
    const int w = threadIdx.x & (kLineW - 1);
    const int64_t rows = (int64_t)a.Z * a.Y, row0 = (int64_t)blockIdx.x * a.cta_rows;
    const LineRow<L> to(a.h, a.pad);
    for (int t0 = 0; t0 < a.tiles * kLineW; t0 += kLineW) {
        const int rl = (t0 + w) / a.C, c = t0 + w - rl * a.C;
        const int64_t row = row0 + rl;
        const bool on = rl < a.cta_rows && row < rows;
        const float2* in = a.in + (on ? row * a.OSX * a.ncol + c : 0);
        LpFirst<L> v;
        lp_load<L>(v, [&](int m, int) -> float2 {
            int j = m + a.h;
            if (j >= L) j -= L;
            return on ? in[j * a.ncol] : make_float2(0.f, 0.f);
        });
        const int z = on ? (int)(row / a.Y) : 0, y = on ? (int)(row - (int64_t)z * a.Y) : 0;
        const float sc = a.apz[z] * a.apy[y] * a.scale;
        const float2* mp = a.maps ? a.maps + (on ? row * a.X * a.C + c : 0) : nullptr;
        lp_pass<L, true, 0, 1, true>(v, sm, tw, [&](int k, float2 r, int) {
            const int x = to(k);
            if ((unsigned)x >= (unsigned)a.X) return;
            const float2 m = mp ? (on ? mp[x * a.C] : make_float2(0.f, 0.f)) : make_float2(on ? sc * a.apx[x] : 0.f, 0.f);
            sm[x * kPitch + w] = cmulc(r, m);
        });
        __syncthreads();
        const int r0 = t0 / a.C, n = min(a.cta_rows, (t0 + kLineW - 1) / a.C + 1) - r0;      // rows in this tile
        for (int i = threadIdx.x; i < n * a.X; i += NT) {
            const int r = r0 + (n == 1 ? 0 : i / a.X), x = i - (r - r0) * a.X;
            if (row0 + r >= rows) break;
            const int k0 = max(r * a.C - t0, 0), k1 = min((r + 1) * a.C - t0, kLineW);
            const float2* p = sm + x * kPitch;
            float2 t = p[k0];
            for (int k = k0 + 1; k < k1; ++k) t = cadd(t, p[k]);
            float2* dst = a.img + (row0 + r) * a.X + x;
            *dst = r * a.C < t0 ? cadd(*dst, t) : t;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ table
template <int L>
LineKernels lp_entry() {
    LineKernels k;
    if constexpr (lp_supported(L)) {
        k.fwd = (const void*)k_lp_line<L, false>;
        k.inv = (const void*)k_lp_line<L, true>;
        k.fwd_x = (const void*)k_lp_fwd_x<L>;
        k.adj_x = (const void*)k_lp_adj_x<L>;
        if constexpr (L >= kLongLen) {
            k.fwd_x_images = (const void*)k_lp_fwd_x_images<L>;
            k.adj_x_one = (const void*)k_lp_adj_x_one<L>;
        }
        k.threads = lp_threads(L);
        k.smem = lp_smem(L);
    }
    return k;
}
template <int PART, int... I>
void lp_fill(LineKernels* table, std::integer_sequence<int, I...>) {
    ((table[PART + I * kLineParts] = lp_entry<PART + I * kLineParts>()), ...);
}
template <int PART>
void lp_fill_part(LineKernels* table) {
    lp_fill<PART>(table, std::make_integer_sequence<int, (kMaxLineLen - PART) / kLineParts + 1>());
}

}  // namespace tr
