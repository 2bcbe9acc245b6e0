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
__host__ __device__ constexpr int lp_smem(int L) { return L * kLineW * 8 + L * 8; }

// One Stockham pass on the [L][16] tile `buf` (in place: the results of a pass are stored after every
// input was read).  The first pass reads its inputs from load(m), the last hands its outputs to
// store(k, v); kSyncLast: store() writes into buf.
template <int L, bool INV, int s, int Ns, bool kSyncLast, class Load, class Store>
__device__ __forceinline__ void lp_pass(float2* buf, const float2* tw, Load& load, Store& store) {
    constexpr int R = lp_radix(L, s), NB = L / R, NT = lp_threads(L), JS = NT / kLineW, IT = (NB + JS - 1) / JS;
    constexpr int STEP = L / (Ns * R);
    constexpr bool last = s == lp_stages(L) - 1;
    const int w = threadIdx.x & (kLineW - 1), j0 = threadIdx.x / kLineW;
    float2 v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = j0 + it * JS;
        if (j < NB) {
            const int k = Ns == 1 ? 0 : j % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if constexpr (s == 0) load.first(j + r * NB, v[it][r]);
                else v[it][r] = buf[(j + r * NB) * kLineW + w];
            }
            if constexpr (s == 0 && Load::kTwo) {          // a second factor, four loads in flight at a time
#pragma unroll
                for (int r0 = 0; r0 < R; r0 += 4) {
                    float2 f[4];
#pragma unroll
                    for (int r = r0; r < r0 + 4 && r < R; ++r) f[r - r0] = load.second(j + r * NB);
#pragma unroll
                    for (int r = r0; r < r0 + 4 && r < R; ++r) v[it][r] = cmul(v[it][r], f[r - r0]);
                }
            }
#pragma unroll
            for (int r = 1; r < R; ++r) {
                if constexpr (s > 0) {
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
                if constexpr (last) store(d0 + r * Ns, v[it][r]);
                else buf[(d0 + r * Ns) * kLineW + w] = v[it][r];
            }
        }
    }
    if constexpr (!last) {
        __syncthreads();
        lp_pass<L, INV, s + 1, Ns * R, kSyncLast>(buf, tw, load, store);
    }
}

// Inputs of a first pass: row (m + h) mod L of the padded line, zero outside [0, n).  Loads are
// predicated, never branched around, so that a thread's loads are all in flight together.
struct LineLoad {
    static constexpr bool kTwo = false;
    const float2* in;
    int64_t stride;
    int n, d, wrap, L;                       // position m + d, less L from m = wrap on
    __device__ __forceinline__ int row(int m) const { return m + d - (m >= wrap ? L : 0); }
    __device__ __forceinline__ void first(int m, float2& v) const {
        const int i = row(m);
        v = (unsigned)i < (unsigned)n ? in[i * stride] : make_float2(0.f, 0.f);
    }
    __device__ __forceinline__ float2 second(int) const { return make_float2(1.f, 0.f); }
};

// ------------------------------------------------------------------ line pass
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
    const int lin = on ? a.Lin : 0, lout = on ? a.Lout : 0, din = a.h - a.p_in, dout = a.h - a.p_out;
    LineLoad load{in, a.inner, lin, din, L - a.h, L};
    auto store = [&](int k, float2 v) {
        int o = k + dout;
        if (k + a.h >= L) o -= L;
        if ((unsigned)o < (unsigned)lout) out[(int64_t)o * a.inner] = v;
    };
    lp_pass<L, INV, 0, 1, false>(sm, tw, load, store);
}

// u times the scaled map, or u times the apodisation where there are no maps.
struct MapLoad {
    static constexpr bool kTwo = true;
    LineLoad u;
    const float2* map;
    const float* apx;
    int C;
    float sc;
    __device__ __forceinline__ void first(int m, float2& v) const { u.first(m, v); }
    __device__ __forceinline__ float2 second(int m) const {
        const int x = u.row(m);
        const bool in = (unsigned)x < (unsigned)u.n;
        if (map) return in ? map[(int64_t)x * C] : make_float2(0.f, 0.f);
        return make_float2(in ? sc * apx[x] : 0.f, 0.f);
    }
};

// ------------------------------------------------------------------ forward x pass
// Sixteen consecutive (row, column) pairs per CTA, columns of a row first, so that any coil count and
// number of images fills the tile.
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_min_ctas(L)) k_lp_fwd_x(FwdXArgs a) {
    extern __shared__ float2 sm[];
    float2* tw = sm + L * kLineW;
    for (int i = threadIdx.x; i < L; i += lp_threads(L)) tw[i] = a.tw[i];
    const int64_t q = (int64_t)blockIdx.x * kLineW + (threadIdx.x & (kLineW - 1));
    const int64_t rows = (int64_t)a.Z * a.Y;
    const bool on = q < rows * a.ncol;
    const int64_t row = on ? q / a.ncol : 0;
    const int col = on ? (int)(q - row * a.ncol) : 0, img = col / a.C, c = col - img * a.C;
    const int z = (int)(row / a.Y), y = (int)(row - (int64_t)z * a.Y);
    const float sc = a.apz[z] * a.apy[y] * a.scale;
    const float2* src = a.img + (int64_t)img * a.img_stride + row * a.X;
    const float2* map = a.maps ? a.maps + row * a.X * a.C + c : nullptr;
    float2* out = a.out + row * a.OSX * a.ncol + col;
    const int nx = on ? a.X : 0, din = a.h - a.pad;
    MapLoad load{{src, 1, nx, din, L - a.h, L}, map, a.apx, a.C, sc};
    auto store = [&](int k, float2 v) {
        int g = k + a.h;
        if (g >= L) g -= L;
        if (on) out[(int64_t)g * a.ncol] = v;
    };
    lp_pass<L, false, 0, 1, false>(sm, tw, load, store);
}

// ------------------------------------------------------------------ adjoint x pass
// One row per CTA, its columns in chunks of 16 (several whole rows where they fit one chunk).  The
// transformed, cropped rows go back into the tile with column w of row x at w ^ (x % 16), which both
// the products with the coil maps (half-warps along the columns of an x) and the write of the
// images (warps along x) read without bank conflicts.  The columns of an image are summed by a
// segmented shuffle; an image whose coils span chunks is added up in its image row.
template <int L>
__global__ void __launch_bounds__(lp_threads(L), lp_min_ctas(L)) k_lp_adj_x(AdjXArgs a) {
    extern __shared__ float2 sm[];
    constexpr int NT = lp_threads(L);
    float2* tw = sm + L * kLineW;
    float2* smap = tw + L;                               // [X][16]: the chunk's coil maps
    for (int i = threadIdx.x; i < L; i += NT) tw[i] = a.tw[i];
    const int w = threadIdx.x & (kLineW - 1);
    const int64_t rows = (int64_t)a.Z * a.Y;
    const int rpc = a.ncol >= kLineW ? 1 : kLineW / a.ncol;                  // rows per CTA
    const int nchunk = a.ncol >= kLineW ? (a.ncol + kLineW - 1) / kLineW : 1;
    const int dout = a.h - a.pad;
    // column w of chunk ch: row, image, coil
    for (int ch = 0; ch < nchunk; ++ch) {
        auto place = [&](int slot, int64_t& row, int& col) {
            const int rl = nchunk > 1 || rpc == 1 ? 0 : slot / a.ncol;
            row = (int64_t)blockIdx.x * rpc + rl;
            col = ch * kLineW + slot - rl * a.ncol;
            return rl < rpc && row < rows && col < a.ncol;
        };
        int64_t row;
        int col;
        const bool on = place(w, row, col);
        const float2* in = a.in + (on ? row * a.OSX * a.ncol + col : 0);
        LineLoad load{in, a.ncol, on ? L : 0, a.h, L - a.h, L};
        auto store = [&](int k, float2 v) {
            int x = k + dout;
            if (k + a.h >= L) x -= L;
            if ((unsigned)x < (unsigned)a.X) sm[x * kLineW + (w ^ (x & 15))] = v;
        };
        const int img = on ? col / a.C : -1, c = on ? col - img * a.C : 0;
        const int seg = on ? (int)(row - (int64_t)blockIdx.x * rpc) * a.n_img + img : -1;
        constexpr int JS = NT / kLineW;
        if (a.maps) {                                      // the columns' maps travel during the transform
            const float2* map = a.maps + (on ? row * a.X * a.C + c : 0);
            for (int x = threadIdx.x / kLineW; x < a.X; x += JS)
                cp_async8(smap + x * kLineW + w, map + (on ? (int64_t)x * a.C : 0), on ? 8 : 0);
        }
        lp_pass<L, true, 0, 1, true>(sm, tw, load, store);
        cp_async_wait_all();
        __syncthreads();
        if (a.maps) {
            const unsigned half = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
            int same = 0;                                  // bit b: lane w + 2^b belongs to the same image
            for (int b = 0; b < 4; ++b) {
                const int other = __shfl_down_sync(half, seg, 1 << b, kLineW);
                same |= (w + (1 << b) < kLineW && other == seg) << b;
            }
            constexpr int U = 4;                           // x positions side by side per thread
            for (int x0 = threadIdx.x / kLineW; x0 < a.X; x0 += U * JS) {
                float2 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int x = x0 + u * JS;
                    v[u] = on && x < a.X ? cmulc(sm[x * kLineW + (w ^ (x & 15))], smap[x * kLineW + w])
                                         : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    if (1 << b >= a.C) break;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float tx = __shfl_down_sync(half, v[u].x, 1 << b, kLineW);
                        const float ty = __shfl_down_sync(half, v[u].y, 1 << b, kLineW);
                        if (same & (1 << b)) v[u] = make_float2(v[u].x + tx, v[u].y + ty);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int x = x0 + u * JS;
                    if (x < a.X) sm[x * kLineW + (w ^ (x & 15))] = v[u];
                }
            }
            __syncthreads();
        }
        // the first column of every image in the chunk holds its sum: write (first coils) or add
        const unsigned heads = __ballot_sync(0xffffffffu, on && (c == 0 || w == 0)) & 0xffffu;
        const int nx = (a.X + 31) / 32, tasks = __popc(heads) * nx;
        for (int t = threadIdx.x >> 5; t < tasks; t += NT / 32) {
            const int hn = t / nx, x = (t - hn * nx) * 32 + (threadIdx.x & 31), slot = __fns(heads, 0, hn + 1);
            int64_t r;
            int cl;
            place(slot, r, cl);
            if (x >= a.X) continue;
            const int im = cl / a.C;
            float2 v = sm[x * kLineW + (slot ^ (x & 15))];
            if (!a.maps) {
                const int z = (int)(r / a.Y), y = (int)(r - (int64_t)z * a.Y);
                v = cscale(v, a.apz[z] * a.apy[y] * a.apx[x] * a.scale);
            }
            float2* dst = a.img + (int64_t)im * a.img_stride + r * a.X + x;
            if (cl - im * a.C > 0) v = cadd(*dst, v);
            *dst = v;
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
        k.threads = lp_threads(L);
        k.smem = lp_smem(L);
        k.smem_adj_x = lp_smem(L) + L * kLineW * 8;
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
