// TVMW spatial wavelet W2 on sm_100a: db6, PyWavelets "zero" mode, level =
// PyWavelets' maximum, over (Z, Y, X) of every (bin, echo) image.
//
// Reference: src/toporecon/algorithms/tvmw.py:196-206 (ptwt wavedec3 /
// waverec3, axes (-3, -2, -1)), the dual step at :447-452 (p += sigma W2 u,
// then _tree_project_linf_complex2ch_ at :162-193 on every sub-band), and the
// primal use of waverec3 as the adjoint substitute at :647-649.
//
// Analysis along one axis:   c[o] = sum_j f[j] x[2o + 1 - j], x = 0 outside,
//                            output length (n + F - 1) / 2.
// Synthesis along one axis:  y[o] = sum_j g_lo[2j + o%2] a[i - j] + g_hi[2j + o%2] d[i - j],
//                            i = o/2 + F/2 - 1, computed only for the lengths
//                            the next finer level needs (PyWavelets' crop).
// Coefficients of one image: [cA_L | 7 detail bands of level L | ... | level 1],
// detail bands ordered aad, ada, add, daa, dad, dda, ddd (z, y, x letters).

#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <vector>

#include "tr_internal.cuh"

namespace tr {

constexpr int kF = 12;          // db6 filter length
constexpr int kMaxLevels = 8;

// Daubechies extremal-phase db6 scaling (reconstruction low-pass) filter,
// obtained by spectral factorisation of P(y) = sum_k C(5 + k, k) y^k
// (Daubechies 1988); sum = sqrt(2), unit norm.
static const double kDb6RecLo[kF] = {
    0.11154074335010940,  0.49462389039845290,  0.75113390802109490,  0.31525035170919800,
    -0.22626469396543930, -0.12976686756726188, 0.09750160558732306,  0.02752286553030561,
    -0.03158203931748598, 0.00055384220116150,  0.00477725751094551,  -0.00107730108530848};

struct Filters {
    float dec_lo[kF], dec_hi[kF], rec_lo[kF], rec_hi[kF];
};

struct WaveletPlan {
    int levels = 0;
    int in_shape[kMaxLevels][3];
    int out_shape[kMaxLevels][3];
    int64_t det_off[kMaxLevels];   // offset of level l's 7 detail bands (l = 0 finest)
    int64_t ncoef = 0;
    Filters f;
    float2* T1 = nullptr;          // z-transformed halves: (nimg, 2, Zo, Yi, Xi)
    float2* A[2] = {nullptr, nullptr};
    int64_t t1_elems = 0, a_elems = 0;
    int nimg = 0;
};

static int dwt_len(int n) { return (n + kF - 1) / 2; }

static int max_level(const int* shape) {
    int lv = 1 << 30;
    for (int i = 0; i < 3; ++i) {
        int l = shape[i] < kF - 1 ? 0 : (int)std::floor(std::log2((double)shape[i] / (kF - 1)));
        lv = std::min(lv, l);
    }
    return std::max(lv, 0);
}

tr_status wavelet_prepare(tr_plan* p) {
    WaveletPlan* w = new WaveletPlan();
    p->wav = w;
    w->levels = std::min(max_level(p->n), kMaxLevels);
    int cur[3] = {p->n[0], p->n[1], p->n[2]};
    for (int l = 0; l < w->levels; ++l) {
        for (int i = 0; i < 3; ++i) {
            w->in_shape[l][i] = cur[i];
            w->out_shape[l][i] = dwt_len(cur[i]);
            cur[i] = w->out_shape[l][i];
        }
    }
    // layout: cA_L, det_L, ..., det_1
    int64_t off = 0;
    if (w->levels > 0) {
        const int* s = w->out_shape[w->levels - 1];
        off = (int64_t)s[0] * s[1] * s[2];
    }
    for (int l = w->levels - 1; l >= 0; --l) {
        const int* s = w->out_shape[l];
        w->det_off[l] = off;
        off += 7LL * s[0] * s[1] * s[2];
    }
    w->ncoef = off;
    for (int j = 0; j < kF; ++j) {
        const double lo = kDb6RecLo[kF - 1 - j];                      // dec_lo = reversed rec_lo
        const double hi = ((j + 1) % 2 ? -1.0 : 1.0) * kDb6RecLo[j];  // dec_hi[j] = (-1)^(j+1) dec_lo[F-1-j]
        w->f.dec_lo[j] = (float)lo;
        w->f.dec_hi[j] = (float)hi;
    }
    for (int j = 0; j < kF; ++j) {
        w->f.rec_lo[j] = w->f.dec_lo[kF - 1 - j];
        w->f.rec_hi[j] = w->f.dec_hi[kF - 1 - j];
    }
    return TR_OK;
}

void wavelet_info(const tr_plan* p, int32_t* levels, int64_t* coeffs) {
    if (levels) *levels = p->wav ? p->wav->levels : 0;
    if (coeffs) *coeffs = p->wav ? p->wav->ncoef : 0;
}

void wavelet_destroy(tr_plan* p) {
    if (!p->wav) return;
    cudaFree(p->wav->T1);
    cudaFree(p->wav->A[0]);
    cudaFree(p->wav->A[1]);
    delete p->wav;
    p->wav = nullptr;
}

static tr_status ensure_wavelet_buffers(tr_plan* p, int nimg) {
    WaveletPlan* w = p->wav;
    if (w->nimg >= nimg && w->T1) return TR_OK;
    cudaFree(w->T1);
    cudaFree(w->A[0]);
    cudaFree(w->A[1]);
    w->T1 = w->A[0] = w->A[1] = nullptr;
    int64_t t1 = 0, a = 0;
    for (int l = 0; l < w->levels; ++l) {
        const int* si = w->in_shape[l];
        const int* so = w->out_shape[l];
        t1 = std::max<int64_t>(t1, 2LL * so[0] * si[1] * si[2]);
        a = std::max<int64_t>(a, (int64_t)so[0] * so[1] * so[2]);       // the approximations between levels
    }
    w->t1_elems = t1 * nimg;
    w->a_elems = a * nimg;
    TR_CUDA(cudaMalloc(&w->T1, w->t1_elems * sizeof(float2)));
    TR_CUDA(cudaMalloc(&w->A[0], w->a_elems * sizeof(float2)));
    TR_CUDA(cudaMalloc(&w->A[1], w->a_elems * sizeof(float2)));
    p->workspace_bytes += (w->t1_elems + 2 * w->a_elems) * (int64_t)sizeof(float2);
    w->nimg = nimg;
    return TR_OK;
}

// Each level is two kernels in either direction, both bound by the memory they must move: a pass along
// z, in which a thread slides a register window over a run of outputs, and a kernel for the other two
// axes of a slice, which hands its first axis's results to the second in shared memory.  One output
// per thread and axis (12 loads per output, 64-bit divisions, every axis through global memory, the
// copy of cA and a memset) took 6.75 ms for the pair on 36 images of 112 x 160 x 160 (3 levels);
// these kernels take 2.1 ms.

// V consecutive complex values (16-byte access for two).
template <int V>
struct CVec {
    float2 v[V];
};
template <int V>
__device__ __forceinline__ CVec<V> cv_load(const float2* p) {
    CVec<V> r;
    if constexpr (V == 2) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        r.v[0] = make_float2(t.x, t.y);
        r.v[1] = make_float2(t.z, t.w);
    } else {
        r.v[0] = *p;
    }
    return r;
}
template <int V>
__device__ __forceinline__ void cv_store(float2* p, const CVec<V>& r) {
    if constexpr (V == 2) *reinterpret_cast<float4*>(p) = make_float4(r.v[0].x, r.v[0].y, r.v[1].x, r.v[1].y);
    else *p = r.v[0];
}
template <int V>
__device__ __forceinline__ CVec<V> cv_zero() {
    CVec<V> r;
#pragma unroll
    for (int k = 0; k < V; ++k) r.v[k] = make_float2(0.f, 0.f);
    return r;
}
template <int V>
__device__ __forceinline__ void cv_fma(CVec<V>& acc, float f, const CVec<V>& x) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
        acc.v[k].x = fmaf(f, x.v[k].x, acc.v[k].x);
        acc.v[k].y = fmaf(f, x.v[k].y, acc.v[k].y);
    }
}

// ------------------------------------------------------------------ analysis
// Outputs per thread along z: 34 loads for 12 instead of the 24 of a whole line; 4 (18 loads) while runs of 12
// are fewer than two blocks a multiprocessor.  One image of 48 x 64 x 64, analysis of two levels: 43 us with
// runs of 12, 36 with 4 (37 with one output a thread before).
constexpr int kDwtRun = 12, kDwtRunShort = 4;
constexpr int kDwtRows = 16;     // output rows (of each half) per CTA of the y + x kernel

// Along z: in (P, n, Q) -> out (P, 2, no, Q) (band 0 = low, 1 = high).
template <int V, int RUN>
__global__ void __launch_bounds__(256) k_dwt_z(const float2* __restrict__ in, float2* __restrict__ out, int64_t P, int n,
                                               int64_t Q, int no, Filters f) {
    const int64_t q = ((int64_t)blockIdx.x * 256 + threadIdx.x) * V;
    if (q >= Q) return;
    const int runs = (no + RUN - 1) / RUN;
    for (int64_t pr = blockIdx.y; pr < P * runs; pr += gridDim.y) {
        const int64_t pp = pr / runs;
        const int o0 = (int)(pr - pp * runs) * RUN;
        const float2* src = in + pp * n * Q + q;
        float2* lo = out + (pp * 2 * no + o0) * Q + q;
        float2* hi = lo + (int64_t)no * Q;
        auto get = [&](int i) { return (unsigned)i < (unsigned)n ? cv_load<V>(src + (int64_t)i * Q) : cv_zero<V>(); };
        CVec<V> w[kF];                               // input i at i mod 12
#pragma unroll
        for (int t = 0; t < kF - 2; ++t) w[(t + 2) % kF] = get(2 * o0 - (kF - 2) + t);
#pragma unroll
        for (int r = 0; r < RUN; ++r) {
            w[(2 * r) % kF] = get(2 * (o0 + r));
            w[(2 * r + 1) % kF] = get(2 * (o0 + r) + 1);
            CVec<V> a = cv_zero<V>(), b = cv_zero<V>();
#pragma unroll
            for (int j = 0; j < kF; ++j) {
                cv_fma<V>(a, f.dec_lo[j], w[(2 * r + 1 - j + 2 * kF) % kF]);
                cv_fma<V>(b, f.dec_hi[j], w[(2 * r + 1 - j + 2 * kF) % kF]);
            }
            if (o0 + r < no) {
                cv_store<V>(lo + (int64_t)r * Q, a);
                cv_store<V>(hi + (int64_t)r * Q, b);
            }
        }
    }
}

// Along y, then x, of one z-transformed slice: T1 (img, bz, Zo, Yi, Xi) -> 8 bands.
// Detail bands (and cA at the coarsest level) update the dual:
//   p <- p + sigma c,  p <- p * min(1, lam / sqrt(|p|^2 + 1e-12))   (lam <= 0: p <- 0)
// with p read from pw2, or zero (fresh).  Band aaa of a non-coarsest level goes to the next level's input.
struct DwtYxArgs {
    const float2* in;
    int nimg, Zo, Yi, Yo, Xi, Xo;
    float2* next;      // (nimg, Zo, Yo, Xo) or null at the coarsest level
    float2* pw2;       // (nimg, ncoef)
    int64_t ncoef, det_off;
    int coarsest, fresh;
    float sigma, lam;
    Filters f;
};

// Shared memory: the y-transformed rows, even x and odd x apart, so that the 12 taps of neighbouring
// outputs are neighbouring values.
__host__ __device__ constexpr int dwt_half(int Xi) { return 6 + (Xi + kF - 1) / 2; }     // zeros past both ends
static size_t dwt_yx_smem(int Xi) { return (size_t)2 * kDwtRows * 2 * dwt_half(Xi) * sizeof(float2); }

__global__ void __launch_bounds__(256) k_dwt_yx(DwtYxArgs a) {
    extern __shared__ float2 rows[];                  // [2 halves][kDwtRows][even | odd]
    const int half = dwt_half(a.Xi);
    const int o0 = blockIdx.x * kDwtRows;
    const int64_t slice = (int64_t)blockIdx.z * gridDim.y + blockIdx.y;      // (img, bz, z)
    if (slice >= (int64_t)a.nimg * 2 * a.Zo) return;
    const float2* src = a.in + slice * a.Yi * a.Xi;
    // zeros past both row ends (odd x: (Xi - 1) / 2 + 1 values, even x: Xi / 2 + ... values)
    for (int i = threadIdx.x; i < 4 * kDwtRows * 6; i += blockDim.x) rows[(i / 6) * half + i % 6] = make_float2(0.f, 0.f);
    for (int i = threadIdx.x; i < 4 * kDwtRows; i += blockDim.x)
        for (int k = 6 + (a.Xi + ((i & 1) ? 0 : 1)) / 2; k < half; ++k) rows[i * half + k] = make_float2(0.f, 0.f);
    for (int x = threadIdx.x; x < a.Xi; x += blockDim.x) {
        float2* dst = rows + (x & 1) * half + 6 + (x >> 1);
        auto get = [&](int i) {
            return (unsigned)i < (unsigned)a.Yi ? src[(int64_t)i * a.Xi + x] : make_float2(0.f, 0.f);
        };
        CVec<1> w[kF];
#pragma unroll
        for (int t = 0; t < kF - 2; ++t) w[(t + 2) % kF].v[0] = get(2 * o0 - (kF - 2) + t);
#pragma unroll
        for (int r = 0; r < kDwtRows; ++r) {          // rows past Yo are computed and not read
            w[(2 * r) % kF].v[0] = get(2 * (o0 + r));
            w[(2 * r + 1) % kF].v[0] = get(2 * (o0 + r) + 1);
            CVec<1> lo = cv_zero<1>(), hi = cv_zero<1>();
#pragma unroll
            for (int j = 0; j < kF; ++j) {
                cv_fma<1>(lo, a.f.dec_lo[j], w[(2 * r + 1 - j + 2 * kF) % kF]);
                cv_fma<1>(hi, a.f.dec_hi[j], w[(2 * r + 1 - j + 2 * kF) % kF]);
            }
            dst[r * 2 * half] = lo.v[0];
            dst[(kDwtRows + r) * 2 * half] = hi.v[0];
        }
    }
    __syncthreads();
    const int64_t zi = slice % a.Zo, ib = slice / a.Zo;
    const int64_t img = ib >> 1;
    const int bz = (int)(ib & 1);
    const int64_t sub = (int64_t)a.Zo * a.Yo * a.Xo;
    const int nrow = min(kDwtRows, a.Yo - o0);
    const float inside = a.lam * a.lam * 0.999999f;   // |p|^2 below this: |p| < lam whatever the rounding
    for (int r = threadIdx.x >> 5; r < 2 * nrow; r += blockDim.x >> 5) {
        const int by = r >= nrow, y = r - by * nrow;
        const float2* even = rows + (by * kDwtRows + y) * 2 * half + 6;
        const float2* odd = even + half;
        const int64_t at = (zi * a.Yo + o0 + y) * a.Xo;
        const int band = bz * 4 + by * 2;
        float2* d1 = a.pw2 + img * a.ncoef + a.det_off + (int64_t)band * sub + at;            // band + 1
        float2* d0 = band ? d1 - sub : (a.coarsest ? a.pw2 + img * a.ncoef + at : a.next + img * sub + at);
        const bool dual0 = band || a.coarsest;
        for (int x = threadIdx.x & 31; x < a.Xo; x += 32) {
            CVec<1> lo = cv_zero<1>(), hi = cv_zero<1>();
#pragma unroll
            for (int j = 0; j < kF; ++j) {            // input 2 x + 1 - j
                CVec<1> v;
                v.v[0] = (j & 1) ? even[x - (j >> 1)] : odd[x - (j >> 1)];
                cv_fma<1>(lo, a.f.dec_lo[j], v);
                cv_fma<1>(hi, a.f.dec_hi[j], v);
            }
            auto put = [&](float2* slot, float2 c) {
                if (a.lam <= 0.f) {
                    *slot = make_float2(0.f, 0.f);
                    return;
                }
                float2 pv = a.fresh ? make_float2(0.f, 0.f) : *slot;
                pv.x += a.sigma * c.x;
                pv.y += a.sigma * c.y;
                const float m2 = pv.x * pv.x + pv.y * pv.y + 1e-12f;
                if (!(m2 < inside)) {                 // else the scale is one
                    const float s = fminf(a.lam / sqrtf(m2), 1.0f);
                    pv = make_float2(pv.x * s, pv.y * s);
                }
                *slot = pv;
            };
            if (dual0) put(d0 + x, lo.v[0]);
            else d0[x] = lo.v[0];
            put(d1 + x, hi.v[0]);
        }
    }
}

// ------------------------------------------------------------------ synthesis
// The low filter's large taps come first, the high filter's last: the low products are added from the last
// tap on, the high ones from the first, so that the large products meet the sum at the end and it rounds
// less.  Relative error of three levels and time of 36 images of 112 x 160 x 160: 0.97e-7, 978 us; both from
// the first tap on: 1.29e-7, 950 us; six pairs, half as many operations again: 1.18e-7, 1040 us.
//
// Along y, then x, of one slice: 8 bands -> T1 (img, bz, Zo, Yi, Xi).
struct IdwtYxArgs {
    const float2* approx;     // band aaa: image i at approx + i * approx_stride
    int64_t approx_stride;
    const float2* pw2;        // (nimg, ncoef)
    int64_t ncoef, det_off;
    int nimg, Zo, Yo, Xo, Yi, Xi;
    int vec;                  // rows of T1 are 16-byte aligned
    float2* out;
    Filters f;
};

// Shared memory: the y-synthesised rows of the low and high x halves, five zeros behind each row.
__host__ __device__ constexpr int idwt_pitch(int Xo) { return Xo + kF / 2 - 1; }
static size_t idwt_yx_smem(int T, int Xo) { return (size_t)2 * T * idwt_pitch(Xo) * sizeof(float2); }

template <int T>
__global__ void __launch_bounds__(256) k_idwt_yx(IdwtYxArgs a) {
    extern __shared__ __align__(16) float2 rows[];            // [bx][T output rows][coarse x]
    const int pitch = idwt_pitch(a.Xo);
    const int o0 = blockIdx.x * T;
    const int64_t slice = (int64_t)blockIdx.z * gridDim.y + blockIdx.y;      // (img, bz, z)
    if (slice >= (int64_t)a.nimg * 2 * a.Zo) return;
    const int64_t zi = slice % a.Zo, ib = slice / a.Zo, img = ib >> 1;
    const int bz = (int)(ib & 1);
    const int64_t sub = (int64_t)a.Zo * a.Yo * a.Xo, at = (zi * a.Yo + o0 / 2) * a.Xo;
    const float2* det = a.pw2 + img * a.ncoef + a.det_off + at;
    for (int i = threadIdx.x; i < 2 * T * (kF / 2 - 1); i += blockDim.x)
        rows[(i / (kF / 2 - 1)) * pitch + a.Xo + i % (kF / 2 - 1)] = make_float2(0.f, 0.f);
    for (int c = threadIdx.x; c < 2 * a.Xo; c += blockDim.x) {
        const int bx = c >= a.Xo, x = c - bx * a.Xo, band = bz * 4 + bx;     // by = 0; by = 1: band + 2
        const float2* lo = (band ? det + (int64_t)(band - 1) * sub : a.approx + img * a.approx_stride + at) + x;
        const float2* hi = det + (int64_t)(band + 1) * sub + x;
        float2* dst = rows + bx * T * pitch + x;
        CVec<1> u[kF / 2], v[kF / 2];                         // coarse row i at i mod 6
        auto get = [&](int t) {
            const bool in = o0 / 2 + t < a.Yo;
            u[t % 6].v[0] = in ? lo[(int64_t)t * a.Xo] : make_float2(0.f, 0.f);
            v[t % 6].v[0] = in ? hi[(int64_t)t * a.Xo] : make_float2(0.f, 0.f);
        };
#pragma unroll
        for (int t = 0; t < kF / 2 - 1; ++t) get(t);
#pragma unroll
        for (int h = 0; h < T / 2; ++h) {                     // outputs 2 h, 2 h + 1: coarse rows h .. h + 5
            get(h + 5);
            CVec<1> e = cv_zero<1>(), o = cv_zero<1>();
#pragma unroll
            for (int j = 0; j < kF / 2; ++j) {
                cv_fma<1>(e, a.f.rec_lo[10 - 2 * j], u[(h + j) % 6]);
                cv_fma<1>(e, a.f.rec_hi[2 * j], v[(h + 5 - j) % 6]);
                cv_fma<1>(o, a.f.rec_lo[11 - 2 * j], u[(h + j) % 6]);
                cv_fma<1>(o, a.f.rec_hi[2 * j + 1], v[(h + 5 - j) % 6]);
            }
            dst[(2 * h) * pitch] = e.v[0];
            dst[(2 * h + 1) * pitch] = o.v[0];
        }
    }
    __syncthreads();
    float2* out = a.out + (slice * a.Yi + o0) * a.Xi;
    for (int r = threadIdx.x >> 5; r < min(T, a.Yi - o0); r += blockDim.x >> 5) {
        const float2* lo = rows + r * pitch;
        const float2* hi = lo + T * pitch;
        float2* row = out + (int64_t)r * a.Xi;
        for (int xp = threadIdx.x & 31; 2 * xp < a.Xi; xp += 32) {           // outputs 2 xp, 2 xp + 1
            CVec<1> e = cv_zero<1>(), o = cv_zero<1>();
#pragma unroll
            for (int j = 0; j < kF / 2; ++j) {
                CVec<1> u, v;
                u.v[0] = lo[xp + j];
                v.v[0] = hi[xp + 5 - j];
                cv_fma<1>(e, a.f.rec_lo[10 - 2 * j], u);
                cv_fma<1>(e, a.f.rec_hi[2 * j], v);
                cv_fma<1>(o, a.f.rec_lo[11 - 2 * j], u);
                cv_fma<1>(o, a.f.rec_hi[2 * j + 1], v);
            }
            if (a.vec) {
                *reinterpret_cast<float4*>(row + 2 * xp) = make_float4(e.v[0].x, e.v[0].y, o.v[0].x, o.v[0].y);
            } else {
                row[2 * xp] = e.v[0];
                if (2 * xp + 1 < a.Xi) row[2 * xp + 1] = o.v[0];
            }
        }
    }
}

constexpr int kIdwtRun = 12;     // output pairs per thread along z

// Along z: in (P, 2, no, Q) -> out (P, ni, Q).
template <int V>
__global__ void __launch_bounds__(256) k_idwt_z(const float2* __restrict__ in, float2* __restrict__ out, int64_t P, int no,
                                                int64_t Q, int ni, Filters f) {
    const int64_t q = ((int64_t)blockIdx.x * 256 + threadIdx.x) * V;
    if (q >= Q) return;
    const int runs = ((ni + 1) / 2 + kIdwtRun - 1) / kIdwtRun;
    for (int64_t pr = blockIdx.y; pr < P * runs; pr += gridDim.y) {
        const int64_t pp = pr / runs;
        const int h0 = (int)(pr - pp * runs) * kIdwtRun;
        const float2* lo = in + pp * 2 * no * Q + q;
        const float2* hi = lo + (int64_t)no * Q;
        float2* dst = out + (pp * ni + 2 * h0) * Q + q;
        CVec<V> u[kF / 2], v[kF / 2];                         // coarse plane i at i mod 6
        auto get = [&](int t) {
            const int i = h0 + t;
            u[t % 6] = i < no ? cv_load<V>(lo + (int64_t)i * Q) : cv_zero<V>();
            v[t % 6] = i < no ? cv_load<V>(hi + (int64_t)i * Q) : cv_zero<V>();
        };
#pragma unroll
        for (int t = 0; t < kF / 2 - 1; ++t) get(t);
#pragma unroll
        for (int h = 0; h < kIdwtRun; ++h) {
            const int o = 2 * (h0 + h);
            if (o >= ni) break;
            get(h + 5);
            CVec<V> e = cv_zero<V>(), d = cv_zero<V>();
#pragma unroll
            for (int j = 0; j < kF / 2; ++j) {
                cv_fma<V>(e, f.rec_lo[10 - 2 * j], u[(h + j) % 6]);
                cv_fma<V>(e, f.rec_hi[2 * j], v[(h + 5 - j) % 6]);
                cv_fma<V>(d, f.rec_lo[11 - 2 * j], u[(h + j) % 6]);
                cv_fma<V>(d, f.rec_hi[2 * j + 1], v[(h + 5 - j) % 6]);
            }
            cv_store<V>(dst + (int64_t)(2 * h) * Q, e);
            if (o + 1 < ni) cv_store<V>(dst + (int64_t)(2 * h + 1) * Q, d);
        }
    }
}

// Threads of the slice kernels: whole warps for one column each, at most 256.
static unsigned slice_threads(int cols) { return (unsigned)std::min(256, std::max(64, (cols + 31) / 32 * 32)); }
static dim3 slice_grid(int tiles, int64_t slices) {
    const int64_t gy = std::min<int64_t>(slices, 32768);
    return dim3((unsigned)tiles, (unsigned)gy, (unsigned)((slices + gy - 1) / gy));
}
static dim3 z_grid(int64_t Q, int V, int64_t runs) {
    return dim3((unsigned)((Q / V + 255) / 256), (unsigned)std::min<int64_t>(runs, 65535));
}
static bool two_wide(int64_t Q, const void* a, const void* b) {
    return Q % 2 == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0;
}

// fresh: the dual starts from zero instead of p_w2's contents.
tr_status wavelet_dual(tr_plan* p, const float2* u_bar, float2* p_w2, float sigma, float lam, cudaStream_t st, bool fresh) {
    WaveletPlan* w = p->wav;
    const int nimg = p->B * p->E;
    if (w->levels == 0) return fail(TR_ERR_UNSUPPORTED, "image too small for a db6 decomposition");
    TR_TRY(ensure_wavelet_buffers(p, nimg));
    const float2* cur = u_bar;
    for (int l = 0; l < w->levels; ++l) {
        const int* si = w->in_shape[l];
        const int* so = w->out_shape[l];
        const int64_t Q = (int64_t)si[1] * si[2];
        const int V = two_wide(Q, cur, w->T1) ? 2 : 1;
        auto runs = [&](int run) { return (int64_t)nimg * ((so[0] + run - 1) / run); };
        const bool few = (Q / V + 255) / 256 * runs(kDwtRun) < 2 * p->sms;
        auto fn = few ? (V == 2 ? k_dwt_z<2, kDwtRunShort> : k_dwt_z<1, kDwtRunShort>)
                      : (V == 2 ? k_dwt_z<2, kDwtRun> : k_dwt_z<1, kDwtRun>);
        fn<<<z_grid(Q, V, runs(few ? kDwtRunShort : kDwtRun)), 256, 0, st>>>(cur, w->T1, nimg, si[0], Q, so[0], w->f);
        TR_CHECK_LAUNCH();
        DwtYxArgs a;
        a.in = w->T1;
        a.nimg = nimg;
        a.Zo = so[0];
        a.Yi = si[1];
        a.Yo = so[1];
        a.Xi = si[2];
        a.Xo = so[2];
        a.coarsest = (l == w->levels - 1);
        a.fresh = fresh;
        a.next = a.coarsest ? nullptr : w->A[l & 1];
        a.pw2 = p_w2;
        a.ncoef = w->ncoef;
        a.det_off = w->det_off[l];
        a.sigma = sigma;
        a.lam = lam;
        a.f = w->f;
        const size_t smem = dwt_yx_smem(si[2]);
        TR_TRY(raise_smem_limit((const void*)k_dwt_yx, smem));
        k_dwt_yx<<<slice_grid((so[1] + kDwtRows - 1) / kDwtRows, (int64_t)nimg * 2 * so[0]), slice_threads(si[2]), smem, st>>>(a);
        TR_CHECK_LAUNCH();
        cur = a.next;
    }
    return TR_OK;
}

tr_status wavelet_adjoint(tr_plan* p, const float2* p_w2, float2* out, cudaStream_t st) {
    WaveletPlan* w = p->wav;
    const int nimg = p->B * p->E;
    if (w->levels == 0) return fail(TR_ERR_UNSUPPORTED, "image too small for a db6 decomposition");
    TR_TRY(ensure_wavelet_buffers(p, nimg));
    const float2* approx = p_w2;                   // cA of the coarsest level leads every image's tree
    int64_t approx_stride = w->ncoef;
    for (int l = w->levels - 1; l >= 0; --l) {
        const int* si = w->in_shape[l];
        const int* so = w->out_shape[l];
        IdwtYxArgs a;
        a.approx = approx;
        a.approx_stride = approx_stride;
        a.pw2 = p_w2;
        a.ncoef = w->ncoef;
        a.det_off = w->det_off[l];
        a.nimg = nimg;
        a.Zo = so[0];
        a.Yo = so[1];
        a.Xo = so[2];
        a.Yi = si[1];
        a.Xi = si[2];
        a.vec = si[2] % 2 == 0;
        a.out = w->T1;
        a.f = w->f;
        // 32 output rows per CTA (from 21 coarse rows), 16 (13) where their shared memory would leave one CTA per SM
        const bool tall = idwt_yx_smem(32, so[2]) <= 100 * 1024;
        const size_t smem = idwt_yx_smem(tall ? 32 : 16, so[2]);
        auto fn = tall ? k_idwt_yx<32> : k_idwt_yx<16>;
        TR_TRY(raise_smem_limit((const void*)fn, smem));
        fn<<<slice_grid((si[1] + (tall ? 31 : 15)) / (tall ? 32 : 16), (int64_t)nimg * 2 * so[0]), slice_threads(2 * so[2]),
             smem, st>>>(a);
        TR_CHECK_LAUNCH();
        const int64_t Q = (int64_t)si[1] * si[2], runs = (int64_t)nimg * (((si[0] + 1) / 2 + kIdwtRun - 1) / kIdwtRun);
        float2* dst = l == 0 ? out : w->A[l & 1];
        if (two_wide(Q, w->T1, dst))
            k_idwt_z<2><<<z_grid(Q, 2, runs), 256, 0, st>>>(w->T1, dst, nimg, so[0], Q, si[0], w->f);
        else
            k_idwt_z<1><<<z_grid(Q, 1, runs), 256, 0, st>>>(w->T1, dst, nimg, so[0], Q, si[0], w->f);
        TR_CHECK_LAUNCH();
        approx = dst;
        approx_stride = (int64_t)si[0] * si[1] * si[2];
    }
    return TR_OK;
}

}  // namespace tr

using namespace tr;

// W2 analysis alone: the dual update of wavelet_dual with a zero dual, unit step
// and an inactive projection (p = 0 + 1 c, scale min(1, FLT_MAX / |c|) = 1) is
// the coefficient tree itself, bit for bit.
extern "C" tr_status tr_wavelet_forward(tr_plan* p, const void* images, void* coeffs, void* stream) {
    if (!p || !images || !coeffs) return fail(TR_ERR_INVALID_ARG, "tr_wavelet_forward: null argument");
    if (!p->wav || p->wav->levels == 0)
        return fail(TR_ERR_UNSUPPORTED, "image too small for a db6 decomposition");
    DeviceGuard g(p->device);
    cudaStream_t st = (cudaStream_t)stream;
    return wavelet_dual(p, (const float2*)images, (float2*)coeffs, 1.0f, FLT_MAX, st, true);
}

extern "C" tr_status tr_wavelet_adjoint(tr_plan* p, const void* coeffs, void* images, void* stream) {
    if (!p || !images || !coeffs) return fail(TR_ERR_INVALID_ARG, "tr_wavelet_adjoint: null argument");
    if (!p->wav || p->wav->levels == 0)
        return fail(TR_ERR_UNSUPPORTED, "image too small for a db6 decomposition");
    DeviceGuard g(p->device);
    return wavelet_adjoint(p, (const float2*)coeffs, (float2*)images, (cudaStream_t)stream);
}
