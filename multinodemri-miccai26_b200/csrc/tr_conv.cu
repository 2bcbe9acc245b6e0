// 3x3x3 convolutions (stride 1, zero padding 1) for the learned PDHG warm start on the
// 5th-generation tensor cores: BF16 operands (tcgen05.mma kind::f16), FP32 accumulators in TMEM.
//
// Layout: activations channels-last (N, D, H, W, C); weights (Cout, 27, Cin) bf16 with tap
// t = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1).
//   forward      y[v, co] = bias[co] + sum_{t, ci} w[co, t, ci] x[v + off_t, ci]
//                (the data gradient is the same kernel with w'[ci, 26 - t, co] = w[co, t, ci])
//   weight grad  dw[co, t, ci] = sum_v gy[v, co] x[v + off_t, ci]
//                split over voxel columns into per-CTA partials, then a fixed-order sum
//                (deterministic).
// Requirements: Cin even, Cout % 8 == 0, Cout <= 128.
//
// Both kernels are implicit GEMMs that never form the 27-fold im2col matrix.  A halo of voxels
// sits in shared memory as planes of 8 channels, [plane][voxel][16 bytes]: the unswizzled
// core-matrix layout of tcgen05 operands, in which 8 x-neighbours are one 128-byte core matrix
// and any 16-byte aligned start address is valid.  A tap (dz, dy, dx) is then just another start
// address in the operand descriptor, so each voxel is read from L2 once per halo instead of once
// per tap.  Forward reads the planes K-major (K = channels), the weight gradient reads the same
// planes MN-major (K = voxels).
//
// Every wait is bounded (kMbarPollLimit polls, or the calling thread's tr_conv3d_set_wait_limit); a CTA
// whose wait runs out writes NaN to its outputs (the error mark a caller sees), lets its MMAs and copies end
// (at most kMbarDrainLimit polls, whatever the limit), frees its TMEM and leaves.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "tr_fft.cuh"
#include "tr_internal.cuh"

namespace {

using tr::kMbarDrainLimit;
using tr::kMbarPollLimit;
using tr::mbar_init;
using tr::mbar_wait_bounded;
using tr::smem_u32;

// ------------------------------------------------------------------ tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {      // one warp, all lanes
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Operand descriptors come as (low, high) words: the loops advance the low words (start addresses) only.
__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi, uint32_t idesc,
                                        bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n setp.ne.b32 p, %6, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}\n" ::"r"(d), "r"(alo), "r"(ahi), "r"(blo), "r"(bhi),
        "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// One lane of a converged warp.  The MMA issue loops run under it in a warp index made uniform
// by a shuffle, fully unrolled: operands then sit in uniform registers.  Issued from a
// `threadIdx.x == 0` branch an MMA costs 144 cycles whatever its shape, this way the cycles its
// operands take to come from shared memory at 128 bytes a cycle (41 for 128 x 32 x 16).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// Arrives on `bar` once every MMA this thread issued before has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// 8 consecutive 32-bit columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// nc (8, 16, 24 or 32) columns of this warp's lanes to each lane's row (16-byte aligned).
__device__ __forceinline__ void tmem_to_rows(uint32_t addr, int nc, float* row) {
    if (nc == 32) {
        uint32_t r[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
              "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
              "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(addr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i)
            reinterpret_cast<uint4*>(row)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        return;
    }
    for (int k = 0; k < nc; k += 8) {
        float v[8];
        tmem_ld8(addr + k, v);
        reinterpret_cast<float4*>(row + k)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(row + k)[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Shared-memory operand descriptor, no swizzle.  lead / stride in bytes:
//   K-major   stride: next 8 rows (M or N), lead: next 8 K elements
//   MN-major  stride: next 8 rows (M or N), lead: next 8 K elements
__device__ __forceinline__ uint64_t op_desc(uint32_t saddr, uint32_t lead, uint32_t stride) {
    return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)((lead >> 4) & 0x3fff) << 16) |
           ((uint64_t)((stride >> 4) & 0x3fff) << 32) | (1ull << 46);
}
// Instruction descriptor: bf16 x bf16 -> f32, M x N.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, bool mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? (1u << 15) | (1u << 16) : 0u) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

struct ConvDims {
    int N, D, H, W, Cin, Cout;
    int64_t V;   // N*D*H*W
};

// An MMA tile's voxels: 8 (x) by 16 (y) of one z slice, halo one voxel wide.
constexpr int kTX = 8, kTY = 16;
constexpr int kHX = kTX + 2, kHY = kTY + 2;
constexpr int kSlice = kHX * kHY;                     // halo voxels per z slice
// Voxels per plane, padded to 2 mod 8: a quarter-warp stores 2 voxels x 4 planes (16 bytes
// each) to eight different bank groups.
__host__ __device__ constexpr int plane_pitch(int voxels) { return voxels + ((2 - voxels % 8) + 8) % 8; }

// ------------------------------------------------------------------ 8 channels of one voxel
// Channels [c, c + 8) at p (the voxel's channel 0), zero past C; VEC: C % 8 == 0 and 16-byte
// aligned rows; else pairs: 4-byte aligned rows.
template <bool VEC>
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p, int c, int C, bool pairs) {
    if constexpr (VEC) {
        return c < C ? *reinterpret_cast<const uint4*>(p + c) : make_uint4(0, 0, 0, 0);
    } else {
        uint32_t r[4] = {0u, 0u, 0u, 0u};
        if (pairs) {
#pragma unroll
            for (int i = 0; i < 4; ++i)               // C is even: pairs never straddle the end
                if (c + 2 * i < C) r[i] = *reinterpret_cast<const uint32_t*>(p + c + 2 * i);
        } else {
            const auto* h = reinterpret_cast<const unsigned short*>(p + c);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c + 2 * i < C) r[i] = h[2 * i] | ((uint32_t)h[2 * i + 1] << 16);
        }
        return make_uint4(r[0], r[1], r[2], r[3]);
    }
}
__host__ __device__ __forceinline__ bool at16(const void* p) { return (uintptr_t)p % 16 == 0; }
__host__ __device__ __forceinline__ bool at4(const void* p) { return (uintptr_t)p % 4 == 0; }
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// The same as it is held between its load and its store to shared memory: float input is
// rounded only then, so that several loads are in flight.
template <class TIn, bool VEC>
struct Piece {
    uint4 v;
    __device__ __forceinline__ void zero() { v = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void load(const __nv_bfloat16* p, int c, int C, bool pairs) { v = load8<VEC>(p, c, C, pairs); }
    __device__ __forceinline__ uint4 bf16() const { return v; }
};
template <bool VEC>
struct Piece<float, VEC> {
    float f[8];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = 0.f;
    }
    __device__ __forceinline__ void load(const float* p, int c, int C, bool) {
        if constexpr (VEC) {
            if (c >= C) return zero();
            const float4 a = *reinterpret_cast<const float4*>(p + c), b = *reinterpret_cast<const float4*>(p + c + 4);
            f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
            f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = c + i < C ? p[c + i] : 0.f;
        }
    }
    __device__ __forceinline__ uint4 bf16() const {
        return make_uint4(bf16_pair(f[0], f[1]), bf16_pair(f[2], f[3]), bf16_pair(f[4], f[5]), bf16_pair(f[6], f[7]));
    }
};

// ------------------------------------------------------------------ forward
// Persistent: one CTA per SM walks over tiles of NZ z slices of 8 x 16 voxels (NZ MMA tiles of
// 128 voxels), every output channel.  Warp roles, joined by mbarrier rings:
//   warps 8-15  halo of the next 16 channels into shared memory (float input becomes bf16 here)
//   warp 1      packed weights of one or three (dz, dy) rows of taps by one bulk copy a stage
//   warps 0, 2  MMAs: 27 taps x 16 channels per halo stage, half of the slices each (one thread's
//               issue, about 30 cycles an MMA with its waits, was slower than the small MMAs)
//   warps 4-7   finished accumulators (two in TMEM where they fit) to global memory, plus bias
// Loads, MMAs and stores of different tiles overlap; with loads, MMAs and the epilogue of a tile in
// sequence and two CTAs per SM the tensor pipe idled more than half of the time.  Bound by the MMAs'
// operand reads from shared memory (128 bytes a cycle: 4 KB of voxels and 32 bytes per output
// channel for 128 x Cout x 16 products), so by the tensor cores only from Cout = 128 on.
// Measured at (1, 128, 256, 256), 64 -> 32 channels, float input (converted by a pass of its own
// before): 21.5 ms with mma.sync fragments gathered from global memory, 1.34 to 1.38 ms with this kernel.
constexpr int kFwdThreads = 512;
constexpr int kLoaders = 256;                         // warps 8-15
constexpr int kHaloStages = 4;
constexpr int kMaxWStages = 4;
constexpr int kRowTaps = 3;                           // a (dz, dy) row: dx = -1, 0, 1
constexpr int kEpPitch = 36;                          // floats per row of the epilogue's staging tile

// Halo voxels per plane, padded to 4 mod 8: a quarter-warp stores 4 voxels x 2 planes (16 bytes
// each) to eight different bank groups.
__host__ __device__ constexpr int halo_pitch(int nz) { return kSlice * (nz + 2) + ((4 - kSlice * (nz + 2) % 8) + 8) % 8; }
__host__ __device__ constexpr int halo_stage_bytes(int nz) { return 2 * halo_pitch(nz) * 16; }
__host__ __device__ constexpr int w_row_bytes(int npad) { return kRowTaps * 2 * npad * 16; }
// Rows per weight stage and stages: a wait per 36 MMAs where three such stages fit beside the halo.
__host__ __device__ constexpr int w_stage_rows(int npad) { return npad <= 64 ? 3 : 1; }
__host__ __device__ constexpr int w_stages(int npad) { return npad <= 64 ? 3 : kMaxWStages; }
static size_t fwd_smem_bytes(int nz, int npad) {
    return (size_t)kHaloStages * halo_stage_bytes(nz) + (size_t)w_stages(npad) * w_stage_rows(npad) * w_row_bytes(npad) +
           4 * 32 * kEpPitch * sizeof(float) + 128;
}

// The MMAs of one row of taps and a 16-channel step on NS z slices.
template <int NS>
__device__ __forceinline__ void fwd_mmas(uint32_t a0, uint32_t ahi, uint32_t b0, uint32_t bhi, uint32_t tmem, int npad,
                                         uint32_t idesc, bool accumulate) {
#pragma unroll
    for (int dx = 0; dx < kRowTaps; ++dx)
#pragma unroll
        for (int m = 0; m < NS; ++m)
            mma_f16(tmem + m * npad, a0 + m * kSlice + dx, ahi, b0 + dx * 2 * npad, bhi, idesc, accumulate || dx > 0);
}

// Weights as the forward kernel streams them: [16 input channels][tap][plane of 8][npad output
// channels][8] bf16, zeros past the channel counts, so that a stage is one contiguous copy.  (TMA
// boxes of the unpacked weights have 16-byte rows and take about four cycles a row, more than a
// stage's MMAs.)  FLIP: the data gradient's weights w'[ci, t, co] = w[co, 26 - t, ci]; nout / nin
// are the output / input channels of the convolution that uses the packed weights.
//
// A last chunk of fewer than 16 channels comes first: its 27 steps add little, and each step of the sum loses a
// share of what is summed so far (24 input channels, 48 outputs: relative error 7.2e-7 with it last, 6.1e-7 first).
__host__ __device__ __forceinline__ int channel_chunk(int step, int cin) {
    const int n = (cin + 15) / 16, c = cin % 16 ? step + n - 1 : step;
    return c < n ? c : c - n;
}
template <class TW, bool FLIP>
__global__ void __launch_bounds__(256) k_conv3d_pack(const TW* __restrict__ w, __nv_bfloat16* __restrict__ packed, int nout,
                                                     int nin, int npad, int total) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int k8 = i & 7, n = (i >> 3) % npad, r = (i >> 3) / npad, pl = r & 1, t = (r >> 1) % 27, ch = (r >> 1) / 27;
    const int k = channel_chunk(ch, nin) * 16 + pl * 8 + k8;
    float v = 0.f;
    if (n < nout && k < nin)
        v = (float)(FLIP ? w[((int64_t)k * 27 + 26 - t) * nout + n] : w[((int64_t)n * 27 + t) * nin + k]);
    packed[i] = __float2bfloat16_rn(v);
}
__host__ __device__ constexpr int conv_npad(int cout) { return (cout + 15) / 16 * 16; }
int64_t packed_elems(int cin, int cout) { return (int64_t)((cin + 15) / 16) * 27 * 16 * conv_npad(cout); }

// VEC: halo rows are read 16 bytes at a time; yvec: y is 16-byte aligned, rows are written so.
// Off: offsets of halo voxels from the halo's corner (64 bits where a halo spans 2^31 voxels or more).
template <int NZ, class TIn, bool VEC, class Off>
__global__ void __launch_bounds__(kFwdThreads, 1) k_conv3d_fwd(const TIn* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ w,
                                                               const float* __restrict__ bias, float* __restrict__ y,
                                                               ConvDims c, int64_t tiles, int npad, int nacc, uint32_t cols,
                                                               int yvec, int poll) {
    extern __shared__ __align__(128) unsigned char smraw_[];
    __shared__ __align__(8) uint64_t hfull[kHaloStages], hempty[kHaloStages], wfull[kMaxWStages],
        wempty[kMaxWStages], afull[2], aempty[2], drained[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;                                   // some wait ran out: tiles from here on are NaN
    unsigned char* halo = smraw_ + ((128 - (smem_u32(smraw_) & 127)) & 127);
    unsigned char* wring = halo + kHaloStages * halo_stage_bytes(NZ);
    const int rows = w_stage_rows(npad), nst = w_stages(npad);
    unsigned char* eps = wring + nst * rows * w_row_bytes(npad);
    constexpr int kP = halo_pitch(NZ);
    constexpr int kIssuers = NZ > 1 ? 2 : 1, kNS = NZ / kIssuers;     // MMA warps, slices of each
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int nchunk = (c.Cin + 15) / 16;                    // halo stages per tile
    const int ntx = (c.W + kTX - 1) / kTX, nty = (c.H + kTY - 1) / kTY, ntz = (c.D + NZ - 1) / NZ;
    volatile int* vfailed = &failed;

    if (warp == 0) tmem_alloc(&tmem_slot, cols);
    if (tid == 32) {
        for (int s = 0; s < kHaloStages; ++s) {
            mbar_init(&hfull[s], kLoaders / 32);
            mbar_init(&hempty[s], kIssuers);
        }
        for (int s = 0; s < nst; ++s) {
            mbar_init(&wfull[s], 1);
            mbar_init(&wempty[s], kIssuers);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&afull[s], kIssuers);
            mbar_init(&aempty[s], 4);
        }
        mbar_init(&drained[0], 1);
        mbar_init(&drained[1], 1);
        failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    // Bounded wait for use number `use` of a ring entry; after a failure nothing waits any more.
    auto wait = [&](uint64_t* bar, int use) {
        if (!ok) return;
        ok = mbar_wait_bounded(bar, use & 1, poll);
        if (!ok) {
            *vfailed = 1;
            __threadfence_block();
        }
    };

    if (warp == 0 || (kIssuers == 2 && warp == 2)) {
        // ---- MMAs of slices [m0, m0 + kNS)
        if (elect_one()) {
            const int m0 = warp ? kNS : 0;
            const uint32_t idesc = instr_desc(128, npad, false);
            const uint64_t ad = op_desc(smem_u32(halo), kP * 16, kHX * 16), bd = op_desc(smem_u32(wring), npad * 16, 128);
            const uint32_t ahi = (uint32_t)(ad >> 32), bhi = (uint32_t)(bd >> 32), alo = (uint32_t)ad + m0 * kSlice;
            const uint32_t row16 = w_row_bytes(npad) >> 4;
            int hs = 0, hu = 0, ws = 0, wu = 0, n = 0;       // ring entries and their use counts
            for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++n) {
                const int as = nacc == 2 ? n & 1 : 0, au = nacc == 2 ? n >> 1 : n;
                if (au > 0) wait(&aempty[as], au - 1);
                const uint32_t acc = tmem + (as * NZ + m0) * npad;
                for (int ch = 0; ch < nchunk && ok; ++ch) {
                    wait(&hfull[hs], hu);
                    const uint32_t a0 = alo + hs * (halo_stage_bytes(NZ) >> 4);
                    for (int g = 0; g < 9; g += rows) {
                        wait(&wfull[ws], wu);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t b0 = (uint32_t)bd + ws * rows * row16;
                        for (int r = 0; r < rows; ++r) {
                            const int row = g + r;           // (dz, dy)
                            fwd_mmas<kNS>(a0 + ((row / 3) * kHY + row % 3) * kHX, ahi, b0 + r * row16, bhi, acc, npad, idesc,
                                          ch + row > 0);
                        }
                        mma_commit(&wempty[ws]);
                        if (++ws == nst) ws = 0, ++wu;
                    }
                    mma_commit(&hempty[hs]);
                    if (++hs == kHaloStages) hs = 0, ++hu;
                }
                mma_commit(&afull[as]);
            }
            // MMAs in flight end before the TMEM is freed, also where only the epilogue's wait ran out
            mma_commit(&drained[warp >> 1]);
            mbar_wait_bounded(&drained[warp >> 1], 0, kMbarDrainLimit);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- weights
        if (elect_one()) {
            const uint32_t bytes = rows * w_row_bytes(npad);
            int ws = 0, wu = 0, last = 0;                    // copies issued (the last nst may be in flight)
            for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const unsigned char* src = reinterpret_cast<const unsigned char*>(w);
                for (int g = 0; g < 9 * nchunk; g += rows, src += bytes) {
                    if (wu > 0) wait(&wempty[ws], wu - 1);
                    if (!ok) break;
                    tr::mbar_expect_tx(&wfull[ws], bytes);
                    tr::bulk_g2s(wring + ws * bytes, src, bytes, &wfull[ws]);
                    ++last;
                    if (++ws == nst) ws = 0, ++wu;
                }
            }
            for (int i = max(0, last - nst); i < last; ++i)  // no copy outlives the CTA
                mbar_wait_bounded(&wfull[i % nst], (i / nst) & 1, kMbarDrainLimit);
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ---- halo: two 16-byte pieces (8 channels) per voxel, consecutive lanes along the channels
        constexpr int kUnits = 2 * kSlice * (NZ + 2), kPer = (kUnits + kLoaders - 1) / kLoaders;
        constexpr int kBatch = 5;                            // pieces in flight per thread
        const int lt = tid - (kFwdThreads - kLoaders), pl = lt & 1;
        const bool pairs = at4(x);
        int hs = 0, hu = 0;
        for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
            int64_t b = t;
            const int x0 = (int)(b % ntx) * kTX - 1;
            b /= ntx;
            const int y0 = (int)(b % nty) * kTY - 1;
            b /= nty;
            const int z0 = (int)(b % ntz) * NZ - 1, img = (int)(b / ntz);
            Off off[kPer];                                   // voxel offset from the halo corner, -1 outside
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int u = lt + k * kLoaders, vox = u >> 1;
                const int hz = vox / kSlice, r = vox - hz * kSlice, hy = r / kHX, hx = r - hy * kHX;
                const bool in = u < kUnits && (unsigned)(z0 + hz) < (unsigned)c.D && (unsigned)(y0 + hy) < (unsigned)c.H &&
                                (unsigned)(x0 + hx) < (unsigned)c.W;
                off[k] = in ? ((Off)hz * c.H + hy) * c.W + hx : -1;
            }
            const TIn* corner = x + ((((int64_t)img * c.D + z0) * c.H + y0) * c.W + x0) * c.Cin;
            for (int ch = 0; ch < nchunk; ++ch) {
                if (hu > 0) wait(&hempty[hs], hu - 1);
                unsigned char* dst = halo + hs * halo_stage_bytes(NZ) + pl * kP * 16;
                const int c0 = (channel_chunk(ch, c.Cin) * 2 + pl) * 8;
#pragma unroll
                for (int k0 = 0; k0 < kPer; k0 += kBatch) {
                    Piece<TIn, VEC> v[kBatch];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
                        if (k0 + k < kPer && off[k0 + k] >= 0) v[k].load(corner + (int64_t)off[k0 + k] * c.Cin, c0, c.Cin, pairs);
                        else v[k].zero();
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const int u = lt + (k0 + k) * kLoaders;
                        if (k0 + k < kPer && u < kUnits) *reinterpret_cast<uint4*>(dst + (u >> 1) * 16) = v[k].bf16();
                    }
                }
                tr::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&hfull[hs]);
                if (++hs == kHaloStages) hs = 0, ++hu;
            }
        }
    } else if (warp >= 4) {
        // ---- epilogue: TMEM -> registers -> [32 voxels][32 channels] per warp -> 128-byte rows
        float* stage = reinterpret_cast<float*>(eps) + (warp & 3) * 32 * kEpPitch;
        const int q = warp & 3;
        int n = 0;
        for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x, ++n) {
            int64_t b = t;
            const int x0 = (int)(b % ntx) * kTX;
            b /= ntx;
            const int y0 = (int)(b % nty) * kTY + q * 4;
            b /= nty;
            const int z0 = (int)(b % ntz) * NZ, img = (int)(b / ntz);
            const int as = nacc == 2 ? n & 1 : 0, au = nacc == 2 ? n >> 1 : n;
            wait(&afull[as], au);
            __syncwarp();
            tc_fence_after();
            const bool bad = __any_sync(0xffffffffu, !ok || *vfailed != 0);
            for (int m = 0; m < NZ && z0 + m < c.D; ++m) {
                float* out = y + ((((int64_t)img * c.D + z0 + m) * c.H + y0) * c.W + x0) * c.Cout;
                for (int c0 = 0; c0 < c.Cout; c0 += 32) {
                    const int nc = min(32, c.Cout - c0);
                    tmem_to_rows(tmem + ((uint32_t)(q * 32) << 16) + (as * NZ + m) * npad + c0, nc, stage + lane * kEpPitch);
                    __syncwarp();
                    // MMA row: x = row % 8, y = row / 8; a lane keeps its columns where nc is a power of two
                    const int n4 = nc >> 2, per = n4 == 6 ? 30 : 32;
                    const int c4 = (lane % n4) * 4, row0 = lane < per ? lane / n4 : 32, step = per / n4;
                    const float4 bv = bias ? make_float4(bias[c0 + c4], bias[c0 + c4 + 1], bias[c0 + c4 + 2], bias[c0 + c4 + 3])
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                    for (int row = row0; row < 32; row += step) {
                        const int xx = row & 7, yy = row >> 3;
                        if (x0 + xx >= c.W || y0 + yy >= c.H) continue;
                        float4 v = *reinterpret_cast<const float4*>(stage + row * kEpPitch + c4);
                        if (bias) v = make_float4(v.x + bv.x, v.y + bv.y, v.z + bv.z, v.w + bv.w);
                        if (bad) v.x = v.y = v.z = v.w = __int_as_float(0x7fffffff);
                        float* dst = out + ((int64_t)yy * c.W + xx) * c.Cout + c0 + c4;
                        if (yvec) {
                            *reinterpret_cast<float4*>(dst) = v;
                        } else {
                            dst[0] = v.x, dst[1] = v.y, dst[2] = v.z, dst[3] = v.w;
                        }
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&aempty[as]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, cols);
}

// ------------------------------------------------------------------ weight gradient
// GEMM with K = voxels: dw_t = X_t^T G.  One CTA marches along z through 8 x 16 voxel columns
// (each x slice is loaded once for the three dz taps that read it), holding the accumulators of
// a group of taps in TMEM: M = 64 channels of the wider side, N = up to 64 channels of the other;
// an M = 64 accumulator fills half of the TMEM lanes, so two taps share a column range.
// Warps 8-15 keep a ring of four items (x slice i, gy slice i - 2) filled, warps 0 and 2 issue
// the MMAs of half of the taps each.  After every run of at most kWgRunSlices slices all warps add the
// accumulators to the CTA's partial, a [27][Cin][Cout] slab piece (in float32, one add per value and run by
// the same thread, so in a fixed order).  Grid: (splits of the voxel columns, tap groups, channel chunks); the
// partials are summed in split order by k_wgrad_reduce.
// Measured, both kernels: (4, 32, 32, 32), 64 -> 32 channels: 453 us with mma.sync (16 voxels a step
// gathered element by element, 27 passes over the voxels), 52 us with these.  (8, 32, 32, 32), 128 -> 128:
// 4.32 ms and a relative error of 1.4e-6 with mma.sync (sums of 2,048 voxels); 290 us and 1.5e-5 with one
// accumulator over a CTA's whole share (14,600 voxels), 367 us and 1.4e-6 with runs.
constexpr int kWgThreads = 512;
constexpr int kWgLoaders = 256;                        // warps 8-15
constexpr int kWgRing = 4;
constexpr int kXPitch = plane_pitch(kSlice);          // voxels per plane of an x slice
constexpr int kGPitch = plane_pitch(kTX * kTY);       // voxels per plane of a gy slice
constexpr int kWgChunk = 64;                          // channels per CTA and side
constexpr int kWgradVox = 2048;                       // voxels per partial that callers' scratch covers at least
// z slices (128 voxels each) that a TMEM accumulator sums.  The tensor core's float32 sums lose about half
// a last bit a step, all in one direction, so that the error grows with the length of a sum.
constexpr int kWgRunSlices = kWgradVox / (kTX * kTY);

struct WgradShape {
    bool mx;             // M side = x (Cin), N side = gy (Cout); else the other way round
    int npad;            // N columns per tap
    int px, pg;          // planes held per slot
    int groups;          // tap groups (grid y)
    int cx, cg;          // channel chunks of each side
    uint32_t cols;
    int64_t cols_n, units;           // (image, y, x) voxel columns; z segments of all of them
    int seg_len, splits;
    int run;                         // units whose voxels one accumulator sums
};

// Tap groups: all 27 taps' accumulators fit TMEM (two per column range) up to 32 columns each.
__host__ __device__ constexpr int wgrad_groups(int npad) { return npad <= 32 ? 1 : 2; }

// The MMAs of one z slice: taps [TA, TB) of the group from T0 on, 16 voxels (two rows of 8) a step.
template <int NPAD, bool MX, int T0, int TA, int TB>
__device__ __forceinline__ void wgrad_mmas(const uint32_t (&xl)[3], uint32_t xhi, uint32_t gl, uint32_t ghi, uint32_t tmem,
                                           uint32_t idesc, bool first) {
#pragma unroll 1
    for (int ks = 0; ks < kTY / 2; ++ks) {
        const uint32_t gk = gl + ks * 2 * kTX, xo = ks * 2 * kHX;
        const bool more = !(first && ks == 0);
#pragma unroll
        for (int t = TA; t < TB; ++t) {
            const uint32_t xk = xl[t / 9] + xo + ((t / 3) % 3 * kHX + t % 3);
            const uint32_t acc = tmem + ((t - T0) >> 1) * NPAD + ((uint32_t)((t - T0) & 1) << 20);
            if (MX) mma_f16(acc, xk, xhi, gk, ghi, idesc, more);
            else mma_f16(acc, gk, ghi, xk, xhi, idesc, more);
        }
    }
}

// Infinite and NaN values in the last x or y of the volume, where a tile reaches past it: the tile's voxels
// outside the volume have gy = 0, and for taps towards smaller x or y the MMAs multiply that zero with the
// last voxels' x, which must not turn a finite sum into NaN.  The loaders put zeros for such values (finite8),
// and a CTA that met some adds their products with the tile's own voxels here.
__device__ __forceinline__ uint4 finite8(uint4 v, int* seen) {
    uint32_t* r = &v.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t m = __vcmpeq2(r[i] & 0x7f807f80u, 0x7f807f80u);
        r[i] &= ~m;
        if (m) *seen = 1;
    }
    return v;
}
__device__ __forceinline__ void wgrad_add_nonfinite(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gy,
                                                 float* __restrict__ dst, const ConvDims& c, const WgradShape& s, int t0,
                                                 int t1, int cx0, int cg0) {
    const int nx = min(kWgChunk, c.Cin - cx0), ng = min(kWgChunk, c.Cout - cg0);
    const int ntx = (c.W + kTX - 1) / kTX, nty = (c.H + kTY - 1) / kTY;
    for (int e = threadIdx.x; e < (t1 - t0) * nx * ng; e += kWgThreads) {
        const int co = cg0 + e % ng, ci = cx0 + e / ng % nx, t = t0 + e / ng / nx;
        const int dz = t / 9 - 1, dy = t / 3 % 3 - 1, dx = t % 3 - 1;
        float sum = 0.f;
        bool any = false;
        for (int64_t u = blockIdx.x; u < s.units; u += s.splits) {
            const int64_t col = u % s.cols_n;
            const int x0 = (int)(col % ntx) * kTX, y0 = (int)((col / ntx) % nty) * kTY;
            const bool ex = x0 + kTX > c.W, ey = y0 + kTY > c.H;
            if (!ex && !ey) continue;
            const int64_t img = col / ((int64_t)ntx * nty);
            const int z0 = (int)(u / s.cols_n) * s.seg_len, z1 = min(z0 + s.seg_len, c.D);
            for (int z = max(z0, -dz); z < min(z1, c.D - dz); ++z)
                for (int y = max(y0, -dy); y < min(y0 + kTY, c.H - max(dy, 0)); ++y)
                    for (int xx = max(x0, -dx); xx < min(x0 + kTX, c.W - max(dx, 0)); ++xx) {
                        if (!(ex && xx + dx == c.W - 1) && !(ey && y + dy == c.H - 1)) continue;
                        const int64_t v = ((img * c.D + z) * c.H + y) * c.W + xx;
                        const float f = __bfloat162float(x[(v + ((int64_t)dz * c.H + dy) * c.W + dx) * c.Cin + ci]);
                        if (isfinite(f)) continue;
                        sum += f * __bfloat162float(gy[v * c.Cout + co]);
                        any = true;
                    }
        }
        if (any) atomicAdd(dst + ((int64_t)t * c.Cin + ci) * c.Cout + co, sum);
    }
}

// XVEC: x is copied 16 bytes at a time; MX: the M side is x (else gy); NPAD: columns per tap; TAIL: some tiles
// reach past the volume (the checks for infinite x cost 7 % at 64 channels on both sides).
template <int NPAD, bool XVEC, bool MX, bool TAIL>
__global__ void __launch_bounds__(kWgThreads) k_conv3d_wgrad(const __nv_bfloat16* __restrict__ x,
                                                             const __nv_bfloat16* __restrict__ gy,
                                                             float* __restrict__ part, ConvDims c, WgradShape s,
                                                             int poll) {
    extern __shared__ __align__(128) unsigned char smraw_[];
    __shared__ __align__(8) uint64_t full[kWgRing], empty[kWgRing], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int nonfinite;                                // some x was left out (finite8)
    unsigned char* sm = smraw_ + ((128 - (smem_u32(smraw_) & 127)) & 127);
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int split = blockIdx.x;
    constexpr int G = wgrad_groups(NPAD);
    const int t0 = G == 1 ? 0 : blockIdx.y * 14, t1 = G == 1 ? 27 : min(27, t0 + 14);
    const int cx0 = (blockIdx.z % s.cx) * kWgChunk, cg0 = (blockIdx.z / s.cx) * kWgChunk;
    const uint32_t xbytes = (uint32_t)s.px * kXPitch * 16, slot = xbytes + (uint32_t)s.pg * kGPitch * 16;
    const int ntx = (c.W + kTX - 1) / kTX, nty = (c.H + kTY - 1) / kTY;

    if (warp == 0) tmem_alloc(&tmem_slot, s.cols);
    if (tid == 0) {
        for (int i = 0; i < kWgRing; ++i) {
            mbar_init(&full[i], kWgLoaders / 32);
            mbar_init(&empty[i], 2);
        }
        mbar_init(&done, 2);
        nonfinite = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int64_t stride = (int64_t)s.run * s.splits;        // units between two runs
    float* dst = part + (int64_t)split * 27 * c.Cin * c.Cout;
    bool ok = true;
    int item0 = 0;                        // ring items before this run

    int run = 0;
    for (int64_t u0 = split; u0 < s.units; u0 += stride, ++run) {
        const int64_t u1 = min(s.units, u0 + stride);
        if (warp == 0 || warp == 2) {
            if (elect_one()) {
                const uint32_t idesc = instr_desc(64, NPAD, true);
                const uint64_t xd = op_desc(smem_u32(sm), kHX * 16, kXPitch * 16);
                const uint64_t gd = op_desc(smem_u32(sm) + xbytes, kTX * 16, kGPitch * 16);
                const uint32_t slot16 = slot >> 4, xhi = (uint32_t)(xd >> 32), ghi = (uint32_t)(gd >> 32);
                bool first = true;
                int item = item0;
                for (int64_t u = u0; u < u1 && ok; u += s.splits) {
                    const int z0 = (int)(u / s.cols_n) * s.seg_len, nz = min(s.seg_len, c.D - z0);
                    for (int k = 0; k < nz && ok; ++k) {
                        for (int i = (k == 0 ? 0 : 2); i < 3 && ok; ++i) {
                            const int j = item + k + i;
                            ok = mbar_wait_bounded(&full[j % kWgRing], (j / kWgRing) & 1, poll);
                        }
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t xl[3] = {(uint32_t)xd + (item + k) % kWgRing * slot16,
                                                (uint32_t)xd + (item + k + 1) % kWgRing * slot16,
                                                (uint32_t)xd + (item + k + 2) % kWgRing * slot16};
                        const uint32_t gl = (uint32_t)gd + (item + k + 2) % kWgRing * slot16;
                        if (G == 1) {
                            if (warp == 0) wgrad_mmas<NPAD, MX, 0, 0, 14>(xl, xhi, gl, ghi, tmem, idesc, first);
                            else wgrad_mmas<NPAD, MX, 0, 14, 27>(xl, xhi, gl, ghi, tmem, idesc, first);
                        } else if (blockIdx.y == 0) {
                            if (warp == 0) wgrad_mmas<NPAD, MX, 0, 0, 7>(xl, xhi, gl, ghi, tmem, idesc, first);
                            else wgrad_mmas<NPAD, MX, 0, 7, 14>(xl, xhi, gl, ghi, tmem, idesc, first);
                        } else {
                            if (warp == 0) wgrad_mmas<NPAD, MX, 14, 14, 21>(xl, xhi, gl, ghi, tmem, idesc, first);
                            else wgrad_mmas<NPAD, MX, 14, 21, 27>(xl, xhi, gl, ghi, tmem, idesc, first);
                        }
                        first = false;
                        mma_commit(&empty[(item + k) % kWgRing]);        // x slice k is not read again
                    }
                    for (int i = 0; i < 2; ++i) mma_commit(&empty[(item + nz + i) % kWgRing]);
                    item += nz + 2;
                }
                mma_commit(&done);
            }
            __syncwarp();
        } else if (warp >= 8) {
            // ---- 16-byte pieces, consecutive lanes along a voxel's channels; a thread's pieces keep their
            // places while the CTA marches along z
            constexpr int kPerX = (kSlice * 8 + kWgLoaders - 1) / kWgLoaders, kPerG = kTX * kTY * 8 / kWgLoaders;
            const int lt = tid - (kWgThreads - kWgLoaders);
            const int nx = min(s.px, 2 * ((min(kWgChunk, c.Cin - cx0) + 15) / 16));     // planes with channels
            const int ng = min(s.pg, 2 * ((min(kWgChunk, c.Cout - cg0) + 15) / 16));
            const int64_t hw = (int64_t)c.H * c.W;
            int item = item0;
            for (int64_t u = u0; u < u1; u += s.splits) {
                const int64_t col = u % s.cols_n;
                const int x0 = (int)(col % ntx) * kTX, y0 = (int)((col / ntx) % nty) * kTY;
                const int img = (int)(col / ((int64_t)ntx * nty));
                const int64_t corner = (int64_t)y0 * c.W + x0;     // of the tile in its slice
                const int z0 = (int)(u / s.cols_n) * s.seg_len, nz = min(s.seg_len, c.D - z0);
                int vx[kPerX], vg[kPerG], dx[kPerX], dg[kPerG];    // row, column in the tile (-1: none); place in the slot
                constexpr int kEdge = 512;                         // added to vx: last x or y, beside voxels outside
#pragma unroll
                for (int k = 0; k < kPerX; ++k) {
                    const int v = lt + k * kWgLoaders, vox = v / nx, pl = v - vox * nx;
                    const int hy = vox / kHX, hx = vox - hy * kHX, yy = y0 - 1 + hy, xx = x0 - 1 + hx;
                    dx[k] = v < kSlice * nx ? (pl * kXPitch + vox) * 16 : -1;
                    vx[k] = dx[k] >= 0 && (unsigned)yy < (unsigned)c.H && (unsigned)xx < (unsigned)c.W ? hy * 16 + hx : -1;
                    if (TAIL && vx[k] >= 0 && ((xx == c.W - 1 && x0 + kTX > c.W) || (yy == c.H - 1 && y0 + kTY > c.H))) vx[k] |= kEdge;
                }
#pragma unroll
                for (int k = 0; k < kPerG; ++k) {
                    const int v = lt + k * kWgLoaders, vox = v / ng, pl = v - vox * ng;
                    dg[k] = v < kTX * kTY * ng ? (pl * kGPitch + vox) * 16 : -1;
                    vg[k] = dg[k] >= 0 && y0 + (vox >> 3) < c.H && x0 + (vox & 7) < c.W ? vox : -1;
                }
                for (int i = 0; i < nz + 2; ++i, ++item) {
                    if (item >= kWgRing)
                        ok = ok && mbar_wait_bounded(&empty[item % kWgRing], (item / kWgRing - 1) & 1, poll);
                    unsigned char* base = sm + (size_t)(item % kWgRing) * slot;
                    const int zx = z0 - 1 + i;
                    const __nv_bfloat16* xs = x + (((int64_t)img * c.D + zx) * hw + corner - c.W - 1) * c.Cin;
                    const __nv_bfloat16* gs = gy + (((int64_t)img * c.D + zx - 1) * hw + corner) * c.Cout;
                    uint4 bx[kPerX], bg[kPerG];
#pragma unroll
                    for (int k = 0; k < kPerX; ++k) {
                        const int ch = cx0 + (dx[k] / (kXPitch * 16)) * 8;
                        bx[k] = make_uint4(0, 0, 0, 0);
                        if (vx[k] >= 0 && (unsigned)zx < (unsigned)c.D)
                            bx[k] = load8<XVEC>(xs + ((int64_t)(vx[k] >> 4 & 31) * c.W + (vx[k] & 15)) * c.Cin, ch, c.Cin, at4(x));
                    }
                    if (i >= 2) {
#pragma unroll
                        for (int k = 0; k < kPerG; ++k) {
                            const int ch = cg0 + (dg[k] / (kGPitch * 16)) * 8;
                            bg[k] = make_uint4(0, 0, 0, 0);
                            const __nv_bfloat16* gv = gs + ((int64_t)(vg[k] >> 3) * c.W + (vg[k] & 7)) * c.Cout;
                            if (vg[k] >= 0)
                                bg[k] = at16(gy) ? load8<true>(gv, ch, c.Cout, true)
                                                 : load8<false>(gv, ch, c.Cout, at4(gy));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kPerX; ++k)
                        if (dx[k] >= 0)
                            *reinterpret_cast<uint4*>(base + dx[k]) = TAIL && vx[k] >= kEdge ? finite8(bx[k], &nonfinite) : bx[k];
                    if (i >= 2) {
#pragma unroll
                        for (int k = 0; k < kPerG; ++k)
                            if (dg[k] >= 0) *reinterpret_cast<uint4*>(base + xbytes + dg[k]) = bg[k];
                    }
                    tr::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[item % kWgRing]);
                }
            }
        }
        for (int64_t u = u0; u < u1; u += s.splits) item0 += min(s.seg_len, c.D - (int)(u / s.cols_n) * s.seg_len) + 2;
        if (tid == 0) ok = ok && mbar_wait_bounded(&done, run & 1, poll);
        const bool bad = __syncthreads_or(!ok) != 0;
        tc_fence_after();
        // ---- part[split][t][ci][co]: lanes 0-15 hold an even accumulator's rows, lanes 16-31 the odd one's
        const int q = warp & 3;
        const int nN = MX ? min(kWgChunk, c.Cout - cg0) : min(kWgChunk, c.Cin - cx0);
        const int nM = MX ? min(kWgChunk, c.Cin - cx0) : min(kWgChunk, c.Cout - cg0);
        float* stage = reinterpret_cast<float*>(sm) + warp * 32 * kEpPitch;      // the ring is idle
        for (int a2 = warp >> 2; 2 * a2 < t1 - t0; a2 += kWgThreads / 128) {
            for (int n0 = 0; n0 < nN; n0 += 32) {
                const int nc = min(32, NPAD - n0);
                tmem_to_rows(tmem + ((uint32_t)(q * 32) << 16) + a2 * NPAD + n0, nc, stage + lane * kEpPitch);
                __syncwarp();
                // four output channels a lane, consecutive lanes along them: the columns (MX) or the rows of a half-warp
                for (int i = lane; i < 8 * nc; i += 32) {
                    const int r = MX ? i / (nc / 4) : (i & 7) * 4, k = MX ? i % (nc / 4) * 4 : i >> 3;
                    const int t = t0 + 2 * a2 + (r >> 4), row = q * 16 + (r & 15);
                    if (t >= t1 || row >= nM || n0 + k >= nN) continue;
                    const int ci = MX ? cx0 + row : cx0 + n0 + k, co = MX ? cg0 + n0 + k : cg0 + row;
                    const float* v = stage + r * kEpPitch + k;
                    constexpr int step = MX ? 1 : kEpPitch;
                    float4 f = make_float4(v[0], v[step], v[2 * step], v[3 * step]);
                    if (bad) f.x = f.y = f.z = f.w = __int_as_float(0x7fffffff);
                    float* d = dst + ((int64_t)t * c.Cin + ci) * c.Cout + co;
                    const bool add = run > 0 && !bad;              // to this thread's own values: nothing is read back
                    if (at16(part)) {
                        if (add) atomicAdd(reinterpret_cast<float4*>(d), f);
                        else *reinterpret_cast<float4*>(d) = f;
                    } else {
                        const float g[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (add) atomicAdd(d + e, g[e]);
                            else d[e] = g[e];
                    }
                }
                __syncwarp();
            }
        }
        if (bad) {
            if (tid == 0) mbar_wait_bounded(&done, run & 1, kMbarDrainLimit);     // MMAs in flight end
            break;
        }
        tc_fence_before();
        __syncthreads();                      // accumulators and ring are free for the next run
        tc_fence_after();
    }
    if (TAIL) __syncthreads();
    if (TAIL && nonfinite) wgrad_add_nonfinite(x, gy, dst, c, s, t0, t1, cx0, cg0);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, s.cols);
}

// dw[co][t][ci] = sum over splits (in order) of part[split][t][ci][co]; consecutive threads read
// consecutive co.
__global__ void __launch_bounds__(128) k_wgrad_reduce(const float* __restrict__ part, float* __restrict__ dw, int nsplit,
                                                      int Cin, int Cout) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = 27 * Cin * Cout;
    if (i >= total) return;
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < nsplit; ++k) s += part[(int64_t)k * total + i];
    const int co = i % Cout, r = i / Cout;
    dw[((int64_t)co * 27 + r / Cin) * Cin + r % Cin] = s;
}

thread_local int wait_polls = kMbarPollLimit;         // of the convolutions that this thread launches

tr_status check_dims(const ConvDims& c) {
    if (c.N < 1 || c.D < 1 || c.H < 1 || c.W < 1) return tr::fail(TR_ERR_INVALID_ARG, "conv3d: empty volume");
    if (c.Cin < 2 || (c.Cin & 1)) return tr::fail(TR_ERR_INVALID_ARG, "conv3d: Cin must be even and >= 2");
    if (c.Cout < 8 || (c.Cout % 8) || c.Cout > 128)
        return tr::fail(TR_ERR_INVALID_ARG, "conv3d: Cout must be a multiple of 8 in [8, 128]");
    return TR_OK;
}

// SMs of the current device (148 on a B200), for the launch shapes.
int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 148;
    return std::max(n, 1);
}

uint32_t tmem_cols(int need) {
    uint32_t n = 32;
    while ((int)n < need) n <<= 1;
    return n;
}

template <int NZ, class TIn, bool VEC, class Off = int>
tr_status launch_fwd(const TIn* x, const __nv_bfloat16* w, const float* bias, float* y, const ConvDims& c, int64_t tiles,
                     cudaStream_t st) {
    auto fn = k_conv3d_fwd<NZ, TIn, VEC, Off>;
    const int npad = conv_npad(c.Cout);
    const size_t smem = fwd_smem_bytes(NZ, npad);
    const int nacc = 2 * NZ * npad <= 512 ? 2 : 1;
    TR_TRY(tr::raise_smem_limit((const void*)fn, smem));
    fn<<<(unsigned)std::min<int64_t>(tiles, sm_count()), kFwdThreads, smem, st>>>(
        x, w, bias, y, c, tiles, npad, nacc, tmem_cols(nacc * NZ * npad), at16(y), wait_polls);
    TR_CHECK_LAUNCH();
    return TR_OK;
}

// z slices per tile, four, two or one: the smallest time of the fullest SM, a tile of k slices
// taking about 2 k + 1 units (its MMAs, and the halo and weights that slices share: 2.1 voxels are
// loaded per output voxel at four slices, 4.2 at one).
template <class TIn>
tr_status conv_fwd(const TIn* x, const __nv_bfloat16* packed, const float* bias, float* y, const ConvDims& c,
                   cudaStream_t st) {
    const int64_t cols = (int64_t)c.N * ((c.W + kTX - 1) / kTX) * ((c.H + kTY - 1) / kTY);
    const int sms = sm_count();
    int nz = 4;
    int64_t tiles = 0, best = INT64_MAX;
    for (int k : {4, 2, 1}) {
        const int64_t n = cols * ((c.D + k - 1) / k), cost = (n + sms - 1) / sms * (2 * k + 1);
        if (cost < best) {
            best = cost;
            nz = k;
            tiles = n;
        }
    }
    const bool vec = c.Cin % 8 == 0 && at16(x);
    if ((int64_t)c.H * c.W > INT32_MAX / 8)              // slices of more than 268 million voxels
        return launch_fwd<1, TIn, false, int64_t>(x, packed, bias, y, c, cols * c.D, st);
#define TR_FWD_NZ(NZV) \
    return vec ? launch_fwd<NZV, TIn, true>(x, packed, bias, y, c, tiles, st) \
               : launch_fwd<NZV, TIn, false>(x, packed, bias, y, c, tiles, st)
    if (nz == 4) TR_FWD_NZ(4);
    if (nz == 2) TR_FWD_NZ(2);
    TR_FWD_NZ(1);
#undef TR_FWD_NZ
}

tr_status pack_weights(const void* w, bool f32, bool flip, __nv_bfloat16* packed, int nin, int nout, cudaStream_t st) {
    const int npad = conv_npad(nout), total = (int)packed_elems(nin, nout);
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (f32) {
        const auto* p = (const float*)w;
        if (flip) k_conv3d_pack<float, true><<<blocks, 256, 0, st>>>(p, packed, nout, nin, npad, total);
        else k_conv3d_pack<float, false><<<blocks, 256, 0, st>>>(p, packed, nout, nin, npad, total);
    } else {
        const auto* p = (const __nv_bfloat16*)w;
        if (flip) k_conv3d_pack<__nv_bfloat16, true><<<blocks, 256, 0, st>>>(p, packed, nout, nin, npad, total);
        else k_conv3d_pack<__nv_bfloat16, false><<<blocks, 256, 0, st>>>(p, packed, nout, nin, npad, total);
    }
    TR_CHECK_LAUNCH();
    return TR_OK;
}

// Launch shape of the weight gradient; at most max_splits partials.
WgradShape wgrad_shape(const ConvDims& c, int64_t max_splits) {
    WgradShape s;
    s.mx = c.Cin >= c.Cout;
    const int cn = s.mx ? c.Cout : c.Cin;
    s.npad = (std::min(cn, kWgChunk) + 15) / 16 * 16;
    // the M side always reads 64 channels (8 planes; rows past the channel count are not written out)
    s.px = s.mx ? 8 : s.npad / 8;
    s.pg = s.mx ? s.npad / 8 : 8;
    s.groups = wgrad_groups(s.npad);
    s.cx = (c.Cin + kWgChunk - 1) / kWgChunk;
    s.cg = (c.Cout + kWgChunk - 1) / kWgChunk;
    s.cols = tmem_cols(14 / s.groups * s.npad);       // two M = 64 accumulators per column range
    s.cols_n = (int64_t)c.N * ((c.W + kTX - 1) / kTX) * ((c.H + kTY - 1) / kTY);
    // one CTA per SM over all groups and chunks; z segments and splits by the slices that the busiest
    // CTA loads (two halo slices a segment; adding a run's accumulators to the partial takes about four)
    const int64_t want = std::max<int64_t>(1, std::min<int64_t>(max_splits, sm_count() / (s.groups * s.cx * s.cg)));
    int64_t best = INT64_MAX;
    const int fewest = (c.D + kWgRunSlices - 1) / kWgRunSlices;
    for (int segs = fewest; segs <= std::max(fewest, std::min(c.D, 64)); ++segs) {
        const int len = (c.D + segs - 1) / segs, run = kWgRunSlices / len;
        const int64_t units = s.cols_n * ((c.D + len - 1) / len), rounds = (units + want - 1) / want;
        const int64_t cost = rounds * (len + 2) + (rounds + run - 1) / run * 4;
        if (cost < best) {
            best = cost;
            s.seg_len = len;
            s.run = run;
            s.units = units;
            s.splits = (int)((units + rounds - 1) / rounds);
        }
    }
    return s;
}

using WgradKernel = void (*)(const __nv_bfloat16*, const __nv_bfloat16*, float*, ConvDims, WgradShape, int);
template <int NPAD, bool TAIL>
WgradKernel wgrad_kernel(bool vec, bool mx) {
    return vec ? (mx ? k_conv3d_wgrad<NPAD, true, true, TAIL> : k_conv3d_wgrad<NPAD, true, false, TAIL>)
               : (mx ? k_conv3d_wgrad<NPAD, false, true, TAIL> : k_conv3d_wgrad<NPAD, false, false, TAIL>);
}
template <bool TAIL>
WgradKernel wgrad_kernel(int npad, bool vec, bool mx) {
    if (npad == 16) return wgrad_kernel<16, TAIL>(vec, mx);
    if (npad == 32) return wgrad_kernel<32, TAIL>(vec, mx);
    if (npad == 48) return wgrad_kernel<48, TAIL>(vec, mx);
    return wgrad_kernel<64, TAIL>(vec, mx);
}

int64_t partial_floats(const ConvDims& c) { return 27LL * c.Cin * c.Cout; }

}  // namespace

// Unpacked weights: packed into stream-ordered scratch (at most 0.9 MB) for the call.
extern "C" tr_status tr_conv3d_fwd(const void* x, const void* w, const float* bias, float* y, int32_t N, int32_t D,
                                   int32_t H, int32_t W, int32_t Cin, int32_t Cout, void* stream) {
    if (!x || !w || !y) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_fwd: null pointer");
    const ConvDims c{N, D, H, W, Cin, Cout, (int64_t)N * D * H * W};
    TR_TRY(check_dims(c));
    cudaStream_t st = (cudaStream_t)stream;
    void* packed = nullptr;
    TR_CUDA(cudaMallocAsync(&packed, (size_t)packed_elems(Cin, Cout) * 2, st));
    tr_status rc = pack_weights(w, false, false, (__nv_bfloat16*)packed, Cin, Cout, st);
    if (rc == TR_OK) rc = conv_fwd((const __nv_bfloat16*)x, (const __nv_bfloat16*)packed, bias, y, c, st);
    TR_CUDA(cudaFreeAsync(packed, st));
    return rc;
}

extern "C" tr_status tr_conv3d_set_wait_limit(int32_t polls) {
    if (polls < 0) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_set_wait_limit: polls must be >= 0");
    wait_polls = polls;
    return TR_OK;
}

extern "C" tr_status tr_conv3d_packed_size(int32_t Cin, int32_t Cout, size_t* bytes) {
    if (!bytes) return tr::fail(TR_ERR_INVALID_ARG, "null bytes");
    TR_TRY(check_dims(ConvDims{1, 1, 1, 1, Cin, Cout, 1}));
    *bytes = (size_t)packed_elems(Cin, Cout) * 2;
    return TR_OK;
}

extern "C" tr_status tr_conv3d_pack(const void* w, int32_t w_f32, int32_t data_grad, void* packed, int32_t Cin,
                                    int32_t Cout, void* stream) {
    if (!w || !packed) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_pack: null pointer");
    TR_TRY(check_dims(ConvDims{1, 1, 1, 1, Cin, Cout, 1}));
    return pack_weights(w, w_f32 != 0, data_grad != 0, (__nv_bfloat16*)packed, Cin, Cout, (cudaStream_t)stream);
}

extern "C" tr_status tr_conv3d_fwd_packed(const void* x, int32_t x_f32, const void* packed, const float* bias, float* y,
                                          int32_t N, int32_t D, int32_t H, int32_t W, int32_t Cin, int32_t Cout,
                                          void* stream) {
    if (!x || !packed || !y) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_fwd_packed: null pointer");
    if ((uintptr_t)packed % 16) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_fwd_packed: packed weights must be 16-byte aligned");
    const ConvDims c{N, D, H, W, Cin, Cout, (int64_t)N * D * H * W};
    TR_TRY(check_dims(c));
    const auto* wp = (const __nv_bfloat16*)packed;
    return x_f32 ? conv_fwd((const float*)x, wp, bias, y, c, (cudaStream_t)stream)
                 : conv_fwd((const __nv_bfloat16*)x, wp, bias, y, c, (cudaStream_t)stream);
}

extern "C" tr_status tr_conv3d_fwd_weights(const void* x, int32_t x_f32, const void* w, int32_t w_f32, int32_t data_grad,
                                           void* packed, const float* bias, float* y, int32_t N, int32_t D, int32_t H,
                                           int32_t W, int32_t Cin, int32_t Cout, void* stream) {
    TR_TRY(tr_conv3d_pack(w, w_f32, data_grad, packed, Cin, Cout, stream));
    return tr_conv3d_fwd_packed(x, x_f32, packed, bias, y, N, D, H, W, Cin, Cout, stream);
}

// Scratch: one partial per kWgradVox voxels, or per split where the launch wants more of them.
extern "C" tr_status tr_conv3d_wgrad_workspace(int32_t N, int32_t D, int32_t H, int32_t W, int32_t Cin,
                                               int32_t Cout, size_t* bytes) {
    if (!bytes) return tr::fail(TR_ERR_INVALID_ARG, "null bytes");
    const ConvDims c{N, D, H, W, Cin, Cout, (int64_t)N * D * H * W};
    int64_t parts = (c.V + kWgradVox - 1) / kWgradVox;
    if (check_dims(c) == TR_OK) parts = std::max<int64_t>(parts, wgrad_shape(c, INT32_MAX).splits);
    *bytes = (size_t)(parts * partial_floats(c) * (int64_t)sizeof(float));
    return TR_OK;
}

extern "C" tr_status tr_conv3d_wgrad(const void* x, const void* gy, float* dw, int32_t N, int32_t D, int32_t H,
                                     int32_t W, int32_t Cin, int32_t Cout, void* workspace, size_t workspace_bytes,
                                     void* stream) {
    if (!x || !gy || !dw || !workspace) return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_wgrad: null pointer");
    const ConvDims c{N, D, H, W, Cin, Cout, (int64_t)N * D * H * W};
    TR_TRY(check_dims(c));
    const int64_t per = partial_floats(c) * (int64_t)sizeof(float);
    if ((int64_t)workspace_bytes < (c.V + kWgradVox - 1) / kWgradVox * per)
        return tr::fail(TR_ERR_INVALID_ARG, "tr_conv3d_wgrad: workspace too small");
    const WgradShape s = wgrad_shape(c, (int64_t)workspace_bytes / per);
    cudaStream_t st = (cudaStream_t)stream;
    const auto* xb = (const __nv_bfloat16*)x;
    const auto* gb = (const __nv_bfloat16*)gy;
    float* part = (float*)workspace;
    const size_t smem = (size_t)kWgRing * 16 * (s.px * kXPitch + s.pg * kGPitch) + 128;
    const bool vec = c.Cin % 8 == 0 && at16(x);
    const bool tail = c.W % kTX || c.H % kTY;
    auto fn = tail ? wgrad_kernel<true>(s.npad, vec, s.mx) : wgrad_kernel<false>(s.npad, vec, s.mx);
    TR_TRY(tr::raise_smem_limit((const void*)fn, smem));
    const dim3 grid((unsigned)s.splits, (unsigned)s.groups, (unsigned)(s.cx * s.cg));
    fn<<<grid, kWgThreads, smem, st>>>(xb, gb, part, c, s, wait_polls);
    TR_CHECK_LAUNCH();
    const int64_t total = partial_floats(c);
    k_wgrad_reduce<<<(unsigned)((total + 127) / 128), 128, 0, st>>>(part, dw, s.splits, Cin, Cout);
    TR_CHECK_LAUNCH();
    return TR_OK;
}
