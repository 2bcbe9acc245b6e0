// FFT passes for every supported oversampled length up to 320: arguments, launch table.
//
// The passes of a NUFFT view their data as [outer][rows][inner] and transform along rows.  The
// kernels of tr_lines_part.cuh take 16 columns per CTA in two (five lengths: three) register
// passes: a thread reads one butterfly's inputs straight from global memory, the tile crosses
// shared memory once, and the last butterfly's outputs go straight back, so every geometry (odd
// lengths, any pad, crop, coil and column count) runs the same code.  Each length is compiled with
// its radices as constants.
#pragma once

#include "tr_internal.cuh"

namespace tr {

constexpr int kMinLineLen = 13;      // oversampled length of the smallest image axis (10)
constexpr int kMaxLineLen = 320;     // longer ones run the runtime-radix kernels
constexpr int kLineW = 16;           // columns per CTA
// z lengths whose empty-column skip also takes column counts that are multiples of 8 only (bin_colmask)
__host__ __device__ constexpr bool lp_mixed_columns(int L) { return L == 240 || L == 320; }

// Arguments of the forward x pass: image * coil map * separable apodisation * scale, centred
// zero-pad, x FFT, centred shift, into the (Z, Y, OSX, ncol) buffer.
struct FwdXArgs {
    const float2* img;      // (n_img, Z, Y, X)
    int64_t img_stride;
    const float2* maps;     // (Z, Y, X, C) or null
    int C;                  // coils per image (1 when maps == null)
    int n_img;
    int Z, Y, X, OSX, h, pad;
    int rows, cc;           // rows per CTA, coils per CTA
    const float* apz;
    const float* apy;
    const float* apx;
    float scale;
    const float2* tw;
    FftStages S;
    float2* out;            // (Z, Y, OSX, ncol)
    int ncol;
    int* err;               // device error word (kDevErr* bits)
    int poll;               // polls before a bounded mbarrier wait gives up
};

// Arguments of a line pass.  Data viewed as [outer][rows][inner]; transforms along rows for W
// consecutive inner elements per CTA.  Input rows present: Lin (pad offset p_in inside the
// length-L line); output rows kept: Lout (crop offset p_out).
struct LineArgs {
    const float2* in;
    float2* out;
    int64_t inner;
    int Lin, Lout, p_in, p_out, h;
    int W;
    int vec16;              // rows are 16-byte aligned: copy two elements per cp.async
    bool inv;
    const float2* tw;
    FftStages S;
    int* err;               // device error word (kDevErr* bits)
    int poll;               // polls before a bounded mbarrier wait gives up
    int kA, kB;             // TMA variant: first transform row of each output box
    // z passes: (y, x) tile columns that no sample's kernel reaches; null: none skipped
    const uint8_t* colmask; // [nt1 * nt2] 1: occupied
    int skip_zero;          // 0: a CTA whose lines are all unoccupied returns (forward: the output is never
                            // read); 1: it writes zeros to its output rows (adjoint: the lines are zero)
    int mcol, mosx, mnt2;   // k-space columns, OSX and tile columns along x of the mask
};

// Empty-column skip of the z passes.  Inner index q of a z pass is
// ((y OSX + x) ncol + column); a line is unoccupied when the tile column
// (y / 4, x / 4) holds no busy tile: gridding wrote no tile there (the line is
// all zeros) and interpolation reads no tap there.  True when every line
// q0 .. q0 + W - 1 (< inner) of the CTA is unoccupied (the same for all threads).
// A CTA that mixes lines of occupied and unoccupied columns (W does not divide
// the column count) must not read the latter's unwritten tiles: k_lp_line
// takes them as zeros, for the other kernels the host passes no mask then.
__device__ __forceinline__ bool lines_unoccupied(const LineArgs& a, int64_t q0, int W) {
    if (!a.colmask) return false;
    const int64_t q1 = min(q0 + W, a.inner) - 1;
    for (int64_t yx = q0 / a.mcol; yx <= q1 / a.mcol; ++yx) {
        const int y = (int)(yx / a.mosx), x = (int)(yx - (int64_t)y * a.mosx);
        if (a.colmask[(y >> 2) * a.mnt2 + (x >> 2)]) return false;
    }
    return true;
}
// The zeros of an unoccupied CTA's output rows (adjoint z pass): [Lout][W] at q0.
__device__ __forceinline__ void lines_write_zeros(const LineArgs& a, int64_t q0, int W, int64_t outer) {
    float2* out = a.out + outer * a.Lout * a.inner;
    for (int i = threadIdx.x; i < a.Lout * W; i += blockDim.x) {
        const int o = i / W, w = i - o * W;
        if (q0 + w < a.inner) out[(int64_t)o * a.inner + q0 + w] = make_float2(0.f, 0.f);
    }
}

// Arguments of the adjoint x pass: x IFFT, centred shift and crop, apodisation, scale,
// conj(coil map) and the coil sum, into the image rows.
struct AdjXArgs {
    const float2* in;       // (Z, Y, OSX, ncol)
    int ncol;
    const float2* maps;     // (Z, Y, X, C) or null
    int C, cc, rows;
    int cta_rows, tiles;    // k_lp_adj_x_one: image rows and 16-column tiles per CTA
    int n_img;
    int Z, Y, X, OSX, h, pad;
    const float* apz;
    const float* apy;
    const float* apx;
    float scale;
    const float2* tw;
    FftStages S;
    float2* img;            // (n_img, Z, Y, X)
    int64_t img_stride;
    int* err;               // device error word (kDevErr* bits)
    int poll;               // polls before a bounded mbarrier wait gives up
};

// Kernels of one length (null where the length is not compiled).
struct LineKernels {
    const void* fwd = nullptr;       // line pass, (LineArgs)
    const void* inv = nullptr;
    const void* fwd_x = nullptr;     // (FwdXArgs)
    const void* fwd_x_images = nullptr;   // several images of one coil with maps; null where fwd_x is used
    const void* adj_x = nullptr;     // (AdjXArgs)
    const void* adj_x_one = nullptr; // the same for one image; null where adj_x is the faster one
    int threads = 0;
    int smem = 0;                    // dynamic shared memory, bytes
};
const LineKernels& line_kernels(int L);
// Forward x pass: image rows in shared memory (odd pitch: rows in different banks), the most distinct rows
// that 16 consecutive (row, coil) pairs meet, and their bytes (two buffers where there are several images).
__host__ __device__ constexpr int lp_row_pitch(int X) { return X | 1; }
__host__ __device__ constexpr int lp_rows_per_cta(int C) { return (kLineW - 1 + C - 1) / C + 1; }
constexpr size_t lp_row_bytes(int X, int C, int n_img) {
    return (size_t)(n_img > 1 ? 2 : 1) * lp_rows_per_cta(C) * lp_row_pitch(X) * sizeof(float2);
}

}  // namespace tr
