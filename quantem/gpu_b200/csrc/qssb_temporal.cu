// qssb_temporal.cu - joining a time series of SSB object waves (sm_100a).
//
// Restates the drift-corrected complex mean of the reference's temporal
// helpers (ssb/temporal.py:77-257 of bobleesj/quantem.gpu):
//   fourier_shift: O'_t = ifft2(fft2(O_t) exp(-2 pi i (f_r s_r + f_c s_c))),
//     f = fftfreq(n, 1) (temporal.py:77-107), as two passes over the stack:
//     the rows' transform, ramp in f_c and inverse transform, then the
//     columns' with the ramp in f_r;
//   join: with phase reference "first", frames t > 0 are multiplied by
//     exp(-i angle(sum_p O'_t conj O'_0)) (temporal.py:154-160; the overlap
//     summed in FP64 in a fixed order), then joined = sum_t w_t O'_t
//     (temporal.py:234).
// Line transforms: the warp FFT at 256..1024 points, groups of 8 lanes at
// 128, the shared-memory Stockham transform at 64.
#include <math.h>

#include "qssb_internal.h"

namespace qssb {

constexpr int kTmpWarps = 8;

template <int N>
__host__ __device__ constexpr int tmp_line() {
    // room for the line and, at N >= 256, the warp FFT's transpose scratch
    return N >= 256 ? (warp_fft_scratch<N>() > N ? warp_fft_scratch<N>() : N) : N;
}

// In-place transform of one line held in shared memory (natural order).
template <int N, int DIR>
__device__ __forceinline__ void line_transform(float2* line, const float2* tw, int lane) {
    if constexpr (N >= 256) {
        constexpr int RPL = N / 32;
        float2 v[RPL];
#pragma unroll
        for (int t = 0; t < RPL; ++t) v[t] = line[lane + 32 * t];
        __syncwarp();
        warp_fft<N, DIR>(v, line, tw, lane);
#pragma unroll
        for (int j = 0; j < RPL; ++j) line[warp_fft_index<N>(lane, j)] = v[j];
        __syncwarp();
    } else {
        line_fft<N, DIR>(line, 1, tw, lane);
    }
}

// exp(-2 pi i f_k shift) / N, f = fftfreq(N, 1), for a line's N frequencies:
// the phase is formed in FP64 and reduced before the float32 sincos (the
// scale is a power of two). Computed once per CTA, whose lines share it.
template <int N>
__device__ __forceinline__ void fill_ramp(float2* ramp, float shift, int tid, int threads) {
    for (int k = tid; k < N; k += threads) {
        double ph = -((double)(k < N / 2 ? k : k - N) * (1.0 / N)) * (double)shift;  // in turns
        ph -= rint(ph);
        float s, co;
        sincospif((float)(2.0 * ph), &s, &co);
        ramp[k] = make_float2(co * (1.0f / N), s * (1.0f / N));
    }
}

// A line of 128 held by a group of 8 lanes as v[n1] = x[s + 8 n1], shifted:
// transform, ramp, inverse transform. Both transforms leave X[s + 8 h + 16 k]
// in v[8 h + k], which is the lane's own value n1 = h + 2 k, so the order
// between and after them is a renaming of registers.
__device__ __forceinline__ void shift_line128(float2 (&v)[16], float2* T, int s, const float2* tw,
                                              const float2* ramp) {
    fft128_g8<-1>(v, T, s, tw);
    float2 u[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const int n1 = (t >> 3) + 2 * (t & 7);
        u[n1] = cmul(v[t], ramp[s + 8 * n1]);
    }
    fft128_g8<+1>(u, T, s, tw);
#pragma unroll
    for (int t = 0; t < 16; ++t) v[(t >> 3) + 2 * (t & 7)] = u[t];
}

// The shift ramp is separable, so each direction is shifted in one pass
// (transform, ramp, inverse transform of a line on chip) and the stack goes
// through memory twice. Row transforms, columns with the 2D ramp and inverse
// row transforms took 23 + 49 + 23 us at 256 frames of 128^2 (all kernels of
// the join 185 us); the join of them with both passes and its reductions here
// takes 92 us in all, against 227.
// Rows: 128 points as four lines per warp in registers; other sizes a warp
// per line in shared memory.
template <int C>
__host__ __device__ constexpr int shift_lines() { return C == 128 ? 4 * kTmpWarps : kTmpWarps; }

template <int C>
__host__ __device__ constexpr size_t shift_smem() {
    return sizeof(float2) * (2 * C + (C == 128 ? (size_t)4 * kTmpWarps * kG8Scratch
                                               : (size_t)kTmpWarps * (tmp_line<C>() | 1)));
}

template <int C>
__global__ void __launch_bounds__(32 * kTmpWarps) k_shift_rows(const float2* __restrict__ in,
                                                               float2* __restrict__ out, int rows,
                                                               const float* __restrict__ shifts) {
    extern __shared__ float2 tmp_smem[];
    float2* tw = tmp_smem;
    float2* ramp = tw + C;
    float2* scratch = ramp + C;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    fill_twiddles<C>(tw, tid, 32 * kTmpWarps);
    fill_ramp<C>(ramp, __ldg(shifts + 2 * blockIdx.y + 1), tid, 32 * kTmpWarps);
    __syncthreads();
    if constexpr (C == 128) {
        const int group = tid >> 3;
        const int s = lane & 7;
        const int r = blockIdx.x * shift_lines<C>() + group;
        const bool on = r < rows;  // whole warps call the transform
        const size_t base = ((size_t)blockIdx.y * rows + (on ? r : 0)) * C;
        float2 v[16];
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1) v[n1] = in[base + s + 8 * n1];
        shift_line128(v, scratch + group * kG8Scratch, s, tw, ramp);
        if (!on) return;
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1) out[base + s + 8 * n1] = v[n1];
    } else {
        const int r = blockIdx.x * shift_lines<C>() + warp;
        if (r >= rows) return;
        const size_t base = ((size_t)blockIdx.y * rows + r) * C;
        float2* line = scratch + warp * (tmp_line<C>() | 1);
        for (int i = lane; i < C; i += 32) line[i] = in[base + i];
        __syncwarp();
        line_transform<C, -1>(line, tw, lane);
        for (int i = lane; i < C; i += 32) line[i] = cmul(line[i], ramp[i]);
        __syncwarp();
        line_transform<C, +1>(line, tw, lane);
        for (int i = lane; i < C; i += 32) out[base + i] = line[i];
    }
}

// Columns, in place. 128 points: four neighbouring columns per warp (whole
// 32-byte sectors) straight into registers; other sizes a strip of
// kTmpWarps columns staged in shared memory, a warp per column.
template <int R>
__global__ void __launch_bounds__(32 * kTmpWarps) k_shift_cols(float2* __restrict__ data, int cols,
                                                               const float* __restrict__ shifts) {
    constexpr int P = tmp_line<R>() | 1;
    extern __shared__ float2 tmp_smem[];
    float2* tw = tmp_smem;
    float2* ramp = tw + R;
    float2* scratch = ramp + R;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int c0 = blockIdx.x * shift_lines<R>();
    float2* d = data + (size_t)blockIdx.y * R * cols;
    fill_twiddles<R>(tw, tid, 32 * kTmpWarps);
    fill_ramp<R>(ramp, __ldg(shifts + 2 * blockIdx.y), tid, 32 * kTmpWarps);
    if constexpr (R == 128) {
        __syncthreads();
        const int s = lane >> 2;  // lanes 4 s + j: column j of the warp's four
        const int group = warp * 4 + (lane & 3);
        const int c = c0 + group;
        const bool on = c < cols;
        float2* col = d + (on ? c : 0);
        float2 v[16];
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1) v[n1] = col[(size_t)(s + 8 * n1) * cols];
        // groups 4 float2 apart mod 16: the half-warp's 4 groups x 4 lanes meet no bank twice
        shift_line128(v, scratch + group * (16 * kG8Pitch + 4), s, tw, ramp);
        if (!on) return;
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1) col[(size_t)(s + 8 * n1) * cols] = v[n1];
    } else {
        const int nc = min(kTmpWarps, cols - c0);
        for (int e = tid; e < R * kTmpWarps; e += 32 * kTmpWarps) {
            const int r = e / kTmpWarps;
            const int c = e - r * kTmpWarps;
            if (c < nc) scratch[c * P + r] = d[(size_t)r * cols + c0 + c];
        }
        __syncthreads();
        if (warp < nc) {
            float2* line = scratch + warp * P;
            line_transform<R, -1>(line, tw, lane);
            for (int r = lane; r < R; r += 32) line[r] = cmul(line[r], ramp[r]);
            __syncwarp();
            line_transform<R, +1>(line, tw, lane);
        }
        __syncthreads();
        for (int e = tid; e < R * kTmpWarps; e += 32 * kTmpWarps) {
            const int r = e / kTmpWarps;
            const int c = e - r * kTmpWarps;
            if (c < nc) d[(size_t)r * cols + c0 + c] = scratch[c * P + r];
        }
    }
}

constexpr int kJoinBlocks = 64;   // overlap partial sums per frame, at most
constexpr int kJoinThreads = 256;

// Blocks per frame of the overlap: 8 pixels per thread and more, so that the
// block's reduction is small beside its reads (one pixel per thread took 30 us
// at 256 frames of 128^2).
static int overlap_blocks(long long n_pix) {
    const long long b = (n_pix + 8 * kJoinThreads - 1) / (8 * kJoinThreads);
    return b < kJoinBlocks ? (int)b : kJoinBlocks;
}

__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    }
    return v;
}

// partial[t][blk] = sum over this block's pixels of a_t conj(a_0), FP64. FULL:
// kJoinBlocks blocks a frame, a stride that the compiler knows, two pixels'
// loads at once (64 frames of 1024^2: 97 us; 137 with four, 118 with a stride of
// gridDim.x).
template <bool FULL>
__global__ void __launch_bounds__(kJoinThreads) k_overlap_partial(const float2* __restrict__ a,
                                                                  long long n_pix,
                                                                  double2* __restrict__ partial) {
    __shared__ double2 red[kJoinThreads / 32];
    const int t = blockIdx.y;
    const float2* at = a + (size_t)t * n_pix;
    double sr = 0.0, si = 0.0;
    const long long stride = (long long)(FULL ? kJoinBlocks : gridDim.x) * kJoinThreads;
#pragma unroll(FULL ? 2 : 1)
    for (long long p = (long long)blockIdx.x * kJoinThreads + threadIdx.x; p < n_pix; p += stride) {
        const float2 v = at[p];
        const float2 r = a[p];
        sr += (double)v.x * r.x + (double)v.y * r.y;
        si += (double)v.y * r.x - (double)v.x * r.y;
    }
    double2 sum = warp_sum(make_double2(sr, si));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kJoinThreads / 32; ++w) {
            sum.x += red[w].x;
            sum.y += red[w].y;
        }
        partial[(size_t)t * gridDim.x + blockIdx.x] = sum;
    }
}

// rot[t] = exp(-i angle(overlap_t)) for t > 0, 1 for frame 0; a warp per frame.
__global__ void __launch_bounds__(128) k_overlap_rotation(const double2* __restrict__ partial,
                                                          int n_blocks, int n_frames,
                                                          float2* __restrict__ rot) {
    const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= n_frames) return;
    if (t == 0) {
        if (lane == 0) rot[0] = make_float2(1.0f, 0.0f);
        return;
    }
    double2 sum = make_double2(0.0, 0.0);
    for (int b = lane; b < n_blocks; b += 32) {
        const double2 v = partial[(size_t)t * n_blocks + b];
        sum.x += v.x;
        sum.y += v.y;
    }
    sum = warp_sum(sum);
    if (lane != 0) return;
    const double ang = atan2(sum.y, sum.x);
    rot[t] = make_float2((float)cos(ang), (float)-sin(ang));
}

// joined[p] = sum_t w_t rot_t a_t[p] in FP32; the rotated frames are written
// back when requested. A block takes 32 pixels and its 8 warps every 8th
// frame, the 8 sums added in order: a thread per pixel over all frames leaves
// 64 blocks at 128^2.
constexpr int kJoinSlices = kJoinThreads / 32;
__global__ void __launch_bounds__(kJoinThreads) k_join(float2* __restrict__ a,
                                                       const float* __restrict__ w,
                                                       const float2* __restrict__ rot,
                                                       int n_frames, long long n_pix,
                                                       float2* __restrict__ joined,
                                                       int write_back) {
    __shared__ float2 red[kJoinSlices][32];
    const int lane = threadIdx.x & 31;
    const int slice = threadIdx.x >> 5;
    const long long p = (long long)blockIdx.x * 32 + lane;
    float sr = 0.0f, si = 0.0f;
    if (p < n_pix) {
#pragma unroll 4
        for (int t = slice; t < n_frames; t += kJoinSlices) {
            float2 v = a[(size_t)t * n_pix + p];
            if (rot) v = cmul(v, __ldg(rot + t));
            if (write_back) a[(size_t)t * n_pix + p] = v;
            const float wt = __ldg(w + t);
            sr = fmaf(wt, v.x, sr);
            si = fmaf(wt, v.y, si);
        }
    }
    red[slice][lane] = make_float2(sr, si);
    __syncthreads();
    if (slice != 0 || p >= n_pix) return;
#pragma unroll
    for (int k = 1; k < kJoinSlices; ++k) {
        sr += red[k][lane].x;
        si += red[k][lane].y;
    }
    joined[p] = make_float2(sr, si);
}

// The same by a thread per pixel, all frames in order.
__global__ void __launch_bounds__(kJoinThreads) k_join_pixels(float2* __restrict__ a,
                                                              const float* __restrict__ w,
                                                              const float2* __restrict__ rot,
                                                              int n_frames, long long n_pix,
                                                              float2* __restrict__ joined,
                                                              int write_back) {
    const long long p = (long long)blockIdx.x * kJoinThreads + threadIdx.x;
    if (p >= n_pix) return;
    float sr = 0.0f, si = 0.0f;
#pragma unroll 4
    for (int t = 0; t < n_frames; ++t) {
        float2 v = a[(size_t)t * n_pix + p];
        if (rot) v = cmul(v, __ldg(rot + t));
        if (write_back) a[(size_t)t * n_pix + p] = v;
        const float wt = __ldg(w + t);
        sr = fmaf(wt, v.x, sr);
        si = fmaf(wt, v.y, si);
    }
    joined[p] = make_float2(sr, si);
}

// Pixels from which a thread each fills the chip. k_join against k_join_pixels,
// us: 256 frames of 128^2 9 / 47, 64 of 256^2 9.0 / 14.4, 256 of 256 x 512 70 /
// 121; 16 of 512^2 10.3 / 8.9 and 64 of them 37 / 36, 1 of 1024^2 20 / 9, 16 of
// them 51 / 37.
constexpr long long kJoinPixels = 1 << 18;

template <int C>
static int launch_rows(const float2* in, float2* out, int n_frames, int rows, const float* shifts,
                       cudaStream_t s) {
    constexpr int lines = shift_lines<C>();
    CUDA_TRY(cudaFuncSetAttribute(k_shift_rows<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)shift_smem<C>()));
    { k_shift_rows<C><<<dim3((rows + lines - 1) / lines, n_frames), 32 * kTmpWarps, shift_smem<C>(), s>>>(
        in, out, rows, shifts); note_launch(); }
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}

template <int R>
static int launch_cols(float2* data, int n_frames, int cols, const float* shifts, cudaStream_t s) {
    constexpr int lines = shift_lines<R>();
    CUDA_TRY(cudaFuncSetAttribute(k_shift_cols<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)shift_smem<R>()));
    { k_shift_cols<R><<<dim3((cols + lines - 1) / lines, n_frames), 32 * kTmpWarps, shift_smem<R>(), s>>>(
        data, cols, shifts); note_launch(); }
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}

static bool tmp_size_ok(int n) {
    return n == 64 || n == 128 || n == 256 || n == 512 || n == 1024;
}

}  // namespace qssb

using namespace qssb;

extern "C" int qssb_fourier_shift(const float* in, float* out, int32_t n_frames, int32_t rows,
                                  int32_t cols, const float* shifts, void* stream) {
    if (!in || !out || !shifts || n_frames <= 0 || n_frames > 65535)
        return set_error(QSSB_ERR_INVALID, "qssb_fourier_shift: null pointer or n_frames outside [1, 65535]");
    if (!tmp_size_ok(rows) || !tmp_size_ok(cols))
        return set_error(QSSB_ERR_UNSUPPORTED, "qssb_fourier_shift: sizes must be 64..1024, powers of two");
    cudaStream_t s = (cudaStream_t)stream;
    auto* i = reinterpret_cast<const float2*>(in);
    auto* o = reinterpret_cast<float2*>(out);
    int rc;
    switch (cols) {
        case 64: rc = launch_rows<64>(i, o, n_frames, rows, shifts, s); break;
        case 128: rc = launch_rows<128>(i, o, n_frames, rows, shifts, s); break;
        case 256: rc = launch_rows<256>(i, o, n_frames, rows, shifts, s); break;
        case 512: rc = launch_rows<512>(i, o, n_frames, rows, shifts, s); break;
        default: rc = launch_rows<1024>(i, o, n_frames, rows, shifts, s); break;
    }
    if (rc) return rc;
    switch (rows) {
        case 64: return launch_cols<64>(o, n_frames, cols, shifts, s);
        case 128: return launch_cols<128>(o, n_frames, cols, shifts, s);
        case 256: return launch_cols<256>(o, n_frames, cols, shifts, s);
        case 512: return launch_cols<512>(o, n_frames, cols, shifts, s);
        default: return launch_cols<1024>(o, n_frames, cols, shifts, s);
    }
}

extern "C" int qssb_join_workspace_bytes(int32_t n_frames, size_t* bytes) {
    if (!bytes || n_frames <= 0 || n_frames > 65535)
        return set_error(QSSB_ERR_INVALID, "qssb_join_workspace_bytes: n_frames must be in [1, 65535]");
    const size_t part = (sizeof(double2) * (size_t)n_frames * kJoinBlocks + 255) & ~(size_t)255;
    *bytes = part + sizeof(float2) * (size_t)n_frames;
    return QSSB_OK;
}

extern "C" int qssb_join_object_waves(float* frames, const float* weights, int32_t n_frames,
                                      int64_t n_pix, int32_t phase_reference, void* workspace,
                                      size_t workspace_bytes, float* joined, int32_t write_back,
                                      void* stream) {
    if (!frames || !weights || !joined || n_frames <= 0 || n_frames > 65535 || n_pix <= 0)
        return set_error(QSSB_ERR_INVALID, "qssb_join_object_waves: null pointer or empty shape");
    if (phase_reference != 0 && phase_reference != 1)
        return set_error(QSSB_ERR_INVALID, "qssb_join_object_waves: phase_reference must be 0 (none) or 1 (first)");
    cudaStream_t s = (cudaStream_t)stream;
    auto* a = reinterpret_cast<float2*>(frames);
    float2* rot = nullptr;
    if (phase_reference == 1) {
        size_t need = 0;
        int rc = qssb_join_workspace_bytes(n_frames, &need);
        if (rc) return rc;
        if (!workspace || workspace_bytes < need)
            return set_error(QSSB_ERR_WORKSPACE, "qssb_join_object_waves: workspace too small");
        if (((uintptr_t)workspace & 255u) != 0)
            return set_error(QSSB_ERR_INVALID, "qssb_join_object_waves: workspace must be 256-byte aligned");
        auto* partial = static_cast<double2*>(workspace);
        const size_t part = (sizeof(double2) * (size_t)n_frames * kJoinBlocks + 255) & ~(size_t)255;
        rot = reinterpret_cast<float2*>(static_cast<char*>(workspace) + part);
        const int n_blocks = overlap_blocks(n_pix);
        auto launch_partial = [&](auto kern) {
            kern<<<dim3(n_blocks, n_frames), kJoinThreads, 0, s>>>(a, n_pix, partial);
            note_launch();
        };
        if (n_blocks == kJoinBlocks)
            launch_partial(k_overlap_partial<true>);
        else
            launch_partial(k_overlap_partial<false>);
        CUDA_TRY(cudaGetLastError());
        { k_overlap_rotation<<<(n_frames + 3) / 4, 128, 0, s>>>(partial, n_blocks, n_frames, rot); note_launch(); }
        CUDA_TRY(cudaGetLastError());
    }
    const int per_block = n_pix < kJoinPixels ? 32 : kJoinThreads;
    const long long blocks = (n_pix + per_block - 1) / per_block;
    if (blocks > 0x7fffffffLL) return set_error(QSSB_ERR_INVALID, "qssb_join_object_waves: too many pixels");
    auto launch = [&](auto kern) {
        kern<<<(unsigned)blocks, kJoinThreads, 0, s>>>(a, weights, rot, n_frames, n_pix,
                                                       reinterpret_cast<float2*>(joined), write_back);
        note_launch();
    };
    if (n_pix < kJoinPixels)
        launch(k_join);
    else
        launch(k_join_pixels);
    CUDA_TRY(cudaGetLastError());
    return QSSB_OK;
}
