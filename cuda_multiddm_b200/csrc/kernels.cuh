// Device kernels of the DDM engine (sm_100a).
//
//   fft_rows_kernel,   (fft.cuh) tile extraction + 2-D R2C FFT per scale (replaces
//   fft_cols_kernel    parseBufferScalePow2 + cufftExecR2C, src/DDM_kernel.cuh:43-78)
//   lag_pipe_kernel    (lag.cuh) |F(a) - F(b)|^2 accumulation for a block of frames
//                      against every tau (replaces processFFT, src/DDM_kernel.cuh:85-101)
//   azimuth_partial_kernel, azimuth_final_kernel
//                      masked azimuthal average of every (scale, tile, lambda, tau) bin over
//                      the annulus index lists, FP64, in two deterministic stages (replaces
//                      maskReduce + the host sums, src/azimuthal_average.cu:292-346)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "layout.cuh"

namespace ddm {

constexpr int kMaxScales = 16;
constexpr int kAzThreads = 256;
constexpr int kMaxJ = 64;          // register frames per element of one lag-kernel launch
constexpr int kPieceFrames = 32;   // frames per ingest piece (FFT group, staging) at most

struct ScaleDesc {
    int s, tiles;
    long long n, off;     // elements per tile, offset of the scale in a frame
    long long isf_off;    // offset of the scale's block in the ISF output
    int q_base;           // index of (scale, q = 0) in counts / chunk_first / chunk_count
    double inv_s4;
    // azimuthal work: the scale's annulus index lists cut into chunks of <= kAzChunk entries (az_chunk_size)
    int nchunks;          // chunks of all q of this scale
    int chunk_off;        // first chunk of the scale in chunk_beg / chunk_end
    long long item_base;  // first (chunk, tile, tau) item of the scale; items are ordered (tile, chunk, tau)
};

// Annulus indices summed by one warp: at most kAzChunk, halved down to kAzMinChunk while the average
// has fewer warps than the GPU holds (a chunk is a serial chain of gathers: 256^2, 20 taus, 10
// lambdas took 16 us with chunks of 1024).
constexpr int kAzChunk = 1024, kAzMinChunk = 128;
// A B200's 148 SMs times 32 warps; fixed, not the device's own count, because the chunk sets the order of the
// FP64 sums: one configuration has the same bits everywhere.
constexpr long long kAzWantWarps = 148 * 32;
constexpr int kAzWarps = kAzThreads / 32;

struct AzArgs {
    int S, T, Q;
    ScaleDesc sc[kMaxScales];
    const float2 *acc;
    AccLayout lay;
    const int *idx;          // element indices within a tile, CSR per (scale, q)
    const int *chunk_beg;    // [chunks] absolute offsets into idx
    const int *chunk_end;
    const int *chunk_first;  // [S*Q] first chunk of (scale, q), relative to the scale
    const int *chunk_count;  // [S*Q]
    const int *counts;       // [S*Q] annulus pixel counts
    const double *norm;      // [T], or null: in the launch's AzNorm
    double *partial;         // [items] stage-1 sums
    double *isf;
    long long items, bins;
};

// The pair counts of up to kAzInlineNorms taus travel with the launch (no upload to wait for).
constexpr int kAzInlineNorms = 128;
struct AzNorm {
    double v[kAzInlineNorms];
};

__device__ __forceinline__ int az_scale_of(const AzArgs &a, long long item) {
    int si = 0;
    while (si + 1 < a.S && item >= a.sc[si + 1].item_base) si++;
    return si;
}

// Stage 1: one warp per (scale, tile, chunk, tau) item sums the accumulator values
// (sum - compensation, in FP64) at the chunk's annulus indices into partial[item]. Neighbouring
// warps take neighbouring taus of one chunk: their accumulators lie side by side in the blocked
// layout, and they share the index list.
__global__ void __launch_bounds__(kAzThreads) azimuth_partial_kernel(AzArgs a) {
    const long long item = static_cast<long long>(blockIdx.x) * kAzWarps + (threadIdx.x >> 5);
    if (item >= a.items) return;
    const int lane = threadIdx.x & 31;
    const int si = az_scale_of(a, item);
    const ScaleDesc &sc = a.sc[si];
    const long long rel = item - sc.item_base;
    const long long tc = rel / a.T;  // tile * nchunks + chunk
    const int t = static_cast<int>(rel - tc * a.T);
    const int tile = static_cast<int>(tc / sc.nchunks), c = static_cast<int>(tc - static_cast<long long>(tile) * sc.nchunks);
    const float2 *row = a.acc + t * a.lay.row;
    const int e0 = static_cast<int>(sc.off + tile * sc.n);  // the tile's first element
    const int beg = a.chunk_beg[sc.chunk_off + c], end = a.chunk_end[sc.chunk_off + c];
    double sum = 0.0;
    for (int i = beg + lane; i < end; i += 32) {
        const int e = e0 + a.idx[i];
        const float2 v = row[(e >> 4) * a.lay.block + (e & 15)];
        sum += static_cast<double>(v.x) - static_cast<double>(v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) a.partial[item] = sum;
}

// Stage 2: one thread per (scale, tile, q, tau) bin adds its chunks' partials in order and
// normalises: ISF = 2 * sum / s^4 / pixel_count / norm[tau] (0 for an empty annulus).
__global__ void __launch_bounds__(kAzThreads) azimuth_final_kernel(AzArgs a, const __grid_constant__ AzNorm inl) {
    const long long bin = static_cast<long long>(blockIdx.x) * kAzThreads + threadIdx.x;
    if (bin >= a.bins) return;
    int si = 0;
    while (si + 1 < a.S && bin >= a.sc[si + 1].isf_off) si++;
    const ScaleDesc &sc = a.sc[si];
    const long long rel = bin - sc.isf_off;  // ((tile * Q + q) * T + t)
    const int t = static_cast<int>(rel % a.T);
    const long long tq = rel / a.T;
    const int q = static_cast<int>(tq % a.Q);
    const int tile = static_cast<int>(tq / a.Q);
    const int first = a.chunk_first[sc.q_base + q], cnt = a.chunk_count[sc.q_base + q];
    const double *p = a.partial + sc.item_base + (static_cast<long long>(tile) * sc.nchunks + first) * a.T + t;
    double sum = 0.0;
    for (int c = 0; c < cnt; c++) sum += p[static_cast<long long>(c) * a.T];
    const int P = a.counts[sc.q_base + q];
    const double nrm = a.norm ? a.norm[t] : inl.v[t];
    a.isf[bin] = (P != 0 && nrm != 0.0) ? 2.0 * sum * sc.inv_s4 / static_cast<double>(P) / nrm : 0.0;
}

// The elements of one frame (blocks of 16, `stride` apart) packed into dst[0..E).
__global__ void gather_frame_kernel(const float2 *__restrict__ src, int stride, float2 *__restrict__ dst, long long E) {
    const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e < E) dst[e] = src[(e >> 4) * stride + (e & 15)];
}

}  // namespace ddm
