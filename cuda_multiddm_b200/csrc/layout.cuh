// Where the spectrum elements of a ring slot and the accumulators live in device memory.
//
// Elements are stored in blocks of 16 (128 bytes). Two layouts of the ring:
//   natural  [slot][element]: what the ring lag kernel's tensor maps read;
//   slabs    [slot / 32][element / 16][slot % 32][16]: the 32 frames of a slab lie next to each
//            other for every 16 elements, so the lag history of an element block is a few
//            contiguous pieces of up to 4 KB. (Read from the natural layout, a block's rows of 128
//            or 256 bytes each lie in a memory page of their own: 2.2 - 4.6 TB/s, bound by address
//            translation; slabs of 8 / 16 / 32 frames: 4.0 / 6.4 / 7.2 TB/s with CTAs out of step.)
// A last slab of fewer than 32 slots is packed by its own height, so both layouts take the same
// memory. The accumulators follow: [tau][element] or [element / 16][tau][16].
#pragma once

#include <cuda_runtime.h>

namespace ddm {

constexpr int kSlabLog2 = 5;
constexpr int kSlab = 1 << kSlabLog2;

struct RingLayout {
    long long E;  // elements of a frame (slabs: rounded up to a multiple of 16)
    int R;        // slots
    int slabs;    // 1: slabs, 0: natural

    // element e of slot s: ring[base(s) + (e >> 4) * stride(s) + (e & 15)]
    __host__ __device__ int slab_height(int slot) const {
        const int left = R - (slot >> kSlabLog2 << kSlabLog2);
        return left < kSlab ? left : kSlab;
    }
    __host__ __device__ long long base(int slot) const {
        return slabs ? (static_cast<long long>(slot >> kSlabLog2) << kSlabLog2) * E + (slot & (kSlab - 1)) * 16
                     : slot * E;
    }
    __host__ __device__ int stride(int slot) const { return slabs ? slab_height(slot) * 16 : 16; }
};

// One frame's elements: element e is *at(e). LINEAR: one after another (a natural slot, or a buffer of
// frames), else blocks of 16 a stride apart.
template <bool LINEAR>
struct FramePtr {
    float2 *p;
    int stride;
    __device__ __forceinline__ FramePtr(float2 *first, int block_stride) : p(first), stride(block_stride) {}
    __device__ __forceinline__ float2 *at(int e) const {
        return LINEAR ? p + e : p + static_cast<long long>(e >> 4) * stride + (e & 15);
    }
    // element e + d, given at_e = at(e), for a d known at compile time: whole blocks are a fixed distance
    __device__ __forceinline__ float2 *step(float2 *at_e, int e, int d) const {
        return LINEAR ? at_e + d : d % 16 == 0 ? at_e + static_cast<long long>(d / 16) * stride : at(e + d);
    }
};

// Accumulators: element e of tau row t at t * row + (e >> 4) * block + (e & 15).
struct AccLayout {
    long long row, block;
    __host__ __device__ long long at(int t, long long e) const { return t * row + (e >> 4) * block + (e & 15); }
};

}  // namespace ddm
