// How the sparse products of the optic lobe (optic.cu, adjoint.cu) lay the flies of a unit on lanes,
// and how their persistent launches hand out work.
#pragma once
#include "common.cuh"

namespace flyb {

// The flies of a unit on the F fly lanes of a row slot: W consecutive flies per vector (a 4-, 8- or
// 16-byte access, W dividing the batch), NV vectors per lane, F vectors apart. A lane's vector is
// inside the batch as a whole or not at all.
template <int W, int NV, int F>
struct Flies {
  static constexpr int FPL = W * NV;                               // flies per lane
  static __device__ __forceinline__ int at(int f, int v) { return (f + v * F) * W; }
};

template <int W>
__device__ __forceinline__ void load_w(const float* p, float* x) {
  if constexpr (W == 1) {
    x[0] = *p;
  } else if constexpr (W == 2) {
    const float2 q = *reinterpret_cast<const float2*>(p); x[0] = q.x; x[1] = q.y;
  } else {
    const float4 q = *reinterpret_cast<const float4*>(p); x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
  }
}

template <int W>
__device__ __forceinline__ void store_w(float* p, const float* x) {
  if constexpr (W == 1) *p = x[0];
  else if constexpr (W == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  else *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}

// Widest vector access a batch and its arrays allow: W flies, W dividing the batch and every array W
// floats aligned.
template <int N>
static int vector_width(int batch, const void* const (&arrays)[N]) {
  for (int w = 4; w > 1; w >>= 1) {
    bool ok = batch % w == 0;
    for (const void* p : arrays) ok = ok && (reinterpret_cast<uintptr_t>(p) & (4 * w - 1)) == 0;
    if (ok) return w;
  }
  return 1;
}

template <int LPR>
struct RowSlots {
  static constexpr int RPW = 32 / LPR;           // row slots per warp
  static constexpr int SLOTS = 8 * RPW;          // row slots per 256-thread block
};

// Items 0 .. items - 1 of pass number `pass` of a persistent launch, handed out to its blocks as they
// come for them: the first gridDim.x <= items by block, the others by `count` (zero at the launch),
// which grows by one per item and so by `items` per pass. Thread 0 asks for the next item beside
// the current one. `next` is the block's shared word; a barrier over the grid separates passes.
template <typename Body>
__device__ __forceinline__ void deal_items(int* count, unsigned pass, long long items, unsigned* next, Body body) {
  for (long long item = blockIdx.x; item < items;) {
    unsigned given = 0;
    if (threadIdx.x == 0) given = (unsigned)atomicAdd(count, 1) - pass * (unsigned)items;
    body(item);
    if (threadIdx.x == 0) *next = given;
    __syncthreads();
    item = (long long)gridDim.x + *next;
    __syncthreads();
  }
}

}  // namespace flyb
