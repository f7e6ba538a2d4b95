// Batches of independent H-matrices: packing, the stages of all parts of a batch
// in one launch each (the bodies of hmvm_multi_kernel and hmvm_dmma_kernel),
// reductions and unpacking.
#pragma once

#include "kernels_dmma.cuh"
#include "kernels_multi.cuh"

namespace hmvm {

// ---- batches of independent H-matrices ----------------------------------------
// A batch runs as block-diagonal H-matrices over concatenated index spaces;
// instance m owns rows [off, off + n) of its class.
struct BatchIO {
  const void* X;  // column c at X + c * ldx
  int64_t ldx;
  void* Y;
  int64_t ldy;
  int64_t off;
  int32_t n, nrhs;
};

// A batch is planned as block-diagonal classes (one plan per pass width), and an
// apply runs each class's passes; every (class, pass) -- a "part" -- has its own
// packed inputs, t, partial sums and concatenated outputs, so all parts run at
// once: each of these kernels reads the batch's part table (global memory) and
// cuts its blocks (or work items) into per-part ranges.  Every buffer access of
// a part is checked against the part's capacities (a miss records error 3 and
// is skipped).
struct BatchPart {
  MultiArgs a;
  int32_t cta0;  // first block of the part in its stage launch
  int32_t nr;    // pass width: 2, 4 or 8
};
template <int WPB, int S, int CHUNK, int MODE, bool VST>
__global__ void __launch_bounds__(
    32 * WPB, (MODE <= kModePlain32 ? dmma_min_blocks<WPB, S, CHUNK>() : multi_min_blocks<WPB, S, CHUNK, kMultiZBytes>()))
    hmvm_batch_multi_kernel(const BatchPart* __restrict__ parts, int nparts) {
  int k = 0;
  while (k + 1 < nparts && (int)blockIdx.x >= parts[k + 1].cta0) k++;
  const MultiArgs a = parts[k].a;
  const int bid = (int)blockIdx.x - parts[k].cta0;
  if constexpr (MODE <= kModePlain32) {
    using T = typename std::conditional<MODE == kModePlain64, double, float>::type;
    dmma_body<T, WPB, S, CHUNK, 0, VST, true>(a, bid, parts[k].nr);
  } else {
    switch (parts[k].nr) {
      case 2: multi_body<WPB, S, CHUNK, 2, MODE, VST, true>(a, bid); break;
      case 4: multi_body<WPB, S, CHUNK, 4, MODE, VST, true>(a, bid); break;
      default: multi_body<WPB, S, CHUNK, 8, MODE, VST, true>(a, bid); break;
    }
  }
}

// The split-tile reductions of every part (hmvm_reduce_multi_kernel's sums, with
// each part's width): work items [w0, w0 + n * nr) are the part's.
struct BatchRedPart {
  const int4* red;
  const void* p;
  void* dst;
  int64_t ldy;
  int64_t w0;
  int64_t pcap, dcap;  // elements of p and dst
  int32_t n, nr;
};
template <typename TP, typename TD, bool VST>
__global__ void hmvm_batch_reduce_kernel(const BatchRedPart* __restrict__ parts, int nparts, int64_t total,
                                         int* err) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
    int q = 0;
    while (q + 1 < nparts && k >= parts[q + 1].w0) q++;
    const BatchRedPart& P = parts[q];
    const int NR = P.nr;
    const int64_t l = k - P.w0;
    const int i = (int)(l / NR), r = (int)(l % NR);
    const int4 e = P.red[i];
    const int64_t last = (int64_t)(e.y + (e.z - 1) * e.w) * NR + r;
    const int64_t d = VST ? (int64_t)e.x * NR + r : (int64_t)e.x + (int64_t)r * P.ldy;
    if (e.y < 0 || e.z < 0 || last >= P.pcap || d < 0 || d >= P.dcap) {
      atomicExch(err, 3);
      continue;
    }
    const TP* p = static_cast<const TP*>(P.p);
    TP sum = TP(0);
    for (int u = 0; u < e.z; u++) sum += p[(int64_t)(e.y + u * e.w) * NR + r];
    static_cast<TD*>(P.dst)[d] = (TD)sum;
  }
}

// One row of the pack / unpack grids (blockIdx.y): an instance in one part.
struct BatchPack {
  int32_t io;       // the instance (index into the batch's BatchIO table)
  int32_t c0;       // first column of the part's pass
  int32_t nr;       // pass width
  int32_t _pad;
  double* x64;      // the part's packed inputs (row-interleaved, nr per row)
  float* x32;
  void* ycat;       // the part's concatenated outputs, column r at ycat + r * ldc
  int64_t ldc;
  int64_t xcap, ycap;  // elements of the packed inputs and of ycat
};
// Columns [c0, c0 + nr) of each instance -> its part's packed inputs (zero past nrhs).
template <typename TI>
__global__ void hmvm_batch_pack_kernel(const BatchIO* __restrict__ io, int nio, const BatchPack* __restrict__ e,
                                       int* err) {
  const BatchPack q = e[blockIdx.y];
  if (q.io < 0 || q.io >= nio) {
    if (threadIdx.x == 0) atomicExch(err, 3);
    return;
  }
  const BatchIO b = io[q.io];
  if (b.off < 0 || (b.off + b.n) * q.nr > q.xcap) {
    if (threadIdx.x == 0) atomicExch(err, 3);
    return;
  }
  const TI* X = static_cast<const TI*>(b.X);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < (int64_t)b.n * q.nr;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k / q.nr;
    const int r = (int)(k % q.nr);
    const double v = q.c0 + r < b.nrhs ? (double)X[i + (int64_t)(q.c0 + r) * b.ldx] : 0.0;
    const int64_t dst = (b.off + i) * q.nr + r;
    if (q.x64) q.x64[dst] = v;
    if (q.x32) q.x32[dst] = (float)v;
  }
}
// Each instance's columns of its part's concatenated outputs -> its own Y.
template <typename T>
__global__ void hmvm_batch_unpack_parts_kernel(const BatchIO* __restrict__ io, int nio,
                                               const BatchPack* __restrict__ e, int* err) {
  const BatchPack q = e[blockIdx.y];
  if (q.io < 0 || q.io >= nio) {
    if (threadIdx.x == 0) atomicExch(err, 3);
    return;
  }
  const BatchIO b = io[q.io];
  if (b.off < 0 || b.off + b.n + (int64_t)(q.nr - 1) * q.ldc > q.ycap) {
    if (threadIdx.x == 0) atomicExch(err, 3);
    return;
  }
  T* Y = static_cast<T*>(b.Y);
  const T* yc = static_cast<const T*>(q.ycat);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < (int64_t)b.n * q.nr;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(k / b.n);
    const int64_t i = k % b.n;
    if (q.c0 + r < b.nrhs) Y[i + (int64_t)(q.c0 + r) * b.ldy] = yc[b.off + i + r * q.ldc];
  }
}

}  // namespace hmvm
