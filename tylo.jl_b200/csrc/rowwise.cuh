// Row-resident building block for the bandwidth kernels (softmax, RMSNorm, LayerNorm).
//
// A row is one Julia column: the contiguous, reduced dimension of length M.  THREADS threads own a row: a CTA, or a warp,
// eight of which share a CTA.  The row is read from HBM exactly once as 16-byte packets that stay in registers, the
// statistics are reduced with warp shuffles plus one shared-memory hop (none within a warp), and the result is written once.
// THREADS x ITERS packets of 16 bytes cover the row; packets past the end are predicated off.
#pragma once
#include "common.cuh"

namespace tylo {

// A row that starts or ends inside a 16-byte packet (M not a multiple of the packet, so that rows of a 16-byte aligned array
// start at every element offset).  Packets are counted from the aligned address at or before the row's start; all but the
// first and the last are whole and move as 16 bytes, those two element by element, so nothing outside the row is touched.
// Every array of a call is aligned alike, so one row has the same offset in all of them.
// Packets are counted in 64 bits: the two-pass kernels take rows as long as memory allows.
template <typename T> struct RaggedRow {
  static constexpr int kVec = Elem<T>::kVec;
  T* base;                 // the aligned address at or before the row's start
  int off;                 // elements of packet 0 that lie before the row
  int64_t end;             // elements from `base` to the row's end
  __device__ __forceinline__ RaggedRow(const T* r, int64_t m)
      : base(reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(r) & ~uintptr_t(15))),
        off((int)((reinterpret_cast<uintptr_t>(r) & 15) / sizeof(T))), end(off + m) {}
  __device__ __forceinline__ int64_t nvec() const { return (end + kVec - 1) / kVec; }
  // elements of packet v inside the row: [first, last)
  __device__ __forceinline__ int first(int64_t v) const { return v == 0 ? off : 0; }
  __device__ __forceinline__ int last(int64_t v) const {
    const int64_t n = end - v * kVec;
    return n >= kVec ? kVec : (n > 0 ? (int)n : 0);
  }
  // packet v, elements outside the row (and packets past it) read as `fill`
  __device__ __forceinline__ Pack<T> load(int64_t v, float fill) const {
    Pack<T> p;
    const int lo = first(v), hi = last(v);
    const T* q = base + v * kVec;
    if (lo == 0 && hi == kVec) { p.raw = ld_stream(q); return p; }
    float f[kVec];
#pragma unroll
    for (int j = 0; j < kVec; ++j) f[j] = j >= lo && j < hi ? Elem<T>::to_f(q[j]) : fill;
    p.pack(f);
    return p;
  }
  __device__ __forceinline__ void store(int64_t v, const Pack<T>& p) const {
    const int lo = first(v), hi = last(v);
    T* q = base + v * kVec;
    if (lo == 0 && hi == kVec) { st_stream(q, p.raw); return; }
    float f[kVec];
    p.unpack(f);
#pragma unroll
    for (int j = 0; j < kVec; ++j)
      if (j >= lo && j < hi) q[j] = Elem<T>::from_f(f[j]);
  }
};

// Rows of one warp share a CTA, eight at a time (a CTA of one warp per row leaves the SM at its limit of 32 CTAs, 32 warps, and
// spends as long on starting CTAs as on the rows: 3.3 TB/s at 512 bf16 elements); longer rows have a CTA each.
constexpr int kWarpRows = 8;
constexpr int row_cta(int threads) { return threads == 32 ? 32 * kWarpRows : threads; }
inline unsigned row_grid(int threads, int64_t rows) { return (unsigned)(threads == 32 ? (rows + kWarpRows - 1) / kWarpRows : rows); }
template <int THREADS> __device__ __forceinline__ int row_thread() { return THREADS == 32 ? (int)(threadIdx.x & 31) : (int)threadIdx.x; }
template <int THREADS> __device__ __forceinline__ size_t row_index() {
  return THREADS == 32 ? (size_t)blockIdx.x * kWarpRows + (threadIdx.x >> 5) : (size_t)blockIdx.x;
}

// (the thread's index is spelled out in the loops below: through row_thread the compiler takes 128 registers instead of 80 for
// 256 x 16 packets, a CTA per SM less)
template <typename T, int THREADS, int ITERS> struct RowRegs {
  static constexpr int kVec = Elem<T>::kVec;
  static constexpr int kMaxElems = THREADS * ITERS * kVec;
  Pack<T> p[ITERS];

  __device__ __forceinline__ void load(const T* __restrict__ row, int nvec) {
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
      const int v = i * THREADS + (THREADS == 32 ? threadIdx.x & 31 : threadIdx.x);
      if (v < nvec) p[i].raw = ld_stream(row + (size_t)v * kVec);
      else p[i].raw = make_uint4(0, 0, 0, 0);
    }
  }
  __device__ __forceinline__ void load(const RaggedRow<T>& row, float fill) {
#pragma unroll
    for (int i = 0; i < ITERS; ++i) p[i] = row.load(i * THREADS + (THREADS == 32 ? threadIdx.x & 31 : threadIdx.x), fill);
  }
  __device__ __forceinline__ void store(const RaggedRow<T>& row) const {
#pragma unroll
    for (int i = 0; i < ITERS; ++i) row.store(i * THREADS + (THREADS == 32 ? threadIdx.x & 31 : threadIdx.x), p[i]);
  }
  __device__ __forceinline__ void store(T* __restrict__ row, int nvec) const {
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
      const int v = i * THREADS + (THREADS == 32 ? threadIdx.x & 31 : threadIdx.x);
      if (v < nvec) st_stream(row + (size_t)v * kVec, p[i].raw);
    }
  }
};

// Load one 16-byte packet of a small, reused vector (weights): default caching.
template <typename T> __device__ __forceinline__ Pack<T> ld_param(const T* p) {
  Pack<T> r;
  r.raw = *reinterpret_cast<const uint4*>(p);
  return r;
}

// Launch-shape table (threads, packets per thread) of the norm forwards: 32-128 bytes of the row in flight per thread, and
// a shape for every power of two of packets up to 4,096, so that the common row lengths leave no thread idle (with 256 x 4
// for 512 packets, half of them were: layer norm 4096 bf16 2.9 TB/s).
struct RowShape { int threads, iters; };
inline bool pick_row_shape(int64_t nvec, RowShape* out) {
  static const RowShape table[] = {{32, 2}, {64, 2}, {128, 2}, {128, 4}, {256, 4}, {512, 4}, {512, 8}, {1024, 8}};
  for (const RowShape& s : table)
    if ((int64_t)s.threads * s.iters >= nvec) { *out = s; return true; }
  return false;
}

}  // namespace tylo
