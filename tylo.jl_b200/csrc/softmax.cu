// Row softmax forward / backward for sm_100a: one read and one write of HBM per element
// (the reference's streaming kernel reads X twice, softmax.jl:6-33).
//
// A row of up to 32,768 (16-bit) / 8,192 (fp32) elements (forward; 8,192 / 4,096 backward) is held in the registers of one
// CTA, or of one warp when it is short; longer rows take two passes, the second of which reads out of L2.  Rows of any
// length and start move as 16-byte packets (see RaggedRow).
//
// exp is evaluated once per element: each thread first takes the max of its own elements,
// exponentiates against that, and the result is rescaled by exp2(m_thread - m_row) / sum
// — one extra exp per thread instead of one per element.
#include <cooperative_groups.h>

#include "rowwise.cuh"

namespace cg = cooperative_groups;

namespace tylo {

constexpr float kLog2e = 1.4426950408889634f;

// Combine a per-thread (max, sum-relative-to-that-max) pair over the row's threads.  Returns the row max and the row sum relative
// to it; the sum is 0 for a row made only of -Inf and NaN for a row that holds a NaN or +Inf, wherever in it (fmaxf passes over
// a NaN, so a part of -Inf and NaN has maximum -Inf and a NaN as its sum).  Differences are taken before the factor log2(e): the
// lowest finite fp32 value would overflow with it.
template <int THREADS>
__device__ __forceinline__ void reduce_max_sum(float& m, float& s, float* smem /* >= 64 floats */) {
  // warp level
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const float mn = fmaxf(m, m2);
    s = (mn == -INFINITY) ? s + s2 : s * exp2f((m - mn) * kLog2e) + s2 * exp2f((m2 - mn) * kLog2e);
    m = mn;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (THREADS > 32) {
    if (lane == 0) { smem[warp] = m; smem[32 + warp] = s; }
    __syncthreads();
    m = lane < THREADS / 32 ? smem[lane] : -INFINITY;
    s = lane < THREADS / 32 ? smem[32 + lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
      const float mn = fmaxf(m, m2);
      s = (mn == -INFINITY) ? s + s2 : s * exp2f((m - mn) * kLog2e) + s2 * exp2f((m2 - mn) * kLog2e);
      m = mn;
    }
  }
  if constexpr (THREADS > 32) __syncthreads();
}

template <typename T, int THREADS, int ITERS, bool RAGGED>
__global__ void __launch_bounds__(row_cta(THREADS))
softmax_fwd_kernel(T* __restrict__ Y, const T* __restrict__ X, int64_t M, int N) {
  constexpr int VEC = Elem<T>::kVec;
  __shared__ float smem[64];
  const size_t row = row_index<THREADS>();
  if (THREADS == 32 && row >= (size_t)N) return;
  const int tid = row_thread<THREADS>();
  int nvec = (int)(M / VEC);

  RowRegs<T, THREADS, ITERS> r;
  if constexpr (RAGGED) {
    const RaggedRow<T> x(X + row * M, M);
    nvec = (int)x.nvec();
    r.load(x, -INFINITY);
  } else {
    r.load(X + row * M, nvec);
  }
  float e[ITERS][VEC];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    r.p[i].unpack(e[i]);
    if (i * THREADS + tid < nvec) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) m = fmaxf(m, e[i][j]);
    }
  }
  const float m_thread = m;
  const float mt = (m_thread == -INFINITY) ? 0.f : m_thread;
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const bool live = i * THREADS + tid < nvec;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      e[i][j] = live ? exp2f((e[i][j] - mt) * kLog2e) : 0.f;
      s += e[i][j];
    }
  }
  reduce_max_sum<THREADS>(m, s, smem);
  // a row made only of -Inf yields zeros (nothing in the reference's tests pins that case); a NaN sum reaches every element
  const float factor = s == 0.f ? 0.f : ((m_thread == -INFINITY) ? 0.f : exp2f((m_thread - m) * kLog2e)) / s;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
#pragma unroll
    for (int j = 0; j < VEC; ++j) e[i][j] *= factor;
    r.p[i].pack(e[i]);
  }
  if constexpr (RAGGED) r.store(RaggedRow<T>(Y + row * M, M));
  else r.store(Y + row * M, nvec);
}

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Forward for 16-bit storage.  The row stays in registers in its packed 16-bit form (half the
// registers of an fp32 copy, so twice the bytes in flight per SM for the same occupancy) and exp is
// evaluated twice per element (once for the sum, once for the output) on the otherwise idle
// special-function unit; its approximate form is ample for a 16-bit result.
// (ragged rows at 16 packets per thread: left alone the compiler takes 226 registers; three CTAs per SM are asked for)
template <typename T, int THREADS, int ITERS, bool RAGGED>
__global__ void __launch_bounds__(row_cta(THREADS), RAGGED && ITERS == 16 ? 3 : 0)
softmax_fwd_packed_kernel(T* __restrict__ Y, const T* __restrict__ X, int64_t M, int N) {
  constexpr int VEC = Elem<T>::kVec;
  __shared__ float smem[32];
  const size_t row = row_index<THREADS>();
  if (THREADS == 32 && row >= (size_t)N) return;
  const int tid = row_thread<THREADS>();
  const int nvec = RAGGED ? (int)RaggedRow<T>(X + row * M, M).nvec() : (int)(M / VEC);
  RowRegs<T, THREADS, ITERS> r;
  if constexpr (RAGGED) r.load(RaggedRow<T>(X + row * M, M), -INFINITY);
  else r.load(X + row * M, nvec);
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    if (i * THREADS + tid < nvec) {
      float f[VEC]; r.p[i].unpack(f);
#pragma unroll
      for (int j = 0; j < VEC; ++j) m = fmaxf(m, f[j]);
    }
  }
  m = block_reduce<THREADS>(m, MaxOp(), -INFINITY, smem);
  const float mo = (m == -INFINITY) ? 0.f : m * kLog2e;
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    if (i * THREADS + tid < nvec) {
      float f[VEC]; r.p[i].unpack(f);
#pragma unroll
      for (int j = 0; j < VEC; ++j) s += ex2_fast(fmaf(f[j], kLog2e, -mo));
    }
  }
  s = block_reduce<THREADS>(s, SumOp(), 0.f, smem);
  const float inv = (m == -INFINITY && s == 0.f) ? 0.f : 1.f / s;     // only -Inf: zeros; NaN or +Inf in the row: NaN throughout
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    float f[VEC]; r.p[i].unpack(f);
#pragma unroll
    for (int j = 0; j < VEC; ++j) f[j] = ex2_fast(fmaf(f[j], kLog2e, -mo)) * inv;
    r.p[i].pack(f);
  }
  if constexpr (RAGGED) r.store(RaggedRow<T>(Y + row * M, M));
  else r.store(Y + row * M, nvec);
}

// Rows too long for one CTA's registers, forward: a pass that keeps a running (max, sum) per thread and a pass that reads
// the row again out of L2 (see the backward's two-pass form below) and writes.
// CLUSTERED: a row is dealt packet by packet over the CTAs of a cluster, which exchange their (max, sum) through distributed
// shared memory; for launches with fewer rows than SMs.  Each thread reads and writes the same packets in both passes.
// ONCE: the row is no longer than U packets per thread, which wait in registers for the second pass.
template <typename T, int THREADS, bool RAGGED, bool CLUSTERED, bool ONCE>
__global__ void __launch_bounds__(THREADS)
softmax_fwd_twopass_kernel(T* __restrict__ Y, const T* __restrict__ X, int64_t M) {
  constexpr int VEC = Elem<T>::kVec, U = 4;
  __shared__ float smem[66];
  int ctas = 1, rank = 0;
  if constexpr (CLUSTERED) { ctas = cg::this_cluster().num_blocks(); rank = cg::this_cluster().block_rank(); }
  const int step = ctas * THREADS, first = rank * THREADS + (int)threadIdx.x;
  const size_t base = (size_t)(blockIdx.x / ctas) * M;
  const RaggedRow<T> x(X + base, M), y(Y + base, M);
  const int64_t nvec = RAGGED ? x.nvec() : M / VEC;
  auto ex2 = [](float v) { return sizeof(T) == 2 ? ex2_fast(v) : exp2f(v); };
  auto load = [&](int64_t v) {
    Pack<T> p;
    if constexpr (RAGGED) return x.load(v, -INFINITY);
    if (v < nvec) { p.raw = __ldg(reinterpret_cast<const uint4*>(X + base) + v); return p; }
    float f[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) f[j] = -INFINITY;
    p.pack(f);
    return p;
  };
  float m = -INFINITY, s = 0.f;
  Pack<T> p[U];
  for (int64_t v0 = first; v0 < nvec; v0 += U * step) {
#pragma unroll
    for (int u = 0; u < U; ++u) p[u] = load(v0 + u * step);
    float mx = -INFINITY;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[VEC]; p[u].unpack(f);
#pragma unroll
      for (int j = 0; j < VEC; ++j) mx = fmaxf(mx, f[j]);
    }
    const float mn = fmaxf(m, mx);
    if (mn != -INFINITY) {
      s *= ex2((m - mn) * kLog2e);
      m = mn;
    }
    const float mo = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[VEC]; p[u].unpack(f);
#pragma unroll
      for (int j = 0; j < VEC; ++j) s += ex2((f[j] - mo) * kLog2e);
    }
  }
  reduce_max_sum<THREADS>(m, s, smem);
  if constexpr (CLUSTERED) {
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0) { smem[64] = m; smem[65] = s; }
    cluster.sync();
    const int lane = threadIdx.x & 31;
    const float* peer = cluster.map_shared_rank(smem, lane < ctas ? lane : 0);
    m = lane < ctas ? peer[64] : -INFINITY;
    s = lane < ctas ? peer[65] : 0.f;
    reduce_max_sum<32>(m, s, smem);
    cluster.sync();               // a CTA may leave, and take its shared memory along, once everyone has read it
  }
  const float inv = s == 0.f ? 0.f : 1.f / s, mo = m == -INFINITY ? 0.f : m;
  for (int64_t v0 = first; v0 < nvec; v0 += U * step) {
    if constexpr (!ONCE) {
#pragma unroll
      for (int u = 0; u < U; ++u) p[u] = load(v0 + u * step);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t v = v0 + u * step;
      float f[VEC]; p[u].unpack(f);
#pragma unroll
      for (int j = 0; j < VEC; ++j) f[j] = ex2((f[j] - mo) * kLog2e) * inv;
      p[u].pack(f);
      if constexpr (RAGGED) y.store(v, p[u]);
      else if (v < nvec) st_stream(Y + base + (size_t)v * VEC, p[u].raw);
    }
  }
}

template <typename T, int THREADS, int ITERS, bool RAGGED>
__global__ void __launch_bounds__(row_cta(THREADS))
softmax_bwd_kernel(T* __restrict__ dX, const T* __restrict__ dY, const T* __restrict__ Y, int64_t M, int N) {
  constexpr int VEC = Elem<T>::kVec;
  __shared__ float smem[32];
  const size_t row = row_index<THREADS>();
  if (THREADS == 32 && row >= (size_t)N) return;
  const int nvec = (int)(M / VEC);

  RowRegs<T, THREADS, ITERS> y, dy;
  if constexpr (RAGGED) {
    y.load(RaggedRow<T>(Y + row * M, M), 0.f);
    dy.load(RaggedRow<T>(dY + row * M, M), 0.f);
  } else {
    y.load(Y + row * M, nvec);
    dy.load(dY + row * M, nvec);
  }
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    float a[VEC], b[VEC];
    y.p[i].unpack(a); dy.p[i].unpack(b);
#pragma unroll
    for (int j = 0; j < VEC; ++j) dot += a[j] * b[j];
  }
  dot = block_reduce<THREADS>(dot, SumOp(), 0.f, smem);
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    float a[VEC], b[VEC];
    y.p[i].unpack(a); dy.p[i].unpack(b);
#pragma unroll
    for (int j = 0; j < VEC; ++j) a[j] = a[j] * (b[j] - dot);
    y.p[i].pack(a);
  }
  if constexpr (RAGGED) y.store(RaggedRow<T>(dX + row * M, M));
  else y.store(dX + row * M, nvec);
}

// Long rows, backward: two passes over Y and dY instead of a register-resident row.  Pass 1 sums y * dy, pass 2
// reads both again — a row pair is 128 KB at 32,768 16-bit elements, a few hundred of them in flight fit L2 many
// times over, so the second read never reaches HBM — and writes dX.  No cluster, no row held in registers: a thread
// keeps eight 16-byte loads in flight and the CTA is free of the all-or-nothing scheduling of a cluster.
template <typename T, int THREADS, bool RAGGED>
__global__ void __launch_bounds__(THREADS)
softmax_bwd_twopass_kernel(T* __restrict__ dX, const T* __restrict__ dY, const T* __restrict__ Y, int64_t M) {
  constexpr int VEC = Elem<T>::kVec, U = 4;
  __shared__ float smem[32];
  const size_t base = (size_t)blockIdx.x * M;
  const RaggedRow<T> ry(Y + base, M), rd(dY + base, M), ro(dX + base, M);
  const int64_t nvec = RAGGED ? ry.nvec() : M / VEC;
  auto load = [&](const T* p, const RaggedRow<T>& r, int64_t v) {
    Pack<T> k;
    if constexpr (RAGGED) return r.load(v, 0.f);
    k.raw = v < nvec ? __ldg(reinterpret_cast<const uint4*>(p + base) + v) : make_uint4(0, 0, 0, 0);
    return k;
  };
  float dot = 0.f;
  for (int64_t v0 = threadIdx.x; v0 < nvec; v0 += U * THREADS) {
    Pack<T> y[U], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { y[u] = load(Y, ry, v0 + u * THREADS); d[u] = load(dY, rd, v0 + u * THREADS); }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float a[VEC], b[VEC];
      y[u].unpack(a); d[u].unpack(b);
#pragma unroll
      for (int j = 0; j < VEC; ++j) dot = fmaf(a[j], b[j], dot);
    }
  }
  dot = block_reduce<THREADS>(dot, SumOp(), 0.f, smem);
  for (int64_t v0 = threadIdx.x; v0 < nvec; v0 += U * THREADS) {
    Pack<T> y[U], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { y[u] = load(Y, ry, v0 + u * THREADS); d[u] = load(dY, rd, v0 + u * THREADS); }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t v = v0 + u * THREADS;
      float a[VEC], b[VEC];
      y[u].unpack(a); d[u].unpack(b);
#pragma unroll
      for (int j = 0; j < VEC; ++j) a[j] = a[j] * (b[j] - dot);
      y[u].pack(a);
      if constexpr (RAGGED) ro.store(v, y[u]);
      else if (v < nvec) st_stream(dX + base + (size_t)v * VEC, y[u].raw);
    }
  }
}

template <typename T, bool FWD, bool RAGGED>
static int32_t softmax_launch(void* out, const void* a, const void* b, int64_t M, int64_t N, cudaStream_t st) {
  constexpr int VEC = Elem<T>::kVec;
  const char* what = FWD ? "softmax_fwd" : "softmax_bwd";
  const int64_t nvec = RAGGED ? (M + 2 * VEC - 2) / VEC : M / VEC;     // packets a row may touch
  // register-resident rows; a shape for every power of two of packets (see pick_row_shape)
#define TYLO_SM_LAUNCH(THREADS, ITERS)                                                                               \
  do {                                                                                                               \
    const unsigned grid = row_grid(THREADS, N), cta = row_cta(THREADS);                                              \
    if constexpr (!FWD) softmax_bwd_kernel<T, THREADS, ITERS, RAGGED><<<grid, cta, 0, st>>>(                         \
        (T*)out, (const T*)a, (const T*)b, M, (int)N);                                                               \
    else if constexpr (VEC == 8) softmax_fwd_packed_kernel<T, THREADS, ITERS, RAGGED><<<grid, cta, 0, st>>>(         \
        (T*)out, (const T*)a, M, (int)N);                                                                            \
    else softmax_fwd_kernel<T, THREADS, ITERS, RAGGED><<<grid, cta, 0, st>>>((T*)out, (const T*)a, M, (int)N);       \
    return check_launch(what);                                                                                       \
  } while (0)
  if (nvec <= 64) TYLO_SM_LAUNCH(32, 2);
  if (nvec <= 128) TYLO_SM_LAUNCH(64, 2);
  if (nvec <= 256) TYLO_SM_LAUNCH(128, 2);
  if (nvec <= 512) TYLO_SM_LAUNCH(128, 4);
  if (nvec <= 1024) TYLO_SM_LAUNCH(256, 4);
  if constexpr (FWD && VEC == 8) {
    if (nvec <= 2048) TYLO_SM_LAUNCH(256, 8);
    if (nvec <= 4096) TYLO_SM_LAUNCH(256, 16);
  } else if constexpr (FWD) {
    if (nvec <= 2048) TYLO_SM_LAUNCH(512, 4);
  }
#undef TYLO_SM_LAUNCH
  // rows too long for one CTA's registers: the two-pass form (backward of 4096 x 32768 bf16: 4,952 GB/s with a clustered
  // register-resident form, 6,225 with this one at 1,024 threads; 5,317 at 512 and 4,042 at 256 threads)
  if constexpr (FWD) {
    // more than 8,192 packets and fewer rows than SMs: each over the largest cluster of 8, 4 or 2 CTAs that leaves an SM per CTA, an
    // eighth of the SMs kept back (clusters do not span the chip's processor groups: 18 clusters of 8 took two waves, 22.5 us for 14.3).
    // fp32, cold, us, one CTA / cluster: 65,536 elements x 1 row 18.4 / 12.3, x 64 18.4 / 16.3; 131,072 x 1 28.7 / 12.3, x 64
    // 30.7 / 24.6; 2^20 x 1 166 / 31.  At 3,072 and 4,096 packets the cluster's two barriers cost more than they save (10.2 / 12.3).
    // Up to 8,192 packets and a quarter as many rows as SMs: clusters of 4 or 8 CTAs of 256 threads that hold the row in registers.
    // us back to back, one CTA / cluster: fp32 16,384 elements x 1 row 5.2 / 4.6, 32,768 x 1 7.1 / 4.7, x 32 7.2 / 6.6; bf16 65,536 x 1
    // 8.8 / 4.7, x 37 9.0 / 7.2.
    auto clusters = [&](auto kern, unsigned c, unsigned threads) -> int32_t {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)N * c); cfg.blockDim = dim3(threads); cfg.stream = st;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr; cfg.numAttrs = 1;
      TYLO_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, (T*)out, (const T*)a, M));
      return TYLO_OK;
    };
    if (nvec <= 8192 && N <= sm_count() / 4)
      return clusters(softmax_fwd_twopass_kernel<T, 256, RAGGED, true, true>, nvec <= 4096 ? 4 : 8, 256);
    unsigned c = nvec > 8192 ? 8 : 1;
    while (c > 1 && 8 * c * N > 7 * sm_count()) c /= 2;
    if (c > 1) return clusters(softmax_fwd_twopass_kernel<T, 1024, RAGGED, true, false>, c, 1024);
    softmax_fwd_twopass_kernel<T, 1024, RAGGED, false, false><<<(unsigned)N, 1024, 0, st>>>((T*)out, (const T*)a, M);
  }
  else softmax_bwd_twopass_kernel<T, 1024, RAGGED><<<(unsigned)N, 1024, 0, st>>>((T*)out, (const T*)a, (const T*)b, M);
  return check_launch(what);
}

}  // namespace tylo

using namespace tylo;

extern "C" int32_t tylo_b200_softmax_fwd(void* Y, const void* X, int64_t M, int64_t N, int32_t dtype,
                                         tylo_stream_t stream) {
  TYLO_REQUIRE(Y && X, TYLO_ERR_INVALID_ARGUMENT, "softmax_fwd: Y and X must be non-null");
  TYLO_REQUIRE(M > 0 && N > 0, TYLO_ERR_INVALID_ARGUMENT, "softmax_fwd: extents must be positive (M=%lld, N=%lld)",
               (long long)M, (long long)N);
  TYLO_REQUIRE(N <= 0x7fffffffLL, TYLO_ERR_UNSUPPORTED, "softmax_fwd: N above 2^31-1 is not supported");
  TYLO_REQUIRE(aligned16(Y) && aligned16(X), TYLO_ERR_MISALIGNED, "softmax_fwd: pointers must be 16-byte aligned");
  TYLO_DISPATCH_DTYPE(dtype, T, return (M % Elem<T>::kVec ? softmax_launch<T, true, true>(Y, X, nullptr, M, N, (cudaStream_t)stream)
                                                       : softmax_launch<T, true, false>(Y, X, nullptr, M, N, (cudaStream_t)stream)));
  return TYLO_OK;
}

extern "C" int32_t tylo_b200_softmax_bwd(void* dX, const void* dY, const void* Y, int64_t M, int64_t N,
                                         int32_t dtype, tylo_stream_t stream) {
  TYLO_REQUIRE(dX && dY && Y, TYLO_ERR_INVALID_ARGUMENT, "softmax_bwd: dX, dY and Y must be non-null");
  TYLO_REQUIRE(M > 0 && N > 0, TYLO_ERR_INVALID_ARGUMENT, "softmax_bwd: extents must be positive (M=%lld, N=%lld)",
               (long long)M, (long long)N);
  TYLO_REQUIRE(N <= 0x7fffffffLL, TYLO_ERR_UNSUPPORTED, "softmax_bwd: N above 2^31-1 is not supported");
  TYLO_REQUIRE(aligned16(dX) && aligned16(dY) && aligned16(Y), TYLO_ERR_MISALIGNED,
               "softmax_bwd: pointers must be 16-byte aligned");
  // argument order of the kernel: (dX, dY, Y)
  TYLO_DISPATCH_DTYPE(dtype, T, return (M % Elem<T>::kVec ? softmax_launch<T, false, true>(dX, dY, Y, M, N, (cudaStream_t)stream)
                                                       : softmax_launch<T, false, false>(dX, dY, Y, M, N, (cudaStream_t)stream)));
  return TYLO_OK;
}
