// RMSNorm and LayerNorm, forward and backward, for sm_100a.
//
// Forward: one pass over HBM (read X once, write Y once); the row lives in registers, the
// statistics are fp32.  LayerNorm's variance is the centred second moment computed from the
// registers, so it has the accuracy of the reference's three-pass kernel without its two
// extra reads (layer_norm.jl:6-46 reads X three times, rms_norm.jl:6-32 twice).
//
// Backward: `n_groups` CTAs stride over the rows.  Each keeps its partial dW (and dB) for the
// columns it owns in registers and writes one row of the fp32 partial buffer at the end; a
// second kernel sums the partial rows.  No locks, no atomics, deterministic
// (the reference serialises the groups on a global spin-lock: rms_norm.jl:68-78,
// layer_norm.jl:102-116).
#include "rowwise.cuh"
#include "sm100_ptx.cuh"


namespace tylo {

#define TYLO_ROW_DISPATCH(shape, ...)                                                          \
  do {                                                                                         \
    if ((shape).threads == 32) { constexpr int THREADS = 32, ITERS = 2; __VA_ARGS__; }                                \
    else if ((shape).threads == 64) { constexpr int THREADS = 64, ITERS = 2; __VA_ARGS__; }                           \
    else if ((shape).threads == 128 && (shape).iters == 2) { constexpr int THREADS = 128, ITERS = 2; __VA_ARGS__; }   \
    else if ((shape).threads == 128) { constexpr int THREADS = 128, ITERS = 4; __VA_ARGS__; }                         \
    else if ((shape).threads == 256) { constexpr int THREADS = 256, ITERS = 4; __VA_ARGS__; }                         \
    else if ((shape).threads == 512 && (shape).iters == 4) { constexpr int THREADS = 512, ITERS = 4; __VA_ARGS__; }   \
    else if ((shape).threads == 512) { constexpr int THREADS = 512, ITERS = 8; __VA_ARGS__; }                         \
    else { constexpr int THREADS = 1024, ITERS = 8; __VA_ARGS__; }                                                    \
  } while (0)

// Merge of two (count, mean, M2) partial statistics.
__device__ __forceinline__ void welford_merge(float& n, float& mu, float& m2, float nb, float mub, float m2b) {
  const float nt = n + nb;
  if (nt > 0.f) {
    const float d = mub - mu, f = nb / nt;
    mu += d * f;
    m2 += m2b + d * d * n * f;
  }
  n = nt;
}
// Same for partial statistics of EQUAL counts (every thread holds the same number of elements, the
// common case): no division, `half_n` = elements per side / 2 ... passed as the per-side count.
template <int THREADS>
__device__ __forceinline__ void welford_block_equal(float per_thread, float& mu, float& m2, float* scratch) {
  float n = per_thread;   // elements per side at this level
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float mub = __shfl_xor_sync(0xffffffffu, mu, o), m2b = __shfl_xor_sync(0xffffffffu, m2, o);
    const float d = mub - mu;
    mu = 0.5f * (mu + mub);
    m2 = m2 + m2b + d * d * (0.5f * n);
    n *= 2.f;
  }
  if constexpr (THREADS > 32) {
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { scratch[warp] = mu; scratch[32 + warp] = m2; }
    __syncthreads();
    mu = scratch[lane & (kWarps - 1)];
    m2 = scratch[32 + (lane & (kWarps - 1))];
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
      const float mub = __shfl_xor_sync(0xffffffffu, mu, o), m2b = __shfl_xor_sync(0xffffffffu, m2, o);
      const float d = mub - mu;
      mu = 0.5f * (mu + mub);
      m2 = m2 + m2b + d * d * (0.5f * n);
      n *= 2.f;
    }
  }
}

// All threads receive the block-wide (count, mean, M2).  `scratch` holds 96 floats.
template <int THREADS>
__device__ __forceinline__ void welford_block(float& n, float& mu, float& m2, float* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float nb = __shfl_xor_sync(0xffffffffu, n, o), mub = __shfl_xor_sync(0xffffffffu, mu, o),
                m2b = __shfl_xor_sync(0xffffffffu, m2, o);
    welford_merge(n, mu, m2, nb, mub, m2b);
  }
  if constexpr (THREADS > 32) {
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { scratch[warp] = n; scratch[32 + warp] = mu; scratch[64 + warp] = m2; }
    __syncthreads();
    n = lane < kWarps ? scratch[lane] : 0.f;
    mu = lane < kWarps ? scratch[32 + lane] : 0.f;
    m2 = lane < kWarps ? scratch[64 + lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float nb = __shfl_xor_sync(0xffffffffu, n, o), mub = __shfl_xor_sync(0xffffffffu, mu, o),
                  m2b = __shfl_xor_sync(0xffffffffu, m2, o);
      welford_merge(n, mu, m2, nb, mub, m2b);
    }
  }
  // the merge is not bit-commutative: every thread takes lane 0's result
  n = __shfl_sync(0xffffffffu, n, 0); mu = __shfl_sync(0xffffffffu, mu, 0); m2 = __shfl_sync(0xffffffffu, m2, 0);
}

// ------------------------------------------------------------------------------------------------
// forward, row in registers
// ------------------------------------------------------------------------------------------------
// (fp32 at 512 threads: two CTAs per SM are asked for; LayerNorm left alone takes 76 registers at 8 packets per thread, one CTA:
// 8,000 rows of 12,288 elements 236 us, 146 so)
template <typename T, int THREADS, int ITERS, bool LAYER>
__global__ void __launch_bounds__(row_cta(THREADS), sizeof(T) == 4 && THREADS == 512 ? 2 : 0)
norm_fwd_kernel(T* __restrict__ Y, const T* __restrict__ X, const T* __restrict__ W,
                const T* __restrict__ Bias, float* __restrict__ Mean, float* __restrict__ Rstd,
                int M, int N, float eps, float offset) {
  constexpr int VEC = Elem<T>::kVec;
  __shared__ float red[32];
  __shared__ float wred[LAYER ? 96 : 1];
  const int nvec = M / VEC, tid = row_thread<THREADS>();
  const size_t row = row_index<THREADS>();
  if (THREADS == 32 && row >= (size_t)N) return;
  RowRegs<T, THREADS, ITERS> x;
  x.load(X + row * M, nvec);

  const float inv_m = 1.0f / (float)M;
  float mean = 0.f;
  float ss = 0.f;
  if constexpr (LAYER) {
    // Per-thread mean and centred second moment from the registers, then ONE reduction round that
    // merges (count, mean, M2) triples (Chan et al.): centred accuracy without a second barrier.
    float cnt = 0.f, s = 0.f;
    // two elements per instruction (packed fp32 pairs): the kernel is close enough to the issue limit
    // for the instruction count to show in its bandwidth
    uint64_t s2 = 0ull;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
      if (i * THREADS + tid < nvec) {
        float f[VEC]; x.p[i].unpack(f);
#pragma unroll
        for (int j = 0; j < VEC; j += 2) s2 = sm100::add_f32x2(s2, sm100::pack_f32x2(f[j], f[j + 1]));
        cnt += (float)VEC;
      }
    }
    { float a, b; sm100::unpack_f32x2(s2, a, b); s = a + b; }
    float mu = cnt > 0.f ? s / cnt : 0.f, m2 = 0.f;
    const uint64_t nmu2 = sm100::pack_f32x2(-mu, -mu);
    uint64_t q2 = 0ull;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
      if (i * THREADS + tid < nvec) {
        float f[VEC]; x.p[i].unpack(f);
#pragma unroll
        for (int j = 0; j < VEC; j += 2) {
          const uint64_t c2 = sm100::add_f32x2(sm100::pack_f32x2(f[j], f[j + 1]), nmu2);
          q2 = sm100::fma_f32x2(c2, c2, q2);
        }
      }
    }
    { float a, b; sm100::unpack_f32x2(q2, a, b); m2 = a + b; }
    if (nvec == THREADS * ITERS) welford_block_equal<THREADS>((float)(ITERS * VEC), mu, m2, wred);
    else welford_block<THREADS>(cnt, mu, m2, wred);
    mean = mu; ss = m2;
  } else {
    uint64_t q2 = 0ull;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
      float f[VEC]; x.p[i].unpack(f);     // packets past the end are zero
#pragma unroll
      for (int j = 0; j < VEC; j += 2) {
        const uint64_t v2 = sm100::pack_f32x2(f[j], f[j + 1]);
        q2 = sm100::fma_f32x2(v2, v2, q2);
      }
    }
    { float a, b; sm100::unpack_f32x2(q2, a, b); ss = a + b; }
    ss = block_reduce<THREADS>(ss, SumOp(), 0.f, red);
  }
  const float rstd = 1.0f / sqrtf(ss * inv_m + eps);
  if (tid == 0) {
    if (Rstd) Rstd[row] = rstd;
    if (LAYER && Mean) Mean[row] = mean;
  }
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const int v = i * THREADS + tid;
    if (v < nvec) {
      float f[VEC], w[VEC], b[VEC];
      x.p[i].unpack(f);
      ld_param(W + (size_t)v * VEC).unpack(w);
      if constexpr (LAYER) ld_param(Bias + (size_t)v * VEC).unpack(b);
      if constexpr (LAYER) {
        // ((x - mean) rstd) w + b on pairs: (x + (-mean)) * (rstd w) + b
        const uint64_t nmean2 = sm100::pack_f32x2(-mean, -mean), rstd2 = sm100::pack_f32x2(rstd, rstd);
#pragma unroll
        for (int j = 0; j < VEC; j += 2) {
          const uint64_t c2 = sm100::add_f32x2(sm100::pack_f32x2(f[j], f[j + 1]), nmean2);
          const uint64_t a2 = sm100::mul_f32x2(sm100::pack_f32x2(w[j], w[j + 1]), rstd2);
          sm100::unpack_f32x2(sm100::fma_f32x2(c2, a2, sm100::pack_f32x2(b[j], b[j + 1])), f[j], f[j + 1]);
        }
      } else {
        const uint64_t rstd2 = sm100::pack_f32x2(rstd, rstd), off2 = sm100::pack_f32x2(offset, offset);
#pragma unroll
        for (int j = 0; j < VEC; j += 2) {
          const uint64_t a2 = sm100::mul_f32x2(sm100::add_f32x2(sm100::pack_f32x2(w[j], w[j + 1]), off2), rstd2);
          sm100::unpack_f32x2(sm100::mul_f32x2(sm100::pack_f32x2(f[j], f[j + 1]), a2), f[j], f[j + 1]);
        }
      }
      x.p[i].pack(f);
    }
  }
  x.store(Y + row * M, nvec);
}

// forward, any M and any row alignment: scalar accesses, X re-read from L2.
template <typename T, bool LAYER>
__global__ void __launch_bounds__(256)
norm_fwd_generic_kernel(T* __restrict__ Y, const T* __restrict__ X, const T* __restrict__ W,
                        const T* __restrict__ Bias, float* __restrict__ Mean,
                        float* __restrict__ Rstd, int64_t M, float eps, float offset) {
  __shared__ float red[32];
  const size_t row = blockIdx.x;
  const T* x = X + row * M;
  const float inv_m = 1.0f / (float)M;
  float mean = 0.f;
  if constexpr (LAYER) {
    float s = 0.f;
    for (int64_t i = threadIdx.x; i < M; i += 256) s += Elem<T>::to_f(x[i]);
    mean = block_reduce<256>(s, SumOp(), 0.f, red) * inv_m;
  }
  float ss = 0.f;
  for (int64_t i = threadIdx.x; i < M; i += 256) {
    const float c = Elem<T>::to_f(x[i]) - mean;
    ss += c * c;
  }
  ss = block_reduce<256>(ss, SumOp(), 0.f, red);
  const float rstd = 1.0f / sqrtf(ss * inv_m + eps);
  if (threadIdx.x == 0) {
    if (Rstd) Rstd[row] = rstd;
    if (LAYER && Mean) Mean[row] = mean;
  }
  for (int64_t i = threadIdx.x; i < M; i += 256) {
    const float f = Elem<T>::to_f(x[i]);
    float y;
    if constexpr (LAYER) y = (f - mean) * rstd * Elem<T>::to_f(W[i]) + Elem<T>::to_f(Bias[i]);
    else y = f * rstd * (Elem<T>::to_f(W[i]) + offset);
    Y[row * M + i] = Elem<T>::from_f(y);
  }
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
// backward, streaming form for rows of exactly THREADS packets (one 16-byte packet of X and of dY per
// thread): the per-thread state is a handful of registers, so the packets of the next TWO rows are
// already in flight while the current row is reduced — the HBM stream never waits for a reduction.
// One barrier per row (the reduction scratch is double-buffered).
template <typename T, int THREADS, bool LAYER>
__global__ void __launch_bounds__(THREADS)
norm_bwd_stream_kernel(T* __restrict__ dX, float* __restrict__ dWp, float* __restrict__ dBp,
                       const T* __restrict__ dY, const T* __restrict__ X, const T* __restrict__ W,
                       const float* __restrict__ Mean, const float* __restrict__ Rstd,
                       int M, int64_t N, float offset) {
  constexpr int VEC = Elem<T>::kVec;
  constexpr int kWarps = THREADS / 32;
  __shared__ float red[2][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t col = (size_t)threadIdx.x * VEC;
  const float inv_m = 1.0f / (float)M;
  float g[VEC], dw[VEC], db[VEC];
  ld_param(W + col).unpack(g);
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    if constexpr (!LAYER) g[j] += offset;
    dw[j] = 0.f; db[j] = 0.f;
  }
  const int64_t stride = gridDim.x;
  Pack<T> x0, d0, x1, d1, x2, d2;
  float r0 = 0.f, r1 = 0.f, r2 = 0.f, m0 = 0.f, m1 = 0.f, m2 = 0.f;
  auto fetch = [&](int64_t r, Pack<T>& x, Pack<T>& d, float& rs, float& mn) {
    if (r < N) {
      x.raw = ld_stream(X + r * M + col); d.raw = ld_stream(dY + r * M + col);
      rs = Rstd[r];
      mn = LAYER ? Mean[r] : 0.f;
    }
  };
  int64_t row = blockIdx.x;
  // rows in flight behind the current one: two for RMSNorm, one for LayerNorm (its extra accumulators
  // and statistics would otherwise push the 1024-thread CTA past 64 registers per thread)
  fetch(row, x0, d0, r0, m0);
  if constexpr (!LAYER) fetch(row + stride, x1, d1, r1, m1);
  for (int par = 0; row < N; row += stride, par ^= 1) {
    if constexpr (LAYER) fetch(row + stride, x1, d1, r1, m1);
    else fetch(row + 2 * stride, x2, d2, r2, m2);
    float s1 = 0.f, s2 = 0.f;
    const uint64_t nm2 = sm100::pack_f32x2(-m0, -m0), r2p = sm100::pack_f32x2(r0, r0);
    {
      // packed fp32 pairs: xhat = (x - mean) rstd, gd = g dy, s1 += xhat gd, s2 += gd
      float xf[VEC], df[VEC];
      x0.unpack(xf); d0.unpack(df);
      uint64_t a1 = 0ull, a2 = 0ull;
#pragma unroll
      for (int j = 0; j < VEC; j += 2) {
        const uint64_t gd2 = sm100::mul_f32x2(sm100::pack_f32x2(g[j], g[j + 1]), sm100::pack_f32x2(df[j], df[j + 1]));
        const uint64_t xh2 = sm100::mul_f32x2(sm100::add_f32x2(sm100::pack_f32x2(xf[j], xf[j + 1]), nm2), r2p);
        a1 = sm100::fma_f32x2(xh2, gd2, a1);
        if constexpr (LAYER) a2 = sm100::add_f32x2(a2, gd2);
      }
      float lo, hi;
      sm100::unpack_f32x2(a1, lo, hi); s1 = lo + hi;
      if constexpr (LAYER) { sm100::unpack_f32x2(a2, lo, hi); s2 = lo + hi; }
    }
    s1 = warp_reduce(s1, SumOp());
    if constexpr (LAYER) s2 = warp_reduce(s2, SumOp());
    if (lane == 0) { red[par][warp] = s1; red[par][32 + warp] = s2; }
    __syncthreads();
    s1 = warp_reduce(lane < kWarps ? red[par][lane] : 0.f, SumOp());
    if constexpr (LAYER) s2 = warp_reduce(lane < kWarps ? red[par][32 + lane] : 0.f, SumOp());
    const float c1 = s1 * inv_m, c2 = LAYER ? s2 * inv_m : 0.f;
    // the packets are unpacked again rather than kept as fp32 across the barrier (registers)
    float xf[VEC], df[VEC], o[VEC];
    x0.unpack(xf); d0.unpack(df);
    const uint64_t nc1 = sm100::pack_f32x2(-c1, -c1), nc2 = sm100::pack_f32x2(-c2, -c2);
#pragma unroll
    for (int j = 0; j < VEC; j += 2) {
      // same formulas as norm_bwd_kernel, two columns per instruction:
      // dx = (g dy - (xhat c1 + c2)) rstd,  dW += dy xhat,  dB += dy
      const uint64_t df2 = sm100::pack_f32x2(df[j], df[j + 1]);
      const uint64_t xh2 = sm100::mul_f32x2(sm100::add_f32x2(sm100::pack_f32x2(xf[j], xf[j + 1]), nm2), r2p);
      const uint64_t t2 = sm100::fma_f32x2(xh2, nc1, nc2);
      const uint64_t o2 = sm100::mul_f32x2(sm100::fma_f32x2(sm100::pack_f32x2(g[j], g[j + 1]), df2, t2), r2p);
      sm100::unpack_f32x2(o2, o[j], o[j + 1]);
      const uint64_t w2 = sm100::fma_f32x2(df2, xh2, sm100::pack_f32x2(dw[j], dw[j + 1]));
      sm100::unpack_f32x2(w2, dw[j], dw[j + 1]);
      if constexpr (LAYER) {
        const uint64_t b2 = sm100::add_f32x2(sm100::pack_f32x2(db[j], db[j + 1]), df2);
        sm100::unpack_f32x2(b2, db[j], db[j + 1]);
      }
    }
    Pack<T> out; out.pack(o);
    st_stream(dX + row * M + col, out.raw);
    x0 = x1; d0 = d1; r0 = r1; m0 = m1;
    if constexpr (!LAYER) { x1 = x2; d1 = d2; r1 = r2; m1 = m2; }
  }
  float4* pw = reinterpret_cast<float4*>(dWp + (size_t)blockIdx.x * M + col);
#pragma unroll
  for (int j = 0; j < VEC; j += 4) pw[j / 4] = make_float4(dw[j], dw[j + 1], dw[j + 2], dw[j + 3]);
  if constexpr (LAYER) {
    float4* pb = reinterpret_cast<float4*>(dBp + (size_t)blockIdx.x * M + col);
#pragma unroll
    for (int j = 0; j < VEC; j += 4) pb[j / 4] = make_float4(db[j], db[j + 1], db[j + 2], db[j + 3]);
  }
}

// Rows of up to 1,024 packets: one 16-byte packet of X and dY per thread, TPR threads (whole warps) per row, R rows per CTA at
// a time.  HBM bound; what it takes is bytes in flight, so short rows share a CTA (a 512-element bf16 row is 64 threads:
// alone in its CTA it left 2 warps per SM, 8 rows give 32) and every row group asks for its next one or two rows before it
// reduces the current one, so that the stream never waits for a reduction.  One named barrier per row (scratch is
// double-buffered); none when a row is one warp.  dW / dB partials stay in registers and are added up over the R groups
// through shared memory at the end.
constexpr int kMaxSmem = 220 * 1024;    // dynamic shared memory asked for at most
constexpr int kNormRowGroups = 15;      // named barriers 1..15

//
// TPR: a thread count known to the compiler, one row per CTA; 0: tpr and R of the launch, which costs registers (in 16 bits the 64
// of a 1,024-thread CTA do not hold the row loop without spills).  FULL: every thread of a row holds a packet.
template <typename T, int TPR, bool LAYER, bool FULL>
__global__ void __launch_bounds__(TPR ? TPR : 1024, TPR == 512 || (TPR && sizeof(T) == 4) ? 2 : 1)
norm_bwd_kernel(T* __restrict__ dX, float* __restrict__ dWp, float* __restrict__ dBp, const T* __restrict__ dY,
                const T* __restrict__ X, const T* __restrict__ W, const float* __restrict__ Mean,
                const float* __restrict__ Rstd, int M, int N, float offset, int tpr_, int R_) {
  constexpr int VEC = Elem<T>::kVec;
  extern __shared__ __align__(16) float sm[];
  const int tpr = TPR ? TPR : tpr_, R = TPR ? 1 : R_;
  const int nvec = FULL ? tpr : M / VEC, wpr = tpr >> 5;
  const int rg = TPR ? 0 : threadIdx.x / tpr, v = TPR ? threadIdx.x : threadIdx.x % tpr, lane = threadIdx.x & 31, wr = v >> 5;
  float* red = sm + rg * 2 * 64;               // [parity][64]
  float* tot = sm + R * 2 * 64;                // the CTA's dW (and dB) partials, R > 1
  // threads past the row's end read its last packet (no branch around the loads) and take no part in the sums and stores
  const bool live = FULL || v < nvec;
  const int col = (live ? v : nvec - 1) * VEC;
  const float inv_m = 1.0f / (float)M;
  float g[VEC], dw[VEC], db[VEC];
  ld_param(W + col).unpack(g);
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    if constexpr (!LAYER) g[j] += offset;
    dw[j] = 0.f; db[j] = 0.f;
  }
  // rows are counted in unsigned: N may be 2^31 - 1, and the row asked for ahead lies up to 2 x 296 x 15 beyond (see the launch)
  const unsigned stride = gridDim.x * (unsigned)R, rows = (unsigned)N;
  Pack<T> x0, d0, x1, d1, x2, d2;
  x0.raw = d0.raw = x1.raw = d1.raw = x2.raw = d2.raw = make_uint4(0, 0, 0, 0);
  float r0 = 0.f, r1 = 0.f, r2 = 0.f, m0 = 0.f, m1 = 0.f, m2 = 0.f;
  auto fetch = [&](unsigned r, Pack<T>& x, Pack<T>& d, float& rs, float& mn) {
    if (r < rows) {
      x.raw = ld_stream(X + (size_t)r * M + col); d.raw = ld_stream(dY + (size_t)r * M + col);
      rs = Rstd[r];
      mn = LAYER ? Mean[r] : 0.f;
    }
  };
  // rows in flight behind the current one: two for RMSNorm; one for LayerNorm (its extra accumulators and statistics would push
  // the 1024-thread CTA past 64 registers per thread) and in 16 bits with launch-time counts (rms bf16 512: 180 us with two, 144)
  constexpr bool kTwo = !LAYER && (TPR || VEC == 4);
  unsigned row = blockIdx.x * (unsigned)R + rg;
  fetch(row, x0, d0, r0, m0);
  if constexpr (kTwo) fetch(row + stride, x1, d1, r1, m1);
  for (int par = 0; row < rows; row += stride, par ^= 1) {
    if constexpr (!kTwo) fetch(row + stride, x1, d1, r1, m1);
    else fetch(row + 2 * stride, x2, d2, r2, m2);
    float s1 = 0.f, s2 = 0.f;
    const uint64_t nm2 = sm100::pack_f32x2(-m0, -m0), r2p = sm100::pack_f32x2(r0, r0);
    {
      // packed fp32 pairs: xhat = (x - mean) rstd, gd = g dy, s1 += xhat gd, s2 += gd
      float xf[VEC], df[VEC];
      x0.unpack(xf); d0.unpack(df);
      uint64_t a1 = 0ull, a2 = 0ull;
#pragma unroll
      for (int j = 0; j < VEC; j += 2) {
        const uint64_t gd2 = sm100::mul_f32x2(sm100::pack_f32x2(g[j], g[j + 1]), sm100::pack_f32x2(df[j], df[j + 1]));
        const uint64_t xh2 = sm100::mul_f32x2(sm100::add_f32x2(sm100::pack_f32x2(xf[j], xf[j + 1]), nm2), r2p);
        a1 = sm100::fma_f32x2(xh2, gd2, a1);
        if constexpr (LAYER) a2 = sm100::add_f32x2(a2, gd2);
      }
      float lo, hi;
      sm100::unpack_f32x2(a1, lo, hi); s1 = lo + hi;
      if constexpr (LAYER) { sm100::unpack_f32x2(a2, lo, hi); s2 = lo + hi; }
      if (!live) { s1 = 0.f; s2 = 0.f; }
    }
    s1 = warp_reduce(s1, SumOp());
    if constexpr (LAYER) s2 = warp_reduce(s2, SumOp());
    if (wpr > 1) {
      float* rp = red + par * 64;
      if (lane == 0) { rp[wr] = s1; rp[32 + wr] = s2; }
      if constexpr (TPR) __syncthreads();
      else asm volatile("bar.sync %0, %1;" ::"r"(rg + 1), "r"(tpr) : "memory");
      s1 = warp_reduce(lane < wpr ? rp[lane] : 0.f, SumOp());
      if constexpr (LAYER) s2 = warp_reduce(lane < wpr ? rp[32 + lane] : 0.f, SumOp());
    }
    const float c1 = s1 * inv_m, c2 = LAYER ? s2 * inv_m : 0.f;
    // the packets are unpacked again rather than kept as fp32 across the barrier (registers)
    float xf[VEC], df[VEC], o[VEC];
    x0.unpack(xf); d0.unpack(df);
    const uint64_t nc1 = sm100::pack_f32x2(-c1, -c1), nc2 = sm100::pack_f32x2(-c2, -c2);
#pragma unroll
    for (int j = 0; j < VEC; j += 2) {
      // RMS: rstd*(dy*g - rstd^2*dd*x) with xhat = x*rstd, c1 = rstd*dd  (test/norm.jl:78-87)
      // LN : (g*dy - (xhat*c1 + c2))*rstd                                  (test/norm.jl:90-102)
      // two columns per instruction; dW += dy xhat,  dB += dy
      const uint64_t df2 = sm100::pack_f32x2(df[j], df[j + 1]);
      const uint64_t xh2 = sm100::mul_f32x2(sm100::add_f32x2(sm100::pack_f32x2(xf[j], xf[j + 1]), nm2), r2p);
      const uint64_t t2 = sm100::fma_f32x2(xh2, nc1, nc2);
      const uint64_t o2 = sm100::mul_f32x2(sm100::fma_f32x2(sm100::pack_f32x2(g[j], g[j + 1]), df2, t2), r2p);
      sm100::unpack_f32x2(o2, o[j], o[j + 1]);
      const uint64_t w2 = sm100::fma_f32x2(df2, xh2, sm100::pack_f32x2(dw[j], dw[j + 1]));
      sm100::unpack_f32x2(w2, dw[j], dw[j + 1]);
      if constexpr (LAYER) {
        const uint64_t b2 = sm100::add_f32x2(sm100::pack_f32x2(db[j], db[j + 1]), df2);
        sm100::unpack_f32x2(b2, db[j], db[j + 1]);
      }
    }
    Pack<T> out; out.pack(o);
    if (live) st_stream(dX + (size_t)row * M + col, out.raw);
    x0 = x1; d0 = d1; r0 = r1; m0 = m1;
    if constexpr (kTwo) { x1 = x2; d1 = d2; r1 = r2; m1 = m2; }
  }
  // sum over the row groups, in their order
  for (int k = 1; k < R; ++k) {
    if (rg == k && live) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) { tot[col + j] = dw[j]; if constexpr (LAYER) tot[M + col + j] = db[j]; }
    }
    __syncthreads();
    if (rg == 0 && live) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) { dw[j] += tot[col + j]; if constexpr (LAYER) db[j] += tot[M + col + j]; }
    }
    __syncthreads();
  }
  if (rg == 0 && live) {
    float4* pw = reinterpret_cast<float4*>(dWp + (size_t)blockIdx.x * M + col);
#pragma unroll
    for (int j = 0; j < VEC; j += 4) pw[j / 4] = make_float4(dw[j], dw[j + 1], dw[j + 2], dw[j + 3]);
    if constexpr (LAYER) {
      float4* pb = reinterpret_cast<float4*>(dBp + (size_t)blockIdx.x * M + col);
#pragma unroll
      for (int j = 0; j < VEC; j += 4) pb[j / 4] = make_float4(db[j], db[j + 1], db[j + 2], db[j + 3]);
    }
  }
}

// Longer rows (up to 4,096 packets, as long as the accumulators fit shared memory): P packets per thread, one row per CTA at
// a time, dW / dB partials in shared memory (each thread is the only one to touch its columns), the weights re-read from
// the first-level cache.
template <typename T, int P, bool LAYER>
__global__ void __launch_bounds__(1024)
norm_bwd_wide_kernel(T* __restrict__ dX, float* __restrict__ dWp, float* __restrict__ dBp, const T* __restrict__ dY,
                     const T* __restrict__ X, const T* __restrict__ W, const float* __restrict__ Mean,
                     const float* __restrict__ Rstd, int M, int64_t N, float offset) {
  constexpr int VEC = Elem<T>::kVec;
  extern __shared__ __align__(16) float sm[];
  const int nvec = M / VEC, nt = blockDim.x, wpr = nt >> 5, lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
  float* red = sm;
  float* aw = sm + 128;
  float* ab = aw + M;
  const float inv_m = 1.0f / (float)M;
  for (int i = threadIdx.x; i < (LAYER ? 2 : 1) * M; i += nt) aw[i] = 0.f;
  __syncthreads();
  int par = 0;
  for (int64_t row = blockIdx.x; row < N; row += gridDim.x, par ^= 1) {
    Pack<T> x[P], d[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int v = i * nt + threadIdx.x;
      x[i].raw = d[i].raw = make_uint4(0, 0, 0, 0);
      if (v < nvec) { x[i].raw = ld_stream(X + row * M + (size_t)v * VEC); d[i].raw = ld_stream(dY + row * M + (size_t)v * VEC); }
    }
    const float rstd = Rstd[row], mean = LAYER ? Mean[row] : 0.f;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int v = i * nt + threadIdx.x;
      if (v < nvec) {
        float xf[VEC], df[VEC], g[VEC];
        x[i].unpack(xf); d[i].unpack(df); ld_param(W + (size_t)v * VEC).unpack(g);
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          const float gd = (LAYER ? g[j] : g[j] + offset) * df[j];
          s1 += (xf[j] - mean) * rstd * gd;
          if constexpr (LAYER) s2 += gd;
        }
      }
    }
    s1 = warp_reduce(s1, SumOp());
    if constexpr (LAYER) s2 = warp_reduce(s2, SumOp());
    float* rp = red + par * 64;
    if (lane == 0) { rp[wr] = s1; rp[32 + wr] = s2; }
    __syncthreads();
    s1 = warp_reduce(lane < wpr ? rp[lane] : 0.f, SumOp());
    if constexpr (LAYER) s2 = warp_reduce(lane < wpr ? rp[32 + lane] : 0.f, SumOp());
    const float c1 = s1 * inv_m, c2 = LAYER ? s2 * inv_m : 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int v = i * nt + threadIdx.x;
      if (v < nvec) {
        float xf[VEC], df[VEC], g[VEC], o[VEC];
        x[i].unpack(xf); d[i].unpack(df); ld_param(W + (size_t)v * VEC).unpack(g);
        float4* pw = reinterpret_cast<float4*>(aw + (size_t)v * VEC);
        float4* pb = reinterpret_cast<float4*>(ab + (size_t)v * VEC);
#pragma unroll
        for (int q = 0; q < VEC; q += 4) {
          float xh[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            xh[e] = (xf[q + e] - mean) * rstd;
            o[q + e] = ((LAYER ? g[q + e] : g[q + e] + offset) * df[q + e] - (xh[e] * c1 + c2)) * rstd;
          }
          float4 w = pw[q / 4];
          w.x += df[q] * xh[0]; w.y += df[q + 1] * xh[1]; w.z += df[q + 2] * xh[2]; w.w += df[q + 3] * xh[3];
          pw[q / 4] = w;
          if constexpr (LAYER) {
            float4 b = pb[q / 4];
            b.x += df[q]; b.y += df[q + 1]; b.z += df[q + 2]; b.w += df[q + 3];
            pb[q / 4] = b;
          }
        }
        Pack<T> out; out.pack(o);
        st_stream(dX + row * M + (size_t)v * VEC, out.raw);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int v = i * nt + threadIdx.x;
    if (v < nvec) {
#pragma unroll
      for (int q = 0; q < VEC; q += 4) {
        const size_t c = (size_t)v * VEC + q;
        *reinterpret_cast<float4*>(dWp + (size_t)blockIdx.x * M + c) = *reinterpret_cast<const float4*>(aw + c);
        if constexpr (LAYER) *reinterpret_cast<float4*>(dBp + (size_t)blockIdx.x * M + c) = *reinterpret_cast<const float4*>(ab + c);
      }
    }
  }
}

// Any M / alignment: element accesses.  While the row and the partials of several CTAs fit shared memory (SMEM), X and dY are read from
// memory once, the row waits in shared memory as fp32 and the partials are added up there; beyond that the CTA's partial row
// is accumulated in global memory (the CTA is its only writer) and the row read twice.
template <typename T, bool LAYER, bool SMEM>
__global__ void __launch_bounds__(512)
norm_bwd_generic_kernel(T* __restrict__ dX, float* __restrict__ dWp, float* __restrict__ dBp,
                        const T* __restrict__ dY, const T* __restrict__ X,
                        const T* __restrict__ W, const float* __restrict__ Mean,
                        const float* __restrict__ Rstd, int64_t M, int64_t N, float offset) {
  constexpr int NT = 512, U = 4;
  __shared__ float red[64];
  extern __shared__ __align__(16) float sm[];
  const float inv_m = 1.0f / (float)M;
  float* mw = SMEM ? sm : dWp + (size_t)blockIdx.x * M;
  float* mb = !LAYER ? nullptr : (SMEM ? sm + M : dBp + (size_t)blockIdx.x * M);
  float* cx = sm + (LAYER ? 2 : 1) * M;        // xhat and dy of the row
  float* cd = cx + M;
  for (int64_t i = threadIdx.x; i < M; i += NT) { mw[i] = 0.f; if (LAYER) mb[i] = 0.f; }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t row = blockIdx.x; row < N; row += gridDim.x) {
    const T* x = X + row * M; const T* dy = dY + row * M;
    const float rstd = Rstd[row];
    const float mean = LAYER ? Mean[row] : 0.f;
    float s1 = 0.f, s2 = 0.f;
    for (int64_t i0 = threadIdx.x; i0 < M; i0 += NT * U) {
      float xv[U], dv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * NT;
        xv[u] = i < M ? Elem<T>::to_f(x[i]) : mean;
        dv[u] = i < M ? Elem<T>::to_f(dy[i]) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * NT;
        if (i < M) {
          const float xh = (xv[u] - mean) * rstd, gd = (Elem<T>::to_f(W[i]) + (LAYER ? 0.f : offset)) * dv[u];
          s1 += xh * gd;
          s2 += gd;
          if (SMEM) { cx[i] = xh; cd[i] = dv[u]; }
        }
      }
    }
    s1 = warp_reduce(s1, SumOp());
    s2 = warp_reduce(s2, SumOp());
    if (lane == 0) { red[warp] = s1; red[32 + warp] = s2; }
    __syncthreads();
    const float c1 = warp_reduce(lane < NT / 32 ? red[lane] : 0.f, SumOp()) * inv_m;
    const float c2 = LAYER ? warp_reduce(lane < NT / 32 ? red[32 + lane] : 0.f, SumOp()) * inv_m : 0.f;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < M; i += NT) {
      const float gi = Elem<T>::to_f(W[i]) + (LAYER ? 0.f : offset);
      const float d = SMEM ? cd[i] : Elem<T>::to_f(dy[i]);
      const float xhat = SMEM ? cx[i] : (Elem<T>::to_f(x[i]) - mean) * rstd;
      dX[row * M + i] = Elem<T>::from_f((gi * d - (xhat * c1 + c2)) * rstd);
      mw[i] += d * xhat;
      if (LAYER) mb[i] += d;
    }
  }
  if (SMEM)
    for (int64_t i = threadIdx.x; i < M; i += NT) {
      dWp[(size_t)blockIdx.x * M + i] = mw[i];
      if (LAYER) dBp[(size_t)blockIdx.x * M + i] = mb[i];
    }
}

// second stage: dW[m] = sum over groups of the partial rows.  32 columns x 32 group lanes per CTA, four rows in flight per
// lane: at 768 columns only 24 CTAs run, and eight lanes adding 37 rows one after the other took 13 us of waiting.
template <typename T>
__global__ void __launch_bounds__(1024)
norm_bwd_reduce_kernel(T* __restrict__ dW, T* __restrict__ dB, const float* __restrict__ dWp,
                       const float* __restrict__ dBp, int64_t M, int n_groups) {
  __shared__ float sw[32][33], sb[32][33];
  const int col = threadIdx.x & 31, gl = threadIdx.x >> 5;
  const int64_t m = (int64_t)blockIdx.x * 32 + col;
  float aw = 0.f, ab = 0.f;
  if (m < M) {
#pragma unroll 4
    for (int g = gl; g < n_groups; g += 32) {
      aw += dWp[(size_t)g * M + m];
      if (dBp) ab += dBp[(size_t)g * M + m];
    }
  }
  sw[gl][col] = aw; sb[gl][col] = ab;
  __syncthreads();
  // warp gl sums column gl over its 32 lanes
  const float tw = warp_reduce(sw[col][gl], SumOp()), tb = warp_reduce(sb[col][gl], SumOp());
  const int64_t mo = (int64_t)blockIdx.x * 32 + gl;
  if (col == 0 && mo < M) {
    dW[mo] = Elem<T>::from_f(tw);
    if (dBp) dB[mo] = Elem<T>::from_f(tb);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// More than 48 KB of shared memory has to be asked for; below that the call would only cost the host time.  The 48 KB hold a
// kernel's static arrays too, so the line for the dynamic part lies 1 KB lower (the kernels here have at most 256 bytes of them).
template <typename K> static int32_t allow_smem(K kern, int64_t bytes) {
  if (bytes > 47 * 1024) TYLO_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return TYLO_OK;
}

template <typename T, bool LAYER>
static int32_t norm_fwd_launch(void* Y, const void* X, const void* W, const void* Bias, float* Mean,
                               float* Rstd, int64_t M, int64_t N, float eps, float offset,
                               cudaStream_t st) {
  constexpr int VEC = Elem<T>::kVec;
  RowShape shape;
  if (M % VEC == 0 && pick_row_shape(M / VEC, &shape)) {
    TYLO_ROW_DISPATCH(shape, norm_fwd_kernel<T, THREADS, ITERS, LAYER><<<row_grid(THREADS, N), row_cta(THREADS), 0, st>>>(
        (T*)Y, (const T*)X, (const T*)W, (const T*)Bias, Mean, Rstd, (int)M, (int)N, eps, offset));
  } else {
    norm_fwd_generic_kernel<T, LAYER><<<(unsigned)N, 256, 0, st>>>(
        (T*)Y, (const T*)X, (const T*)W, (const T*)Bias, Mean, Rstd, M, eps, offset);
  }
  return check_launch(LAYER ? "layer_norm_fwd" : "rms_norm_fwd");
}

template <typename T, bool LAYER>
static int32_t norm_bwd_launch(void* dX, void* dW, void* dB, const void* dY, const void* X,
                               const void* W, const float* Mean, const float* Rstd, float* dWp,
                               float* dBp, int n_groups, int64_t M, int64_t N, float offset,
                               cudaStream_t st) {
  constexpr int VEC = Elem<T>::kVec;
  const int sms = sm_count();
  const char* what = LAYER ? "layer_norm_bwd" : "rms_norm_bwd";
  const int64_t nvec = M % VEC == 0 ? M / VEC : 0;
  const int64_t acc_bytes = (LAYER ? 2 : 1) * M * 4;
  auto walkers = [&](int64_t rows, int per_sm) {     // CTAs: no more than there are rows or partial rows, or fit at once
    int64_t g = n_groups < rows ? n_groups : rows;
    return (unsigned)(g < (int64_t)sms * per_sm ? g : (int64_t)sms * per_sm);
  };
  unsigned grid;
  if (nvec == 1024 || nvec == 512) {
    // a kernel of their own for whole CTAs: 2^27 bytes of X in us, backward, here / in norm_bwd_kernel at 1,024 or 512 threads: RMS
    // bf16 1,024 packets 152 / 160, 512 149 / 152, fp32 512 145 / 152; LayerNorm is level (172 / 172, 160 / 158)
    grid = walkers(N, nvec == 1024 ? 1 : 2);
    if (nvec == 1024)
      norm_bwd_stream_kernel<T, 1024, LAYER><<<grid, 1024, 0, st>>>(
          (T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, (int)M, N, offset);
    else
      norm_bwd_stream_kernel<T, 512, LAYER><<<grid, 512, 0, st>>>(
          (T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, (int)M, N, offset);
  } else if (nvec > (VEC == 8 ? 256 : 512) && nvec <= (VEC == 8 ? 1024 : 768)) {
    // thread counts known to the compiler, up to a quarter of them idle; fp32 fits two such CTAs per SM.  us, launch-time counts /
    // these: RMS bf16 300 packets 290 / 219, 513 347 / 208, 1,000 245 / 166; LayerNorm bf16 1,000 273 / 173; fp32 RMS 513 209 / 162,
    // 768 164 / 137 (850 at 896 threads, where only one CTA fits, 167 / 166: left on launch-time counts)
    auto run = [&](auto kern, int threads, int per_sm) {
      grid = walkers(N, per_sm);
      kern<<<grid, threads, 2 * 64 * 4, st>>>((T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, (int)M, (int)N, offset, 0, 1);
    };
    if constexpr (VEC == 8) {
      if (nvec <= 512) run(norm_bwd_kernel<T, 512, LAYER, false>, 512, 2);
      else if (nvec <= 640) run(norm_bwd_kernel<T, 640, LAYER, false>, 640, 1);
      else if (nvec <= 768) run(norm_bwd_kernel<T, 768, LAYER, false>, 768, 1);
      else if (nvec <= 896) run(norm_bwd_kernel<T, 896, LAYER, false>, 896, 1);
      else run(norm_bwd_kernel<T, 1024, LAYER, false>, 1024, 1);
    } else {
      if (nvec <= 640) run(norm_bwd_kernel<T, 640, LAYER, false>, 640, 2);
      else run(norm_bwd_kernel<T, 768, LAYER, false>, 768, 2);
    }
  } else if (nvec >= 1 && nvec <= 1024) {
    const int tpr = (int)(nvec + 31) / 32 * 32;
    // as many rows per CTA as make 512 threads, fewer when there are not enough rows to occupy every SM with that
    int R = 512 / tpr;
    if (R > kNormRowGroups) R = kNormRowGroups;
    const int64_t per_sm = (N + sms - 1) / sms;
    if (R > per_sm) R = (int)per_sm;
    if (R < 1) R = 1;
    grid = walkers((N + R - 1) / R, tpr * R > 512 ? 1 : 2);
    const size_t smem = (size_t)R * 2 * 64 * 4 + (R > 1 ? acc_bytes : 0);
    auto kern = nvec == tpr ? norm_bwd_kernel<T, 0, LAYER, true> : norm_bwd_kernel<T, 0, LAYER, false>;
    // (several rows per CTA means rows of at most 256 packets: below the 48 KB that need no attribute)
    kern<<<grid, tpr * R, smem, st>>>((T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, (int)M, (int)N,
                                      offset, tpr, R);
  } else if (nvec > 1024 && nvec <= 4096 && acc_bytes + 512 <= kMaxSmem) {
    grid = walkers(N, 1);
#define TYLO_BWD_WIDE(P)                                                                                              \
  do {                                                                                                                \
    auto kern = norm_bwd_wide_kernel<T, P, LAYER>;                                                                    \
    if (int32_t rc = allow_smem(kern, acc_bytes + 512)) return rc;                                                    \
    kern<<<grid, (unsigned)((nvec + P - 1) / P + 31) / 32 * 32, acc_bytes + 512, st>>>(                               \
        (T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, (int)M, N, offset);                     \
  } while (0)
    if (nvec <= 2048) TYLO_BWD_WIDE(2); else TYLO_BWD_WIDE(4);
#undef TYLO_BWD_WIDE
  } else {
    // through shared memory while three CTAs (RMSNorm) or two (LayerNorm, whose partials are twice the traffic in global memory) fit
    // an SM; with fewer, the rows wait for one another longer than the second read takes.  us, shared / global memory, 2^26
    // elements: RMSNorm bf16 7,001 elements 333 / 291, 16,383 576 / 320, fp32 9,401 723 / 375; LayerNorm bf16 7,001 (two CTAs)
    // 342 / 415, 8,101 (one) 575 / 430.
    const int64_t smem = acc_bytes + 2 * M * 4;
    const bool in_smem = smem <= kMaxSmem / (LAYER ? 2 : 3);
    grid = walkers(N, smem <= kMaxSmem / 3 ? 3 : 2);
    if (in_smem) {
      auto kern = norm_bwd_generic_kernel<T, LAYER, true>;
      if (int32_t rc = allow_smem(kern, smem)) return rc;
      kern<<<grid, 512, smem, st>>>((T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, M, N, offset);
    } else {
      norm_bwd_generic_kernel<T, LAYER, false><<<grid, 512, 0, st>>>(
          (T*)dX, dWp, dBp, (const T*)dY, (const T*)X, (const T*)W, Mean, Rstd, M, N, offset);
    }
  }
  if (int32_t rc = check_launch(what)) return rc;
  norm_bwd_reduce_kernel<T><<<(unsigned)((M + 31) / 32), 1024, 0, st>>>((T*)dW, (T*)dB, dWp, LAYER ? dBp : nullptr, M, (int)grid);
  return check_launch("norm_bwd_reduce");
}

static int32_t check_mn(int64_t M, int64_t N) {
  TYLO_REQUIRE(M > 0 && N > 0, TYLO_ERR_INVALID_ARGUMENT, "extents must be positive (M=%lld, N=%lld)",
               (long long)M, (long long)N);
  TYLO_REQUIRE(N <= 0x7fffffffLL && M <= 0x7fffffffLL, TYLO_ERR_UNSUPPORTED,
               "extents above 2^31-1 are not supported (M=%lld, N=%lld)", (long long)M, (long long)N);
  return TYLO_OK;
}

}  // namespace tylo

using namespace tylo;

extern "C" int32_t tylo_b200_rms_norm_fwd(void* Y, const void* X, const void* W, float* Rstd, int64_t M,
                                          int64_t N, float eps, float offset, int32_t dtype,
                                          tylo_stream_t stream) {
  TYLO_REQUIRE(Y && X && W, TYLO_ERR_INVALID_ARGUMENT, "rms_norm_fwd: Y, X and W must be non-null");
  if (int32_t rc = check_mn(M, N)) return rc;
  TYLO_REQUIRE(aligned16(Y) && aligned16(X) && aligned16(W), TYLO_ERR_MISALIGNED,
               "rms_norm_fwd: pointers must be 16-byte aligned");
  TYLO_DISPATCH_DTYPE(dtype, T, return (norm_fwd_launch<T, false>(Y, X, W, nullptr, nullptr, Rstd, M, N, eps,
                                                                  offset, (cudaStream_t)stream)));
  return TYLO_OK;
}

extern "C" int32_t tylo_b200_layer_norm_fwd(void* Y, const void* X, const void* W, const void* Bias,
                                            float* Mean, float* Rstd, int64_t M, int64_t N, float eps,
                                            int32_t dtype, tylo_stream_t stream) {
  TYLO_REQUIRE(Y && X && W && Bias, TYLO_ERR_INVALID_ARGUMENT,
               "layer_norm_fwd: Y, X, W and B must be non-null");
  if (int32_t rc = check_mn(M, N)) return rc;
  TYLO_REQUIRE(aligned16(Y) && aligned16(X) && aligned16(W) && aligned16(Bias), TYLO_ERR_MISALIGNED,
               "layer_norm_fwd: pointers must be 16-byte aligned");
  TYLO_DISPATCH_DTYPE(dtype, T, return (norm_fwd_launch<T, true>(Y, X, W, Bias, Mean, Rstd, M, N, eps, 0.f,
                                                                 (cudaStream_t)stream)));
  return TYLO_OK;
}

extern "C" int32_t tylo_b200_rms_norm_bwd(void* dX, void* dW, const void* dY, const void* X,
                                          const void* W, const float* Rstd, float* dW_partial,
                                          int32_t n_groups, int64_t M, int64_t N, float offset,
                                          int32_t dtype, tylo_stream_t stream) {
  TYLO_REQUIRE(dX && dW && dY && X && W && Rstd && dW_partial, TYLO_ERR_INVALID_ARGUMENT,
               "rms_norm_bwd: all pointers must be non-null (Rstd comes from the forward's checkpoints)");
  if (int32_t rc = check_mn(M, N)) return rc;
  TYLO_REQUIRE(n_groups > 0, TYLO_ERR_INVALID_ARGUMENT, "rms_norm_bwd: n_groups must be positive");
  TYLO_REQUIRE(aligned16(dX) && aligned16(dW) && aligned16(dY) && aligned16(X) && aligned16(W) &&
                   aligned16(dW_partial), TYLO_ERR_MISALIGNED,
               "rms_norm_bwd: pointers must be 16-byte aligned");
  TYLO_DISPATCH_DTYPE(dtype, T, return (norm_bwd_launch<T, false>(dX, dW, nullptr, dY, X, W, nullptr, Rstd,
                                                                  dW_partial, nullptr, n_groups, M, N, offset,
                                                                  (cudaStream_t)stream)));
  return TYLO_OK;
}

extern "C" int32_t tylo_b200_layer_norm_bwd(void* dX, void* dW, void* dB, const void* dY, const void* X,
                                            const void* W, const float* Mean, const float* Rstd,
                                            float* dW_partial, float* dB_partial, int32_t n_groups,
                                            int64_t M, int64_t N, int32_t dtype, tylo_stream_t stream) {
  TYLO_REQUIRE(dX && dW && dB && dY && X && W && Mean && Rstd && dW_partial && dB_partial,
               TYLO_ERR_INVALID_ARGUMENT,
               "layer_norm_bwd: all pointers must be non-null (Mean/Rstd come from the forward's checkpoints)");
  if (int32_t rc = check_mn(M, N)) return rc;
  TYLO_REQUIRE(n_groups > 0, TYLO_ERR_INVALID_ARGUMENT, "layer_norm_bwd: n_groups must be positive");
  TYLO_REQUIRE(aligned16(dX) && aligned16(dW) && aligned16(dB) && aligned16(dY) && aligned16(X) &&
                   aligned16(W) && aligned16(dW_partial) && aligned16(dB_partial), TYLO_ERR_MISALIGNED,
               "layer_norm_bwd: pointers must be 16-byte aligned");
  TYLO_DISPATCH_DTYPE(dtype, T, return (norm_bwd_launch<T, true>(dX, dW, dB, dY, X, W, Mean, Rstd, dW_partial,
                                                                 dB_partial, n_groups, M, N, 0.f,
                                                                 (cudaStream_t)stream)));
  return TYLO_OK;
}
