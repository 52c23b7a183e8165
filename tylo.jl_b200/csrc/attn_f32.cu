// Attention forward / backward for fp32 storage in true fp32 arithmetic: register-tiled FMA kernels for head dims that
// are multiples of 4 up to 128 (Dk = Dv), every mask and score mod without a host-built
// block list.  The rest of the fp32 calls runs on attn_generic.cu.
//
// Bound: the FMA pipes (128 per clock and SM; tensor cores have no fp32 operands) next to shared memory, which hands 32
// values per clock to the registers of an SM whatever is broadcast: a kernel needs four FMAs per value read.  A CTA owns 64
// rows (queries, or keys for dK / dV) and streams tiles of the other side through shared memory with cp.async.  A thread owns
// 8 rows x 8 columns of a score tile (6 or 3 in the backward, where shared memory limits the streamed tile) and 8 x 8 of the
// output: 4 FMAs per value (a 2 x 2 patch, as in attn_generic.cu, has one).  Groups of 64 threads (128 at head dim 128) take
// the streamed tiles in turn, each with its own tiles, statistics and accumulators, and are merged once at the end: small
// problems have about one CTA per SM, and one group's loads and exponentials run under the other groups' FMAs.
//
// Packed pairs (fma.rn.f32x2) are used where their accumulators fit: they take half the issue slots, and with 32 warps per SM
// twice the rate (242 FMA per clock; with the eight warps that the registers allow here 125, as many as fmaf).  Every sum is
// kept in short chains (see dot_tile and acc_tile).  Forward + backward of B2 H8 S512 D64: 825 us on the 2 x 2 patches of
// attn_generic.cu, 174 here; eight warps per SM do not hide the shared-memory latency.
//
// Forward: online softmax per group.  Backward: no atomics on dQ / dK / dV; dK / dV CTAs (own 64 keys, sum the query heads
// of the group) and dQ CTAs (own 64 queries) share one launch, heaviest first, so that both fill the SMs together.
#include "attn_dispatch.cuh"
#include "sm100_ptx.cuh"

namespace tylo {
namespace f32 {

constexpr int BR = 64, RT = 8;     // rows a CTA owns, rows of a thread
constexpr int kThreads = 256;
constexpr int LDU = BR + 4;        // probabilities / score gradients: [streamed row][own row]
// Up to so many keys, and at head dim 128, dot_tile takes its finer form (template argument FINE): the fewer keys, the more the
// rounding of the scores outweighs that of the sums over the keys, and at 128 it costs nothing.  Relative error of O against 64
// bits, D 64: 144 keys 1.96e-7 (2.09e-7 otherwise, 2.06e-7 in attn_generic.cu), 512 keys 2.20e-7 without it (2.28e-7 there).
constexpr int kFineKeys = 384;

// TX threads side by side over a tile's columns, 8 of them down its rows: a group of 64 or 128 threads.
template <int D> struct Shape {
  static constexpr int TX = D == 128 ? 16 : 8, OC = D / TX;      // OC: output columns of a thread
  static constexpr int kGT = (BR / RT) * TX, kGroups = kThreads / kGT;
  int grp, tid, lane, ty, tx;
  __device__ __forceinline__ Shape()
      : grp(threadIdx.x / kGT), tid(threadIdx.x % kGT), lane(threadIdx.x & 31), ty(tid / TX), tx(tid % TX) {}
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(kGT) : "memory"); }
};
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ROWS x D tile of a (rows x Dr) fp32 array into shared memory (row pitch D + 4), zeros beyond `nrows` rows and Dr columns.
template <int D, int ROWS, int THREADS>
__device__ __forceinline__ void load_tile(float* dst, const float* __restrict__ src, int row0, int nrows, int Dr, int tid) {
  constexpr int C = D / 4;
  for (int i = tid; i < ROWS * C; i += THREADS) {
    const int r = i / C, c = (i % C) * 4;
    const int row = row0 + r;
    const bool ok = row < nrows && c < Dr;
    const float* s = ok ? src + (size_t)row * Dr + c : src;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sm100::smem_addr(dst + r * (D + 4) + c)), "l"(s),
                 "r"(ok ? 16 : 0) : "memory");
  }
}

// out[i][j] = X[8 ty + i] . Y[tx + TX j].  PAIR: even and odd columns of the head dim in the two halves of packed pairs
// (fma.rn.f32x2: half the instructions), for twice the accumulators.  FINE: the products of four columns are summed on their own
// before they join the accumulator, so that it rounds D / 4 times and not D / 2 times per half: an instruction more per four
// columns and pair (512 x 512, D 64: 43 -> 49 us forward; at D 128, where the loads hide it, 74 either way).  The fine form is
// paired in every kernel, spilling or not: scores that round alike in the forward and in both halves of the backward make P of a
// row with few keys exact (dV of 49 causal rows, D 64: error 1.13 times that of attn_generic.cu otherwise, 0.94 so).
template <int D, int NJ, bool PAIR, bool FINE>
__device__ __forceinline__ void dot_tile(const float* __restrict__ X, const float* __restrict__ Y, int ty, int tx, float (&out)[RT][NJ]) {
  constexpr int TX = Shape<D>::TX;
  const float* x = X + RT * ty * (D + 4);
  const float* y = Y + tx * (D + 4);
  if constexpr (PAIR) {
    uint64_t acc[RT][NJ];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[i][j] = 0ull;
#pragma unroll 1
    for (int c = 0; c < D; c += 4) {
      ulonglong2 a[RT];
#pragma unroll
      for (int i = 0; i < RT; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(x + i * (D + 4) + c);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(y + j * TX * (D + 4) + c);
#pragma unroll
        for (int i = 0; i < RT; ++i)
          acc[i][j] = FINE ? sm100::add_f32x2(acc[i][j], sm100::fma_f32x2(a[i].y, b.y, sm100::mul_f32x2(a[i].x, b.x)))
                           : sm100::fma_f32x2(a[i].y, b.y, sm100::fma_f32x2(a[i].x, b.x, acc[i][j]));
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) { float lo, hi; sm100::unpack_f32x2(acc[i][j], lo, hi); out[i][j] = lo + hi; }
    return;
  }
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) out[i][j] = 0.f;
#pragma unroll 2
  for (int c = 0; c < D; c += 4) {
    float4 a[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) a[i] = *reinterpret_cast<const float4*>(x + i * (D + 4) + c);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float4 b = *reinterpret_cast<const float4*>(y + j * TX * (D + 4) + c);
#pragma unroll
      for (int i = 0; i < RT; ++i)
        out[i][j] += fmaf(a[i].w, b.w, fmaf(a[i].z, b.z, fmaf(a[i].y, b.y, a[i].x * b.x)));      // (short chains: D / 4 sums)
    }
  }
}

// acc[i], columns 4 j + e (in pairs) = acc[i] f[i] (f only with SCALE) + sum_n U[n][8 ty + i] Y[n][4 TX j + 4 tx + e].  The rows are
// summed in PARTS sums of their own, in the registers of the scores, which are free by then: an accumulator that runs through
// all rows rounds once per row (dK of 1,200 rows, D 128: error 6.4e-7 in one chain, 3.7e-7 so; of 512, D 64: 4.0e-7, 3.5e-7).
template <int D, int ROWS, int PARTS, bool SCALE>
__device__ __forceinline__ void acc_tile(const float* __restrict__ U, const float* __restrict__ Y, int ty, int tx,
                                         uint64_t (&acc)[RT][Shape<D>::OC / 2], const float (&f)[RT]) {
  constexpr int TX = Shape<D>::TX, OC = Shape<D>::OC, N = ROWS / PARTS;
  static_assert(ROWS % PARTS == 0, "whole parts");
  const float* u = U + RT * ty;
  const float* y = Y + 4 * tx;
#pragma unroll 1
  for (int part = 0; part < PARTS; ++part) {
    uint64_t t[RT][OC / 2];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int e = 0; e < OC / 2; ++e) t[i][e] = 0ull;
#pragma unroll 4
    for (int n = part * N; n < (part + 1) * N; ++n) {
      const float4 p0 = *reinterpret_cast<const float4*>(u + n * LDU), p1 = *reinterpret_cast<const float4*>(u + n * LDU + 4);
      const float pi[RT] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
      for (int j = 0; j < OC / 4; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(y + n * (D + 4) + 4 * TX * j);
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const uint64_t p2 = sm100::pack_f32x2(pi[i], pi[i]);
          t[i][2 * j] = sm100::fma_f32x2(p2, v.x, t[i][2 * j]);
          t[i][2 * j + 1] = sm100::fma_f32x2(p2, v.y, t[i][2 * j + 1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const float fi = part == 0 ? f[i] : 1.f;
      const uint64_t f2 = sm100::pack_f32x2(fi, fi);
#pragma unroll
      for (int e = 0; e < OC / 2; ++e) acc[i][e] = SCALE ? sm100::fma_f32x2(acc[i][e], f2, t[i][e]) : sm100::add_f32x2(acc[i][e], t[i][e]);
    }
  }
}
template <int D, int ROWS, int PARTS>
__device__ __forceinline__ void acc_tile(const float* __restrict__ U, const float* __restrict__ Y, int ty, int tx, uint64_t (&acc)[RT][Shape<D>::OC / 2]) {
  const float none[RT] = {};
  acc_tile<D, ROWS, PARTS, false>(U, Y, ty, tx, acc, none);
}
// U[tx + TX j][8 ty + i] = v[i][j]
template <int D, int NJ>
__device__ __forceinline__ void put_transposed(float* U, int ty, int tx, const float (&v)[RT][NJ]) {
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float4* u = reinterpret_cast<float4*>(U + (tx + Shape<D>::TX * j) * LDU + RT * ty);
    u[0] = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
    u[1] = make_float4(v[4][j], v[5][j], v[6][j], v[7][j]);
  }
}
template <int D, int NJ>
__device__ __forceinline__ void get_transposed(const float* U, int ty, int tx, float (&v)[RT][NJ]) {
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const float4* u = reinterpret_cast<const float4*>(U + (tx + Shape<D>::TX * j) * LDU + RT * ty);
    const float4 a = u[0], b = u[1];
    v[0][j] = a.x; v[1][j] = a.y; v[2][j] = a.z; v[3][j] = a.w; v[4][j] = b.x; v[5][j] = b.y; v[6][j] = b.z; v[7][j] = b.w;
  }
}
// a thread's output patch to / from a BR x D tile in shared memory (row pitch D + 4)
template <int D>
__device__ __forceinline__ void put_rows(float* dst, int ty, int tx, const uint64_t (&a)[RT][Shape<D>::OC / 2]) {
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < Shape<D>::OC / 4; ++j)
      *reinterpret_cast<ulonglong2*>(dst + (RT * ty + i) * (D + 4) + 4 * (Shape<D>::TX * j + tx)) = make_ulonglong2(a[i][2 * j], a[i][2 * j + 1]);
}

__device__ __forceinline__ int clamp_len(const int32_t* lens, int b, int S) {
  if (!lens) return S;
  const int v = lens[b];
  return v < 0 ? 0 : (v > S ? S : v);
}
// attention.jl:25-26 skips whole 64-row query blocks that start at or beyond q_lengths[b].
__device__ __forceinline__ int q_row_limit(const AttnParams& p, int b) {
  if (!p.q_lengths) return p.Sq;
  return min(p.Sq, (clamp_len(p.q_lengths, b, p.Sq) + 63) / 64 * 64);
}
// Whether a tile of queries from row q0 and keys [kv0, kv0 + keys) holds pairs that the mask may drop: exact for the causal
// mask (the usual one), always for the other terms.
__device__ __forceinline__ bool needs_mask(const AttnParams& p, int q0, int kv0, int keys) {
  if (p.n_or > 0 || (p.mask_flags & ~(uint32_t)TYLO_MASK_CAUSAL)) return true;
  return (p.mask_flags & TYLO_MASK_CAUSAL) && kv0 + keys - 1 > q0 + p.input_pos;
}
__device__ __forceinline__ uint32_t low_bits(int n) { return (1u << max(0, min(n, RT))) - 1u; }
// Which of the pairs (q + i, kv), or (q, kv + i) with OWN_KEYS, that are set in `live` a clause keeps: mask_keep for the RT own
// rows of a column at once.  Every term but the documents is an interval of i, so a column costs a few instructions instead of a
// few per pair; pairs that are not live are not looked up in the id tables.
template <bool OWN_KEYS>
__device__ __forceinline__ uint32_t clause_bits(uint32_t live, uint32_t flags, int window, int prefix_len, const int32_t* doc_q,
                                                const int32_t* doc_kv, long long doc_stride, int b, int q, int kv) {
  constexpr uint32_t kAll = (1u << RT) - 1u;
  const int d = q - kv, w = min(window, 1 << 30);                                   // (positions are far below 2^30)
  const uint32_t past = OWN_KEYS ? low_bits(d + 1) : kAll & ~low_bits(-d);          // query position >= key position
  const uint32_t prefix = OWN_KEYS ? low_bits(prefix_len - kv) : (kv < prefix_len ? kAll : 0u);
  if (flags & (TYLO_MASK_CAUSAL | TYLO_MASK_SLIDING)) live &= past;
  if (flags & TYLO_MASK_SLIDING) live &= OWN_KEYS ? kAll & ~low_bits(d - w) : low_bits(w - d + 1);
  if (flags & TYLO_MASK_PREFIX) live &= prefix;
  if (flags & TYLO_MASK_PREFIX_LM) live &= past | prefix;
  if ((flags & TYLO_MASK_DOCUMENT) && live) {
    const int32_t* own = (OWN_KEYS ? doc_kv + kv : doc_q + q) + (size_t)b * doc_stride;
    const int id = OWN_KEYS ? doc_q[(size_t)b * doc_stride + q] : doc_kv[(size_t)b * doc_stride + kv];
    int ids[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) ids[i] = (live >> i) & 1u ? own[i] : id;
#pragma unroll
    for (int i = 0; i < RT; ++i) live &= ~((ids[i] != id ? 1u : 0u) << i);
  }
  return live;
}
// Bit 8 j + i: pair (i, j) of a thread's patch takes part.  own0: first own row of the thread, str0: its first streamed row,
// columns TX apart.  The loop over the columns is rolled: with a mask test per pair written out, one masked tile cost more
// in fetching its code (64 copies) than in computing: causal with a window, B1 H4 S50 D64, forward, cold: 86 us against 23
// rolled.
template <int TX, int NJ, bool OWN_KEYS>
__device__ __forceinline__ uint64_t keep_bits(const AttnParams& p, int b, int own0, int str0, int q_lim, int k_len, bool masked) {
  uint64_t bits = 0;
#pragma unroll 1
  for (int j = 0; j < NJ; ++j) {
    const int str = str0 + TX * j;
    const uint32_t live = OWN_KEYS ? (str < q_lim ? low_bits(k_len - own0) : 0u) : (str < k_len ? low_bits(q_lim - own0) : 0u);
    uint32_t keep = live;
    if (masked && live) {
      const int q = (OWN_KEYS ? str : own0) + p.input_pos, kv = OWN_KEYS ? own0 : str;
      keep = clause_bits<OWN_KEYS>(live, p.mask_flags, p.window, p.prefix_len, p.doc_q, p.doc_kv, p.doc_stride, b, q, kv);
      for (int i = 0; i < p.n_or; ++i) {
        const MaskClause& o = p.or_clause[i];
        keep |= clause_bits<OWN_KEYS>(live, o.flags, o.window, o.prefix_len, o.doc_q, o.doc_kv, o.doc_stride, b, q, kv);
      }
    }
    bits |= (uint64_t)keep << (RT * j);
  }
  return bits;
}
// The score mods of one (batch entry, query head): score_additive, score_apply and score_vjp with the table's base worked out
// once and one tanh for a score and its derivative.
struct ScoreMods {
  float slope;
  const float* bias;           // table of this batch entry and head, or null
  size_t bias0;
  __device__ __forceinline__ ScoreMods(const AttnParams& p, int b, int h)
      : slope((p.score_flags & TYLO_SCORE_ALIBI) ? p.slopes[h] : 0.f), bias(nullptr), bias0(0) {
    if (p.score_flags & TYLO_SCORE_BIAS) { bias0 = bias_index(p, b, h, 0, 0); bias = p.bias + bias0; }
  }
  // the additive mods of four pairs: keys kv.. of one row with KEYS, rows row.. at one key otherwise.  Pairs outside the problem
  // take the nearest one inside (the table is not read beyond its end); their scores are not used.
  template <bool KEYS>
  __device__ __forceinline__ void additive(const AttnParams& p, int row, int kv, float (&add)[4]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) add[i] = slope * (float)((KEYS ? row : row + i) + p.input_pos - (KEYS ? kv + i : kv));
    if (bias) {          // one branch for the four, so that their loads are in flight together
      float t[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) t[i] = bias[(size_t)min(KEYS ? row : row + i, p.Sq - 1) * p.Sk + min(KEYS ? kv + i : kv, p.Sk - 1)];
#pragma unroll
      for (int i = 0; i < 4; ++i) add[i] += t[i];
    }
  }
  // the modded score of the scaled score s0; d_add, d_s0: its derivatives by the additive mods and by s0
  __device__ __forceinline__ float apply(const AttnParams& p, float s0, float add, float& d_add, float& d_s0) const {
    d_add = 1.f; d_s0 = 1.f;
    if (!(p.score_flags & TYLO_SCORE_SOFTCAP)) return s0 + add;
    const bool cap_first = p.score_flags & TYLO_SCORE_SOFTCAP_FIRST;
    const float th = tanhf((cap_first ? s0 : s0 + add) / p.cap), d = 1.f - th * th;
    d_s0 = d;
    if (!cap_first) d_add = d;
    return cap_first ? p.cap * th + add : p.cap * th;
  }
};
template <int TX, typename Op> __device__ __forceinline__ float row_reduce(float v, Op op) {
#pragma unroll
  for (int o = TX / 2; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------------
template <int D> struct FwdSmem {
  static constexpr int kTile = BR * (D + 4), kU = BR * LDU;           // floats
  static constexpr int kGroup = 2 * kTile + kU;                        // K, V, P of one group
  static constexpr int kBytes = (kTile + Shape<D>::kGroups * kGroup) * 4;      // 149 KB, 221 KB, 199 KB for D = 32, 64, 128
  static constexpr int kParts = 4;                                     // sums of 16 keys
};

template <int D, bool FINE>
__global__ void __launch_bounds__(kThreads, 1)
fwd_kernel(float* __restrict__ O, const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
           float* __restrict__ Mout, float* __restrict__ Lout, const AttnParams p) {
  using SM = FwdSmem<D>;
  using SH = Shape<D>;
  constexpr int TX = SH::TX, OC = SH::OC, NG = SH::kGroups, GT = SH::kGT, NJ = BR / TX;
  extern __shared__ __align__(16) float sm[];
  const SH sh;
  const int grp = sh.grp, tid = sh.tid, ty = sh.ty, tx = sh.tx;
  float* sQ = sm;
  float* sK = sm + SM::kTile + grp * SM::kGroup;
  float* sV = sK + SM::kTile;
  float* sP = sV + SM::kTile;

  const int nqt = (p.Sq + BR - 1) / BR, hbs = p.H * p.B;
  const int qt = nqt - 1 - (int)(blockIdx.x / hbs), hb = blockIdx.x % hbs;   // the last query blocks (causal: the longest) first
  const int b = hb / p.H, h = hb % p.H, hk = h / p.G;
  const int q0 = qt * BR;
  if (q0 >= q_row_limit(p, b)) return;
  const int k_len = clamp_len(p.k_lengths, b, p.Sk);
  const float* Qg = Q + (size_t)(b * p.H + h) * p.Sq * p.Dk;
  const float* Kg = K + (size_t)(b * p.Hkv + hk) * p.Sk * p.Dk;
  const float* Vg = V + (size_t)(b * p.Hkv + hk) * p.Sk * p.Dk;
  const ScoreMods mods(p, b, h);
  const bool modded = p.score_flags != 0;
  const float c = p.scale * kLog2e;


  int lo, hi;
  kv_range(p, q0 + p.input_pos, min(q0 + BR, p.Sq) - 1 + p.input_pos, k_len, &lo, &hi);
  const int t0 = lo / BR, t1 = hi > lo ? (hi - 1) / BR + 1 : t0;

  float m[RT], l[RT];
  uint64_t o[RT][OC / 2];
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int e = 0; e < OC / 2; ++e) o[i][e] = 0ull;
  }

  load_tile<D, BR, kThreads>(sQ, Qg, q0, p.Sq, p.Dk, threadIdx.x);
  if (t0 + grp < t1) load_tile<D, BR, GT>(sK, Kg, (t0 + grp) * BR, k_len, p.Dk, tid);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  for (int t = t0 + grp; t < t1; t += NG) {
    const int kv0 = t * BR;
    cp_wait<0>();
    sh.sync();                 // K of this tile is there; everyone is done with the last tile's V
    load_tile<D, BR, GT>(sV, Vg, kv0, k_len, p.Dk, tid);
    cp_commit();
    float s[RT][NJ];
    dot_tile<D, NJ, true, FINE>(sQ, sK, ty, tx, s);
    __syncwarp();              // a warp writes and reads only its own rows of P
    if (modded) {
      // through the thread's own elements of P, four at a time in a rolled loop (see keep_bits); columns that no row can
      // see are left as they are
      put_transposed<D, NJ>(sP, ty, tx, s);
      const int ne = 2 * min(NJ, (hi - kv0 + TX - 1) / TX);
#pragma unroll 1
      for (int e = 0; e < ne; ++e) {
        const int j = e >> 1, i0 = 4 * (e & 1);
        float4* u = reinterpret_cast<float4*>(sP + (tx + TX * j) * LDU + RT * ty + i0);
        const float4 raw = *u;
        float add[4], da, ds;
        mods.additive<false>(p, q0 + RT * ty + i0, kv0 + tx + TX * j, add);
        *u = make_float4(mods.apply(p, raw.x * p.scale, add[0], da, ds) * kLog2e, mods.apply(p, raw.y * p.scale, add[1], da, ds) * kLog2e,
                         mods.apply(p, raw.z * p.scale, add[2], da, ds) * kLog2e, mods.apply(p, raw.w * p.scale, add[3], da, ds) * kLog2e);
      }
      get_transposed<D, NJ>(sP, ty, tx, s);
    } else {
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) s[i][j] *= c;
    }
    const bool masked = needs_mask(p, q0, kv0, BR);
    if (masked || kv0 + BR > k_len) {
      const uint64_t bits = keep_bits<TX, NJ, false>(p, b, q0 + RT * ty, kv0 + tx, p.Sq, k_len, masked);
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) s[i][j] = (bits >> (RT * j + i)) & 1u ? s[i][j] : -INFINITY;
    }
    float f[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      float mx = s[i][0];
#pragma unroll
      for (int j = 1; j < NJ; ++j) mx = fmaxf(mx, s[i][j]);
      const float mn = fmaxf(m[i], row_reduce<TX>(mx, MaxOp()));
      const float alpha = (mn == -INFINITY) ? 1.f : exp2f(m[i] - mn);
      float ps = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        s[i][j] = (s[i][j] == -INFINITY) ? 0.f : exp2f(s[i][j] - mn);
        ps += s[i][j];
      }
      l[i] = l[i] * alpha + ps;
      m[i] = mn;
      f[i] = alpha;
    }
    put_transposed<D, NJ>(sP, ty, tx, s);
    cp_wait<0>();
    sh.sync();                 // V is there; everyone is done with K
    if (t + NG < t1) load_tile<D, BR, GT>(sK, Kg, (t + NG) * BR, k_len, p.Dk, tid);
    cp_commit();
    acc_tile<D, BR, SM::kParts, true>(sP, sV, ty, tx, o, f);
  }

  // merge of the groups: each leaves its rows in its own K tile and its statistics in its own P; every thread then takes an
  // equal share of the output
  sh.sync();
  put_rows<D>(sK, ty, tx, o);
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    l[i] = row_reduce<TX>(l[i], SumOp());
    if (tx == 0) { sP[RT * ty + i] = m[i]; sP[BR + RT * ty + i] = l[i]; }
  }
  __syncthreads();
  const float* x0 = sm + SM::kTile;
  for (int idx = threadIdx.x; idx < BR * (D / 4); idx += kThreads) {
    const int r = idx / (D / 4), col = idx % (D / 4) * 4, row = q0 + r;
    if (row >= p.Sq) break;
    float mg[NG], mn = -INFINITY, lt = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int g = 0; g < NG; ++g) { mg[g] = x0[g * SM::kGroup + 2 * SM::kTile + r]; mn = fmaxf(mn, mg[g]); }
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const float a = mg[g] == -INFINITY ? 0.f : exp2f(mg[g] - mn);
      const float4 x = *reinterpret_cast<const float4*>(x0 + g * SM::kGroup + r * (D + 4) + col);
      lt += x0[g * SM::kGroup + 2 * SM::kTile + BR + r] * a;
      acc.x += x.x * a; acc.y += x.y * a; acc.z += x.z * a; acc.w += x.w * a;
    }
    const float inv = lt > 0.f ? 1.f / lt : 0.f;
    const size_t si = (size_t)(b * p.H + h) * p.Sq + row;
    if (col < p.Dk) *reinterpret_cast<float4*>(O + si * p.Dk + col) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    if (col == 0) {
      if (Mout) Mout[si] = p.natural_stats ? mn * kLn2 : mn;
      if (Lout) Lout[si] = lt;
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------------------
// Streamed tiles are 64 rows at head dim 32 and 48 rows above, which is what fits four (two at 128) groups into shared memory.
// P and dS of a tile share one buffer: dV is summed before dS takes P's place.
template <int D> struct BwdSmem {
  static constexpr int SB = D <= 32 ? 64 : 48;
  static constexpr int kOwn = BR * (D + 4), kTile = SB * (D + 4), kU = SB * LDU;
  static constexpr int kGroup = 2 * kTile + kU + 2 * SB;               // Y1, Y2, P / dS, statistics
  static constexpr int kParts = D == 128 ? 1 : 2;                      // sums of 48 rows, 24 (64), 32 (32)
  static constexpr int kBytes = (2 * kOwn + 2 * BR + Shape<D>::kGroups * kGroup) * 4;
  static_assert(kGroup >= kOwn, "a group's sum is left in its own tiles");
};

// Delta[row] = sum_d dO * O, eight lanes per row
__global__ void __launch_bounds__(256)
delta_kernel(float* __restrict__ Delta, const float* __restrict__ O, const float* __restrict__ dO, long long rows, int Dr) {
  const int sub = threadIdx.x & 7;                     // 8 lanes per row
  const long long row = (long long)blockIdx.x * 32 + (threadIdx.x >> 3);
  float s = 0.f;
  if (row < rows)
    for (int d = sub * 4; d < Dr; d += 32) {
      const float4 a = *reinterpret_cast<const float4*>(O + row * Dr + d), g = *reinterpret_cast<const float4*>(dO + row * Dr + d);
      s += a.x * g.x + a.y * g.y + (a.z * g.z + a.w * g.w);
    }
  s = row_reduce<8>(s, SumOp());
  if (sub == 0 && row < rows) Delta[row] = s;
}

// OWN_KEYS: own 64 keys of a KV head, stream the queries of its group (dV += P^T dO, dK += dS^T Q); otherwise own 64 queries,
// stream keys (dQ += dS K).  Own rows are the rows of T1 = X1 Y1^T (scores) and T2 = X2 Y2^T (dP).
template <int D, bool OWN_KEYS, bool FINE>
__device__ __forceinline__ void bwd_tiles(float* sm, float* __restrict__ dA, float* __restrict__ dB, const float* __restrict__ Q,
                                          const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ dO,
                                          const float* __restrict__ Mst, const float* __restrict__ Lst,
                                          const float* __restrict__ Delta, const AttnParams& p, const int b, const int hx, const int own0) {
  using SM = BwdSmem<D>;
  using SH = Shape<D>;
  constexpr int TX = SH::TX, OC = SH::OC, NG = SH::kGroups, GT = SH::kGT, SB = SM::SB, NJ = SB / TX;
  const SH sh;
  const int grp = sh.grp, tid = sh.tid, ty = sh.ty, tx = sh.tx;
  float* sX1 = sm;
  float* sX2 = sX1 + SM::kOwn;
  float* sOwn = sX2 + SM::kOwn;                       // own queries' log-sum-exp and Delta
  float* gs = sOwn + 2 * BR;
  float* sY1 = gs + grp * SM::kGroup;
  float* sY2 = sY1 + SM::kTile;
  float* sU = sY2 + SM::kTile;
  float* sStat = sU + SM::kU;                          // streamed queries' statistics

  const int hk = OWN_KEYS ? hx : hx / p.G, h0 = OWN_KEYS ? hx * p.G : hx;
  const int k_len = clamp_len(p.k_lengths, b, p.Sk), q_lim = q_row_limit(p, b);
  const float* Kg = K + (size_t)(b * p.Hkv + hk) * p.Sk * p.Dk;
  const float* Vg = V + (size_t)(b * p.Hkv + hk) * p.Sk * p.Dk;
  const bool modded = p.score_flags != 0;
  const float c = p.scale * kLog2e;
  auto lse2_of = [&](size_t si) {
    const float L = Lst[si];
    return L > 0.f ? (p.natural_stats ? Mst[si] * kLog2e : Mst[si]) + log2f(L) : INFINITY;      // no keys: P = 0
  };

  int lo = 0, hi = 0;
  if (OWN_KEYS) {
    if (own0 < k_len) q_range(p, own0, min(own0 + BR, k_len) - 1, q_lim, &lo, &hi);
  } else if (own0 < q_lim) {
    kv_range(p, own0 + p.input_pos, min(own0 + BR, q_lim) - 1 + p.input_pos, k_len, &lo, &hi);
  }
  const int t0 = lo / SB, nt = hi > lo ? (hi - 1) / SB + 1 - t0 : 0;

  uint64_t acc1[RT][OC / 2], acc2[RT][OC / 2];        // (acc1: dV, OWN_KEYS only)
  float slope_acc = 0.f;

  // (Y1, Y2) of streamed tile n: queries and their dO of query head h, or keys and values
  auto load_y = [&](int n, int h) {
    const int row0 = (t0 + n) * SB;
    if (OWN_KEYS) {
      const size_t hq = (size_t)(b * p.H + h) * p.Sq;
      load_tile<D, SB, GT>(sY1, Q + hq * p.Dk, row0, q_lim, p.Dk, tid);
      load_tile<D, SB, GT>(sY2, dO + hq * p.Dk, row0, q_lim, p.Dk, tid);
      if (tid < SB) {
        const int row = row0 + tid;
        sStat[tid] = row < q_lim ? lse2_of(hq + row) : INFINITY;
        sStat[SB + tid] = row < q_lim ? Delta[hq + row] : 0.f;
      }
    } else {
      load_tile<D, SB, GT>(sY1, Kg, row0, k_len, p.Dk, tid);
      load_tile<D, SB, GT>(sY2, Vg, row0, k_len, p.Dk, tid);
    }
  };

  if (nt > 0) {
    if (OWN_KEYS) {
      load_tile<D, BR, kThreads>(sX1, Kg, own0, k_len, p.Dk, threadIdx.x);
      load_tile<D, BR, kThreads>(sX2, Vg, own0, k_len, p.Dk, threadIdx.x);
    } else {
      const size_t hq = (size_t)(b * p.H + h0) * p.Sq;
      load_tile<D, BR, kThreads>(sX1, Q + hq * p.Dk, own0, q_lim, p.Dk, threadIdx.x);
      load_tile<D, BR, kThreads>(sX2, dO + hq * p.Dk, own0, q_lim, p.Dk, threadIdx.x);
      if (threadIdx.x < BR) {
        const int row = own0 + threadIdx.x;
        sOwn[threadIdx.x] = row < q_lim ? lse2_of(hq + row) : INFINITY;
        sOwn[BR + threadIdx.x] = row < q_lim ? Delta[hq + row] : 0.f;
      }
    }
  }
  cp_commit();
  cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int e = 0; e < OC / 2; ++e) { acc1[i][e] = 0ull; acc2[i][e] = 0ull; }
  // dK / dV: the tiles of all query heads of the group are dealt over the groups of threads (head by head, groups of threads
  // idled whenever a head has fewer tiles than there are groups, and every head paid for a merge)
  const int total = OWN_KEYS ? nt * p.G : nt;
  for (int u = grp; u < total; u += NG) {
    const int n = OWN_KEYS ? u % nt : u, h = OWN_KEYS ? h0 + u / nt : h0;
    const int str0 = (t0 + n) * SB;
    sh.sync();                  // everyone is done with the tile before
    load_y(n, h);
    cp_commit();
    cp_wait<0>();
    sh.sync();
    const int q0 = OWN_KEYS ? str0 : own0, kv0 = OWN_KEYS ? own0 : str0;
    const bool masked = needs_mask(p, q0, kv0, OWN_KEYS ? BR : SB);
    const bool partial = masked || kv0 + (OWN_KEYS ? BR : SB) > k_len || q0 + (OWN_KEYS ? SB : BR) > q_lim;
    const ScoreMods mods(p, b, h);
    auto lse_of = [&](int i, int j) { return OWN_KEYS ? sStat[tx + TX * j] : sOwn[RT * ty + i]; };
    auto delta_of = [&](int i, int j) { return OWN_KEYS ? sStat[SB + tx + TX * j] : sOwn[BR + RT * ty + i]; };
    const uint64_t bits = partial ? keep_bits<TX, NJ, OWN_KEYS>(p, b, own0 + RT * ty, str0 + tx, q_lim, k_len, masked) : ~0ull;
    float s[RT][NJ];
    dot_tile<D, NJ, !OWN_KEYS || FINE, FINE>(sX1, sY1, ty, tx, s);
    if (!modded) {
      // P into shared memory, dV from it; dS takes its place element by element (each thread its own)
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) s[i][j] = exp2f(fmaf(s[i][j], c, -lse_of(i, j)));
      if (partial) {
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < NJ; ++j) s[i][j] = (bits >> (RT * j + i)) & 1u ? s[i][j] : 0.f;
      }
      put_transposed<D, NJ>(sU, ty, tx, s);
      __syncwarp();             // a warp writes and reads only its own rows of P and dS
      if constexpr (OWN_KEYS) acc_tile<D, SB, SM::kParts>(sU, sY2, ty, tx, acc1);
      dot_tile<D, NJ, !OWN_KEYS || FINE, FINE>(sX2, sY2, ty, tx, s);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        float4* u = reinterpret_cast<float4*>(sU + (tx + TX * j) * LDU + RT * ty);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float4 w = u[q];
          // (a masked pair's dS is zero whatever its dP is)
          w.x = w.x == 0.f ? 0.f : w.x * ((s[4 * q][j] - delta_of(4 * q, j)) * p.scale);
          w.y = w.y == 0.f ? 0.f : w.y * ((s[4 * q + 1][j] - delta_of(4 * q + 1, j)) * p.scale);
          w.z = w.z == 0.f ? 0.f : w.z * ((s[4 * q + 2][j] - delta_of(4 * q + 2, j)) * p.scale);
          w.w = w.w == 0.f ? 0.f : w.w * ((s[4 * q + 3][j] - delta_of(4 * q + 3, j)) * p.scale);
          u[q] = w;
        }
      }
    } else {
      // score mods: the raw products wait in shared memory; P, then dS with the mods' derivative at them.  Four elements
      // at a time in rolled loops (see keep_bits)
      put_transposed<D, NJ>(sU, ty, tx, s);
      auto row_of = [&](int i, int j) { return OWN_KEYS ? str0 + tx + TX * j : own0 + RT * ty + i; };
      auto key_of = [&](int i, int j) { return OWN_KEYS ? own0 + RT * ty + i : str0 + tx + TX * j; };
      auto element = [&](float raw, float add, int i, int j, float dp, float& ds) {       // returns p
        ds = 0.f;
        if (!((bits >> (RT * j + i)) & 1u)) return 0.f;
        float d_add, d_s0;
        const float pr = exp2f(mods.apply(p, raw * p.scale, add, d_add, d_s0) * kLog2e - lse_of(i, j));
        const float g = pr * (dp - delta_of(i, j)), at_add = g * d_add;
        ds = g * d_s0 * p.scale;
        if (!OWN_KEYS) {      // parameter gradients: the dQ side meets every pair once (mods.jl:296-313)
          const int row = row_of(i, j), kv = key_of(i, j);
          slope_acc += at_add * (float)(row + p.input_pos - kv);
          if (mods.bias && p.d_bias) atomicAdd(p.d_bias + mods.bias0 + (size_t)row * p.Sk + kv, at_add);
        }
        return pr;
      };
      if constexpr (OWN_KEYS) {
        float ds;
        // (P of this thread's elements goes to its place, and the raw products back)
#pragma unroll 1
        for (int e = 0; e < 2 * NJ; ++e) {
          const int j = e >> 1, i0 = 4 * (e & 1);
          float4* u = reinterpret_cast<float4*>(sU + (tx + TX * j) * LDU + RT * ty + i0);
          float4 w = *u;
          float add[4];
          mods.additive<OWN_KEYS>(p, row_of(i0, j), key_of(i0, j), add);
          w.x = element(w.x, add[0], i0, j, 0.f, ds); w.y = element(w.y, add[1], i0 + 1, j, 0.f, ds);
          w.z = element(w.z, add[2], i0 + 2, j, 0.f, ds); w.w = element(w.w, add[3], i0 + 3, j, 0.f, ds);
          *u = w;
        }
        __syncwarp();
        acc_tile<D, SB, SM::kParts>(sU, sY2, ty, tx, acc1);
        __syncwarp();
        put_transposed<D, NJ>(sU, ty, tx, s);
      }
      dot_tile<D, NJ, !OWN_KEYS || FINE, FINE>(sX2, sY2, ty, tx, s);
#pragma unroll 1
      for (int e = 0; e < 2 * NJ; ++e) {
        const int j = e >> 1, i0 = 4 * (e & 1);
        float4* u = reinterpret_cast<float4*>(sU + (tx + TX * j) * LDU + RT * ty + i0);
        const float4 raw = *u;
        float4 w;
        float add[4];
        mods.additive<OWN_KEYS>(p, row_of(i0, j), key_of(i0, j), add);
        element(raw.x, add[0], i0, j, s[0][0], w.x); element(raw.y, add[1], i0 + 1, j, s[1][0], w.y);
        element(raw.z, add[2], i0 + 2, j, s[2][0], w.z); element(raw.w, add[3], i0 + 3, j, s[3][0], w.w);
        *u = w;
        // the next four dP move up to the front (registers cannot be indexed)
#pragma unroll
        for (int k = 0; k < NJ; ++k)
#pragma unroll
          for (int i = 0; i < 4; ++i) { s[i][k] = s[i + 4][k]; if (k + 1 < NJ) s[i + 4][k] = s[i][k + 1]; }
      }
    }
    __syncwarp();
    acc_tile<D, SB, SM::kParts>(sU, sY1, ty, tx, acc2);
  }

  // sums over the groups, one output at a time, through each group's own tiles
  const int S = OWN_KEYS ? p.Sk : p.Sq;
  const size_t base = (size_t)(OWN_KEYS ? b * p.Hkv + hk : b * p.H + h0) * S;
  auto merge = [&](const uint64_t (&a)[RT][OC / 2], float* __restrict__ out) {
    __syncthreads();
    put_rows<D>(gs + grp * SM::kGroup, ty, tx, a);
    __syncthreads();
    for (int idx = threadIdx.x; idx < BR * (D / 4); idx += kThreads) {
      const int r = idx / (D / 4), col = idx % (D / 4) * 4, row = own0 + r;
      if (row >= S) break;
      float4 t = *reinterpret_cast<const float4*>(gs + r * (D + 4) + col);
#pragma unroll
      for (int k = 1; k < NG; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(gs + k * SM::kGroup + r * (D + 4) + col);
        t.x += x.x; t.y += x.y; t.z += x.z; t.w += x.w;
      }
      if (col < p.Dk) *reinterpret_cast<float4*>(out + (base + row) * p.Dk + col) = t;
    }
  };
  if constexpr (OWN_KEYS) merge(acc1, dB);
  merge(acc2, dA);
  if (!OWN_KEYS && p.d_slopes && (p.score_flags & TYLO_SCORE_ALIBI)) {
    slope_acc = warp_reduce(slope_acc, SumOp());
    if (sh.lane == 0 && slope_acc != 0.f) atomicAdd(p.d_slopes + h0, slope_acc);
  }
}

template <int D, bool FINE>
__global__ void __launch_bounds__(kThreads, 1)
bwd_kernel(float* __restrict__ dQ, float* __restrict__ dK, float* __restrict__ dV, const float* __restrict__ Q,
           const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ dO, const float* __restrict__ Mst,
           const float* __restrict__ Lst, const float* __restrict__ Delta, const AttnParams p, const int n_keys) {
  extern __shared__ __align__(16) float sm[];
  // dK / dV CTAs come first (four tile products per pair against three, G heads each); under a causal mask the first
  // key blocks and the last query blocks see the most
  if ((int)blockIdx.x < n_keys) {
    const int heads = p.Hkv * p.B, hb = blockIdx.x % heads;
    bwd_tiles<D, true, FINE>(sm, dK, dV, Q, K, V, dO, Mst, Lst, Delta, p, hb / p.Hkv, hb % p.Hkv, (int)(blockIdx.x / heads) * BR);
  } else {
    const int i = blockIdx.x - n_keys, heads = p.H * p.B, hb = i % heads, nqt = (p.Sq + BR - 1) / BR;
    bwd_tiles<D, false, FINE>(sm, dQ, nullptr, Q, K, V, dO, Mst, Lst, Delta, p, hb / p.H, hb % p.H, (nqt - 1 - i / heads) * BR);
  }
}

template <int D>
static int32_t launch_fwd(float* O, const float* Q, const float* K, const float* V, float* M, float* L, const AttnParams& p,
                          cudaStream_t st) {
  auto kern = D == 128 || p.Sk <= kFineKeys ? fwd_kernel<D, true> : fwd_kernel<D, D == 128>;
  TYLO_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdSmem<D>::kBytes));
  const long long grid = (long long)((p.Sq + BR - 1) / BR) * p.H * p.B;
  TYLO_REQUIRE(grid <= 0x7fffffffLL, TYLO_ERR_UNSUPPORTED, "attention: problem too large for one launch");
  kern<<<(unsigned)grid, kThreads, FwdSmem<D>::kBytes, st>>>(O, Q, K, V, M, L, p);
  return check_launch("attn_fwd_f32");
}

template <int D>
static int32_t launch_bwd(float* dQ, float* dK, float* dV, const float* Q, const float* K, const float* V, const float* O,
                          const float* dO, const float* M, const float* L, float* Delta, const AttnParams& p, cudaStream_t st) {
  const long long rows = (long long)p.Sq * p.H * p.B;
  const long long n_keys = (long long)((p.Sk + BR - 1) / BR) * p.Hkv * p.B, n_q = (long long)((p.Sq + BR - 1) / BR) * p.H * p.B;
  TYLO_REQUIRE(n_keys + n_q <= 0x7fffffffLL, TYLO_ERR_UNSUPPORTED, "attention backward: problem too large");
  delta_kernel<<<(unsigned)((rows + 31) / 32), 256, 0, st>>>(Delta, O, dO, rows, p.Dk);
  if (int32_t rc = check_launch("attn_bwd_f32_delta")) return rc;
  auto kern = D == 128 || p.Sk <= kFineKeys ? bwd_kernel<D, true> : bwd_kernel<D, D == 128>;
  TYLO_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdSmem<D>::kBytes));
  kern<<<(unsigned)(n_keys + n_q), kThreads, BwdSmem<D>::kBytes, st>>>(dQ, dK, dV, Q, K, V, dO, M, L, Delta, p, (int)n_keys);
  return check_launch("attn_bwd_f32");
}

}  // namespace f32

// (the entry points refuse arrays that are not 16-byte aligned)
static bool f32_covers(const AttnParams& p, int32_t dtype) {
  return dtype == TYLO_F32 && p.Dk == p.Dv && p.Dk % 4 == 0 && p.Dk >= 4 && p.Dk <= 128 && !p.bm_count;
}

// Where the 32 x 32 tiles of attn_generic.cu are still the better ones: calls of one key tile, in which one group of threads
// works while the others (three of four at head dims up to 64) wait, on one CTA per SM where the general kernel has four or
// more.  Times in us, general kernel / this one, B 64 H 8 unless stated:
bool attn_fwd_f32_preferred(const AttnParams& p, int32_t dtype) {
  if (!f32_covers(p, dtype)) return false;
  const bool cap = p.score_flags & TYLO_SCORE_SOFTCAP;
  const bool waves = (long long)((p.Sq + f32::BR - 1) / f32::BR) * p.H * p.B > sm_count();      // more CTAs than SMs
  if (p.Dk > 64)               // two groups: S 32 D 128 55 / 57, with a soft cap 57 / 71; from 33 on ours: 109 / 62
    return !(waves && p.Sq <= 32 && p.Sk <= 32);
  if (p.Sk <= 32) return false;                                      // S 32 D 64: 37 / 60; 1 x 32: 33 / 65; B 1 H 4 1 x 32 warm: 7.4 / 10
  if (cap && p.Sk <= 64) return false;                               // (64 tanh in a row per thread) S 50 D 64: 84 / 117
  if (waves && p.Sq <= 32) return !(p.Sk <= 64 || (cap && p.Sk <= 256));    // bias 8 x 64 D 64: 35 / 50; soft cap 32 x 100: 58 / 72
  return true;
}
bool attn_bwd_f32_preferred(const AttnParams& p, int32_t dtype) {
  if (!f32_covers(p, dtype)) return false;
  // score mods on a single half-empty tile, CTAs for more than three waves: bias S 32 D 64 152 / 180 (B 20: 82 / 73, B 1: 53 / 29)
  return !(p.Dk <= 64 && p.score_flags && p.Sq <= 32 && p.Sk <= 32 && (long long)(p.H + p.Hkv) * p.B > 3 * sm_count());
}

int32_t attn_fwd_f32(void* O, const void* Q, const void* K, const void* V, float* M, float* L, const AttnParams& p, cudaStream_t st) {
  auto run = p.Dk > 64 ? f32::launch_fwd<128> : (p.Dk > 32 ? f32::launch_fwd<64> : f32::launch_fwd<32>);
  return run((float*)O, (const float*)Q, (const float*)K, (const float*)V, M, L, p, st);
}

int32_t attn_bwd_f32(void* dQ, void* dK, void* dV, const void* Q, const void* K, const void* V, const void* O, const void* dO,
                     const float* M, const float* L, float* Delta, const AttnParams& p, cudaStream_t st) {
  auto run = p.Dk > 64 ? f32::launch_bwd<128> : (p.Dk > 32 ? f32::launch_bwd<64> : f32::launch_bwd<32>);
  return run((float*)dQ, (float*)dK, (float*)dV, (const float*)Q, (const float*)K, (const float*)V, (const float*)O,
             (const float*)dO, M, L, Delta, p, st);
}

}  // namespace tylo
