// Rational attention on the CUDA cores (fp32 accumulation): the path for float32 tensors
// (tensor cores cannot hold the 1e-5 bar in one pass), for head sizes the tcgen05 kernels
// do not cover, and the on-device cross-check of the tcgen05 path.
//
// What bounds it: the FMA pipe, as long as shared memory, issue slots and latencies keep up.  A CTA owns kOwn = 32 queries
// (forward, d_q) or keys (d_k/d_v) and streams tiles of kStream = 64 rows of the other side.  Short own tiles, handed out
// longest first over all heads, because small problems have few of them: 2x12 heads of 512 tokens are 384 CTAs of 1-8 steps;
// 64-row tiles left 192 for 148 SMs and twice the longest one's time.  (The backward of heads beyond 64, whose tiles leave an SM one
// CTA of four warps, takes 64 own rows where a launch has enough of them: long_tiles.)  Four threads per own row; a warp covers 16 x 32 scores, a thread
// 4 x 4 (rows 4 apart, columns 8 apart), so that no shared load has bank conflicts.  FMAs are issued as float32 pairs
// (fma.rn.f32x2: same pipe time, half the issue slots): along the head dimension in the score products, along the output
// columns in the others, whose weights lie doubled (w, w) in shared memory so that no register moves build the pairs.
// float32 tiles arrive by cp.async, each while a contraction that does not need its buffer runs; rows that cannot be moved in
// 16-byte pieces have kernels of their own (VEC), with eight element loads in flight (D = 70, 4x16x512, forward + backward: 1647 ->
// 852 us with the longer tiles; D = 30: 361 -> 290) and none of that code in the others.
// 2x12 heads, 512 tokens, D = 64, float32: forward 97 -> 57 us, d_q 133 -> 79 us, d_k/d_v 152 -> 78 us (64-row tiles of 256
// threads with synchronous loads before); eight steps of the contractions unrolled instead of four and the wider pitch of the
// doubled weights bring forward + backward from 201 to 193 us (sixteen steps: 199, two: 208).  With four steps: FMA pipe 40-45 % busy on an
// active SM at 8 warps per SM (before: 15-20 %): latency of the shared loads, and an SM's share of the CTAs (71 % of the longest SM's time on average).
// Backward is two kernels without atomics: a query-major one (Delta, d_q) and a key-major one (d_k, d_v), each
// recomputing the scores it needs.  No running maximum anywhere (sigma^4 <= 1).
#include <algorithm>

#include "attn_common.cuh"

namespace fat {
namespace {

constexpr int kOwn = 32, kStream = 64;           // (the backward also has tiles of 64 own rows: OWN)
constexpr int kPairLd = 2 * kStream + 16;       // pitch of the doubled weights [OWN][kStream] in floats: neighbouring rows half the banks apart

typedef unsigned long long f32x2;
__device__ __forceinline__ void upk2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

// This thread's place: score rows row(i) of the own tile, score columns col(j) of the streamed tile.
struct Lane {
  int ly, lx, wy, wx;
  __device__ __forceinline__ Lane() : ly((threadIdx.x & 31) >> 3), lx(threadIdx.x & 7), wy(threadIdx.x >> 6), wx((threadIdx.x >> 5) & 1) {}
  __device__ __forceinline__ int row(int i) const { return wy * 16 + ly + 4 * i; }
  __device__ __forceinline__ int col(int j) const { return wx * 32 + lx + 8 * j; }
};

// The CTA's tile: the grid runs over (tile, batch, head) with the tile slowest, whatever the caller wants first.
struct Tile { int b, h, tile; };
template <int OWN>
__device__ __forceinline__ Tile this_tile(const AttnParams& p) {
  const int tiles = (p.T + OWN - 1) / OWN, group = gridDim.x / tiles;         // H * B, or H with the batch on the y axis
  const int bh = blockIdx.y * group + blockIdx.x % group;
  return Tile{bh / p.H, bh % p.H, int(blockIdx.x) / group};
}

// dst[ROWS][DP + 4] = rows row0.. of base as float, zeros beyond T_len and D.  float32 rows that can be moved in 16-byte
// pieces are copied asynchronously (the caller waits with copies_done), everything else is there on return.
template <typename T, int DP, int ROWS, int NT, bool VEC>
__device__ __forceinline__ void load_tile(float* __restrict__ dst, const T* __restrict__ base,
                                          int64_t row_stride, int row0, int T_len, int D) {
  constexpr int LD = DP + 4;
  constexpr int W = 16 / sizeof(T);
  if constexpr (VEC) {
    constexpr int PPR = DP / W;
    if constexpr (sizeof(T) == 4) {
      const uint32_t s0 = uint32_t(__cvta_generic_to_shared(dst));
#pragma unroll 8
      for (int idx = threadIdx.x; idx < ROWS * PPR; idx += NT) {
        const int r = idx / PPR, c = (idx % PPR) * W, row = row0 + r;
        const bool in = row < T_len && c < D;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s0 + uint32_t(r * LD + c) * 4u),
                     "l"(base + (in ? int64_t(row) * row_stride + c : 0)), "r"(in ? 16u : 0u) : "memory");
      }
    } else {
#pragma unroll 2
      for (int idx = threadIdx.x; idx < ROWS * PPR; idx += NT) {
        const int r = idx / PPR, c = (idx % PPR) * W, row = row0 + r;
        float vals[W];
        if (row < T_len && c < D) {
          load_pack_cached<T, W>(base + int64_t(row) * row_stride + c, vals);
        } else {
#pragma unroll
          for (int j = 0; j < W; ++j) vals[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < W; j += 4)
          *reinterpret_cast<float4*>(&dst[r * LD + c + j]) = make_float4(vals[j], vals[j + 1], vals[j + 2], vals[j + 3]);
      }
    }
  } else {
#pragma unroll 8
    for (int idx = threadIdx.x; idx < ROWS * DP; idx += NT) {
      const int r = idx / DP, c = idx % DP, row = row0 + r;
      dst[r * LD + c] = (row < T_len && c < D) ? Elem<T>::to_c(base[int64_t(row) * row_stride + c]) : 0.f;
    }
  }
}
// Every copy of this thread has landed / those of all threads are visible.
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void copies_visible() { copies_done(); __syncthreads(); }

// s[i][j] = sum_d A[row(i)][d] * Bm[col(j)][d]     (A is [own][DP+4], Bm is [kStream][DP+4])
template <int DP>
__device__ __forceinline__ void gemm_nt(float (&s)[4][4], const float* __restrict__ A, const float* __restrict__ Bm, const Lane& ln) {
  constexpr int LD = DP + 4;
  f32x2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const float* a0 = A + ln.row(0) * LD;
  const float* b0 = Bm + ln.col(0) * LD;
#pragma unroll 8
  for (int d = 0; d < DP; d += 4) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a0 + 4 * i * LD + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(b0 + 8 * j * LD + d);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].y, b[j].y, acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      upk2(acc[i][j], lo, hi);
      s[i][j] = lo + hi;
    }
}

// Columns of the [own][DP] outputs: a warp has one half of them, a lane VW neighbours in each of NCH chunks.
template <int DP> struct OutCols {
  static constexpr int VW = DP >= 64 ? 4 : 2;
  static constexpr int NCH = DP / 16 / VW;
  static constexpr int NP = DP / 32;                                            // pairs per thread and row
  static __device__ __forceinline__ int col(const Lane& ln, int c) { return ln.wx * (DP / 2) + c * 8 * VW + ln.lx * VW; }
};
template <int DP> struct Out { f32x2 v[4][OutCols<DP>::NP]; };
template <int DP> __device__ __forceinline__ void clear(Out<DP>& o) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int n = 0; n < OutCols<DP>::NP; ++n) o.v[i][n] = 0ull;
}

// o[row(i)][*] += sum_k W[row(i)][k] * V[k][*]     (W doubled, V is [kStream][DP+4])
template <int DP>
__device__ __forceinline__ void gemm_nn(Out<DP>& o, const float* __restrict__ W, const float* __restrict__ V, const Lane& ln) {
  using OC = OutCols<DP>;
  constexpr int LD = DP + 4;
  const float* w0 = W + ln.row(0) * kPairLd;
#pragma unroll 8
  for (int k = 0; k < kStream; k += 2) {
    ulonglong2 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const ulonglong2*>(w0 + 4 * i * kPairLd + 2 * k);
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      f32x2 v[OC::NP];
#pragma unroll
      for (int c = 0; c < OC::NCH; ++c) {
        const float* at = V + (k + kk) * LD + OC::col(ln, c);
        if constexpr (OC::VW == 4) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(at);
          v[2 * c] = t.x;
          v[2 * c + 1] = t.y;
        } else {
          v[c] = *reinterpret_cast<const f32x2*>(at);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int n = 0; n < OC::NP; ++n) o.v[i][n] = fma2(kk ? w[i].y : w[i].x, v[n], o.v[i][n]);
    }
  }
}

// Writes o*mul to `base`; when `lo` is given also writes the rounding residual round(o*mul - stored).
template <typename T, int DP>
__device__ __forceinline__ void store_rows(T* __restrict__ base, int64_t row_stride, int row0, int T_len, int D,
                                           const Out<DP>& o, const float (&mul)[4], const Lane& ln, T* __restrict__ lo = nullptr) {
  using OC = OutCols<DP>;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + ln.row(i);
    if (row >= T_len) continue;
#pragma unroll
    for (int n = 0; n < OC::NP; ++n) {
      float val[2];
      upk2(o.v[i][n], val[0], val[1]);
      const int col = OC::col(ln, 2 * n / OC::VW) + 2 * n % OC::VW;
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (col + e < D) {
          const float x = val[e] * mul[i];
          const T hi = Elem<T>::from_c(x);
          base[int64_t(row) * row_stride + col + e] = hi;
          if (lo) lo[int64_t(row) * row_stride + col + e] = Elem<T>::from_c(x - Elem<T>::to_c(hi));
        }
    }
  }
}

__device__ __forceinline__ void put_pair(float* W, int row, int col, float w) {
  *reinterpret_cast<float2*>(W + row * kPairLd + 2 * col) = make_float2(w, w);
}

struct Score { float f, k; };   // f = sigma^4, k = 2 sigma^3 r^2 (derivative of f w.r.t. the score)

__device__ __forceinline__ Score score_terms(float qk, float scale, float slope, int row, int col) {
  const float s = qk * scale - slope * fabsf(float(row - col));
  const float r = rcp1p_abs(s);
  const float sg = rsigmoid(s, r);
  const float s2 = sg * sg;
  return Score{s2 * s2, 2.f * s2 * sg * r * r};
}

// ------------------------------------------------------------------ forward
template <typename T, int DP, bool VEC>
__global__ void __launch_bounds__(4 * kOwn, DP > 64 ? 2 : 3) attn_fwd_simt_kernel(AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = DP + 4, NT = 4 * kOwn;
  float* Qs = smem; float* Ks = Qs + kOwn * LD; float* Vs = Ks + kStream * LD; float* Ps = Vs + kStream * LD;
  const Lane ln;
  const Tile tl = this_tile<kOwn>(p);
  const int b = tl.b, h = tl.h, n_tiles = (p.T + kOwn - 1) / kOwn;
  const int q0 = (n_tiles - 1 - tl.tile) * kOwn;                               // long rows first
  const T* qb = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const T* kb = static_cast<const T*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const T* vb = static_cast<const T*>(p.v) + b * p.vs[0] + h * p.vs[1];
  T* ob = static_cast<T*>(p.out) + b * p.os[0] + h * p.os[1];
  const float slope = p.slopes[h];

  load_tile<T, DP, kOwn, NT, VEC>(Qs, qb, p.qs[2], q0, p.T, p.D);
  load_tile<T, DP, kStream, NT, VEC>(Ks, kb, p.ks[2], 0, p.T, p.D);
  Out<DP> o;
  clear(o);
  float l[4] = {0.f, 0.f, 0.f, 0.f};
  const int k_end = p.causal ? min(p.T, q0 + kOwn) : p.T;
#pragma unroll 1
  for (int k0 = 0; k0 < k_end; k0 += kStream) {
    copies_visible();                                                          // K is there, V and the weights are free
    load_tile<T, DP, kStream, NT, VEC>(Vs, vb, p.vs[2], k0, p.T, p.D);
    float s[4][4];
    gemm_nt<DP>(s, Qs, Ks, ln);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = k0 + ln.col(j);
      const bool kept = col < p.T && key_kept(p, b, col);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = q0 + ln.row(i);
        const bool live = kept && row < p.T && (!p.causal || col <= row);
        const float f = live ? score_terms(s[i][j], p.scale, slope, row, col).f : 0.f;
        l[i] += f;
        put_pair(Ps, ln.row(i), ln.col(j), f);
      }
    }
    copies_visible();                                                          // V is there, K is free
    if (k0 + kStream < k_end) load_tile<T, DP, kStream, NT, VEC>(Ks, kb, p.ks[2], k0 + kStream, p.T, p.D);
    gemm_nn<DP>(o, Ps, Vs, ln);
  }
  // a row's sum: over the eight lanes that share it, then over the two warps
  float* part = Qs;                                                            // (every score has been formed)
  float inv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], m);
    if (ln.lx == 0) part[ln.wx * kOwn + ln.row(i)] = l[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float sum = part[ln.row(i)] + part[kOwn + ln.row(i)];
    inv[i] = 1.f / (sum + p.eps);
    const int row = q0 + ln.row(i);
    if (ln.wx == 0 && ln.lx == 0 && row < p.T) p.L[(int64_t(b) * p.H + h) * p.T + row] = sum;
  }
  T* olo = p.out_lo ? static_cast<T*>(p.out_lo) + b * p.os[0] + h * p.os[1] : nullptr;
  store_rows<T, DP>(ob, p.os[2], q0, p.T, p.D, o, inv, ln, olo);
}

// ------------------------------------------------------------------ backward, query-major: Delta and d_q
template <typename T, int DP, bool VEC, int OWN>
__global__ void __launch_bounds__(4 * OWN, OWN > 32 ? 1 : DP > 64 ? 2 : 3) attn_bwd_dq_simt_kernel(AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = DP + 4, NT = 4 * OWN;
  float* Qs = smem; float* dOs = Qs + OWN * LD; float* Ks = dOs + OWN * LD; float* Vs = Ks + kStream * LD;
  float* dSs = Vs + kStream * LD; float* rowInv = dSs + OWN * kPairLd; float* rowD = rowInv + OWN;
  const Lane ln;
  const Tile tl = this_tile<OWN>(p);
  const int b = tl.b, h = tl.h, n_tiles = (p.T + OWN - 1) / OWN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = (n_tiles - 1 - tl.tile) * OWN;
  const T* qb = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const T* kb = static_cast<const T*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const T* vb = static_cast<const T*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const T* ob = static_cast<const T*>(p.out) + b * p.os[0] + h * p.os[1];
  const T* olo = p.out_lo ? static_cast<const T*>(p.out_lo) + b * p.os[0] + h * p.os[1] : nullptr;
  const T* dob = static_cast<const T*>(p.d_out) + b * p.dos[0] + h * p.dos[1];
  T* dqb = static_cast<T*>(p.d_q) + b * p.dqs[0] + h * p.dqs[1];
  const int64_t stat0 = (int64_t(b) * p.H + h) * p.T;
  const float slope = p.slopes[h];

  load_tile<T, DP, OWN, NT, VEC>(Qs, qb, p.qs[2], q0, p.T, p.D);
  load_tile<T, DP, OWN, NT, VEC>(dOs, dob, p.dos[2], q0, p.T, p.D);
  load_tile<T, DP, kStream, NT, VEC>(Ks, kb, p.ks[2], 0, p.T, p.D);
  load_tile<T, DP, kStream, NT, VEC>(Vs, vb, p.vs[2], 0, p.T, p.D);
#pragma unroll 2
  for (int r = warp * 8; r < warp * 8 + 8; ++r) {                              // Delta = d_out . (out + its rounding residual)
    const int row = q0 + r;
    float s = 0.f;
    if (row < p.T) {
#pragma unroll
      for (int d = lane; d < DP; d += 32)
        if (d < p.D) {
          float o = Elem<T>::to_c(ob[int64_t(row) * p.os[2] + d]);
          if (olo) o += Elem<T>::to_c(olo[int64_t(row) * p.os[2] + d]);
          s = fmaf(Elem<T>::to_c(dob[int64_t(row) * p.dos[2] + d]), o, s);
        }
    }
    s = warp_sum(s);
    if (lane == 0) {
      rowD[r] = s;
      rowInv[r] = row < p.T ? 1.f / (p.L[stat0 + row] + p.eps) : 0.f;
      if (row < p.T) p.delta[stat0 + row] = s;
    }
  }

  Out<DP> dq;
  clear(dq);
  const int k_end = p.causal ? min(p.T, q0 + OWN) : p.T;
#pragma unroll 1
  for (int k0 = 0; k0 < k_end; k0 += kStream) {
    copies_visible();
    float s[4][4], dp[4][4];
    gemm_nt<DP>(s, Qs, Ks, ln);
    gemm_nt<DP>(dp, dOs, Vs, ln);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = k0 + ln.col(j);
      const bool kept = col < p.T && key_kept(p, b, col);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int rl = ln.row(i), row = q0 + rl;
        const bool live = kept && row < p.T && (!p.causal || col <= row);
        put_pair(dSs, rl, ln.col(j), live ? score_terms(s[i][j], p.scale, slope, row, col).k * (dp[i][j] - rowD[rl]) * rowInv[rl] : 0.f);
      }
    }
    __syncthreads();                                                           // dS is there, V is free
    const bool more = k0 + kStream < k_end;
    if (more) load_tile<T, DP, kStream, NT, VEC>(Vs, vb, p.vs[2], k0 + kStream, p.T, p.D);
    gemm_nn<DP>(dq, dSs, Ks, ln);
    __syncthreads();                                                           // K and dS are free
    if (more) load_tile<T, DP, kStream, NT, VEC>(Ks, kb, p.ks[2], k0 + kStream, p.T, p.D);
  }
  copies_done();
  const float mul[4] = {p.scale, p.scale, p.scale, p.scale};
  store_rows<T, DP>(dqb, p.dqs[2], q0, p.T, p.D, dq, mul, ln);
}

// ------------------------------------------------------------------ backward, key-major: d_k and d_v
template <typename T, int DP, bool VEC, int OWN>
__global__ void __launch_bounds__(4 * OWN, OWN > 32 ? 1 : 2) attn_bwd_dkv_simt_kernel(AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = DP + 4, NT = 4 * OWN;
  float* Ks = smem; float* Vs = Ks + OWN * LD; float* Qs = Vs + OWN * LD; float* dOs = Qs + kStream * LD;
  float* PsT = dOs + kStream * LD; float* dSsT = PsT + OWN * kPairLd;
  const Lane ln;
  const Tile tl = this_tile<OWN>(p);                                                // early key tiles are the long ones
  const int b = tl.b, h = tl.h, k0 = tl.tile * OWN;
  const T* qb = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const T* kb = static_cast<const T*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const T* vb = static_cast<const T*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const T* dob = static_cast<const T*>(p.d_out) + b * p.dos[0] + h * p.dos[1];
  T* dkb = static_cast<T*>(p.d_k) + b * p.dks[0] + h * p.dks[1];
  T* dvb = static_cast<T*>(p.d_v) + b * p.dvs[0] + h * p.dvs[1];
  const int64_t stat0 = (int64_t(b) * p.H + h) * p.T;
  const float slope = p.slopes[h];

  int q0 = p.causal ? k0 / kStream * kStream : 0;
  load_tile<T, DP, OWN, NT, VEC>(Ks, kb, p.ks[2], k0, p.T, p.D);
  load_tile<T, DP, OWN, NT, VEC>(Vs, vb, p.vs[2], k0, p.T, p.D);
  load_tile<T, DP, kStream, NT, VEC>(Qs, qb, p.qs[2], q0, p.T, p.D);
  load_tile<T, DP, kStream, NT, VEC>(dOs, dob, p.dos[2], q0, p.T, p.D);
  bool kept[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int col = k0 + ln.row(i);
    kept[i] = col < p.T && key_kept(p, b, col);
  }
  Out<DP> dk, dv;
  clear(dk);
  clear(dv);
#pragma unroll 1
  for (; q0 < p.T; q0 += kStream) {
    float L[4], dlt[4];                                                        // of this thread's four queries
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = q0 + ln.col(j);
      L[j] = row < p.T ? p.L[stat0 + row] : 0.f;
      dlt[j] = row < p.T ? p.delta[stat0 + row] : 0.f;
    }
    copies_visible();
    float s[4][4], dp[4][4];
    gemm_nt<DP>(s, Ks, Qs, ln);
    gemm_nt<DP>(dp, Vs, dOs, ln);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = q0 + ln.col(j);
      const float inv = 1.f / (L[j] + p.eps);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cl = ln.row(i), col = k0 + cl;
        const bool live = kept[i] && row < p.T && (!p.causal || col <= row);
        const Score sc = score_terms(s[i][j], p.scale, slope, row, col);
        put_pair(PsT, cl, ln.col(j), live ? sc.f * inv : 0.f);
        put_pair(dSsT, cl, ln.col(j), live ? sc.k * (dp[i][j] - dlt[j]) * inv : 0.f);
      }
    }
    __syncthreads();
    gemm_nn<DP>(dv, PsT, dOs, ln);
    __syncthreads();                                                           // dO is free
    const bool more = q0 + kStream < p.T;
    if (more) load_tile<T, DP, kStream, NT, VEC>(dOs, dob, p.dos[2], q0 + kStream, p.T, p.D);
    gemm_nn<DP>(dk, dSsT, Qs, ln);
    __syncthreads();                                                           // Q and the weights are free
    if (more) load_tile<T, DP, kStream, NT, VEC>(Qs, qb, p.qs[2], q0 + kStream, p.T, p.D);
  }
  copies_done();
  const float one[4] = {1.f, 1.f, 1.f, 1.f};
  const float mul[4] = {p.scale, p.scale, p.scale, p.scale};
  store_rows<T, DP>(dvb, p.dvs[2], k0, p.T, p.D, dv, one, ln);
  store_rows<T, DP>(dkb, p.dks[2], k0, p.T, p.D, dk, mul, ln);
}

template <typename T>
bool tiles_vectorisable(const AttnParams& p, bool bwd) {
  constexpr int W = 16 / sizeof(T);
  if (p.D % W) return false;
  auto ok = [&](const void* ptr, const int64_t* s) {
    return aligned16(ptr) && s[0] % W == 0 && s[1] % W == 0 && s[2] % W == 0;
  };
  bool v = ok(p.q, p.qs) && ok(p.k, p.ks) && ok(p.v, p.vs);
  if (bwd) v = v && ok(p.out, p.os) && ok(p.d_out, p.dos);
  return v;
}

template <int OWN, typename Kern>
int launch(Kern kern, const AttnParams& p, size_t smem, cudaStream_t st, const char* what) {
  if (int rc = ready_kernel(reinterpret_cast<const void*>(kern), smem, what)) return rc;
  const int64_t column = int64_t((p.T + OWN - 1) / OWN) * p.H;
  const bool flat = column * p.B < (int64_t(1) << 31);                          // (otherwise the longest go first within a batch element)
  const dim3 grid(unsigned(flat ? column * p.B : column), unsigned(flat ? 1 : p.B));
  kern<<<grid, 4 * OWN, smem, st>>>(p);
  return check_launch(what);
}

// Whether the backward takes tiles of 64 own rows (256 threads) instead of 32.  From D = 65 on the tiles of either size leave room for
// one CTA per SM, and 32 rows are four warps: half the streamed rows per own row and twice the warps make a 64-row tile cost 1.5
// times a 32-row one, so it pays where a launch has enough tiles to keep every SM busy (waves of equal tiles, or the longest
// tile against an SM's share where the tiles are triangular).  D = 128 float32 backward, us, 32 / 64 rows: 4x16x512 741 / 582,
// 16x24x128 563 / 409, 2x8x512 175 / 251; not causal: 2x8x512 317 / 251, 2x12x512 468 / 493, 4x16x777 2800 / 2405.  D <= 64 has room for
// two to three CTAs of 32 rows, which always win (4x16x512, D = 64: 291 / 331); so they do in the forward (D = 128: 154 / 159).
bool long_tiles(const AttnParams& p) {
  const int64_t n = int64_t((p.T + 63) / 64) * p.B * p.H, sms = num_sms();
  auto waves = [&](int64_t tiles) { return p.causal ? std::max(1.0, 0.5 * double(tiles) / double(sms)) : double((tiles + sms - 1) / sms); };
  return 1.5 * waves(n) < waves(2 * n);
}

template <typename T, int DP, bool VEC>
int fwd_t(const AttnParams& p, cudaStream_t st) {
  constexpr size_t smem = (size_t(kOwn + 2 * kStream) * (DP + 4) + kOwn * kPairLd) * sizeof(float);
  return launch<kOwn>(attn_fwd_simt_kernel<T, DP, VEC>, p, smem, st, "attn_fwd_simt");
}

template <typename T, int DP, bool VEC, int OWN>
int bwd_own(const AttnParams& p, cudaStream_t st) {
  constexpr size_t tiles = size_t(2) * (OWN + kStream) * (DP + 4);
  constexpr size_t smem_dq = (tiles + OWN * kPairLd + 2 * OWN) * sizeof(float);
  constexpr size_t smem_dkv = (tiles + 2 * OWN * kPairLd) * sizeof(float);
  if (int rc = launch<OWN>(attn_bwd_dq_simt_kernel<T, DP, VEC, OWN>, p, smem_dq, st, "attn_bwd_dq_simt")) return rc;
  return launch<OWN>(attn_bwd_dkv_simt_kernel<T, DP, VEC, OWN>, p, smem_dkv, st, "attn_bwd_dkv_simt");
}
template <typename T, int DP, bool VEC>
int bwd_t(const AttnParams& p, cudaStream_t st) {
  if constexpr (DP > 64)
    if (long_tiles(p)) return bwd_own<T, DP, VEC, 64>(p, st);
  return bwd_own<T, DP, VEC, kOwn>(p, st);
}

template <typename T, int DP>
int dispatch_vec(const AttnParams& p, bool bwd, cudaStream_t st) {
  if (tiles_vectorisable<T>(p, bwd)) return bwd ? bwd_t<T, DP, true>(p, st) : fwd_t<T, DP, true>(p, st);
  return bwd ? bwd_t<T, DP, false>(p, st) : fwd_t<T, DP, false>(p, st);
}

template <typename T>
int dispatch_d(const AttnParams& p, bool bwd, cudaStream_t st) {
  if (p.D <= 32) return dispatch_vec<T, 32>(p, bwd, st);
  if (p.D <= 64) return dispatch_vec<T, 64>(p, bwd, st);
  if (p.D <= 128) return dispatch_vec<T, 128>(p, bwd, st);
  set_error("attention: head size %d is not supported (D <= 128)", p.D);
  return FAT_ERR_UNSUPPORTED;
}

int dispatch(const AttnParams& p, int dtype, bool bwd, cudaStream_t st) {
  switch (dtype) {
    case FAT_F32: return dispatch_d<float>(p, bwd, st);
    case FAT_BF16: return dispatch_d<__nv_bfloat16>(p, bwd, st);
    case FAT_F16: return dispatch_d<__half>(p, bwd, st);
    default: set_error("attention: unsupported dtype tag %d", dtype); return FAT_ERR_DTYPE;
  }
}

}  // namespace

int attn_fwd_simt(const AttnParams& p, int dtype, cudaStream_t st) { return dispatch(p, dtype, false, st); }
int attn_bwd_simt(const AttnParams& p, int dtype, cudaStream_t st) { return dispatch(p, dtype, true, st); }

}  // namespace fat
