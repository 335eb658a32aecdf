// One decode step of the whole language model - embedding, every block, final norm and head - for a handful of sequences,
// as ONE cooperative kernel.
//
// A step of generate() (algebraic_model.py:239-265) with a key/value cache moves every weight once through the GPU for 1-16
// tokens: for the small model (110 M parameters, 8 sequences, 530 cached tokens) 219 MB of weights and 160 MB of cache,
// 58 us at the copy bandwidth.  Issued operator by operator it is about 110 launches of 2-9 us that each wait for the one
// before: 455 us on the GPU and 2.6 ms on the host (this kernel: 373 us).  What bounds it is latency, so this kernel keeps one CTA per SM
// resident for the whole step and the CTAs hand their results on through L2, five times per block of the model:
//   P1  h += pending, y = norm(h) (every CTA for itself), qkv = y Wqkv^T
//   P2  attention of the new token over the cache, one (batch, head) pair - or a share of its keys - per CTA; appends the row
//   P3  o = attention Wo^T
//   P4  h += o, y' = norm(h), act = swiglu(y' Wgate^T, y' Wvalue^T)
//   P5  pending = act Wdown^T
// and, after the last block, the final norm and the head.
// Hand-over: every 4 bytes travel with a 4-byte tag (launch, layer, phase) in one 8-byte word, and whoever needs a word polls
// that word; there is no grid-wide barrier.  A hand-over takes about 2.5 us of a phase's 6.  Buffers alternate between even and odd
// layers: a word of layer l is overwritten in layer l + 2 only after a chain of all-to-all phases that contains every reader
// of layer l (each CTA owns a P1 unit, the grid is cut to that), so no tag is lost.
// Weights and old cache rows do not depend on the phase before: every thread streams the 16-byte pieces it will use itself
// through a private ring in shared memory with cp.async, up to four chunks of four pieces ahead of their use, across phases and
// layers, so that they are there when the words of the phase before arrive.
// The code is one loop over the phases in which every routine appears once: with the phases written out one after the other
// (210 KB of instructions, more than the caches hold) fetching instructions took most of the time.
// Contractions: mma.sync m16n8k16 with the tokens as the 16 rows and 8 output columns per unit; a unit's K range is split
// over 8 or 16 warps and summed in shared memory in a fixed order (results are reproducible).  tcgen05 has nothing to give
// here: at 8-16 rows the tensor pipe idles either way, and registers can be filled before the wait.  The order of K inside
// an MMA is free, so a lane takes 8 consecutive elements (one 16-byte load) of a weight row as its share of two MMAs.
// Roundings: h, qkv, o, gate, value and pending are rounded to 16 bits where the operator-by-operator path rounds them (operands,
// cached rows and logits are 16-bit anyway), in every block, so that a step may run either way.  The two differ in the order of
// float32 sums; now and then that tips a rounding, which moves every later one: two such evaluations drift apart while both keep
// their distance from the exact result.  bfloat16 logits of 16-32 steps, 2-norm, this kernel / operators against 64 bits, and
// against each other: 2 blocks of width 768 0.0095 / 0.0095, 0.0062; 5 blocks 0.0142 / 0.0143, 0.0112; 12 blocks 0.0205 / 0.0205,
// 0.0187; 8 blocks of 1024 0.0220 / 0.0224, 0.0180.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace fat {
namespace {

constexpr int kLmThreads = 512, kLmWarps = kLmThreads / 32;
constexpr int kPieces = 4;                      // 16-byte pieces per chunk; a thread's ring holds 4, 2 or 1 chunks, whatever shared memory leaves
constexpr size_t kChunkBytes = size_t(kPieces) * kLmThreads * 16;
constexpr size_t kLmSmemLimit = 220 * 1024;
#ifdef FAT_LM_POLL_LIMIT                        // (test builds only)
constexpr int kPollLimit = FAT_LM_POLL_LIMIT;
#else
constexpr int kPollLimit = 1 << 21;             // about a second
#endif

struct LmLayerArgs {
  const void *norm1, *qkv, *out, *norm2, *gate_val, *down;
  void *k_cache, *v_cache;
  const void* slopes;
};
struct LmArgs {
  LmLayerArgs layer[FAT_LM_MAX_LAYERS];
  const int64_t* ids; const void* embed; const void* norm; const void* head; void* logits; int* n_cached; int* status;
  unsigned* ctl;                                // [0] launches so far, [1] CTAs that have left this one, [2] one of them gave up waiting (both 0 between launches),
                                                // [3] some step since the workspace was zeroed gave up
  // tagged words, two copies each (even / odd layers): float32 values qkv [B][3C], o [B][C], pend [B][C], part [B*H][n_split]
  // [D + 2] (n_split > 1); pairs of 16-bit values att [B][C/2], act [B][act_words]
  uint2 *qkv, *o, *pend, *att, *act, *part;
  int64_t ids_stride, cs_b, cs_h, cs_t;
  int L, B, C, H, F, V, capacity, act_words, n_split, slopes_f32, a_stride, down_bytes;
  float scale, eps_norm, eps_attn;
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void upk2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

template <typename T> struct Pair16;
template <> struct Pair16<__nv_bfloat16> {
  static __device__ __forceinline__ float2 get(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
  static __device__ __forceinline__ uint32_t put(float a, float b) { __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <> struct Pair16<__half> {
  static __device__ __forceinline__ float2 get(uint32_t w) { return __half22float2(*reinterpret_cast<__half2*>(&w)); }
  static __device__ __forceinline__ uint32_t put(float a, float b) { __half2 v = __floats2half2_rn(a, b); return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

// BYTES (4 or 16) from global to shared memory without waiting; zeros if !in.
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src, bool in) {
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16u : 0u) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4u : 0u) : "memory");
}

// ------------------------------------------------------------------------------------------------- tagged words
// A word is one 64-bit element of every access, so that its value and its tag are seen together (a vector access promises that
// for each of its elements, not for the whole).  Two neighbouring words: (value, tag, value, tag).
__device__ __forceinline__ uint4 ld_words(const uint2* p) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
}
__device__ __forceinline__ uint64_t word_of(uint32_t value, unsigned tag) { return uint64_t(tag) << 32 | value; }
__device__ __forceinline__ void st_words(uint2* p, uint32_t a, uint32_t b, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(word_of(a, tag)), "l"(word_of(b, tag)) : "memory");
}
__device__ __forceinline__ void st_word(uint2* p, uint32_t a, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(word_of(a, tag)) : "memory");
}

struct Poller {
  volatile int* failed;                          // shared memory: a wait has run out in this CTA (later waits return at once)
  int* status;
  __device__ __forceinline__ void give_up() const {
    *failed = 1;
    if (status) atomicCAS(status, 0, (FAT_DEV_WAIT_TIMEOUT << 24) | 300);
  }
  // v[i] = the words at src + i * step (words), i < n <= NB, once all of them carry the tag.  The first is polled alone, so
  // that waiting threads ask for 16 bytes at a time.  ODD: the last pair's second word does not exist.
  template <int NB>
  __device__ __forceinline__ void wait(uint4 (&v)[NB], const uint2* src, int step, int n, unsigned tag, bool odd = false) const {
    if (n <= 0) return;
    int it = 0;
#pragma unroll 1
    for (; it < kPollLimit; ++it) {
      v[0] = ld_words(src);
      if (v[0].y == tag && (v[0].w == tag || (odd && n == 1))) break;
      if (*failed) return;
    }
    if (NB > 1) {
      bool ok = false;
#pragma unroll 1
      for (; it < kPollLimit && !ok; ++it) {
        ok = true;
#pragma unroll
        for (int i = 1; i < NB; ++i)
          if (i < n) v[i] = ld_words(src + i * step);
#pragma unroll
        for (int i = 1; i < NB; ++i)
          if (i < n) ok = ok && v[i].y == tag && (v[i].w == tag || (odd && i == n - 1));
        if (*failed) return;
      }
    }
    if (it >= kPollLimit) give_up();
  }
};

template <typename T> __device__ __forceinline__ float as_stored(float v) { return Elem<T>::to_c(Elem<T>::from_c(v)); }

// A[token][0..C) = norm(h) for all tokens, h = the tokens' embedding rows (add == nullptr) or h + add; every CTA keeps the residual
// stream h [token][C] for itself in shared memory.  16 / (8 MR) warps per token; a thread owns the same columns every time.
template <typename T, int MR>
__device__ __forceinline__ void norm_into(unsigned char* A, int a_stride, float* h, float* sums, const LmArgs& p, const Poller& poll, const uint2* add,
                                          unsigned tag, const void* weight) {
  constexpr int WPT = 2 / MR, NT = 32 * WPT, NB = 6;
  const int warp = threadIdx.x >> 5, tok = warp / WPT, idx = threadIdx.x % NT, C2 = p.C / 2;
  float sum = 0.f;
  float2* hr = reinterpret_cast<float2*>(h + tok * p.C);
  if (tok < p.B) {
    if (!add) {
      const int64_t id = p.ids[tok * p.ids_stride];
      const bool known = id >= 0 && id < p.V;     // an id outside the vocabulary makes the token's logits NaN
      const uint32_t* row = reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.embed) + (known ? id : 0) * p.C);
#pragma unroll 1
      for (int c = idx; c < C2; c += NT) {
        float2 a = Pair16<T>::get(__ldg(row + c));
        if (!known) a.x = a.y = __int_as_float(0x7fc00000);
        sum += fabsf(a.x) + fabsf(a.y);
        hr[c] = a;
      }
    } else {
#pragma unroll 1
      for (int c0 = idx; c0 < C2; c0 += NT * NB) {
        uint4 v[NB];
        poll.wait<NB>(v, add + int64_t(tok) * p.C + 2 * c0, 2 * NT, min(NB, (C2 - c0 + NT - 1) / NT), tag);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int c = c0 + i * NT;
          if (c < C2) {
            float2 a = hr[c];
            a.x = as_stored<T>(a.x + __uint_as_float(v[i].x));
            a.y = as_stored<T>(a.y + __uint_as_float(v[i].z));
            sum += fabsf(a.x) + fabsf(a.y);
            hr[c] = a;
          }
        }
      }
    }
  }
  sum = warp_sum(sum);
  if (WPT > 1) {
    if ((threadIdx.x & 31) == 0) sums[warp] = sum;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + tok), "r"(NT) : "memory");
    sum = sums[warp & ~1] + sums[warp | 1];
  }
  if (tok < p.B) {
    const float inv = 1.0f / (sum / float(p.C) + p.eps_norm);
    uint32_t* ar = reinterpret_cast<uint32_t*>(A + tok * a_stride);
#pragma unroll 2
    for (int c = idx; c < C2; c += NT) {
      const float2 a = hr[c], g = Pair16<T>::get(__ldg(static_cast<const uint32_t*>(weight) + c));
      ar[c] = Pair16<T>::put(a.x * inv * g.x, a.y * inv * g.y);
    }
  }
}

// A[token] = rows of 16-bit pairs, `words` tagged words per row (rows an even number of words apart)
template <int MR>
__device__ __forceinline__ void rows_into(unsigned char* A, int a_stride, const LmArgs& p, const Poller& poll, const uint2* src, int words, unsigned tag) {
  constexpr int WPT = 2 / MR, NT = 32 * WPT, NB = 4;
  const int tok = (threadIdx.x >> 5) / WPT, idx = threadIdx.x % NT, per_row = (words + 1) >> 1;
  if (tok >= p.B) return;
#pragma unroll 1
  for (int c0 = idx; c0 < per_row; c0 += NT * NB) {
    uint4 v[NB];
    const int n = min(NB, (per_row - c0 + NT - 1) / NT), last = c0 + (n - 1) * NT;
    const bool odd = 2 * last + 1 >= words;      // the row's last pair lacks its second word
    poll.wait<NB>(v, src + 2 * (int64_t(tok) * per_row + c0), 2 * NT, n, tag, odd);
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (i < n) *reinterpret_cast<uint2*>(A + tok * a_stride + (c0 + i * NT) * 8) = make_uint2(v[i].x, odd && i == n - 1 ? 0u : v[i].z);
  }
}

// ------------------------------------------------------------------------------------------------- attention
// A (batch, head) pair, or a share of its cached rows.
struct Item { int64_t rows; int b, h, share, n, lo, hi; };                 // rows: offset of the pair in the caches; n: cached rows, -1 = no room
__device__ __noinline__ Item item_at(const LmArgs& p, int item) {
  Item r;
  r.share = item % p.n_split;
  const int pair = item / p.n_split;
  r.b = pair / p.H;
  r.h = pair - r.b * p.H;
  r.rows = r.b * p.cs_b + r.h * p.cs_h;
  r.n = __ldcg(p.n_cached + r.b);
  if (r.n < 0 || r.n >= p.capacity) r.n = -1;
  const int n = max(r.n, 0), per = ((n + p.n_split - 1) / p.n_split + 15) / 16 * 16;
  r.lo = r.share * per;
  r.hi = min(n, r.lo + per);
  return r;
}

// A = attention rows from the partial sums of the key shares
template <typename T, int D>
__device__ __forceinline__ void combine_into(unsigned char* A, int a_stride, const LmArgs& p, const Poller& poll, const uint2* part, unsigned tag) {
#pragma unroll 1
  for (int i = threadIdx.x; i < p.B * p.C / 2; i += kLmThreads) {
    const int b = i / (p.C / 2), c = 2 * (i - b * (p.C / 2)), h = c / D, d = c % D;
    const uint2* pt = part + int64_t(b * p.H + h) * p.n_split * (D + 2);
    float a0 = 0.f, a1 = 0.f, L = 0.f;
#pragma unroll 1
    for (int s = 0; s < p.n_split; ++s) {
      uint4 v[1], l[1];
      poll.wait<1>(v, pt + s * (D + 2) + d, 0, 1, tag);
      poll.wait<1>(l, pt + s * (D + 2) + D, 0, 1, tag, true);
      a0 += __uint_as_float(v[0].x);
      a1 += __uint_as_float(v[0].z);
      L += __uint_as_float(l[0].x);
    }
    *reinterpret_cast<uint32_t*>(A + b * a_stride + c * 2) = Pair16<T>::put(a0 / (L + p.eps_attn), a1 / (L + p.eps_attn));
  }
}

// ------------------------------------------------------------------------------------------------- the step
// One contraction: W is `sets` blocks of N rows of K elements; warps share a unit of 8 output columns (1 << wpu_log2 of them)
// and each takes every such block of 32 elements of K, kPieces of them per chunk.
struct Contraction { const void* W; int N, K, wpu_log2, sets; };
__device__ __forceinline__ Contraction contraction(const LmArgs& p, int li, int ph) {     // ph: 0 qkv (or the head), 1 out, 2 gate/value, 3 down
  if (li == p.L) return {p.head, p.V, p.C, 3, 1};
  const LmLayerArgs& ly = p.layer[li];
  if (ph == 0) return {ly.qkv, 3 * p.C, p.C, 3, 1};
  if (ph == 1) return {ly.out, p.C, p.C, 4, 1};
  if (ph == 2) return {ly.gate_val, p.F, p.C, 3, 2};
  return {ly.down, p.C, p.F, 4, 1};
}

// The stream of chunks of one warp, in the order of their use: li, ph as above, with the cached rows (ph 4) before ph 1.
template <typename T, int D, int kStages>
struct Stream {
  static constexpr int LPR = D / 8, RPW = 32 / LPR, kStep = kLmWarps * RPW * kPieces;      // lanes per cache row, rows per warp and piece, rows per step
  const LmArgs& p;
  uint32_t ring;                                 // this thread's first slot
  int ask_stage, use_stage;
  int li, ph, unit, sub;                         // what is asked for next
  Contraction c;
  Item it;
  int item;

  __device__ __forceinline__ Stream(const LmArgs& args, unsigned char* smem) : p(args) {
    ring = uint32_t(__cvta_generic_to_shared(smem)) + threadIdx.x * 16;
    ask_stage = use_stage = 0;
    li = 0;
    start(0);
  }
  __device__ __forceinline__ int first_unit(int wpu_log2) const { return int(blockIdx.x) + ((threadIdx.x >> 5) >> wpu_log2) * int(gridDim.x); }
  __device__ __forceinline__ int unit_step(int wpu_log2) const { return int(gridDim.x) * (kLmWarps >> wpu_log2); }
  __device__ __forceinline__ static int chunks_per_set(const Contraction& c) {
    const int blocks = (c.K + 31) >> 5, per = kPieces << c.wpu_log2;
    return (blocks + per - 1) >> (c.wpu_log2 + 2);
  }
  __device__ __forceinline__ void start(int phase) {
    ph = phase;
    sub = 0;
    if (ph == 4) {
      item = blockIdx.x;
      if (item < p.B * p.H * p.n_split) it = item_at(p, item);
    } else {
      c = contraction(p, li, ph);
      unit = first_unit(c.wpu_log2);
    }
  }
  // Asks for the next chunk (an empty one after the last: the waits count chunks).
  __device__ __forceinline__ void ask() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t dst = ring + uint32_t(ask_stage) * uint32_t(kChunkBytes);
    ask_stage = (ask_stage + 1) % kStages;
    while (li <= p.L) {
      if (ph == 4) {                             // rows it.lo + (sub / 2) kStep .. of the keys (sub even) or values (odd)
        if (item < p.B * p.H * p.n_split) {
          const int base = it.lo + (sub >> 1) * kStep;
          if (base < it.hi) {
            const T* rows = static_cast<const T*>((sub & 1) ? p.layer[li].v_cache : p.layer[li].k_cache) + it.rows + (lane % LPR) * 8;
#pragma unroll
            for (int u = 0; u < kPieces; ++u) {
              const int j = base + (u * kLmWarps + warp) * RPW + lane / LPR;
              copy_async<16>(dst + u * (kLmThreads * 16), rows + (j < it.hi ? j : it.lo) * p.cs_t, j < it.hi);
            }
            ++sub;
            break;
          }
          item += gridDim.x;
          sub = 0;
          if (item < p.B * p.H * p.n_split) it = item_at(p, item);
          continue;
        }
      } else if (unit * 8 < c.N) {
        const int g = lane >> 2, t = lane & 3, part = warp & ((1 << c.wpu_log2) - 1), per_set = chunks_per_set(c);
        const int set = sub >= per_set ? 1 : 0, first = (sub - set * per_set) * kPieces;
        const int n = unit * 8 + g;
        const bool row_ok = n < c.N;
        const T* row = static_cast<const T*>(c.W) + (int64_t(set) * c.N + (row_ok ? n : 0)) * c.K;
        const int k0 = ((part + (first << c.wpu_log2)) << 5) + t * 8, kstep = 32 << c.wpu_log2;
        if (ph != 3 || p.down_bytes == 16) {
#pragma unroll
          for (int i = 0; i < kPieces; ++i) {
            const int k = k0 + i * kstep;
            const bool in = row_ok && k < c.K;
            copy_async<16>(dst + i * (kLmThreads * 16), row + (in ? k : 0), in);
          }
        } else if (p.down_bytes == 4) {
#pragma unroll 1
          for (int i = 0; i < kPieces * 4; ++i) {
            const int k = k0 + (i >> 2) * kstep + (i & 3) * 2;
            const bool in = row_ok && k < c.K;
            copy_async<4>(dst + (i >> 2) * (kLmThreads * 16) + (i & 3) * 4, row + (in ? k : 0), in);
          }
        } else {
          const uint16_t* r16 = reinterpret_cast<const uint16_t*>(row);
#pragma unroll 1
          for (int i = 0; i < kPieces; ++i) {
            const int k = k0 + i * kstep;
#pragma unroll 2
            for (int j = 0; j < 8; ++j) {
              const uint16_t e = row_ok && k + j < c.K ? __ldg(r16 + k + j) : uint16_t(0);
              asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + i * (kLmThreads * 16) + j * 2), "h"(e) : "memory");
            }
          }
        }
        if (++sub == per_set * c.sets) { sub = 0; unit += unit_step(c.wpu_log2); }
        break;
      }
      if (ph == 3 || li == p.L) { if (++li <= p.L) start(0); }
      else start(ph == 0 ? 4 : ph == 4 ? 1 : ph + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // The oldest chunk, once it has arrived (kStages chunks are always outstanding before).
  __device__ __forceinline__ void use(uint4 (&v)[kPieces]) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
    const uint32_t src = ring + uint32_t(use_stage) * uint32_t(kChunkBytes);
    use_stage = (use_stage + 1) % kStages;
#pragma unroll
    for (int i = 0; i < kPieces; ++i)
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w) : "r"(src + i * (kLmThreads * 16)) : "memory");
  }
};

// Attention of one item: scores, weights and weighted values of the cached rows from the stream and of the new row from the
// projection's words; appends the new row.
template <typename T, int D, int kStages>
__device__ __forceinline__ void attend(const LmArgs& p, const LmLayerArgs& ly, const Poller& poll, Stream<T, D, kStages>& st, const Item& r, int item, float* red,
                                       const uint2* qkv_words, uint2* att_words, uint2* part_words, unsigned tag_in, unsigned tag_out) {
  using S = Stream<T, D, kStages>;
  constexpr int LPR = S::LPR, RPW = S::RPW;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane / LPR, c = lane % LPR;
  const uint2* qkv = qkv_words + int64_t(r.b) * 3 * p.C + r.h * D + c * 8;
  const float slope = p.slopes_f32 ? static_cast<const float*>(ly.slopes)[r.h] : Elem<T>::to_c(static_cast<const T*>(ly.slopes)[r.h]);
  f32x2 q2[4], acc2[4];
  {
    uint4 w[4];
    poll.wait<4>(w, qkv, 2, 4, tag_in);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q2[i] = pk2(__uint_as_float(w[i].x) * p.scale, __uint_as_float(w[i].z) * p.scale);
      acc2[i] = pk2(0.f, 0.f);
    }
  }
  auto dot = [&](const uint4& raw) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&raw);
    f32x2 t = pk2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = Pair16<T>::get(w[i]); t = fma2(q2[i], pk2(f.x, f.y), t); }
    float a, d;
    upk2(t, a, d);
    return a + d;
  };
  auto add = [&](float f, const uint4& raw) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&raw);
    const f32x2 f2 = pk2(f, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 e = Pair16<T>::get(w[i]); acc2[i] = fma2(f2, pk2(e.x, e.y), acc2[i]); }
  };
  auto weight = [&](float x, int j) {                                      // sigma(x - slope (n - j))^4
    const float sc = x - slope * float(r.n - j);
    const float sig = fmaf(sc * rcp1p_abs(sc), 0.5f, 0.5f);
    const float s2 = sig * sig;
    return s2 * s2;
  };
  float l = 0.f;
  // four rows per lane group: their sums over LPR lanes by a transpose reduction, one sigmoid for the row this lane ends up with
  const bool up_a = (c & (LPR / 2)) != 0, up_b = (c & (LPR / 4)) != 0;
  const int my_u = 2 * int(up_a) + int(up_b), group0 = lane & ~(LPR - 1);
#pragma unroll 1
  for (int base = r.lo; base < r.hi; base += S::kStep) {
    uint4 w[kPieces];
    st.use(w);
    float d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) d[u] = dot(w[u]);
    const float a0 = (up_a ? d[2] : d[0]) + __shfl_xor_sync(0xffffffffu, up_a ? d[0] : d[2], LPR / 2);
    const float a1 = (up_a ? d[3] : d[1]) + __shfl_xor_sync(0xffffffffu, up_a ? d[1] : d[3], LPR / 2);
    float x = (up_b ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up_b ? a0 : a1, LPR / 4);
#pragma unroll
    for (int o = LPR / 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int j = base + (my_u * kLmWarps + warp) * RPW + g;
    const float f = j < r.hi ? weight(x, j) : 0.f;
    l += f;                                      // (every row is counted by LPR/4 lanes; undone after the loop)
#pragma unroll 1
    for (int again = 0; again < 2; ++again) {    // (one copy of the code that asks)
      if (again) {
        st.use(w);
#pragma unroll
        for (int u = 0; u < 4; ++u) add(__shfl_sync(0xffffffffu, f, group0 + (u >> 1) * (LPR / 2) + (u & 1) * (LPR / 4)), w[u]);
      }
      st.ask();
    }
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  l *= 4.0f / float(LPR);
  if (r.share == 0 && warp == 0 && r.n >= 0) {   // the new row (one lane group counts it)
    uint4 knew, vnew;
    {
      uint4 w[4], u[4];
      poll.wait<4>(w, qkv + p.C, 2, 4, tag_in);
      poll.wait<4>(u, qkv + 2 * p.C, 2, 4, tag_in);
      auto pair = [&](const uint4& e) { return Pair16<T>::put(__uint_as_float(e.x), __uint_as_float(e.z)); };      // as the cache keeps it
      knew = make_uint4(pair(w[0]), pair(w[1]), pair(w[2]), pair(w[3]));
      vnew = make_uint4(pair(u[0]), pair(u[1]), pair(u[2]), pair(u[3]));
    }
    float x = dot(knew);
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const float f = g == 0 ? weight(x, r.n) : 0.f;
    l += f;
    add(f, vnew);
    if (g == 0) {
      const int64_t at = r.rows + r.n * p.cs_t + c * 8;
      *reinterpret_cast<uint4*>(static_cast<T*>(ly.k_cache) + at) = knew;
      *reinterpret_cast<uint4*>(static_cast<T*>(ly.v_cache) + at) = vnew;
    }
  }
  if (r.n < 0 && r.share == 0 && tid == 0 && p.status) atomicOr(p.status, int(FAT_DEV_CACHE_FULL));
  float acc[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) upk2(acc2[i], acc[2 * i], acc[2 * i + 1]);
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
  }
  __syncthreads();                               // (whatever used `red` before is done)
  if (g == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) red[warp * (D + 1) + c * 8 + i] = acc[i];
    if (c == 0) red[warp * (D + 1) + D] = l;
  }
  __syncthreads();
  if (p.n_split > 1) {
    if (tid <= D) {
      float a = 0.f;
#pragma unroll 4
      for (int w = 0; w < kLmWarps; ++w) a += red[w * (D + 1) + tid];
      st_word(part_words + int64_t(item) * (D + 2) + tid, __float_as_uint(a), tag_out);
    }
  } else if (tid < D / 2) {
    float a0 = 0.f, a1 = 0.f, L = 0.f;
#pragma unroll 4
    for (int w = 0; w < kLmWarps; ++w) {
      a0 += red[w * (D + 1) + 2 * tid];
      a1 += red[w * (D + 1) + 2 * tid + 1];
      L += red[w * (D + 1) + D];
    }
    st_word(att_words + (int64_t(r.b) * p.C + r.h * D) / 2 + tid, Pair16<T>::put(a0 / (L + p.eps_attn), a1 / (L + p.eps_attn)), tag_out);
  }
}

// MR: 1 = up to 8 tokens, 2 = up to 16.
template <typename T, int D, int MR, int kStages>
__global__ void __launch_bounds__(kLmThreads, 1)
lm_decode_kernel(const __grid_constant__ LmArgs p) {
  extern __shared__ __align__(16) unsigned char lm_smem[];
  __shared__ int failed, last;
  __shared__ float sums[kLmWarps];
  constexpr int kTile = MR * 64;                 // partial sums of a warp: [row 0..MR*8)[col 0..8)
  unsigned char* A = lm_smem + kStages * kChunkBytes;
  const int as = p.a_stride;
  float* h = reinterpret_cast<float*>(A + MR * 8 * as);
  float* red = h + MR * 8 * p.C;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  Stream<T, D, kStages> st(p, lm_smem);
#pragma unroll 1
  for (int i = 0; i < kStages; ++i) st.ask();
  if (threadIdx.x == 0) failed = 0;
  const Poller poll{&failed, p.status};
  const int B = p.B, C = p.C, items = B * p.H * p.n_split;
#pragma unroll 1
  for (int i = threadIdx.x * 16; i < MR * 8 * as; i += kLmThreads * 16) *reinterpret_cast<uint4*>(A + i) = make_uint4(0u, 0u, 0u, 0u);
  const unsigned launch = __ldcg(p.ctl) << 10;
  Item mine{};
  if (int(blockIdx.x) < items) mine = item_at(p, blockIdx.x);
  __syncthreads();
  const uint2* add = nullptr;
#pragma unroll 1
  for (int step = 0; step <= 4 * p.L; ++step) {
    const int li = step >> 2, ph = step & 3;
    const LmLayerArgs& ly = p.layer[li < p.L ? li : 0];
    const unsigned tag = launch + li * 8 + 1;    // qkv words; + 1 attention, + 2 o, + 3 act, + 4 pending
    const int64_t odd = li & 1;
    uint2 *att = p.att + odd * B * C / 2, *part = p.part + odd * items * (D + 2), *act = p.act + odd * B * p.act_words;
    const Contraction cn = contraction(p, li, ph);
    const bool owner = int(blockIdx.x) * 8 < cn.N;         // (slot 0 has the CTA's first unit)
    if (ph == 1) {
#pragma unroll 1
      for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const Item it = item == int(blockIdx.x) ? mine : item_at(p, item);
        attend<T, D, kStages>(p, ly, poll, st, it, item, red, p.qkv + odd * B * 3 * C, att, part, tag, tag + 1);
      }
    }
    if (ph & 1) {
      if (owner) {
        if (ph == 1 && p.n_split > 1) combine_into<T, D>(A, as, p, poll, part, tag + 1);
        else rows_into<MR>(A, as, p, poll, ph == 1 ? att : act, ph == 1 ? C / 2 : (p.F + 1) / 2, ph == 1 ? tag + 1 : tag + 3);
      }
    } else {
      const void* w = li == p.L ? p.norm : ph == 0 ? ly.norm1 : ly.norm2;
      norm_into<T, MR>(A, as, h, sums, p, poll, add, ph == 0 ? tag - 4 : tag + 2, w);        // (tag - 4: the pending words of the layer before)
    }
    __syncthreads();
    // ---- this step's contraction
    {
      const int wpu = 1 << cn.wpu_log2, slot = warp >> cn.wpu_log2, wpart = warp & (wpu - 1), per_set = Stream<T, D, kStages>::chunks_per_set(cn);
      const int in_slot = wpart * 32 + lane;
      int buf = 0;                               // (the slots may count differently: every step starts over)
#pragma unroll 1
      for (int unit = st.first_unit(cn.wpu_log2); unit * 8 < cn.N; unit += st.unit_step(cn.wpu_log2)) {
        float* mine_red = red + buf * (kLmWarps * 2 * kTile) + slot * (wpu * 2 * kTile);     // [buf][slot][part][set]
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        int first = 0;
#pragma unroll 1
        for (int sub = 0; sub < per_set * cn.sets; ++sub) {
          uint4 w[kPieces];
          st.use(w);
#pragma unroll
          for (int i = 0; i < kPieces; ++i) {
            const int kb = wpart + ((first + i) << cn.wpu_log2);
            if (kb * 32 < cn.K) {                                          // the same for the whole warp
              const unsigned char* a = A + g * as + kb * 64 + t * 16;
              const uint4 lo = *reinterpret_cast<const uint4*>(a);
              const uint4 hi = MR == 2 ? *reinterpret_cast<const uint4*>(a + 8 * as) : make_uint4(0u, 0u, 0u, 0u);
              Pair16<T>::mma(acc, lo.x, hi.x, lo.y, hi.y, w[i].x, w[i].y);
              Pair16<T>::mma(acc, lo.z, hi.z, lo.w, hi.w, w[i].z, w[i].w);
            }
          }
          st.ask();
          first += kPieces;
          if (sub + 1 == per_set || sub + 1 == 2 * per_set) {              // a set is complete
            float* d = mine_red + (wpart * 2 + (sub + 1 == per_set ? 0 : 1)) * kTile + g * 8 + t * 2;
            *reinterpret_cast<float2*>(d) = make_float2(acc[0], acc[1]);
            if (MR == 2) *reinterpret_cast<float2*>(d + 64) = make_float2(acc[2], acc[3]);
            acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
            first = 0;
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(wpu * 32) : "memory");
        const int tok = in_slot >> 2, n = unit * 8 + (in_slot & 3) * 2;
        if (tok < B && n < cn.N) {
          float2 v0 = make_float2(0.f, 0.f), v1 = v0;
#pragma unroll 4
          for (int q = 0; q < wpu; ++q) {
            const float2 a = *reinterpret_cast<const float2*>(mine_red + q * 2 * kTile + in_slot * 2);
            v0.x += a.x;
            v0.y += a.y;
          }
          if (cn.sets == 2) {
#pragma unroll 4
            for (int q = 0; q < wpu; ++q) {
              const float2 a = *reinterpret_cast<const float2*>(mine_red + (q * 2 + 1) * kTile + in_slot * 2);
              v1.x += a.x;
              v1.y += a.y;
            }
          }
          if (li == p.L) {
            T* out = static_cast<T*>(p.logits) + int64_t(tok) * p.V + n;
            if (p.V % 2 == 0) *reinterpret_cast<uint32_t*>(out) = Pair16<T>::put(v0.x, v0.y);
            else {
              out[0] = Elem<T>::from_c(v0.x);
              if (n + 1 < p.V) out[1] = Elem<T>::from_c(v0.y);
            }
          } else {
            v0.x = as_stored<T>(v0.x);
            v0.y = as_stored<T>(v0.y);
            if (ph == 2) {
              const float a0 = v0.x * rsigmoid(v0.x, rcp1p_abs(v0.x)) * as_stored<T>(v1.x);
              const float a1 = v0.y * rsigmoid(v0.y, rcp1p_abs(v0.y)) * as_stored<T>(v1.y);
              st_word(act + int64_t(tok) * p.act_words + n / 2, Pair16<T>::put(a0, a1), tag + 3);
            } else {
#ifdef FAT_TEST_LM_WITHHOLD_UNIT
              // test builds only (never the shipped library): the words of this unit of the first block's projection are not written, so
              // every wait for them runs out
              if (li != 0 || ph != 0 || unit != FAT_TEST_LM_WITHHOLD_UNIT) {
#else
              {
#endif
              uint2* out = ph == 0 ? p.qkv + odd * B * 3 * C : ph == 1 ? p.o + odd * B * C : p.pend + odd * B * C;
              st_words(out + int64_t(tok) * cn.N + n, __float_as_uint(v0.x), __float_as_uint(v0.y), ph == 0 ? tag : ph == 1 ? tag + 2 : tag + 4);
              }
            }
          }
        }
        buf ^= 1;                                // (a buffer is written again only after the next barrier)
      }
    }
    __syncthreads();                             // A and `red` are free
    add = ph == 1 ? p.o + odd * B * C : ph == 3 ? p.pend + odd * B * C : nullptr;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // The last CTA to leave: nobody reads the lengths and the launch number any more.  A step in which a wait ran out (the words
  // behind it are whatever the CTA had in its registers, and spread) gives NaN logits and does not count.
  if (threadIdx.x == 0) {
    if (failed) atomicExch(p.ctl + 2, 1u);
    __threadfence();
    last = atomicAdd(p.ctl + 1, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const bool bad = __ldcg(p.ctl + 2) != 0u;
    if (bad)
#pragma unroll 1
      for (int64_t i = threadIdx.x; i < int64_t(B) * p.V; i += kLmThreads) static_cast<T*>(p.logits)[i] = Elem<T>::from_c(__int_as_float(0x7fc00000));
    __syncthreads();                             // (everyone has read the mark)
    if (threadIdx.x == 0) {
      if (bad) p.ctl[3] = 1u;
      p.ctl[2] = 0u;
      p.ctl[1] = 0u;
      p.ctl[0] += 1u;
#pragma unroll 1
      for (int b = 0; b < B; ++b)
        if (!bad && p.n_cached[b] >= 0 && p.n_cached[b] < p.capacity) p.n_cached[b] += 1;      // (a sequence without room has been given no row)
    }
  }
}

size_t round128(size_t n) { return (n + 127) / 128 * 128; }
int row_bytes(int K) { return (K * 2 + 127) / 128 * 128 + 64; }            // 8 lanes of a 16-byte shared load (two rows) cover all banks

struct Plan { size_t smem; int rows, stages, n_split, act_words, grid; };
// Whether the kernel takes the shape, and its layout.
bool plan_step(int B, int C, int H, int D, int F, int V, int L, int capacity, Plan* out) {
  if (B < 1 || B > 16 || L < 1 || L > FAT_LM_MAX_LAYERS || (D != 64 && D != 128) || C != H * D || F < 1 || V < 1 || capacity < 1) return false;
  const int rows = B <= 8 ? 8 : 16, wide = F > C ? F : C;
  out->rows = rows;
  out->smem = size_t(rows) * (row_bytes((wide + 31) / 32 * 32) + size_t(C) * sizeof(float)) + size_t(2 * kLmWarps * 2) * rows * 8 * sizeof(float);
  out->stages = 4;
  while (out->stages > 1 && out->smem + out->stages * kChunkBytes > kLmSmemLimit) out->stages /= 2;
  out->smem += out->stages * kChunkBytes;
  out->act_words = ((F + 1) / 2 + 1) / 2 * 2;
  out->grid = num_sms() < (3 * C + 7) / 8 ? num_sms() : (3 * C + 7) / 8;       // every CTA owns a unit of P1
  // a (batch, head) pair per CTA; with few pairs their keys are shared out, 64 rows of a full cache at least per share
  int s = out->grid / (B * H);
  if (s > 16) s = 16;
  while (s > 1 && capacity / s < 64) --s;
  out->n_split = s < 1 ? 1 : s;
  return out->smem <= kLmSmemLimit;
}

template <typename T, int D, int MR>
int launch_step(LmArgs& a, const Plan& pl, cudaStream_t st) {
  void (*kern)(const LmArgs) = pl.stages == 4 ? lm_decode_kernel<T, D, MR, 4> : pl.stages == 2 ? lm_decode_kernel<T, D, MR, 2> : lm_decode_kernel<T, D, MR, 1>;
  if (int rc = ready_kernel(reinterpret_cast<const void*>(kern), pl.smem, "lm_decode")) return rc;
  void* args[] = {&a};
  cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(unsigned(pl.grid)), dim3(kLmThreads), args, pl.smem, st);
  return check_launch("lm_decode");
}

template <typename T>
int launch_step_t(LmArgs& a, int D, const Plan& pl, cudaStream_t st) {
  if (D == 64) return pl.rows == 8 ? launch_step<T, 64, 1>(a, pl, st) : launch_step<T, 64, 2>(a, pl, st);
  return pl.rows == 8 ? launch_step<T, 128, 1>(a, pl, st) : launch_step<T, 128, 2>(a, pl, st);
}

}  // namespace
}  // namespace fat

using namespace fat;

extern "C" size_t fat_lm_decode_workspace_bytes(int B, int C, int H, int D, int F, int V, int n_layers, int capacity, int dtype) {
  Plan pl;
  if ((dtype != FAT_BF16 && dtype != FAT_F16) || !plan_step(B, C, H, D, F, V, n_layers, capacity, &pl)) return 0;
  const size_t row = size_t(B) * C;
  return 128 + 2 * sizeof(uint2) * (3 * row + row + row + row / 2 + size_t(B) * pl.act_words + (pl.n_split > 1 ? size_t(B) * H * pl.n_split * (D + 2) : 0)) + 6 * 128;
}

extern "C" int fat_lm_decode_step(const fat_lm_layer* layers, int n_layers, const int64_t* ids, int64_t ids_stride, const void* embed,
                                  const void* norm, const void* head, void* logits, int32_t* n_cached, const int64_t* cache_strides,
                                  int slopes_f32, void* workspace, size_t workspace_bytes, int B, int C, int H, int D, int F, int V,
                                  int capacity, double scale, double eps_norm, double eps_attn, int dtype, int* status, void* stream) {
  Plan pl;
  if (dtype != FAT_BF16 && dtype != FAT_F16) { set_error("lm_decode_step: unsupported dtype tag %d", dtype); return FAT_ERR_DTYPE; }
  if (!plan_step(B, C, H, D, F, V, n_layers, capacity, &pl)) {
    set_error("lm_decode_step: unsupported shape B=%d C=%d H=%d D=%d F=%d V=%d layers=%d capacity=%d", B, C, H, D, F, V, n_layers, capacity);
    return FAT_ERR_UNSUPPORTED;
  }
  if (!layers || !ids || !embed || !norm || !head || !logits || !n_cached || !cache_strides) { set_error("lm_decode_step: null pointer"); return FAT_ERR_NULL; }
  const size_t need = fat_lm_decode_workspace_bytes(B, C, H, D, F, V, n_layers, capacity, dtype);
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 127)) {
    set_error("lm_decode_step: workspace of %zu bytes (128-byte aligned, zeroed once) required, got %zu at %p", need, workspace_bytes, workspace);
    return FAT_ERR_WORKSPACE;
  }
  LmArgs a{};
  bool aligned = aligned16(embed) && aligned16(norm) && aligned16(head);
  for (int i = 0; i < 3; ++i) aligned = aligned && cache_strides[i] % 8 == 0;
  for (int i = 0; i < n_layers; ++i) {
    const fat_lm_layer& l = layers[i];
    if (!l.norm1 || !l.qkv || !l.out || !l.norm2 || !l.gate_val || !l.down || !l.k_cache || !l.v_cache || !l.slopes) {
      set_error("lm_decode_step: null pointer in layer %d", i);
      return FAT_ERR_NULL;
    }
    aligned = aligned && aligned16(l.norm1) && aligned16(l.qkv) && aligned16(l.out) && aligned16(l.norm2) && aligned16(l.gate_val) &&
              aligned16(l.down) && aligned16(l.k_cache) && aligned16(l.v_cache);
    a.layer[i] = {l.norm1, l.qkv, l.out, l.norm2, l.gate_val, l.down, l.k_cache, l.v_cache, l.slopes};
  }
  if (!aligned) { set_error("lm_decode_step: parameters and caches must be 16-byte aligned"); return FAT_ERR_ALIGNMENT; }
  unsigned char* w = static_cast<unsigned char*>(workspace);
  auto take = [&](size_t bytes) { unsigned char* r = w; w += round128(bytes); return r; };
  a.ctl = reinterpret_cast<unsigned*>(take(128));
  const size_t row = size_t(B) * C;
  auto words = [&](size_t n) { return reinterpret_cast<uint2*>(take(2 * n * sizeof(uint2))); };      // even and odd layers
  a.qkv = words(3 * row); a.o = words(row); a.pend = words(row); a.att = words(row / 2); a.act = words(size_t(B) * pl.act_words);
  a.part = pl.n_split > 1 ? words(size_t(B) * H * pl.n_split * (D + 2)) : nullptr;
  a.ids = ids; a.ids_stride = ids_stride; a.embed = embed; a.norm = norm; a.head = head; a.logits = logits; a.n_cached = n_cached; a.status = status;
  a.cs_b = cache_strides[0]; a.cs_h = cache_strides[1]; a.cs_t = cache_strides[2];
  a.L = n_layers; a.B = B; a.C = C; a.H = H; a.F = F; a.V = V; a.capacity = capacity; a.act_words = pl.act_words; a.n_split = pl.n_split;
  a.slopes_f32 = slopes_f32;
  a.down_bytes = F % 8 == 0 ? 16 : F % 2 == 0 ? 4 : 2;          // what the alignment of the down projection's rows allows
  a.a_stride = row_bytes(((F > C ? F : C) + 31) / 32 * 32);
  a.scale = float(scale); a.eps_norm = float(eps_norm); a.eps_attn = float(eps_attn);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == FAT_BF16 ? launch_step_t<__nv_bfloat16>(a, D, pl, st) : launch_step_t<__half>(a, D, pl, st);
}
