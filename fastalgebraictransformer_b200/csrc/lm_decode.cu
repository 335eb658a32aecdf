// One decode step of the whole language model - embedding, every block, final norm and head - for a handful of sequences,
// as ONE cooperative kernel.
//
// A step of generate() (algebraic_model.py:239-265) with a key/value cache moves every weight once through the GPU for 1-16
// tokens: for the small model (110 M parameters, 8 sequences, 530 cached tokens) 219 MB of weights and 160 MB of cache,
// 58 us at the copy bandwidth.  Issued operator by operator it is about 110 launches of 2-9 us that each wait for the one
// before: 449 us on the GPU and 2.6 ms on the host (this kernel: 197 us).  What bounds it is latency, so this kernel keeps one CTA per SM
// resident for the whole step and the CTAs hand their results on through L2, five times per block of the model:
//   P1  h += pending, y = norm(h) (every CTA for itself), qkv = y Wqkv^T
//   P2  attention of the new token over the cache, one (batch, head) pair - or a share of its keys - per CTA; appends the row
//   P3  o = attention Wo^T
//   P4  h += o, y' = norm(h), act = swiglu(y' Wgate^T, y' Wvalue^T)
//   P5  pending = act Wdown^T
// and, after the last block, the final norm and the head.
// Hand-over: every 4 bytes travel with a 4-byte tag (launch, layer, phase) in one 8-byte word, and whoever needs a word polls
// that word; there is no grid-wide barrier.  A hand-over takes 0.7 to 1 us, 2 us for the words of act (65 KB per CTA that wants
// them).  Buffers alternate between even and odd layers: a word of layer l is overwritten in layer l + 2 only after a chain of all-to-all
// phases that contains every reader of layer l (each CTA owns a P1 unit, the grid is cut to that), so no tag is lost.
// Weights and old cache rows do not depend on the phase before: one warp streams them through a ring of chunks in shared memory with
// bulk copies, up to five chunks (165 KB) ahead of their use, across phases and layers, and the computing warps take their first
// pieces into registers before they wait for the words.  When every thread asked for its own pieces (cp.async) and worked out their
// addresses between the products and the hand-over, a step took 373 us: a warp issues an instruction every ten cycles here, so what
// counts is how few of them stand between the words and the results.  That is also why the usual widths are compiled in, why
// h, o, pending and qkv travel as the 16-bit pairs that they are rounded to anyway, and why scores come from the tensor cores.
// us per step, 12 blocks of 768, 512 cached tokens, before / after: 1 sequence 415 / 212, 8 sequences 379 / 197, 16 sequences 571 / 287;
// 8 sequences, 64 cached tokens 341 / 170, 1800 tokens 480 / 261.
// Taken back: fetching the next block's weights and rows into L2 ahead of the ring (8 sequences 212 -> 272, one sequence a little
// faster); keys of the next rows loaded behind the sums of these (registers spill); a copy of the tries on a barrier by one lane
// instead of 32 (slower to wake up).
// Contractions: mma.sync m16n8k16 with the tokens as the 16 rows and 8 output columns per unit; a unit's K range is split
// over 8 or 16 warps and summed in shared memory in a fixed order (results are reproducible).  tcgen05 has nothing to give
// here: at 8-16 rows the tensor pipe idles either way, and registers can be filled before the wait.  The order of K inside
// an MMA is free, so a lane takes 8 consecutive elements (one 16-byte load) of a weight row as its share of two MMAs.
// Roundings: h, qkv, o, gate, value and pending are rounded to 16 bits where the operator-by-operator path rounds them (operands,
// cached rows and logits are 16-bit anyway), in every block, so that a step may run either way.  The two differ in the order of
// float32 sums; now and then that tips a rounding, which moves every later one: two such evaluations drift apart while both keep
// their distance from the exact result.  bfloat16 logits of 16 steps, mean of four seeds, 2-norm, this kernel / the one whose scores were summed by
// float32 FMAs / operators against 64 bits, and this kernel against the operators: 2 blocks of width 768 0.00959 / 0.00958 / 0.00960, 0.0061; 5 blocks
// (heads of 128) 0.01444 / 0.01442 / 0.01443, 0.0114; 12 blocks 0.02062 / 0.02066 / 0.02059, 0.0184; 8 blocks of 1024 0.02154 / 0.02141 / 0.02181, 0.0183.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace fat {
namespace {

constexpr int kLmThreads = 512, kLmWarps = kLmThreads / 32;     // the warps that compute
constexpr int kLmBlock = kLmThreads + 128;     // and a warpgroup of which one warp loads (all four where cached rows are apart in memory)
constexpr int kLaunchRegs = 96, kComputeRegs = 104, kLoadRegs = 56;       // registers per thread: at launch (65536 / 640 threads), after the two groups have shared them out
static_assert(kLmThreads * kComputeRegs + 128 * kLoadRegs <= kLmBlock * kLaunchRegs, "the register shares must fit in what the launch allocates");
constexpr int kPieces = 4;                      // 16-byte pieces that a computing thread takes from a chunk
// A chunk of weights: for a unit of 8 output columns that 8 warps share, 8 rows of 1024 elements, and two such units; of one that 16
// warps share, 8 rows of 2048.  Rows are 64 bytes further apart than they are long: eight lanes of a 16-byte load (two rows) cover all banks.
__host__ __device__ constexpr int row_pitch(int wpu_log2) { return (kPieces * 64 << wpu_log2) + 64; }
constexpr int kChunkBytes = 16 * row_pitch(3);
static_assert(kChunkBytes >= 8 * row_pitch(4) && kChunkBytes >= kPieces * kLmThreads * 16, "a chunk holds 2 x 8 rows, 8 long rows, or cached rows");
constexpr int kMaxStages = 5;
constexpr size_t kLmSmemLimit = 226 * 1024;
constexpr size_t kTileLimit = 188 * 1024;      // of that, what the tokens' rows may take (see plan_step)
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
  // tagged words, two copies each (even / odd layers): pairs of 16-bit values qkv [B][3C/2], o [B][C/2], pend [B][C/2], att [B][C/2],
  // act [B][act_words]; float32 values part [B*H][n_split][D + 2] (n_split > 1)
  uint2 *qkv, *o, *pend, *att, *act, *part;
  int64_t ids_stride, cs_b, cs_h, cs_t;
  int L, B, C, H, F, V, capacity, act_words, n_split, slopes_f32, a_stride;
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

// ------------------------------------------------------------------------------------------------- tagged words
// A word is one 64-bit element of every access, so that its value and its tag are seen together (a vector access promises that
// for each of its elements, not for the whole).  Two neighbouring words: (value, tag, value, tag).
__device__ __forceinline__ uint4 ld_words(const uint2* p) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
}
__device__ __forceinline__ uint64_t word_of(uint32_t value, unsigned tag) { return uint64_t(tag) << 32 | value; }
__device__ __forceinline__ void st_word(uint2* p, uint32_t a, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(word_of(a, tag)) : "memory");
}

struct Poller {
  volatile int* failed;                          // shared memory: a wait has run out in this CTA (later waits return at once)
  // v[i] = the two words at src + at(i), i < n <= NB, once all of them carry the tag.
  template <int NB, typename At>
  __device__ __forceinline__ void wait(uint4 (&v)[NB], const uint2* src, At at, unsigned tag, int n = NB) const {
#pragma unroll 1
    for (int it = 0; it < kPollLimit; ++it) {
      bool ok = true;
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < n) v[i] = ld_words(src + at(i));
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < n) ok = ok && v[i].y == tag && v[i].w == tag;
      if (ok || *failed) return;
    }
    *failed = 1;
  }
};

// Adds the words of the phase before to the residual stream (ADD; otherwise the stream is there already), and A[token][0..C) = norm(h).
// Every CTA keeps the stream h [token][C] for itself in shared memory, as 16-bit values (it is rounded anyway).  16 / (8 MR) warps per
// token; a thread owns the same groups of four columns every time, NC MR of them where C = 256 NC (NC = 0: any number).
template <typename T, int MR, int NC, bool ADD>
__device__ __forceinline__ void norm_into(unsigned char* A, int a_stride, uint2* h, float* sums, const LmArgs& p, const Poller& poll, const uint2* add,
                                          unsigned tag, const uint2* weight) {
  constexpr int WPT = 2 / MR, NT = 32 * WPT, NB = NC ? NC * MR : 4;
  const int C = NC ? NC * 256 : p.C, C4 = C / 4;
  const int warp = threadIdx.x >> 5, tok = warp / WPT, idx = threadIdx.x % NT;
  float sum = 0.f;
  uint2* hr = h + tok * C4 + idx;
  weight += idx;
  if (tok < p.B) {
    const uint2* src = ADD ? add + tok * (C / 2) + 2 * idx : nullptr;
#pragma unroll 1
    for (int c0 = 0; c0 < (NC ? 1 : C4 - idx); c0 += NT * NB) {
      const int n = NC ? NB : min(NB, (C4 - idx - c0 + NT - 1) / NT);
      uint2 w[NB];
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (NC || i < n) w[i] = hr[c0 + i * NT];
      if (ADD) {
        uint4 v[NB];
        poll.wait<NB>(v, src + 2 * c0, [](int i) { return 2 * NT * i; }, tag, n);
#pragma unroll
        for (int i = 0; i < NB; ++i)
          if (NC || i < n) {
            const float2 a = Pair16<T>::get(w[i].x), b = Pair16<T>::get(w[i].y), da = Pair16<T>::get(v[i].x), db = Pair16<T>::get(v[i].z);
            w[i] = make_uint2(Pair16<T>::put(a.x + da.x, a.y + da.y), Pair16<T>::put(b.x + db.x, b.y + db.y));
            hr[c0 + i * NT] = w[i];
          }
      }
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (NC || i < n) {
          const float2 a = Pair16<T>::get(w[i].x), b = Pair16<T>::get(w[i].y);
          sum += (fabsf(a.x) + fabsf(a.y)) + (fabsf(b.x) + fabsf(b.y));
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
    const float inv = 1.0f / (sum / float(C) + p.eps_norm);
    uint2* ar = reinterpret_cast<uint2*>(A + tok * a_stride) + idx;
    auto scaled = [&](int c) {
      const uint2 w = hr[c], gw = weight[c];
      const float2 a = Pair16<T>::get(w.x), b = Pair16<T>::get(w.y), ga = Pair16<T>::get(gw.x), gb = Pair16<T>::get(gw.y);
      ar[c] = make_uint2(Pair16<T>::put(a.x * inv * ga.x, a.y * inv * ga.y), Pair16<T>::put(b.x * inv * gb.x, b.y * inv * gb.y));
    };
    if (NC) {
#pragma unroll
      for (int i = 0; i < NB; ++i) scaled(i * NT);
    } else {
#pragma unroll 1
      for (int c = 0; c < C4 - idx; c += NT) scaled(c);
    }
  }
}

// The residual stream of the first block: the tokens' embedding rows.
template <typename T, int MR>
__device__ __forceinline__ void embed_into(uint2* h, const LmArgs& p) {
  constexpr int NT = 32 * (2 / MR);
  const int tok = (threadIdx.x >> 5) / (2 / MR), C4 = p.C / 4;
  if (tok >= p.B) return;
  const int64_t id = p.ids[tok * p.ids_stride];
  const bool known = id >= 0 && id < p.V;         // an id outside the vocabulary makes the token's logits NaN
  const uint2* row = reinterpret_cast<const uint2*>(static_cast<const T*>(p.embed) + (known ? id : 0) * p.C);
  const uint32_t nan2 = Pair16<T>::put(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
#pragma unroll 1
  for (int c = threadIdx.x % NT; c < C4; c += NT) h[tok * C4 + c] = known ? __ldg(row + c) : make_uint2(nan2, nan2);
}

// A[token] = rows of 16-bit pairs, `words` tagged words per row (an even number); NB (or fewer) pairs of words per thread at a time.
// ALL: NB are exactly a thread's share.
template <int MR, int NB, bool ALL>
__device__ __forceinline__ void rows_into(unsigned char* A, int a_stride, const LmArgs& p, const Poller& poll, const uint2* src, int words, unsigned tag) {
  constexpr int WPT = 2 / MR, NT = 32 * WPT;
  const int tok = (threadIdx.x >> 5) / WPT, idx = threadIdx.x % NT, per_row = ALL ? NB * NT : words >> 1;
  if (tok >= p.B) return;
  src += 2 * (tok * per_row + idx);
  uint2* ar = reinterpret_cast<uint2*>(A + tok * a_stride) + idx;
#pragma unroll 1
  for (int c0 = 0; c0 < (ALL ? 1 : per_row - idx); c0 += NT * NB) {
    uint4 v[NB];
    const int n = ALL ? NB : min(NB, (per_row - idx - c0 + NT - 1) / NT);
    poll.wait<NB>(v, src + 2 * c0, [](int i) { return 2 * NT * i; }, tag, n);
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (ALL || i < n) ar[c0 + i * NT] = make_uint2(v[i].x, v[i].z);
  }
}

// All computing warps.
__device__ __forceinline__ void sync_computing() { asm volatile("bar.sync 15, %0;" ::"n"(kLmThreads) : "memory"); }

// ------------------------------------------------------------------------------------------------- attention
// A (batch, head) pair, or a share of its cached rows.
struct Item { int64_t rows; int b, h, share, n, lo, hi; };                 // rows: offset of the pair in the caches; n: cached rows, -1 = no room
__device__ __forceinline__ Item item_at(const LmArgs& p, const int* lens, int item) {
  Item r;
  r.share = item % p.n_split;
  const int pair = item / p.n_split;
  r.b = pair / p.H;
  r.h = pair - r.b * p.H;
  r.rows = r.b * p.cs_b + r.h * p.cs_h;
  r.n = lens[r.b];                              // (as the launch found it)
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
      poll.wait<1>(v, pt + s * (D + 2) + d, [](int) { return 0; }, tag);
      poll.wait<1>(l, pt + s * (D + 2) + D, [](int) { return 0; }, tag);
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
// A number that the compiler takes for unknown: it writes a copy of a loop for every value that it knows a number to have, and there is no
// room for copies in the instruction caches.
__device__ __forceinline__ int opaque(int v) { asm volatile("" : "+r"(v)); return v; }
__device__ __forceinline__ Contraction contraction(const LmArgs& p, int li, int ph) {     // ph: 0 qkv (or the head), 1 out, 2 gate/value, 3 down
  const LmLayerArgs& ly = p.layer[li < p.L ? li : 0];
  const bool head = li == p.L;
  const void* W = head ? p.head : ph == 0 ? ly.qkv : ph == 1 ? ly.out : ph == 2 ? ly.gate_val : ly.down;
  const int N = head ? p.V : ph == 0 ? 3 * p.C : ph == 2 ? p.F : p.C;
  return {W, opaque(N), opaque(ph == 3 ? p.F : p.C), opaque(ph == 3 ? 4 : 3), opaque(ph == 2 ? 2 : 1)};
}

// ------------------------------------------------------------------------------------------------- the ring
// Chunks of weights or cached rows in the order of their use: `full` waits for the bytes that the loading warp has asked for, `empty`
// counts the computing warps that have taken their pieces.  Norm weights have two buffers of their own.
struct RingBars { uint64_t full[kMaxStages], empty[kMaxStages], norm_full[2], norm_empty[2]; };

// Bounded like the polls: gives up after kWaitSpins tries (then the wait counts as run out).
struct RingWait {
  volatile int *ring_failed, *failed;            // shared memory: a wait for the ring has run out in this CTA (later ones return at once)
#ifdef FAT_TEST_LM_NO_RING_WAIT
  bool gives_up;                                 // test builds only: with that many words in the vocabulary the computing warps' first wait runs out
#endif
  __device__ __forceinline__ bool operator()(uint64_t* bar, uint32_t parity) const {
    bool ok = false;
#ifdef FAT_TEST_LM_NO_RING_WAIT
    if (gives_up && int(threadIdx.x) < kLmThreads) {
      *ring_failed = 1;
      *failed = 1;
      return false;
    }
#endif
#pragma unroll 1
    for (uint32_t i = 0; i < tc::kWaitSpins; ++i) {
      ok = tc::mbar_try_wait(bar, parity);
      if (ok || *ring_failed) break;
    }
    if (!ok) {
      *ring_failed = 1;
      *failed = 1;
    }
    return ok;
  }
};

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// The computing warps' end of the ring.
struct Ring {
  RingBars& bars;
  const RingWait& wait;
  uint32_t base;                                 // the stage to be used next
  int stage, stages;
  uint32_t parity;
  __device__ __forceinline__ uint32_t arrived() const {                    // the chunk's address, once it is there
    wait(&bars.full[stage], parity);
    return base;
  }
  __device__ __forceinline__ void taken() {                                // this warp has read its pieces
    __syncwarp();
    if ((threadIdx.x & 31) == 0) tc::mbar_arrive(&bars.empty[stage]);
    base += kChunkBytes;
    if (++stage == stages) {
      base -= uint32_t(stages) * kChunkBytes;
      stage = 0;
      parity ^= 1u;
    }
  }
};

// A chunk of keys or values holds kRows cached rows for each computing warp, row after row.  Keys are read as an A operand of mma.sync
// (piece u of lane (g, t) = lane / 4, lane % 4: row 8 (u / kKeyPieces) + g, elements 32 (u % kKeyPieces) + 8 t); of the values piece u is row
// kRowsPerPiece u + lane / kLanes, elements 8 (lane % kLanes).
template <int D> struct Rows {
  static constexpr int kKeyPieces = D / 32, kLanes = D / 8, kRowsPerPiece = 32 / kLanes, kRows = kPieces * kRowsPerPiece, kStep = kLmWarps * kRows;
};
__device__ __forceinline__ int chunks_per_set(const Contraction& c) {
  const int blocks = (c.K + 31) >> 5, per = kPieces << c.wpu_log2;
  return (blocks + per - 1) >> (c.wpu_log2 + 2);
}
__device__ __forceinline__ int units_per_round(int wpu_log2) { return int(gridDim.x) * (kLmWarps >> wpu_log2); }

// kFetchers warps (this one is number `part`): n rows of D elements, cs_t elements apart, in 16-byte pieces that do not wait; `bar` gets
// an arrival of every lane when its pieces are there.  (A lane's pieces have the same place in every so many rows.)
constexpr int kFetchers = 4;
template <typename T, int D>
__device__ __forceinline__ void fetch_rows(uint32_t dst, const T* src, int64_t cs_t, int n, uint64_t* bar, int part) {
  using R = Rows<D>;
  const int at = part * 32 + int(threadIdx.x & 31), row0 = at / R::kLanes;
  src += row0 * cs_t + at % R::kLanes * 8;
  dst += uint32_t(at) * 16u;
#pragma unroll 8
  for (int row = row0; row < n; row += kFetchers * R::kRowsPerPiece) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    src += kFetchers * R::kRowsPerPiece * cs_t;
    dst += kFetchers * 512u;
  }
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// The loading warp: every chunk of the launch in the order in which the computing warps use them, as bulk copies (whole rows, one per
// lane, or all of a chunk's cached rows at once).  What is copied starts and ends on 16-byte boundaries: around a row of the down
// projection that does not, up to 14 bytes of its neighbours come along (the matrix itself starts and ends on one).
// Cached rows that are apart in memory are too small for bulk copies: then all warps of the group run this, and fetch those together;
// part 0 does the rest, the others say on every chunk's barrier that they have nothing to add.
template <typename T, int D>
__device__ __forceinline__ void load_all(const LmArgs& p, unsigned char* smem, unsigned char* norm_w, const int* lens, RingBars& bars, const RingWait& wait, int stages, int part) {
  using R = Rows<D>;
  const int lane = threadIdx.x & 31;
  int stage = 0, sent = 0, norm1_sent = 0, norm2_sent = 0;
  uint32_t parity = 1;
  bool ok = true;
  auto copy = [&](uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
  };
  // the next stage, free; every lane says how many bytes it will ask for
  auto next = [&](uint32_t bytes) {
    ok = ok && wait(&bars.empty[stage], parity);
    if (p.cs_t != D) tc::fence_async_smem();     // (ordinary copies may have written to the stage)
    if (ok) tc::mbar_expect_tx(&bars.full[stage], bytes);
    return tc::smem_u32(smem) + uint32_t(stage) * kChunkBytes;
  };
  auto asked = [&]() {
    if (!ok) return;
    ++sent;
    if (++stage == stages) { stage = 0; parity ^= 1u; }
  };
#pragma unroll 1
  for (int step = 0; step <= 4 * p.L && ok; ++step) {
    const int li = step >> 2, ph = opaque(step & 3);
    if (!(ph & 1) && part == 0) {
      const int buf = ph >> 1;
      ok = wait(&bars.norm_empty[buf], (li & 1) ^ 1);
      if (ok && lane == 0) {
        ++(buf ? norm2_sent : norm1_sent);
        tc::mbar_expect_tx(&bars.norm_full[buf], uint32_t(p.C) * 2u);
        copy(tc::smem_u32(norm_w) + uint32_t(buf * p.C) * 2u, li == p.L ? p.norm : ph ? p.layer[li].norm2 : p.layer[li].norm1, uint32_t(p.C) * 2u, &bars.norm_full[buf]);
      }
    }
    if (ph == 1) {                               // the cached rows of this CTA's items: kStep rows of the keys, then of the values, and so on
#pragma unroll 1
      for (int item = blockIdx.x; item < p.B * p.H * p.n_split; item += gridDim.x) {
        const Item it = item_at(p, lens, item);
#pragma unroll 1
        for (int sub = 0; it.lo + (sub >> 1) * R::kStep < it.hi && ok; ++sub) {
          // Rows that lie next to each other are one copy of up to 32 KB: what bounds a long context is how many copies there are.  us per step,
          // 4 blocks of 768, 8 sequences, 8000 cached tokens: 32 copies of 1 KB per chunk 383 (24 GB/s per SM), 8 of 4 KB 217, one 189 (65 GB/s).
          // Rows apart: a bulk copy for each of 128 bytes 2008, one warp fetching 16-byte pieces 314, four 216.
          const int j = it.lo + (sub >> 1) * R::kStep, n = min(R::kStep, it.hi - j);
          const T* src = static_cast<const T*>((sub & 1) ? p.layer[li].v_cache : p.layer[li].k_cache) + it.rows + j * p.cs_t;
          uint64_t* bar = &bars.full[stage];
          if (p.cs_t == D) {
            const uint32_t bytes = lane == 0 ? uint32_t(n) * (D * 2) : 0u, dst = next(bytes);
            if (ok && bytes) copy(dst, src, bytes, bar);
          } else {
            ok = ok && wait(&bars.empty[stage], parity);
            if (ok) fetch_rows<T, D>(tc::smem_u32(smem) + uint32_t(stage) * kChunkBytes, src, p.cs_t, n, bar, part);
          }
          asked();
        }
      }
    }
    const Contraction c = contraction(p, li, ph);
    const int slots = kLmWarps >> c.wpu_log2, per_set = chunks_per_set(c), cols = 32 * kPieces << c.wpu_log2;
#pragma unroll 1
    for (int unit0 = blockIdx.x; unit0 * 8 < c.N; unit0 += int(gridDim.x) * slots)
#pragma unroll 1
      for (int sub = 0; sub < c.sets * per_set && ok; ++sub) {
        const int set = sub >= per_set, n = (unit0 + (lane >> 3) * int(gridDim.x)) * 8 + (lane & 7), k = (sub - set * per_set) * cols;
        const int64_t row = (int64_t(set) * c.N + n) * c.K;
        const uint64_t lo = uint64_t(row + k) * 2 & ~uint64_t(15), hi = (uint64_t(row + min(k + cols, c.K)) * 2 + 15) & ~uint64_t(15);
        const uint32_t bytes = part == 0 && lane < 8 * slots && n < c.N ? uint32_t(hi - lo) : 0u;
        uint64_t* bar = &bars.full[stage];
        const uint32_t dst = next(bytes) + uint32_t(lane) * uint32_t((cols + 32) * 2);
        if (ok && bytes) copy(dst, static_cast<const unsigned char*>(c.W) + lo, bytes, bar);
        asked();
      }
  }
  // Nothing may be on its way into shared memory when the CTA leaves: the computing warps have waited for all of it unless something
  // ran out, on either side.  One limit for all of these waits.
  uint32_t left = tc::kWaitSpins;
  auto landed = [&](uint64_t* bar, uint32_t phase) {
    while (left != 0u && !tc::mbar_try_wait(bar, phase)) --left;
  };
  for (int i = 0; i < min(sent, stages); ++i) {
    stage = (stage == 0 ? stages : stage) - 1;
    if (stage == stages - 1) parity ^= 1u;
    landed(&bars.full[stage], parity ^ 1u);
  }
  if (norm1_sent > 0) landed(&bars.norm_full[0], (norm1_sent - 1) & 1);
  if (norm2_sent > 0) landed(&bars.norm_full[1], (norm2_sent - 1) & 1);
}

// Attention of one item: scores (keys from the ring as the A operand, the query in every column of B, so that a lane finds the scores
// of its rows g and g + 8 without exchanging anything), weights and weighted values (float32 on the CUDA cores) of the cached rows, and
// of the new row from the projection's words; appends the new row.
template <typename T, int D>
__device__ __forceinline__ void attend(const LmArgs& p, const LmLayerArgs& ly, const Poller& poll, Ring& st, const Item& r, float slope, int item, float* red,
                                       const uint2* qkv_words, uint2* att_words, uint2* part_words, unsigned tag_in, unsigned tag_out) {
  using R = Rows<D>;
  constexpr int KP = R::kKeyPieces, kRed = D + 4;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, vg = lane / R::kLanes, vc = lane % R::kLanes;
  const uint2* qkv = qkv_words + (r.b * 3 * p.C + r.h * D) / 2;
  const float scale = p.scale;
  uint32_t q[KP][4];
  // (a lane's share of a row of words: elements 8 t .. of every 32)
  auto at_row = [&](int i) { return (i >> 1) * 16 + (i & 1) * 2; };
  {
    uint4 v[2 * KP];
    poll.wait<2 * KP>(v, qkv + t * 4, at_row, tag_in);
#pragma unroll
    for (int i = 0; i < 2 * KP; ++i) { q[i >> 1][(i & 1) * 2] = v[i].x; q[i >> 1][(i & 1) * 2 + 1] = v[i].z; }
  }
  f32x2 acc2[4] = {pk2(0.f, 0.f), pk2(0.f, 0.f), pk2(0.f, 0.f), pk2(0.f, 0.f)};
  auto add = [&](float f, const uint4& raw) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&raw);
    const f32x2 f2 = pk2(f, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 e = Pair16<T>::get(w[i]); acc2[i] = fma2(f2, pk2(e.x, e.y), acc2[i]); }
  };
  auto weight = [&](float dot, int j) {                                    // sigma(dot scale - slope (n - j))^4
    const float sc = fmaf(dot, scale, -slope * float(r.n - j));
    const float sig = fmaf(sc * rcp1p_abs(sc), 0.5f, 0.5f);
    const float s2 = sig * sig;
    return s2 * s2;
  };
  float l = 0.f;                                 // (the same in the four lanes of a row)
#pragma unroll 1
  for (int base = r.lo + warp * R::kRows; base - warp * R::kRows < r.hi; base += R::kStep) {
    // (rows from r.hi on hold whatever the stage held before)
    uint4 w[kPieces];
    const uint32_t keys = st.arrived() + uint32_t((warp * R::kRows + g) * (D * 2) + t * 16);
#pragma unroll
    for (int u = 0; u < kPieces; ++u) w[u] = lds128(keys + u / KP * (8 * D * 2) + u % KP * 64);
    st.taken();
    float s[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const uint4 lo = w[i], hi = KP < kPieces ? w[kPieces - KP + i] : make_uint4(0u, 0u, 0u, 0u);
      Pair16<T>::mma(s, lo.x, hi.x, lo.y, hi.y, q[i][0], q[i][1]);
      Pair16<T>::mma(s1, lo.z, hi.z, lo.w, hi.w, q[i][2], q[i][3]);
    }
    const uint32_t values = st.arrived() + uint32_t(warp * R::kRows * (D * 2) + lane * 16);
#pragma unroll
    for (int u = 0; u < kPieces; ++u) w[u] = lds128(values + u * 512);
    st.taken();
    if (base < r.hi) {                           // (the same for the whole warp)
      const int j = base + g;
      float f[2];
      f[0] = j < r.hi ? weight(s[0] + s1[0], j) : 0.f;
      f[1] = KP < kPieces && j + 8 < r.hi ? weight(s[2] + s1[2], j + 8) : 0.f;
      l += f[0] + f[1];
#pragma unroll
      for (int u = 0; u < kPieces; ++u) {
        const int row = u * R::kRowsPerPiece;    // + vg
        const float fu = __shfl_sync(0xffffffffu, f[row / 8], (row % 8 + vg) * 4);
        if (base + row + vg < r.hi) add(fu, w[u]);
      }
    }
  }
  if (r.share == 0 && warp == kLmWarps - 1 && r.n >= 0) {                  // the new row (this warp has the fewest cached ones)
    uint32_t k[KP][4];
    uint4 vnew;
    {
      uint4 v[2 * KP + 2];
      poll.wait<2 * KP + 2>(v, qkv + p.C / 2, [&](int i) { return i < 2 * KP ? t * 4 + at_row(i) : p.C / 2 + vc * 4 + (i - 2 * KP) * 2; }, tag_in);
#pragma unroll
      for (int i = 0; i < 2 * KP; ++i) { k[i >> 1][(i & 1) * 2] = v[i].x; k[i >> 1][(i & 1) * 2 + 1] = v[i].z; }
      vnew = make_uint4(v[2 * KP].x, v[2 * KP].z, v[2 * KP + 1].x, v[2 * KP + 1].z);       // as the cache keeps it
    }
    float s[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      Pair16<T>::mma(s, k[i][0], 0u, k[i][1], 0u, q[i][0], q[i][1]);
      Pair16<T>::mma(s1, k[i][2], 0u, k[i][3], 0u, q[i][2], q[i][3]);
    }
    const float f = weight(s[0] + s1[0], r.n);   // (in every lane)
    l += g == 0 ? f : 0.f;
    add(vg == 0 ? f : 0.f, vnew);
    const int64_t at = r.rows + r.n * p.cs_t;
    if (g == 0)
#pragma unroll
      for (int i = 0; i < KP; ++i)
        *reinterpret_cast<uint4*>(static_cast<T*>(ly.k_cache) + at + i * 32 + t * 8) = make_uint4(k[i][0], k[i][1], k[i][2], k[i][3]);
    if (vg == 0) *reinterpret_cast<uint4*>(static_cast<T*>(ly.v_cache) + at + vc * 8) = vnew;
  }
  if (r.n < 0 && r.share == 0 && tid == 0 && p.status) atomicOr(p.status, int(FAT_DEV_CACHE_FULL));
  float acc[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) upk2(acc2[i], acc[2 * i], acc[2 * i + 1]);
#pragma unroll
  for (int o = R::kLanes; o < 32; o <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if (item != int(blockIdx.x)) sync_computing(); // (the item before has been read)
  if (vg == 0) {
    float4* d = reinterpret_cast<float4*>(red + warp * kRed + vc * 8);
    d[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    d[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    if (lane == 0) red[warp * kRed + D] = l;
  }
  sync_computing();
  if (tid < 2 * D) {                             // four threads per pair of columns, four warps' sums each
    const int c = tid >> 2;
    float a0 = 0.f, a1 = 0.f, L = 0.f;
#pragma unroll
    for (int i = 0; i < kLmWarps / 4; ++i) {
      const float* d = red + ((tid & 3) * (kLmWarps / 4) + i) * kRed;
      const float2 a = *reinterpret_cast<const float2*>(d + 2 * c);
      a0 += a.x;
      a1 += a.y;
      L += d[D];
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      a1 += __shfl_xor_sync(0xffffffffu, a1, o);
      L += __shfl_xor_sync(0xffffffffu, L, o);
    }
    if (p.n_split > 1) {
      if ((tid & 3) == 0) {
        uint2* out = part_words + item * (D + 2);
        st_word(out + 2 * c, __float_as_uint(a0), tag_out);
        st_word(out + 2 * c + 1, __float_as_uint(a1), tag_out);
        if (c < 2) st_word(out + D + c, c ? 0u : __float_as_uint(L), tag_out);             // (an even number of words)
      }
    } else {
      const float v = ((tid & 1) ? a1 : a0) / (L + p.eps_attn), other = __shfl_xor_sync(0xffffffffu, v, 1);
      if ((tid & 3) == 0) st_word(att_words + (r.b * p.C + r.h * D) / 2 + c, Pair16<T>::put(v, other), tag_out);
    }
  }
}

// This thread's pieces of the weights in the chunk at the head of the ring: elements 32 (k kPieces + i) kWpu + 32 wpart + 8 t .. of the unit's
// row g, which is row n of the matrix.  NP: only the first NP pieces are wanted, and they lie within the row.
template <int kWpuLog2, int NP = 0>
__device__ __forceinline__ void take_weights(uint4 (&w)[kPieces], int K, int n, int k, Ring& st) {
  constexpr int kWpu = 1 << kWpuLog2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, wpart = warp & (kWpu - 1);
  const uint32_t row = st.arrived() + uint32_t(((warp >> kWpuLog2) * 8 + g) * row_pitch(kWpuLog2) + wpart * 64 + t * 16);
  if constexpr (NP > 0) {
#pragma unroll
    for (int i = 0; i < NP; ++i) w[i] = lds128(row + i * (kWpu * 64));
  } else {
    const int left = K - ((k * kPieces * kWpu + wpart) * 32 + t * 8);      // elements of the row from the first piece on
    if (kWpuLog2 == 3 || K % 8 == 0) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) w[i] = lds128(row + i * (kWpu * 64));
      if (left < (kPieces - 1) * kWpu * 32 + 8)  // (beyond the row the stage holds whatever it held before)
#pragma unroll
        for (int i = 0; i < kPieces; ++i)
          if (left <= i * kWpu * 32) w[i] = make_uint4(0u, 0u, 0u, 0u);
    } else {                                     // the row starts up to 14 bytes behind a 16-byte boundary
      const uint32_t off = (uint32_t(n) * uint32_t(K) * 2u) & 15u, from = row + (off & 12u), shift = (off & 2u) * 8u;
#pragma unroll 1
      for (int i = 0; i < kPieces; ++i) {
        uint32_t e[5], o[4];
#pragma unroll
        for (int j = 0; j < 5; ++j) e[j] = lds32(from + i * (kWpu * 64) + j * 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rest = left - i * kWpu * 32 - 2 * j;
          o[j] = rest <= 0 ? 0u : __funnelshift_r(e[j], e[j + 1], shift) & (rest == 1 ? 0xffffu : 0xffffffffu);
        }
#pragma unroll
        for (int u = 0; u < kPieces; ++u)        // (registers have no index)
          if (u == i) w[u] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
  st.taken();
}

// The units of one contraction that this CTA owns: kSets matrices of N rows of K elements; kWpu warps share a unit.  take() takes the first
// chunk of each set ahead of the wait for the words, run() does the rest.  NP: K is 32 kWpu NP (0: any number).
// store(token, column, sums of the first set, sums of the second).
template <typename T, int MR, int kWpuLog2, int kSets, int NP>
struct Contract {
  static constexpr int kTile = MR * 64, kWpu = 1 << kWpuLog2, kStride = kTile + 8, kFirst = NP ? kSets : 1, kUsed = NP ? NP : kPieces;
  const int N, K;
  Ring& st;
  uint4 w[kFirst][kPieces];
  __device__ __forceinline__ int unit_of(int unit0) const { return unit0 + int((threadIdx.x >> 5) >> kWpuLog2) * int(gridDim.x); }
  __device__ __forceinline__ void take(int unit0) {
    const int n = unit_of(unit0) * 8 + ((threadIdx.x & 31) >> 2);
#pragma unroll
    for (int i = 0; i < kFirst; ++i) take_weights<kWpuLog2, NP>(w[i], K, n, 0, st);
  }
  __device__ __forceinline__ bool owner() const { return int(blockIdx.x) * 8 < N; }       // (slot 0 has the CTA's first unit)
  template <typename Store>
  __device__ __forceinline__ void run(const unsigned char* a_lane, int as, float* red, int B, Store store) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slot = warp >> kWpuLog2, wpart = warp & (kWpu - 1), in_slot = wpart * 32 + lane;
    const int tok = in_slot >> 2, col = (in_slot & 3) * 2;
    float* part0 = red + slot * (kWpu * 2 * kStride);                      // [slot][warp][set][token][8]
    float* part = part0 + wpart * 2 * kStride + (lane >> 2) * 8 + (lane & 3) * 2;
    part0 += in_slot * 2;
    const unsigned char* a0 = a_lane + wpart * 64;
    int other = 0;
#pragma unroll 1
    for (int unit0 = blockIdx.x; unit0 * 8 < N; unit0 += units_per_round(kWpuLog2)) {     // (the same count for all warps, as the ring wants it)
      if (unit0 != int(blockIdx.x)) take(unit0);
      float acc[kSets][2][4] = {};
      auto multiply = [&](float (&c)[2][4], const uint4 (&b)[kPieces], const uint4 (&lo)[kUsed], const uint4 (&hi)[kUsed]) {
#pragma unroll
        for (int i = 0; i < kUsed; ++i) {
          Pair16<T>::mma(c[0], lo[i].x, hi[i].x, lo[i].y, hi[i].y, b[i].x, b[i].y);
          Pair16<T>::mma(c[1], lo[i].z, hi[i].z, lo[i].w, hi[i].w, b[i].z, b[i].w);
        }
      };
      auto load_a = [&](uint4 (&lo)[kUsed], uint4 (&hi)[kUsed], int k) {
#pragma unroll
        for (int i = 0; i < kUsed; ++i) {
          const int kb = (k * kPieces + i) * kWpu;                         // + wpart: the block of 32 elements
          const bool in = NP || (kb + wpart) * 32 < K;                     // (the weights beyond are zeros)
          lo[i] = in ? *reinterpret_cast<const uint4*>(a0 + kb * 64) : make_uint4(0u, 0u, 0u, 0u);
          hi[i] = MR == 2 && in ? *reinterpret_cast<const uint4*>(a0 + kb * 64 + 8 * as) : make_uint4(0u, 0u, 0u, 0u);
        }
      };
      uint4 lo[kUsed], hi[kUsed];
      if constexpr (NP > 0) {
        load_a(lo, hi, 0);
#pragma unroll
        for (int set = 0; set < kSets; ++set) multiply(acc[set], w[set], lo, hi);
      } else {
        const int per_set = (((K + 31) >> 5) + kPieces * kWpu - 1) / (kPieces * kWpu);
#pragma unroll
        for (int set = 0; set < kSets; ++set)
#pragma unroll 1
          for (int k = 0; k < per_set; ++k) {
            if (set + k) take_weights<kWpuLog2>(w[0], K, unit_of(unit0) * 8 + (lane >> 2), k, st);
            load_a(lo, hi, k);
            multiply(acc[set], w[0], lo, hi);
          }
      }
#pragma unroll
      for (int set = 0; set < kSets; ++set) {
        float* d = part + (kSets == 2 ? set : other) * kStride;
        *reinterpret_cast<float2*>(d) = make_float2(acc[set][0][0] + acc[set][1][0], acc[set][0][1] + acc[set][1][1]);
        if (MR == 2) *reinterpret_cast<float2*>(d + 64) = make_float2(acc[set][0][2] + acc[set][1][2], acc[set][0][3] + acc[set][1][3]);
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(kWpu * 32) : "memory");
      const int n = unit_of(unit0) * 8 + col;
      if (in_slot < 32 * MR) {                   // (whole warps)
        float2 v[kSets];
#pragma unroll
        for (int set = 0; set < kSets; ++set) {
          const float* d = part0 + (kSets == 2 ? set : other) * kStride;
          float2 q[kWpu];
#pragma unroll
          for (int i = 0; i < kWpu; ++i) q[i] = *reinterpret_cast<const float2*>(d + i * 2 * kStride);
          v[set] = q[0];
#pragma unroll
          for (int i = 1; i < kWpu; ++i) { v[set].x += q[i].x; v[set].y += q[i].y; }
        }
        if (tok < B && n < N) store(tok, n, v[0], v[kSets - 1]);
      }
      // with one set the other set's place is the other buffer (one is written again only after the next barrier)
      if (kSets == 2) asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(kWpu * 32) : "memory");
      else other ^= 1;
    }
  }
};

// MR: 1 = up to 8 tokens, 2 = up to 16.  NC: the width is 256 NC (0: any other), known where it saves the loops and their tests.
template <typename T, int D, int MR, int NC>
__global__ void __launch_bounds__(kLmBlock, 1)
lm_decode_kernel(const __grid_constant__ LmArgs p, int stages) {
  extern __shared__ __align__(128) unsigned char lm_smem[];
  __shared__ int failed, ring_failed, last, lens[16];
  __shared__ float sums[kLmWarps];
  __shared__ RingBars bars;
  constexpr int kRed = kLmWarps * 2 * (MR * 64 + 8) > kLmWarps * (D + 4) ? kLmWarps * 2 * (MR * 64 + 8) : kLmWarps * (D + 4);      // partial sums: [warp][set][token][8], or [warp][D + 4]
  unsigned char* A = lm_smem + stages * kChunkBytes;
  const int as = p.a_stride;
  float* red = reinterpret_cast<float*>(A + MR * 8 * as);
  uint2* h = reinterpret_cast<uint2*>(red + kRed);
  unsigned char* norm_w = reinterpret_cast<unsigned char*>(h) + MR * 8 * p.C * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Poller poll{&failed};
#ifdef FAT_TEST_LM_NO_RING_WAIT
  const RingWait ring_wait{&ring_failed, &failed, p.V == FAT_TEST_LM_NO_RING_WAIT};
#else
  const RingWait ring_wait{&ring_failed, &failed};
#endif
  const int B = p.B, C = NC ? NC * 256 : p.C, items = B * p.H * p.n_split, loaders = p.cs_t == D ? 1 : kFetchers;
  if (threadIdx.x == 0) {
    failed = ring_failed = 0;
    for (int i = 0; i < kMaxStages; ++i) { tc::mbar_init(&bars.full[i], 32 * loaders); tc::mbar_init(&bars.empty[i], kLmWarps); }
    for (int i = 0; i < 2; ++i) { tc::mbar_init(&bars.norm_full[i], 1); tc::mbar_init(&bars.norm_empty[i], kLmWarps); }
    tc::mbar_fence_init();
  }
  if (int(threadIdx.x) < B) lens[threadIdx.x] = __ldcg(p.n_cached + threadIdx.x);
  if (warp < kLmWarps)
#pragma unroll 1
    for (int i = threadIdx.x * 16; i < MR * 8 * as; i += kLmThreads * 16) *reinterpret_cast<uint4*>(A + i) = make_uint4(0u, 0u, 0u, 0u);
  const unsigned launch = __ldcg(p.ctl) << 10;
  __syncthreads();
  if (warp >= kLmWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLoadRegs));
    if (warp - kLmWarps < loaders) load_all<T, D>(p, lm_smem, norm_w, lens, bars, ring_wait, stages, warp - kLmWarps);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kComputeRegs));
    Ring st{bars, ring_wait, tc::smem_u32(lm_smem), 0, stages, 0u};
    const unsigned char* a_lane = A + (lane >> 2) * as + (lane & 3) * 16;
    const uint2 *norm1_w = reinterpret_cast<const uint2*>(norm_w), *norm2_w = reinterpret_cast<const uint2*>(norm_w + C * 2);
    auto norm_taken = [&](int buf) {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars.norm_empty[buf]);
    };
    auto slope_of = [&](const LmLayerArgs& ly, int head) { return p.slopes_f32 ? static_cast<const float*>(ly.slopes)[head] : Elem<T>::to_c(static_cast<const T*>(ly.slopes)[head]); };
    const Item mine = item_at(p, lens, int(blockIdx.x) < items ? int(blockIdx.x) : 0);
    embed_into<T, MR>(h, p);
#pragma unroll 1
    for (int li = 0; li < p.L; ++li) {
      const LmLayerArgs& ly = p.layer[li];
      const unsigned tag = launch + li * 8 + 1;  // qkv words; + 1 attention, + 2 o, + 3 act, + 4 pending
      const int odd = li & 1, BC2 = B * C / 2;
      uint2 *qkv = p.qkv + odd * 3 * BC2, *att = p.att + odd * BC2, *o = p.o + odd * BC2, *act = p.act + odd * B * p.act_words, *part = p.part + odd * items * (D + 2);
      float slope = slope_of(ly, mine.h);        // (in time for P2)
      {                                          // P1
        Contract<T, MR, 3, 1, NC> c{3 * C, C, st};
        if (c.owner()) c.take(blockIdx.x);
        ring_wait(&bars.norm_full[0], odd);
        if (li == 0) norm_into<T, MR, NC, false>(A, as, h, sums, p, poll, nullptr, 0u, norm1_w);
        else norm_into<T, MR, NC, true>(A, as, h, sums, p, poll, p.pend + (odd ^ 1) * BC2, tag - 4, norm1_w);     // (tag - 4: the pending words of the layer before)
        norm_taken(0);
        sync_computing();
        c.run(a_lane, as, red, B, [&](int tok, int n, float2 v, float2) {
#ifdef FAT_TEST_LM_WITHHOLD_UNIT
          // test builds only (never the shipped library): the words of this unit of the first block's projection are not written, so
          // every wait for them runs out
          if (li == 0 && n / 8 == FAT_TEST_LM_WITHHOLD_UNIT) return;
#endif
          st_word(qkv + (tok * 3 * C + n) / 2, Pair16<T>::put(v.x, v.y), tag);
        });
        sync_computing();                        // A and `red` are free
      }
      Item it = mine;
#pragma unroll 1
      for (int item = blockIdx.x; item < items; item += gridDim.x) {       // P2
        if (item != int(blockIdx.x)) {
          it = item_at(p, lens, item);
          slope = slope_of(ly, it.h);
        }
        attend<T, D>(p, ly, poll, st, it, slope, item, red, qkv, att, part, tag, tag + 1);
      }
      {                                          // P3
        Contract<T, MR, 3, 1, NC> c{C, C, st};
        if (c.owner()) {
          c.take(blockIdx.x);
          if (p.n_split > 1) combine_into<T, D>(A, as, p, poll, part, tag + 1);
          else rows_into<MR, NC ? NC * MR : 4, NC != 0>(A, as, p, poll, att, C / 2, tag + 1);
          sync_computing();
          c.run(a_lane, as, red, B, [&](int tok, int n, float2 v, float2) { st_word(o + (tok * C + n) / 2, Pair16<T>::put(v.x, v.y), tag + 2); });
          sync_computing();
        }
      }
      {                                          // P4
        Contract<T, MR, 3, 2, NC> c{p.F, C, st};
        if (c.owner()) c.take(blockIdx.x);
        ring_wait(&bars.norm_full[1], odd);
        norm_into<T, MR, NC, true>(A, as, h, sums, p, poll, o, tag + 2, norm2_w);
        norm_taken(1);
        sync_computing();
        c.run(a_lane, as, red, B, [&](int tok, int n, float2 v0, float2 v1) {
          const float2 gate = Pair16<T>::get(Pair16<T>::put(v0.x, v0.y)), value = Pair16<T>::get(Pair16<T>::put(v1.x, v1.y));
          if (n + 2 >= p.F && p.act_words > n / 2 + 1) st_word(act + tok * p.act_words + n / 2 + 1, 0u, tag + 3);          // (rows have an even number of words)
          // (column F of an odd width comes from a ring row that nothing was copied to: its weight in P5 is zero, which a NaN does not mind)
          const float second = n + 1 < p.F ? gate.y * rsigmoid(gate.y, rcp1p_abs(gate.y)) * value.y : 0.f;
          st_word(act + tok * p.act_words + n / 2, Pair16<T>::put(gate.x * rsigmoid(gate.x, rcp1p_abs(gate.x)) * value.x, second), tag + 3);
        });
        sync_computing();
      }
      {                                          // P5
        Contract<T, MR, 4, 1, 0> c{C, p.F, st};
        if (c.owner()) {
          c.take(blockIdx.x);
          rows_into<MR, 8, false>(A, as, p, poll, act, p.act_words, tag + 3);
          sync_computing();
          c.run(a_lane, as, red, B, [&](int tok, int n, float2 v, float2) { st_word(p.pend + odd * BC2 + (tok * C + n) / 2, Pair16<T>::put(v.x, v.y), tag + 4); });
          sync_computing();
        }
      }
    }
    {                                            // final norm and head
      const int odd = p.L & 1;
      Contract<T, MR, 3, 1, NC> c{p.V, C, st};
      if (c.owner()) c.take(blockIdx.x);
      ring_wait(&bars.norm_full[0], odd);
      norm_into<T, MR, NC, true>(A, as, h, sums, p, poll, p.pend + (odd ^ 1) * (B * C / 2), launch + p.L * 8 - 3, norm1_w);
      sync_computing();
      c.run(a_lane, as, red, B, [&](int tok, int n, float2 v, float2) {
        T* out = static_cast<T*>(p.logits) + int64_t(tok) * p.V + n;
        if (p.V % 2 == 0) *reinterpret_cast<uint32_t*>(out) = Pair16<T>::put(v.x, v.y);
        else {
          out[0] = Elem<T>::from_c(v.x);
          if (n + 1 < p.V) out[1] = Elem<T>::from_c(v.y);
        }
      });
    }
  }
  __syncthreads();
  // The last CTA to leave: nobody reads the lengths and the launch number any more.  A step in which a wait ran out (the words
  // behind it are whatever the CTA had in its registers, and spread) gives NaN logits and does not count.
  if (threadIdx.x == 0) {
    if (failed) {
      atomicExch(p.ctl + 2, 1u);
      if (p.status) atomicCAS(p.status, 0, (FAT_DEV_WAIT_TIMEOUT << 24) | 300);
    }
    __threadfence();
    last = atomicAdd(p.ctl + 1, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    __threadfence();
    const bool bad = __ldcg(p.ctl + 2) != 0u;
    if (bad)
#pragma unroll 1
      for (int64_t i = threadIdx.x; i < int64_t(B) * p.V; i += kLmBlock) static_cast<T*>(p.logits)[i] = Elem<T>::from_c(__int_as_float(0x7fc00000));
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
  // The tokens' activations, stream and partial sums.  Beyond this line one chunk or two are left for the ring, so that little streams
  // ahead, and the operators, issued one by one, win at long contexts: us per step, fused / operators, 16 sequences, 8 blocks of 1280 with
  // heads of 128: 64 cached tokens 630 / 1186, 1800 tokens 1209 / 1117, 4000 tokens 1825 / 1182.
  if (size_t(rows) * (row_bytes((wide + 31) / 32 * 32) + size_t(C) * 4 + 2048) > kTileLimit) return false;
  const size_t red = size_t(kLmWarps) * (2 * (rows * 8 + 8) > D + 4 ? 2 * (rows * 8 + 8) : D + 4) * sizeof(float);
  out->smem = size_t(rows) * (row_bytes((wide + 31) / 32 * 32) + size_t(C) * 2) + red + size_t(2 * C) * 2;
  if (out->smem + kChunkBytes > kLmSmemLimit) return false;
  out->stages = int((kLmSmemLimit - out->smem) / kChunkBytes);
  if (out->stages > kMaxStages) out->stages = kMaxStages;
  out->smem += size_t(out->stages) * kChunkBytes;
  out->act_words = ((F + 1) / 2 + 1) / 2 * 2;
  out->grid = num_sms() < (3 * C + 7) / 8 ? num_sms() : (3 * C + 7) / 8;       // every CTA owns a unit of P1
  // a (batch, head) pair per CTA; with few pairs their keys are shared out, 64 rows of a full cache at least per share
  int s = out->grid / (B * H);
  if (s > 16) s = 16;
  while (s > 1 && capacity / s < 64) --s;
  out->n_split = s < 1 ? 1 : s;
  return true;
}

// The usual widths are compiled in.  The instance for any other width keeps its loops and spills 420-610 bytes a thread; run at the usual widths, us per
// step, 12 blocks, 512 cached tokens, compiled in / general: 512 wide, 8 sequences 218 / 314; 768 wide, 1 sequence 225 / 298, 8 198 / 308, 16 288 / 481;
// 1024 wide, 8 sequences 263 / 401.
template <typename T, int D, int MR>
int launch_step(LmArgs& a, const Plan& pl, cudaStream_t st) {
  void (*kern)(const LmArgs, int) = a.C == 512 ? lm_decode_kernel<T, D, MR, 2> : a.C == 768 ? lm_decode_kernel<T, D, MR, 3>
                                  : a.C == 1024 ? lm_decode_kernel<T, D, MR, 4> : lm_decode_kernel<T, D, MR, 0>;
  int regs = 0;
  if (int rc = ready_kernel(reinterpret_cast<const void*>(kern), pl.smem, "lm_decode", &regs)) return rc;
  if (regs < kLaunchRegs) {                      // the computing warps could never collect their share
    set_error("lm_decode_step: built with %d registers per thread, the register hand-over needs %d", regs, kLaunchRegs);
    return FAT_ERR_LAUNCH;
  }
  int stages = pl.stages;
  void* args[] = {&a, &stages};
  cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(unsigned(pl.grid)), dim3(kLmBlock), args, pl.smem, st);
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
  return 128 + 2 * sizeof(uint2) * (3 * row / 2 + row / 2 + row / 2 + row / 2 + size_t(B) * pl.act_words + (pl.n_split > 1 ? size_t(B) * H * pl.n_split * (D + 2) : 0)) + 6 * 128;
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
  a.qkv = words(3 * row / 2); a.o = words(row / 2); a.pend = words(row / 2); a.att = words(row / 2); a.act = words(size_t(B) * pl.act_words);
  a.part = pl.n_split > 1 ? words(size_t(B) * H * pl.n_split * (D + 2)) : nullptr;
  a.ids = ids; a.ids_stride = ids_stride; a.embed = embed; a.norm = norm; a.head = head; a.logits = logits; a.n_cached = n_cached; a.status = status;
  a.cs_b = cache_strides[0]; a.cs_h = cache_strides[1]; a.cs_t = cache_strides[2];
  a.L = n_layers; a.B = B; a.C = C; a.H = H; a.F = F; a.V = V; a.capacity = capacity; a.act_words = pl.act_words; a.n_split = pl.n_split;
  a.slopes_f32 = slopes_f32;
  a.a_stride = row_bytes(((F > C ? F : C) + 31) / 32 * 32);
  a.scale = float(scale); a.eps_norm = float(eps_norm); a.eps_attn = float(eps_attn);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == FAT_BF16 ? launch_step_t<__nv_bfloat16>(a, D, pl, st) : launch_step_t<__half>(a, D, pl, st);
}
