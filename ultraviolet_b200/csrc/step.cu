// All transformer layers of one decode step of a small batch in one cooperative launch.
//
// What bounds a step: with a few rows every kernel of a layer is a 3-5 us chain of dependent round trips on a mostly idle
// GPU, and 70 of them in a row took 255-310 us at 1-48 rows, against 17 us of weight traffic.  Here a layer is six hops
// between CTAs of 0.6-1.2 us each with 0.3-0.5 us of work in between (the attention: 2.3 us), and from some 16 rows on the
// loads of CTAs that all read all rows (from L2, at a sixth of its rate): 100 us at 1 row, 110 at 8, 143 at 16, 175 at 32, 209
// at 48 (UV-50M, contexts of 200-900).
//
// Split: one CTA per multiprocessor.  In the projections a CTA owns one 8-wide tile of output features (of gate | up up to
// two pairs of tiles; UV-50M has 80, 80, 208 pairs and 80) for all rows, its weights in shared memory, fetched a layer
// ahead (the region of a phase is refilled as soon as the phase has used it).  The 16 warps are row tiles
// of 16 times slices of K, whose sums meet in shared memory (with the tiles one after the other, 16 slices each, 32 rows took
// 202 us and 48 took 258).  In the attention phase the last CTAs own a row each, a warp
// per head for what is done head by head, chunks of keys dealt out to the warps in between.
//
// Exchange: activations change hands through L2 without barriers, fences or flags on the way.  The workspace starts out
// filled with a value no projection can produce (a word of two 0xffff half-precision NaNs; a NaN result is stored as
// another NaN), and a reader simply loads what it needs, straight into MMA fragments, until none of it is that value:
// a word is its own flag.  Every layer has its own buffers, so a word is written once per launch.  Buffers are laid out so
// that a line has one writer: with a line shared by the 16-byte pieces of eight CTAs, words were seen 1-3 us late.
//
// Matrix instructions: warp-level mma.sync, because operands go from L2 to registers and results from registers to L2 in
// the phase's critical path of a few hundred cycles.  tcgen05 with its TMA tiles, commits and TMEM reads cost 2-3 thousand
// cycles a phase at these sizes (23 us a layer at one row against 10 here).  What counts is the number of instructions on
// the path of a warp: about six cycles each.  Hence fixed tile counts, sums of squares out of
// the tensor cores, and a code size that the instruction caches hold.
//
// Attention: a warp takes 32-key chunks of one row straight from the cache into MMA fragments (whole 64-byte key rows, one
// round trip); the first chunk of every warp is requested before the QKV projection is waited for, and the next layer's
// cache rows are prefetched to L2.  The entry at the row's own position is taken from shared memory.
//
// Rounding points are those of the per-kernel folded step (engine.py): projections round to the activation dtype, norms
// scale the rounded projection, the residual stream adds it.  The sums before them go in other orders (slices of K, chunks of
// keys, lanes), the MLP's norm comes from the tensor cores, and SwiGLU and the gates divide with __fdividef (the rounded
// division: 2 us more a step at one row): hidden states differ by 0.4 % in bf16 and 0.06 % in fp16 after ten layers, and both
// kinds of step are equally far from 64-bit arithmetic (0.7 %, 0.08 - 0.09 %).
//
// Every wait is bounded (200 ms); a CTA that gives up sets status bit 3, skips its later waits for words (not those for its
// own weight copies) and still ends.
#include <mutex>
#include <type_traits>

#include "attn_math.cuh"
#include "qkv_post.cuh"

namespace uv {

constexpr int ST_WARPS = 16;
constexpr int ST_THREADS = ST_WARPS * 32;
constexpr int ST_MAXL = 16;                 // layers per launch (kernel parameter space)
// Rows of a batch: three row tiles, the largest batch that the tests cover.  Up to 64 rows, where the 16 warps still take the
// row tiles side by side, it is faster than one launch per operation (209 against 310 us at 48 rows, 232 : 309 at 64, 294 : 337
// at 64 of 8192 keys); from 65 on, with two passes over the weights, no longer by much or at all (288 : 312, 320 : 315 at 96).
constexpr int ST_ROWS = 48;
constexpr int ST_XCH = 128;                 // leading channels of a row that the gates may read
constexpr int ST_HD = 64;
constexpr int ST_PAIRS = 2;                 // 8-wide gate | up tile pairs a CTA can have (one tile of the other projections)
constexpr unsigned ST_NAP = 100;              // ns between two looks for a missing word: the stores need the L2 too
constexpr uint32_t ST_EMPTY = 0xffffffffu;
constexpr unsigned long long ST_WAIT_NS = 200ull * 1000ull * 1000ull;

enum { PH_QKV = 0, PH_WO = 1, PH_GU = 2, PH_DN = 3 };

struct StepLayerK {
  const void* w[4];
  const void *ve_gate, *gate_w;
  const float* xsa_alpha;
  int8_t *kc, *vc;
  uint16_t *ks, *vs;
  int S, S_alloc, ring, window, rope, pad_;
};

struct StepP {
  StepLayerK layer[ST_MAXL];
  const int64_t *tok, *pos, *starts, *row_map;
  const void *embed, *value_embed;
  const float* inv_freq;
  void* buf;                       // of every layer: x, x after attention, qkv, z, act of all B rows; and the last x
  void* xn;
  int *oob, *status;
  int64_t vocab, stride;           // stride: elements of a layer's buffers
  int off[5];                      // element offsets of the five in them
  int B, L, d, H, f, n_pairs, gate_ch, ve_ch, ring_S;
  int K[4], base[4], rem[4];       // per phase: reduction length; feature tiles (of gate | up: pairs) of every CTA, and how
                                   // many CTAs have one more
  int region[4];                   // byte offsets of the phases' weights in shared memory
  float scale_log2, xsa_eps;
};

// Two values at a time through the packed converters: the scalar ones go to the quarter-rate unit.
template <typename T> __device__ __forceinline__ uint32_t st_pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t st_pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t st_pack2<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ float2 st_unpack2(uint32_t u);
template <> __device__ __forceinline__ float2 st_unpack2<__nv_bfloat16>(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 st_unpack2<__half>(uint32_t u) {
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}
template <typename T> __device__ __forceinline__ float2 st_rnd2(float a, float b) { return st_unpack2<T>(st_pack2<T>(a, b)); }
template <typename T> __device__ __forceinline__ void st_unpack8(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = st_unpack2<T>(w[k]);
    v[2 * k] = f.x, v[2 * k + 1] = f.y;
  }
}
template <typename T> __device__ __forceinline__ uint4 st_pack8(const float (&v)[8]) {
  return make_uint4(st_pack2<T>(v[0], v[1]), st_pack2<T>(v[2], v[3]), st_pack2<T>(v[4], v[5]), st_pack2<T>(v[6], v[7]));
}
// x <- rnd(x * s)
template <typename T> __device__ __forceinline__ void st_scale8(float (&x)[8], float s) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const float2 f = st_rnd2<T>(x[k] * s, x[k + 1] * s);
    x[k] = f.x, x[k + 1] = f.y;
  }
}


template <typename T, int ROWS, int LGM> struct StepSmem {
  alignas(16) T vcur[ST_HD];              // unquantised value of the owned row's token
  float vinv2;                            // 1 / |it|^2
  alignas(16) int8_t qi[2][8][ST_HD];     // its query heads in two int8 parts (split_q, attn_math.cuh)
  float qf[8];                            // the scale of the first part (the second's is 1/254 of it)
  alignas(16) int8_t q8[2][ST_HD];        // its quantised key and value
  uint16_t sc[2];
  alignas(16) StepLayerK layer[ST_MAXL];  // (from the constant bank every first touch of a layer costs ~500 cycles)
  // partial sums: [tile][row][feature pair][slice of K], rows of 2^LGM row tiles; their sums of squares: [row][slice]
  static constexpr int MROWS = ROWS << LGM, KS = ST_WARPS >> LGM, LD = KS == 4 ? 4 : KS + 2, TILE = MROWS * 4 * LD;
  alignas(16) float2 red[2][2 * ST_PAIRS * TILE];
  alignas(16) float ssq[2][MROWS * KS];
  float mg_m[8][ST_WARPS], mg_l[8][ST_WARPS], mg_o[ST_WARPS][8][ST_HD];        // the attention's per-warp results
  uint64_t full[4];                       // weights of a phase have landed
  int dead;
};
// Behind it: the phases' weights (rows of K values + 64 bytes: conflict-free 16-byte reads).

// One warp's share of one row's keys: 32-key chunks straight from the cache into MMA fragments.
struct StepRow {
  const int8_t *k, *v;
  const uint16_t *ks, *vs;
  int lo, hi, newest, S, S_alloc, ring;   // newest: the row's own position when it is attended (taken from shared memory), else -1
};
struct StepChunk {
  uint4 k[4];
  uint2 v[2][4];
  uint16_t sk, sv;               // fp16 scales of key `lane`
};

// the slot of key `key` of the chunk whose first key sits at slot s0: a ring chunk may run past the last slot (rings have
// at least 32 slots: once), a linear row may end inside it (such keys are masked: any slot will do)
__device__ __forceinline__ int step_slot(const StepRow& R, int s0, int key) {
  const int s = s0 + key;
  return s < R.S ? s : R.ring ? s - R.S : s0;
}
__device__ __forceinline__ void step_load_k(const StepRow& R, StepChunk& c, int s0, int lane) {
  const int r = lane >> 2, q = lane & 3;
  if (s0 + 32 <= R.S_alloc) {    // all 32 slots exist in a row: keys past hi are read, and masked later
    const int8_t* k = R.k + (int64_t)(s0 + r) * ST_HD + q * 16;
#pragma unroll
    for (int t = 0; t < 4; ++t) c.k[t] = *reinterpret_cast<const uint4*>(k + t * 8 * ST_HD);
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      c.k[t] = *reinterpret_cast<const uint4*>(R.k + (int64_t)step_slot(R, s0, 8 * t + r) * ST_HD + q * 16);
  }
}
__device__ __forceinline__ void step_load_v(const StepRow& R, StepChunk& c, int s0, int lane) {
  const int r = lane >> 2, q = lane & 3;
  if (s0 + 32 <= R.S_alloc) {
    const int8_t* v = R.v + (int64_t)(s0 + 2 * q) * ST_HD + r * 8;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        c.v[u][j] = *reinterpret_cast<const uint2*>(v + (16 * u + (j & 1) + (j >> 1) * 8) * ST_HD);
  } else {
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        c.v[u][j] = *reinterpret_cast<const uint2*>(
            R.v + (int64_t)step_slot(R, s0, 16 * u + 2 * q + (j & 1) + (j >> 1) * 8) * ST_HD + r * 8);
  }
}
__device__ __forceinline__ void step_load_scales(const StepRow& R, StepChunk& c, int s0, int lane) {
  const int s = step_slot(R, s0, lane);
  c.sk = R.ks[s], c.sv = R.vs[s];
}
__device__ __forceinline__ void step_load(const StepRow& R, StepChunk& c, int s0, int lane) {
  step_load_k(R, c, s0, lane);
  step_load_scales(R, c, s0, lane);
  step_load_v(R, c, s0, lane);
}

struct StepAcc {
  float o[8][4];
  float m, l;
};

// Chunk t0 of the row.  The next chunk (at slot s_next, if >= 0) is requested into the same registers as soon as the tensor cores have
// taken the current one: K and scales under the softmax and P V, V under the next chunk's Q K^T.
template <typename Smem>
__device__ __forceinline__ void step_chunk(const StepRow& R, const Smem& sm, StepChunk& ch, StepAcc& A,
                                           const uint32_t (&q1)[4], const uint32_t (&q2)[4], float f1, float f2, int t0,
                                           int s_next, int lane) {
  const int r = lane >> 2, q = lane & 3;
  const int hi_rel = R.hi - t0, key_new = R.newest - t0;
  const bool newest = R.newest >= t0 && key_new < 32;   // the row's own position: its entry comes from shared memory
  if (newest) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (8 * t + r == key_new) ch.k[t] = *reinterpret_cast<const uint4*>(&sm.q8[0][q * 16]);
    if (lane == key_new) ch.sk = sm.sc[0], ch.sv = sm.sc[1];
  }
  int acc[4][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[t][e] = 0x4b400000;   // 1.5 * 2^23: the sums (|s| < 2^21) are read as floats below
    imma16832(acc[t], q1[0], q2[0], q1[1], q2[1], ch.k[t].x, ch.k[t].y);
    imma16832(acc[t], q1[2], q2[2], q1[3], q2[3], ch.k[t].z, ch.k[t].w);
  }
  // (keys past hi may carry anything: no scale, no weight)
  const uint32_t scales = lane <= hi_rel ? (uint32_t)ch.sk | ((uint32_t)ch.sv << 16) : 0u;
  if (s_next >= 0) step_load_k(R, ch, s_next, lane);
  float sc[4][2], mx = -INFINITY;
  uint32_t vsh[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int kk = 8 * t + 2 * q;
    const uint32_t s0 = __shfl_sync(0xffffffffu, scales, kk), s1 = __shfl_sync(0xffffffffu, scales, kk + 1);
    vsh[t] = __byte_perm(s0, s1, 0x7632);
    const float k0 = __half2float(__ushort_as_half((unsigned short)(s0 & 0xffffu)));
    const float k1 = __half2float(__ushort_as_half((unsigned short)(s1 & 0xffffu)));
    constexpr float MAGIC = 12582912.f;
    const float v0 = ((__int_as_float(acc[t][0]) - MAGIC) * f1 + (__int_as_float(acc[t][2]) - MAGIC) * f2) * k0;
    const float v1 = ((__int_as_float(acc[t][1]) - MAGIC) * f1 + (__int_as_float(acc[t][3]) - MAGIC) * f2) * k1;
    sc[t][0] = v0, sc[t][1] = v1;
    if (hi_rel < 31) {                 // last chunk of the row
      if (kk > hi_rel) sc[t][0] = -INFINITY;
      if (kk + 1 > hi_rel) sc[t][1] = -INFINITY;
    }
    mx = fmaxf(mx, fmaxf(sc[t][0], sc[t][1]));
  }
  if (s_next >= 0) step_load_scales(R, ch, s_next, lane);
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  if (__any_sync(0xffffffffu, mx > A.m + RESCALE_GAP)) {   // the running maximum is raised lazily (decode_attn.cu)
    const float m_new = mx > A.m + RESCALE_GAP ? mx : A.m;
    const float alpha = ex2(A.m - m_new);
    A.l *= alpha;
#pragma unroll
    for (int i = 0; i < 8; ++i) A.o[i][0] *= alpha, A.o[i][1] *= alpha;
    A.m = m_new;
  }
  uint32_t pa[2][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float p0 = ex2(sc[t][0] - A.m), p1 = ex2(sc[t][1] - A.m);
    A.l += p0 + p1;
    const __half2 pv = __hmul2(__floats2half2_rn(p0, p1), *reinterpret_cast<const __half2*>(&vsh[t]));
    pa[t / 2][2 * (t & 1)] = *reinterpret_cast<const uint32_t*>(&pv);
    pa[t / 2][2 * (t & 1) + 1] = 0u;
  }
  if (newest) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (16 * u + 2 * q + (j & 1) + (j >> 1) * 8 == key_new)
          ch.v[u][j] = *reinterpret_cast<const uint2*>(&sm.q8[1][r * 8]);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint32_t xa = (w ? ch.v[u][0].y : ch.v[u][0].x) ^ 0x80808080u;
      const uint32_t xb = (w ? ch.v[u][1].y : ch.v[u][1].x) ^ 0x80808080u;
      const uint32_t xc = (w ? ch.v[u][2].y : ch.v[u][2].x) ^ 0x80808080u;
      const uint32_t xd = (w ? ch.v[u][3].y : ch.v[u][3].x) ^ 0x80808080u;
#pragma unroll
      for (int hw = 0; hw < 2; ++hw) {
        const uint32_t tab = __byte_perm(xa, xb, hw ? 0x7362 : 0x5140);
        const uint32_t tcd = __byte_perm(xc, xd, hw ? 0x7362 : 0x5140);
#pragma unroll
        for (int e = 0; e < 2; ++e)
          mma16816(A.o[4 * w + 2 * hw + e], pa[u][0], pa[u][1], pa[u][2], pa[u][3],
                   bias_pair(tab, e ? 0x4342 : 0x4140), bias_pair(tcd, e ? 0x4342 : 0x4140));
      }
    }
  if (s_next >= 0) step_load_v(R, ch, s_next, lane);
}


// ------------------------------------------------------------------------------------------------ exchange
__device__ __forceinline__ uint4 st_peek(const void* p) {   // L2, never an L1 line
  uint4 u;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(p) : "memory");
  return u;
}
__device__ __forceinline__ void st_put(void* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// two results as a published word: the one pattern that means "not there yet" is a pair of NaNs; another NaN says the same
template <typename T> __device__ __forceinline__ uint32_t st_word(float a, float b) {
  const uint32_t w = st_pack2<T>(a, b);
  return w == ST_EMPTY ? 0x7fff7fffu : w;
}
__device__ __forceinline__ void st_prefetch(const void* p, uint32_t bytes) {   // both multiples of 16
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <typename T>
__device__ __forceinline__ void st_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1);
template <>
__device__ __forceinline__ void st_mma<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  mma16816(d, a0, a1, a2, a3, b0, b1);
}
template <>
__device__ __forceinline__ void st_mma<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                      uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// a wait that began at t_begin (0: just now) has taken too long
__device__ __forceinline__ bool st_late(unsigned long long& t_begin) {
  unsigned long long now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
  if (t_begin == 0) t_begin = now;
  return now - t_begin > ST_WAIT_NS;
}
// it has, or another one had
__device__ __forceinline__ bool st_late(unsigned long long& t_begin, volatile int* dead) {
  if (!*dead && !st_late(t_begin)) return false;
  *dead = 1;
  return true;
}
// Load N pieces of 16 bytes until none holds an empty word (the largest unsigned one), again only what did.  Warp-collective.
template <int N, typename At>
__device__ __forceinline__ void st_take(uint4 (&u)[N], At at, volatile int* dead) {
  unsigned long long t_begin = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) u[j] = st_peek(at(j));
#pragma unroll 1
  for (int i = 0;; ++i) {
    bool missing[N], any = false;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      missing[j] = __any_sync(0xffffffffu, max(max(u[j].x, u[j].y), max(u[j].z, u[j].w)) == ST_EMPTY);
      any |= missing[j];
    }
    if (!any) return;
    if ((i & 31) == 31 && __any_sync(0xffffffffu, st_late(t_begin, dead))) return;
    __nanosleep(ST_NAP);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (missing[j]) u[j] = st_peek(at(j));
  }
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ------------------------------------------------------------------------------------------------ the kernel
// HALF: at most 8 rows (the lower half of the MMA's 16; 110 us at 6 rows with it).
template <typename T, bool HALF, int LGM>
__global__ void __launch_bounds__(ST_THREADS, 1) step_kernel(const __grid_constant__ StepP P) {
  constexpr int ROWS = HALF ? 8 : 16, NR = HALF ? 1 : 2;
  // the warps are 2^LGM row tiles times KS slices of K
  using Smem = StepSmem<T, ROWS, LGM>;
  constexpr int MG = 1 << LGM, MROWS = Smem::MROWS, KS = Smem::KS, LD = Smem::LD, TILE = Smem::TILE;
  constexpr int SL = KS / 4, FROWS = 8 / SL;            // threads a feature pair's sums take, rows of a warp there
  extern __shared__ __align__(128) unsigned char st_smem[];
  Smem& sm = *reinterpret_cast<Smem*>(st_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = blockIdx.x, C = gridDim.x;
  const bool own = C - 1 - rank < P.B;                  // the last CTAs own a row each (the first ones have a tile of
  const int64_t orow = C - 1 - rank;                    // every projection)
  volatile int* const dead = &sm.dead;
  const int NQ = (P.H + 2) * ST_HD, NZ = P.H * ST_HD;
  const int r = lane >> 2, q = lane & 3;                // MMA fragment row and column pair
  // finishing a projection: SL threads for each pair of features of a row of a tile (or pair)
  const int sl = tid & (SL - 1), fq = (tid / SL) & 3, frow = (tid / (4 * SL)) & (MROWS - 1), ft = tid / (4 * SL * MROWS);
  const int mg = warp & (MG - 1), ks = warp >> LGM;

  // ---- weights of phase p, layer l into the phase's region: a bulk copy a row, dealt out over the warps (one issues some 25
  //      cycles apart, and would be late for the next phase with all of them)
  auto fetch = [&](int p, int l) {
    const int K = P.K[p], n = (P.base[p] + (rank < P.rem[p])) * (p == PH_GU ? 16 : 8), row = warp + ST_WARPS * lane;
    if (l >= P.L || row >= n) return;
    const uint32_t bar = smem_addr(&sm.full[p]), bytes = (uint32_t)(2 * K);
    if (row == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes * (uint32_t)n) : "memory");
    const int from = p == PH_GU ? ((row >> 3) & 1) * P.f + (rank + (row >> 4) * C) * 8 + (row & 7) : rank * 8 + row;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(st_smem + P.region[p]) + (uint32_t)row * (bytes + 64u)),
                 "l"(static_cast<const T*>(sm.layer[l].w[p]) + (int64_t)from * K), "r"(bytes), "r"(bar)
                 : "memory");
  };
  auto weights_ready = [&](int p, int l) {              // of phase p, layer l (also after another wait has given up: no CTA
                                                        // may end with copies on their way to its memory)
    const uint32_t bar = smem_addr(&sm.full[p]);
    unsigned long long t_begin = 0;
#pragma unroll 1
    for (int i = 0;; ++i) {
      uint32_t ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(ok) : "r"(bar), "r"((uint32_t)(l & 1)) : "memory");
      if (ok) return;
      if ((i & 63) == 63 && st_late(t_begin)) {
        *dead = 1;
        return;
      }
    }
  };

  for (int i = tid; i < P.L * (int)(sizeof(StepLayerK) / 8); i += ST_THREADS)
    reinterpret_cast<uint64_t*>(sm.layer)[i] = reinterpret_cast<const uint64_t*>(P.layer)[i];
  if (tid == 0) {
    sm.dead = 0;
    for (int p = 0; p < 4; ++p)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[p])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
#pragma unroll 1
  for (int p = 0; p < 4; ++p) fetch(p, 0);

  // ---- the owned row: token, position, cache row
  int pos = 0, start = 0, pmod = 0;                     // pmod: position modulo the ring length of the first local layer
  int64_t tok = 0, crow = 0;
  float2 cs = make_float2(1.f, 1.f), sn = make_float2(0.f, 0.f);   // rotation of this lane's two dimensions of a head
  if (own) {
    tok = P.tok[orow];
    if (tok < 0 || tok >= P.vocab) tok = 0;
    const int64_t st = P.starts[orow];
    pos = (int)P.pos[orow], start = st > 0 ? (int)st : 0, crow = P.row_map ? P.row_map[orow] : orow;
    pmod = P.ring_S > 0 && pos >= 0 ? pos % P.ring_S : 0;
    if (lane < P.n_pairs) {
      const int i = (2 * lane) & (P.n_pairs - 1);
      const float t0 = (float)pos * P.inv_freq[i], t1 = (float)pos * P.inv_freq[i + 1];
      cs = st_rnd2<T>(cosf(t0), cosf(t1)), sn = st_rnd2<T>(sinf(t0), sinf(t1));
      if (2 * lane < P.n_pairs) sn.x = -sn.x, sn.y = -sn.y;
    }
  }
  // keys and values that layer l will read for it, on their way to L2 (whole warp)
  auto prefetch_kv = [&](int l) {
    const StepLayerK& Y = sm.layer[l];
    int a = start, e = pos;                             // slots [a, e)
    if (Y.ring && pos >= Y.S) a = 0, e = Y.S;
    if (e > Y.S) e = Y.S;
    a &= ~7, e = (e + 7) & ~7;
    if ((Y.S_alloc & 7) == 0 && ((reinterpret_cast<uintptr_t>(Y.ks) | reinterpret_cast<uintptr_t>(Y.vs)) & 15) == 0) {
      const int64_t at = crow * Y.S_alloc;
#pragma unroll 1
      for (int s = a + 256 * lane; s < e; s += 256 * 32) {
        const uint32_t n = (uint32_t)(e - s < 256 ? e - s : 256);
        st_prefetch(Y.kc + (at + s) * ST_HD, n * ST_HD);
        st_prefetch(Y.vc + (at + s) * ST_HD, n * ST_HD);
        st_prefetch(Y.ks + at + s, n * 2);
        st_prefetch(Y.vs + at + s, n * 2);
      }
    }
    __syncwarp();
  };
  // a row of x, 16-byte pieces; returns its RMS-norm factor (whole warp)
  auto row_rs = [&](const T* x, uint4 (&u)[4]) {
    st_take<4>(u, [&](int j) { return x + (8 * lane + 256 * j < P.d ? (lane + 32 * j) * (ROWS * 8) : 0); }, dead);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (8 * lane + 256 * j < P.d) {
        float v[8];
        st_unpack8<T>(u[j], v);
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
      }
    return rsqrtf(warp_sum(ss) / (float)P.d + RMS_EPS);
  };
  // one word (whole warp; p: null where a lane wants none)
  auto word = [&](const T* p) {
    uint32_t v = 0u;
    unsigned long long t_begin = 0;
#pragma unroll 1
    for (int i = 0;; ++i) {
      if (p) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
      if (!__any_sync(0xffffffffu, v == ST_EMPTY)) return v;
      __nanosleep(ST_NAP);
      if ((i & 31) == 31 && __any_sync(0xffffffffu, st_late(t_begin, dead))) return v;
    }
  };

  // a buffer of `width` features is row tiles of [8 features][ROWS rows][8]: what one CTA publishes of a row tile is one or
  // two whole lines.  Lines with several writers were seen 1-3 us late.
  auto at_row = [](int row, int width) { return (row / ROWS) * (width * ROWS) + (row & (ROWS - 1)) * 8; };
  // ---- embedding and its norm
  T* const ws = static_cast<T*>(P.buf);
  if (own && warp == 0) {
    const T* e = static_cast<const T*>(P.embed) + tok * P.d;
    float v[4][8], ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 8 * lane + 256 * j;
      st_unpack8<T>(c < P.d ? __ldg(reinterpret_cast<const uint4*>(e + c)) : make_uint4(0u, 0u, 0u, 0u), v[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += v[j][k] * v[j][k];
    }
    const float inv = rsqrtf(warp_sum(ss) / (float)P.d + RMS_EPS);
    T* x = ws + P.off[0] + at_row(orow, P.d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 8 * lane + 256 * j;
      if (c < P.d)
#pragma unroll
        for (int k = 0; k < 8; k += 2)
          st_put(x + c * ROWS + k, st_word<T>(v[j][k] * inv, v[j][k + 1] * inv));
    }
  }
  if (own && warp == ST_WARPS - 1) prefetch_kv(0);
  // ---- the residual stream: two values of a row at the thread that finishes their sums
  const bool has_x = rank < P.rem[PH_WO] || P.base[PH_WO] > 0;
  const bool fin = frow < P.B && sl == 0;
  float2 res = make_float2(0.f, 0.f);
  if (has_x && ft == 0 && (frow & ~(FROWS - 1)) < P.B)
    res = st_unpack2<T>(word(frow < P.B ? ws + P.off[0] + rank * (ROWS * 8) + at_row(frow, P.d) + 2 * fq : nullptr));

  // ---- a projection: rows of `in` (row stride K) times this CTA's tiles of phase p; done(sums of this thread's pair of
  //      features (gate | up: of both), the row's norm factor (gate | up))
  int odd = 0;                                          // areas for partial sums take turns
  auto project = [&](auto phase, int l, const T* in, auto&& done) {
    constexpr int p = decltype(phase)::value, NT = p == PH_GU ? 2 * ST_PAIRS : 1;
    // pieces of 32 K values in flight
    constexpr int J = LGM == 0 ? (p == PH_DN ? 4 : 2) : LGM == 1 ? (p == PH_DN ? 4 : 3) : (p == PH_WO ? 4 : 5);
    const int mine = P.base[p] + (rank < P.rem[p]);     // tiles or pairs of this CTA: at most one, at most ST_PAIRS
    if (mine == 0) return;
    const int K = P.K[p], ld = 2 * K + 64;
    uint32_t w = smem_addr(st_smem + P.region[p]) + (uint32_t)(r * ld + ks * 64 + q * 16);
    constexpr int PIECE = KS * (p == PH_WO ? 32 : 32 * ROWS);   // elements between a warp's pieces
    weights_ready(p, l);
    // this lane's rows of the A fragments (past the batch: the last row again, whose sums nobody reads)
    const int mt = mg * ROWS, ra = mt + r < P.B ? mt + r : P.B - 1, rb = mt + r + 8 < P.B ? mt + r + 8 : P.B - 1;
    const int to_b = (rb - ra) * (p == PH_WO ? K : 8);
    const T* pa = p == PH_WO ? in + ra * K + ks * 32 + 8 * q : in + (ks * 4 + q) * (ROWS * 8) + at_row(ra, K);
    float2* const red = sm.red[odd];
    float* const ssq = sm.ssq[odd];
    odd ^= 1;
    float acc[NT][4], gram[2][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n) gram[n][0] = gram[n][1] = gram[n][2] = gram[n][3] = 0.f;
#pragma unroll 1
    for (int left = mt < P.B ? ((K >> 5) - ks + KS - 1) / KS : 0; left > 0; left -= J) {
      uint4 u[J * NR];
      st_take<J * NR>(u, [&](int j) { return pa + (j / NR < left ? (j / NR) * PIECE : 0) + (j % NR ? to_b : 0); }, dead);
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (j < left) {
          const uint4 a = u[j * NR], b = HALF ? make_uint4(0u, 0u, 0u, 0u) : u[j * NR + NR - 1];
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            if (MG > 1 && n > 1 && mine == 1) continue;
            uint4 b4;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(b4.x), "=r"(b4.y), "=r"(b4.z), "=r"(b4.w)
                         : "r"(w + (uint32_t)(n * 8 * ld + j * KS * 64)));
            st_mma<T>(acc[n], a.x, b.x, a.y, b.y, b4.x, b4.y);
            st_mma<T>(acc[n], a.z, b.z, a.w, b.w, b4.z, b4.w);
          }
          if (p == PH_GU) {                             // sums of squares of the rows: the diagonal of rows times rows
            st_mma<T>(gram[0], a.x, b.x, a.y, b.y, a.x, a.y);
            st_mma<T>(gram[0], a.z, b.z, a.w, b.w, a.z, a.w);
            if (!HALF) {
              st_mma<T>(gram[1], a.x, b.x, a.y, b.y, b.x, b.y);
              st_mma<T>(gram[1], a.z, b.z, a.w, b.w, b.z, b.w);
            }
          }
        }
      pa += J * PIECE, w += J * KS * 64;
    }
    float2* at = red + (mg * ROWS * 4 + lane) * LD + ks;  // lane = row * 4 + pair
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      at[n * TILE] = make_float2(acc[n][0], acc[n][1]);
      if (!HALF) at[n * TILE + 32 * LD] = make_float2(acc[n][2], acc[n][3]);
    }
    if (p == PH_GU && q == (r >> 1)) {                  // columns 2 q, 2 q + 1
      ssq[(mg * ROWS + r) * KS + ks] = r & 1 ? gram[0][1] : gram[0][0];
      if (!HALF) ssq[(mg * ROWS + r + 8) * KS + ks] = r & 1 ? gram[1][3] : gram[1][2];
    }
    __syncthreads();
    if (ft < mine && (frow & ~(FROWS - 1)) < P.B) {                // (whole warps)
      auto sum4 = [&](const float2* at) {               // of the four slices that are this thread's
        const float4 x = reinterpret_cast<const float4*>(at)[0], y = reinterpret_cast<const float4*>(at)[1];
        return make_float2((x.x + x.z) + (y.x + y.z), (x.y + x.w) + (y.y + y.w));
      };
      auto sum_lanes = [](float2& v) {
#pragma unroll
        for (int o = 1; o < SL; o *= 2)
          v.x += __shfl_xor_sync(0xffffffffu, v.x, o), v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      };
      const float2* from = red + (p == PH_GU ? 2 * ft * TILE : 0) + (frow * 4 + fq) * LD + 4 * sl;
      float2 s0 = sum4(from), s1 = s0;
      float ss = 0.f;
      if (p == PH_GU) {
        s1 = sum4(from + TILE);
        const float4 g = *reinterpret_cast<const float4*>(ssq + frow * KS + 4 * sl);
        ss = (g.x + g.y) + (g.z + g.w);
#pragma unroll
        for (int o = 1; o < SL; o *= 2) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        sum_lanes(s1);
      }
      sum_lanes(s0);
      done(s0, s1, p == PH_GU ? rsqrtf(ss / (float)P.d + RMS_EPS) : 0.f);
    }
    fetch(p, l + 1);                                    // (every warp is done with the weights)
  };

  T* x0 = ws + P.off[0];                                // this layer's buffers
#pragma unroll 1                                        // (the code of a layer fits the instruction caches, four do not)
  for (int l = 0; l < P.L; ++l, x0 += P.stride) {
    const StepLayerK& Ly = sm.layer[l];
    T *const x1 = x0 + P.off[1], *const qkv = x0 + P.off[2], *const zb = x0 + P.off[3], *const actb = x0 + P.off[4];
    // ---- before the QKV projection: the first keys of this warp's share of the attention are requested
    StepRow row;
    StepChunk cur;
    int c0 = 0, c1 = 0, nw = 0, slot = 0;               // this warp's chunks; warps that have any
    if (own) {
      int lo = start, hi = pos;
      if (Ly.window > 0 && pos - Ly.window + 1 > lo) lo = pos - Ly.window + 1;
      if (Ly.ring) {
        if (pos - Ly.S + 1 > lo) lo = pos - Ly.S + 1;
      } else if (hi > Ly.S - 1) {
        hi = Ly.S - 1;
      }
      const int64_t at = crow * Ly.S_alloc;
      row.k = Ly.kc + at * ST_HD, row.v = Ly.vc + at * ST_HD, row.ks = Ly.ks + at, row.vs = Ly.vs + at;
      row.lo = lo, row.hi = hi, row.newest = hi == pos ? pos : -1, row.S = Ly.S, row.S_alloc = Ly.ring ? Ly.S : Ly.S_alloc;
      row.ring = Ly.ring;
      if (hi >= lo) {
        const int n = ((hi - lo) >> 5) + 1, each = (n + ST_WARPS - 1) / ST_WARPS;
        c0 = warp * each;
        c1 = c0 + each < n ? c0 + each : n;
        nw = each == 1 ? n : (n + each - 1) / each;
      }
      slot = lo + c0 * 32;                              // chunks count from the first key (a window is whole chunks)
      if (row.ring && c0 < c1) {                        // the slot of that position, which lies less than S below p
        slot = (row.S == P.ring_S ? pmod : pos % row.S) - (pos - slot);
        if (slot < 0) slot += row.S;
      }
      if (c0 < c1) step_load(row, cur, slot, lane);
      if (warp == ST_WARPS - 1 && l + 1 < P.L) prefetch_kv(l + 1);
    }
    // ---- QKV projection
    project(std::integral_constant<int, PH_QKV>{}, l, x0, [&](float2 a, float2, float) {
      if (fin) st_put(qkv + rank * (ROWS * 8) + at_row(frow, NQ) + 2 * fq, st_word<T>(a.x, a.y));
    });
    if (own) {
      // ---- the owned row, a warp a head (queries, key, value), two dimensions a lane: QK norm, RoPE, value embedding, int8
      //      append (qkv_post.cuh), and the head's gate
      const int h = warp;
      const bool isv = h == P.H + 1, adds = isv && Ly.ve_gate != nullptr;
      float g = 1.0f;                                   // 2 sigmoid(w . the leading normalised channels)
      if (h < P.H + 2) {
        const T* const xr = x0 + at_row(orow, P.d);
        const T* const gw = h < P.H ? static_cast<const T*>(Ly.gate_w) : adds ? static_cast<const T*>(Ly.ve_gate) : nullptr;
        const int n = h < P.H ? P.gate_ch : P.ve_ch;
        const T* const w = gw + (h < P.H ? h * n : 0);
        const bool quads = gw != nullptr && (n & 3) == 0;
        uint2 w4 = make_uint2(0u, 0u);
        uint32_t ve = 0u;
        if (quads && 4 * lane < n) w4 = __ldg(reinterpret_cast<const uint2*>(w + 4 * lane));
        if (adds)
          ve = __ldg(reinterpret_cast<const unsigned int*>(static_cast<const T*>(P.value_embed) + tok * ST_HD + 2 * lane));
        uint4 u[4];
        const float rs = row_rs(xr, u);
        if (gw != nullptr) {
          float dot = 0.f;
          if (quads) {                                  // channels 4 lane .. 4 lane + 3, from the lane that has them
            const uint32_t a = __shfl_sync(0xffffffffu, u[0].x, lane >> 1), b = __shfl_sync(0xffffffffu, u[0].y, lane >> 1);
            const uint32_t c = __shfl_sync(0xffffffffu, u[0].z, lane >> 1), d = __shfl_sync(0xffffffffu, u[0].w, lane >> 1);
            const float2 v0 = st_unpack2<T>(lane & 1 ? c : a), v1 = st_unpack2<T>(lane & 1 ? d : b);
            const float2 y0 = st_rnd2<T>(v0.x * rs, v0.y * rs), y1 = st_rnd2<T>(v1.x * rs, v1.y * rs);
            const float2 a0 = st_unpack2<T>(w4.x), a1 = st_unpack2<T>(w4.y);
            dot = (a0.x * y0.x + a0.y * y0.y) + (a1.x * y1.x + a1.y * y1.y);
          } else {
            for (int c = lane; c < n; c += 32) {
              const unsigned short v = __ldcg(reinterpret_cast<const unsigned short*>(xr + (c >> 3) * (ROWS * 8) + (c & 7)));
              dot += to_f32<T>(w[c]) * rnd<T>(to_f32<T>(*reinterpret_cast<const T*>(&v)) * rs);
            }
          }
          g = rnd<T>(2.0f * rnd<T>(__fdividef(1.0f, 1.0f + __expf(-rnd<T>(warp_sum(dot))))));
        }
        float2 x = st_unpack2<T>(word(qkv + (h * 8 + (lane >> 2)) * (ROWS * 8) + at_row(orow, NQ) + 2 * (lane & 3)));
        x = st_rnd2<T>(x.x * rs, x.y * rs);
        if (!isv) {
          const float inv = rsqrtf(warp_sum(x.x * x.x + x.y * x.y) / (float)ST_HD + RMS_EPS);
          x = st_rnd2<T>(x.x * inv, x.y * inv);
          if (Ly.rope) {                                // dim j < n_pairs turns with dim j + n_pairs: x1 c - x2 s, x1 s + x2 c,
            const float o0 = __shfl_xor_sync(0xffffffffu, x.x, P.n_pairs / 2);   // every product and sum rounded
            const float o1 = __shfl_xor_sync(0xffffffffu, x.y, P.n_pairs / 2);
            const float2 a = st_rnd2<T>(x.x * cs.x, x.y * cs.y), d = st_rnd2<T>(o0 * sn.x, o1 * sn.y);
            const float2 y = st_rnd2<T>(a.x + d.x, a.y + d.y);
            if (lane < P.n_pairs) x = y;
          }
        } else if (adds) {
          const float2 e = st_unpack2<T>(ve), a = st_rnd2<T>(g * e.x, g * e.y);
          x = st_rnd2<T>(x.x + a.x, x.y + a.y);
        }
        const float amax = warp_max(fmaxf(fabsf(x.x), fabsf(x.y)));
        if (h < P.H) {
          // the query head in two int8 parts, as split_q (attn_math.cuh): adding 1.5 * 2^23 rounds to an integer whose
          // low byte is the part
          const float s1 = amax > 0.f ? amax / 127.0f : 1.0f, inv1 = 1.0f / s1, inv2 = 254.0f / s1;
          constexpr float MAGIC = 12582912.f;
          const float ra1 = fmaf(x.x, inv1, MAGIC), rb1 = fmaf(x.y, inv1, MAGIC);
          const float ra2 = fmaf(fmaf(-(ra1 - MAGIC), s1, x.x), inv2, MAGIC);
          const float rb2 = fmaf(fmaf(-(rb1 - MAGIC), s1, x.y), inv2, MAGIC);
          *reinterpret_cast<uint16_t*>(&sm.qi[0][h][2 * lane]) =
              (uint16_t)__byte_perm(__float_as_uint(ra1), __float_as_uint(rb1), 0x0040);
          *reinterpret_cast<uint16_t*>(&sm.qi[1][h][2 * lane]) =
              (uint16_t)__byte_perm(__float_as_uint(ra2), __float_as_uint(rb2), 0x0040);
          if (lane == 0) sm.qf[h] = s1 * P.scale_log2;
        } else {
          // key / value: quantize_lane (common.cuh), to shared memory and to the cache
          const __half s16 = __float2half_rn(__fdiv_rn(amax, 127.0f));
          const float sf = fmaxf(__half2float(s16), 1e-30f);
          const float a = fminf(fmaxf(rintf(__fdiv_rn(x.x, sf)), -127.0f), 127.0f);
          const float b = fminf(fmaxf(rintf(__fdiv_rn(x.y, sf)), -127.0f), 127.0f);
          const uint16_t w8 = (uint16_t)(((uint32_t)__float2int_rn(a) & 0xffu) | (((uint32_t)__float2int_rn(b) & 0xffu) << 8));
          *reinterpret_cast<uint16_t*>(&sm.q8[isv][2 * lane]) = w8;
          if (lane == 0) sm.sc[isv] = __half_as_ushort(s16);
          int p = pos;
          if (Ly.ring) p = p >= 0 && Ly.S == P.ring_S ? pmod : (p % Ly.S + Ly.S) % Ly.S;
          if (p < 0 || p >= Ly.S) {
            if (lane == 0 && P.oob) atomicAdd(P.oob, 1);
          } else {
            const int64_t dst = crow * Ly.S_alloc + p;
            *reinterpret_cast<uint16_t*>((isv ? Ly.vc : Ly.kc) + dst * ST_HD + 2 * lane) = w8;
            if (lane == 0) (isv ? Ly.vs : Ly.ks)[dst] = __half_as_ushort(s16);
          }
          if (isv) {                                    // for XSA: the value and 1 / |v|^2
            *reinterpret_cast<uint32_t*>(&sm.vcur[2 * lane]) = st_pack2<T>(x.x, x.y);
            const float vinv = 1.0f / fmaxf(sqrtf(warp_sum(x.x * x.x + x.y * x.y)), P.xsa_eps);
            if (lane == 0) sm.vinv2 = vinv * vinv;
          }
        }
      }
      __syncthreads();
      // ---- attention
      if (c0 < c1) {
        StepAcc A;
#pragma unroll
        for (int i = 0; i < 8; ++i) A.o[i][0] = A.o[i][1] = A.o[i][2] = A.o[i][3] = 0.f;
        A.m = -INFINITY, A.l = 0.f;
        uint32_t q1[4] = {0u, 0u, 0u, 0u}, q2[4] = {0u, 0u, 0u, 0u};
        float f1 = 0.f;
        if (r < P.H) {
          const uint4 a = *reinterpret_cast<const uint4*>(&sm.qi[0][r][16 * q]);
          const uint4 c = *reinterpret_cast<const uint4*>(&sm.qi[1][r][16 * q]);
          q1[0] = a.x, q1[1] = a.y, q1[2] = a.z, q1[3] = a.w, q2[0] = c.x, q2[1] = c.y, q2[2] = c.z, q2[3] = c.w;
          f1 = sm.qf[r];
        }
        const float f2 = f1 * (1.0f / 254.0f);
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
          slot += 32;
          if (row.ring && slot >= row.S) slot -= row.S;
          step_chunk(row, sm, cur, A, q1, q2, f1, f2, row.lo + c * 32, c + 1 < c1 ? slot : -1, lane);
        }
        float lsum = A.l;
        lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
        lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
        if (q == 0) sm.mg_m[r][warp] = A.m, sm.mg_l[r][warp] = lsum;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<float4*>(&sm.mg_o[warp][r][(2 * q + e) * 8 + 4 * j]) =
                make_float4(A.o[4 * j][e], A.o[4 * j + 1][e], A.o[4 * j + 2][e], A.o[4 * j + 3][e]);
      }
      __syncthreads();
      // ---- the warps' results merged, then XSA and the head gate (finalize_row, decode_attn.cu)
      if (h < P.H) {
        const float m = lane < nw ? sm.mg_m[h][lane] : -INFINITY;
        const float mx = warp_max(m), wt = m == -INFINITY ? 0.f : ex2(m - mx);
        const float sum = warp_sum(lane < nw ? wt * sm.mg_l[h][lane] : 0.f), inv = sum > 0.f ? 1.0f / sum : 0.f;
        float2 z = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int w = 0; w < nw; ++w) {
          const float ww = __shfl_sync(0xffffffffu, wt, w);
          const float2 a = *reinterpret_cast<const float2*>(&sm.mg_o[w][h][2 * lane]);
          z.x += ww * a.x, z.y += ww * a.y;
        }
        z = st_rnd2<T>(z.x * inv, z.y * inv);
        if (Ly.xsa_alpha != nullptr) {
          const float2 v = st_unpack2<T>(*reinterpret_cast<const uint32_t*>(&sm.vcur[2 * lane]));
          const float ad = __ldg(Ly.xsa_alpha + h) * warp_sum(z.x * v.x + z.y * v.y) * sm.vinv2;
          z = st_rnd2<T>(z.x - ad * v.x, z.y - ad * v.y);
        }
        st_put(zb + orow * NZ + h * ST_HD + 2 * lane, st_word<T>(z.x * g, z.y * g));
      }
    }
    // ---- output projection, gate | up, down
    auto residual = [&](T* out) {                       // x += sums
      return [&, out](float2 a, float2, float) {
        a = st_rnd2<T>(a.x, a.y);
        const uint32_t w = st_word<T>(res.x + a.x, res.y + a.y);
        res = st_unpack2<T>(w);
        if (fin) st_put(out + rank * (ROWS * 8) + at_row(frow, P.d) + 2 * fq, w);
      };
    };
    project(std::integral_constant<int, PH_WO>{}, l, zb, residual(x1));
    project(std::integral_constant<int, PH_GU>{}, l, x1, [&](float2 g, float2 u, float s) {
      float2 g2 = st_rnd2<T>(g.x, g.y), u2 = st_rnd2<T>(u.x, u.y);
      g2 = st_rnd2<T>(g2.x * s, g2.y * s), u2 = st_rnd2<T>(u2.x * s, u2.y * s);
      const float2 a = st_rnd2<T>(__fdividef(g2.x, 1.0f + __expf(-g2.x)), __fdividef(g2.y, 1.0f + __expf(-g2.y)));
      if (fin)
        st_put(actb + (rank + ft * C) * (ROWS * 8) + at_row(frow, P.f) + 2 * fq, st_word<T>(a.x * u2.x, a.y * u2.y));
    });
    project(std::integral_constant<int, PH_DN>{}, l, actb, residual(x0 + P.stride));
  }
  // ---- the final norm of the owned row
  if (own && warp == 0) {
    uint4 u[4];
    const float rs = row_rs(x0 + at_row(orow, P.d), u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 8 * lane + 256 * j;
      float v[8];
      st_unpack8<T>(u[j], v);
      if (c < P.d) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] *= rs;
        *reinterpret_cast<uint4*>(static_cast<T*>(P.xn) + orow * P.d + c) = st_pack8<T>(v);
      }
    }
  }
  __syncthreads();
  if (tid == 0 && sm.dead && P.status) atomicOr(P.status, 8);
}

// ------------------------------------------------------------------------------------------------ host side
constexpr size_t ST_SMEM_MAX = 227 * 1024;

typedef void (*StepKernel)(const StepP);
template <typename T> static StepKernel step_variant_of(int rows) {
  return rows <= 8 ? step_kernel<T, true, 0> : rows <= 16 ? step_kernel<T, false, 0> : rows <= 32 ? step_kernel<T, false, 1>
                                                                                                  : step_kernel<T, false, 2>;
}
static StepKernel step_variant(bool f16, int rows) {
  return f16 ? step_variant_of<__half>(rows) : step_variant_of<__nv_bfloat16>(rows);
}
static size_t step_state_bytes(int rows) {
  return rows <= 8 ? sizeof(StepSmem<__half, 8, 0>) : rows <= 16 ? sizeof(StepSmem<__half, 16, 0>)
                   : rows <= 32 ? sizeof(StepSmem<__half, 16, 1>) : sizeof(StepSmem<__half, 16, 2>);
}

// Multiprocessors of the current device (0: it cannot run the kernel), asked for once per device.
static int step_sms() {
  constexpr int MAXDEV = 64;
  static int known[MAXDEV];
  static bool done[MAXDEV];
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAXDEV) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    int sms = 0, coop = 0;
    bool ok = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop;
    for (int k = 0; k < 8; ++k)
      ok = ok && cudaFuncSetAttribute(step_variant(k & 1, 8 << (k >> 1)), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)ST_SMEM_MAX) == cudaSuccess;
    if (!ok) cudaGetLastError();
    known[dev] = ok ? sms : 0, done[dev] = true;
  }
  return known[dev];
}

// The split and the shared-memory map; false: these shapes do not go this way.
static bool step_plan(const uv_step_args* a, StepP* P, size_t* smem, int* sms) {
  if (a->B > ST_ROWS) return false;
  if (a->dtype != UV_F16 && a->dtype != UV_BF16) return false;
  if (a->hd != ST_HD || a->K != 1 || a->H < 1 || a->H > 8 || a->n_layers < 1 || a->n_layers > ST_MAXL) return false;
  // K in pieces of 32 whose padded rows start 64 bytes apart from a multiple of 128
  if (a->d % 64 || a->d > 1024 || a->f % 64 || a->gate_ch > ST_XCH || a->ve_ch > ST_XCH || a->gate_ch > a->d || a->ve_ch > a->d)
    return false;
  for (int l = 0; l < a->n_layers; ++l) {
    const uv_step_layer& y = a->h_layers[l];
    if (y.S < 1 || (y.ring && y.S < 32)) return false;
    if (y.rope && a->n_pairs != 8 && a->n_pairs != 16 && a->n_pairs != 32) return false;
  }
  *sms = step_sms();
  if (*sms < a->B) return false;
  P->B = a->B, P->L = a->n_layers, P->d = a->d, P->H = a->H, P->f = a->f;
  P->K[PH_QKV] = P->K[PH_GU] = a->d, P->K[PH_WO] = a->H * ST_HD, P->K[PH_DN] = a->f;
  const int tiles[4] = {(a->H + 2) * ST_HD / 8, a->d / 8, a->f / 8, a->d / 8};
  size_t at = (step_state_bytes(a->B) + 127) & ~(size_t)127;
  for (int p = 0; p < 4; ++p) {
    const int most = p == PH_GU ? ST_PAIRS : 1;
    P->region[p] = (int)at;
    P->base[p] = tiles[p] / *sms, P->rem[p] = tiles[p] % *sms;
    if (P->base[p] + (P->rem[p] > 0) > most) return false;
    at += (size_t)most * (p == PH_GU ? 16 : 8) * (2 * P->K[p] + 64);
  }
  *smem = at;
  return at <= ST_SMEM_MAX;
}

}  // namespace uv

static int step_rows(int B) { return B <= 8 ? 8 : (B + 15) / 16 * 16; }   // rows as stored

extern "C" size_t uv_decode_step_workspace_bytes(const uv_step_args* a) {
  if (!a || a->B < 1) return 0;
  return (size_t)2 * step_rows(a->B) * (a->n_layers * (2 * a->d + (2 * a->H + 2) * (size_t)a->hd + a->f) + a->d);
}

extern "C" int uv_decode_step_supported(const uv_step_args* a) {
  using namespace uv;
  if (!a || a->B < 1 || !a->h_layers) return 0;
  StepP P{};
  size_t smem;
  int sms;
  return step_plan(a, &P, &smem, &sms) ? 1 : 0;
}

extern "C" int uv_decode_step(const uv_step_args* a, void* stream) {
  using namespace uv;
  if (!a) return UV_ERR_ARG;
  if (a->B == 0) return UV_OK;
  if (a->B < 0 || !a->h_layers || !a->tok || !a->pos || !a->starts || !a->embed || !a->xn || a->vocab < 1) return UV_ERR_ARG;
  StepP P{};
  size_t smem = 0;
  int sms = 0;
  if (!step_plan(a, &P, &smem, &sms)) return UV_ERR_SHAPE;
  const size_t ws = uv_decode_step_workspace_bytes(a);
  if (!a->workspace || a->workspace_bytes < ws) return UV_ERR_WORKSPACE;
  if (!aligned16(a->workspace) || !aligned16(a->embed) || !aligned16(a->xn)) return UV_ERR_ALIGN;
  P.tok = a->tok, P.pos = a->pos, P.starts = a->starts, P.row_map = a->row_map;
  P.embed = a->embed, P.value_embed = a->value_embed, P.inv_freq = a->inv_freq, P.xn = a->xn;
  P.oob = a->oob_count, P.status = a->status, P.vocab = a->vocab;
  P.n_pairs = a->n_pairs, P.gate_ch = a->gate_ch, P.ve_ch = a->ve_ch;
  P.scale_log2 = a->scale * LOG2E, P.xsa_eps = a->xsa_eps;
  const int64_t width[5] = {a->d, a->d, (a->H + 2) * ST_HD, a->H * ST_HD, a->f};
  for (int b = 0; b < 5; ++b) P.off[b] = (int)P.stride, P.stride += width[b] * step_rows(a->B);
  P.buf = a->workspace;
  bool rope = false;
  for (int l = a->n_layers - 1; l >= 0; --l) {
    const uv_step_layer& y = a->h_layers[l];
    StepLayerK& o = P.layer[l];
    if (!y.wqkv || !y.wo || !y.gu || !y.down || !y.k_cache || !y.v_cache || !y.k_scale || !y.v_scale) return UV_ERR_ARG;
    if ((y.ve_gate && (!a->value_embed || a->ve_ch < 1)) || (y.attn_gate && a->gate_ch < 1)) return UV_ERR_ARG;
    for (const void* q : {y.wqkv, y.wo, y.gu, y.down, y.ve_gate, y.ve_gate ? a->value_embed : nullptr, y.attn_gate,
                          (const void*)y.k_cache, (const void*)y.v_cache})
      if (!aligned16(q)) return UV_ERR_ALIGN;
    o.w[PH_QKV] = y.wqkv, o.w[PH_WO] = y.wo, o.w[PH_GU] = y.gu, o.w[PH_DN] = y.down;
    o.ve_gate = y.ve_gate, o.gate_w = y.attn_gate, o.xsa_alpha = y.xsa_alpha;
    o.kc = y.k_cache, o.vc = y.v_cache, o.ks = y.k_scale, o.vs = y.v_scale;
    o.S = y.S, o.S_alloc = y.S_alloc > y.S ? y.S_alloc : y.S, o.ring = y.ring, o.window = y.window, o.rope = y.rope;
    if (y.ring) P.ring_S = y.S;
    rope = rope || y.rope;
  }
  if (!rope) P.n_pairs = 0;
  if (rope && !a->inv_freq) return UV_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(a->workspace, 0xff, ws, st);   // every word "not there yet"
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sms), cfg.blockDim = dim3(ST_THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;                   // its CTAs wait for one another: all of them or none
  attr[0].val.cooperative = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, step_variant(a->dtype == UV_F16, a->B), P);
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_last_cuda_error((int)e);
    return UV_ERR_CUDA;
  }
  return check_launch();
}
