// Linear recurrences with a matrix state S (d x dv) per head over prompt portions, in tiles of 64 tokens on the tensor cores: the gated
// delta rule (delta_rule.cu: a decay per head), the delta rule with a decay per key channel and the token-shift recurrence with a bonus
// for the current token (recurrence.cu).  With P_t the product of the tile's decays up to t (a vector over the key channels; P_t / P_j
// below stands for the product of the decays behind j up to t, never for a division) and S0 the state at the tile's start,
//   A_tj = beta_t (P_t / P_j o k_t) . k_j  (j < t),   Q_tj = (P_t / P_j o q_t) . k_j  (j <= t),   T = (I + A)^-1 diag(beta),
//   w = U - W S0 with U = T V, W = T (P o K);   o = (P o Q) S0 + Q w;   S = P_last o S0 + (P_last / P o K)^T w.
// The bonus recurrence has w = v; its read-out sees the decays up to t - 1 and Q_tt = (u o q_t) . k_t.
//
// Two kernels.  (1) All tiles side by side: everything above that does not depend on S0.  (2) A CTA per 32 value columns of a head of
// a sequence walks the tiles; four products a tile are left: W S0, (P o Q) S0, Q w and the state's update.
//
// Everything is float32 as in the kernels that walk: a float32 operand goes into mma.sync as three bfloat16 terms (mma_split.cuh) and a
// product of two of them as the six products of terms that reach the last bit of float32, the five small ones into sums of their own.
// Products of decays are only ever multiplied together (at most 1, underflow to zero is right): for tokens t and j in different blocks of 16
// the decays behind j are split at a border between the blocks, those behind it go with t, those in front of it with j; blocks of 16 are
// taken on the CUDA cores, split at their middle, and the halves of 8 by running products.
// A masked weight is 0, and 0 times an infinity or a NaN is a NaN; an infinity in three terms is one too.  So a CTA of the second kernel looks
// at what it computed: where a read-out or the state is not finite, it walks its columns again token after token (walk_again), and infinities
// and NaNs appear where the recurrence has them.  Looking costs a multiply-add for each result.
//
// What bounds it, and what it measured.  (1) takes a CTA an SM (228 KB) about 50,000 clocks a tile and head of 128 with a decay per channel, in
// steps that wait on one another: 14,000 until the rows are there as unit vectors and decays (their loads 5,000, the exponentials 4,800), the diagonal
// blocks 5,600, products of decays 7,700, blocks below the diagonal 3,300, the inverse 6,100, W and U 7,600, W's way out 2,200.  (2) takes 3.7 us a
// tile (4.9 with 32 columns a CTA), by mma.sync (318 a tile and warp) and its operands' arrival (157 KB by bulk copies; with a cp.async per 16 bytes, 6.5 us).
// Against the kernels that walk, us: decay per head in bfloat16 (kernels of its own, below), 16 heads of 128, one prompt of 2,048 tokens 773 -> 134;
// decay per channel, prompts of 1,400 and 2,100 1,050 -> 320, one of 2,048 1,005 -> 204; bonus, 16 heads of 64, float32, prompts of 200 and 301 108 -> 28,
// 4,096 1,333 -> 207.  Short portions, and many of them in a wide model, are walked (ops.recurrence_form says where the line lies).
// Errors against 64 bits are the walks' or smaller (decay per channel, 2,048 tokens: o 4.9e-7 and S 5.0e-7, walked 5.4e-7 and 5.4e-7).
#include "common.cuh"
#include "mma_split.cuh"
#include <type_traits>

using namespace dli;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int TOKENS = 64;            // of a tile
constexpr int Q_TILE = 16 * 32;       // bytes of a term of a 16 x 16 block (two 16-byte halves a row, exchanged in rows 4..7 and 12..15)
constexpr int Q_TERM = 10 * Q_TILE;   // the ten blocks on and below the diagonal
constexpr int F_ROW = TOKENS + 4;     // floats of a row of a 64 x 64 matrix in shared memory

enum Mode { HEAD_DELTA = 0, CHANNEL_DELTA = 1, BONUS = 2 };

template <int KD> struct Rows {  // a matrix of 64 x KD in three terms, in bytes, rows padded so that ldmatrix reads different banks
  static constexpr int ROW = KD * 2 + 16, TERM = TOKENS * ROW, MATRIX = 3 * TERM;
};
// What the first kernel leaves for a (tile, head), in bytes, laid out as the second one wants it in shared memory, so that a bulk copy brings
// a whole part: the matrices (W of the delta rules only), U in runs of the columns of a CTA of the second kernel, Q in blocks, P_last.
template <int KD, bool DELTA> struct Left : Rows<KD> {
  static constexpr int MATRIX = Rows<KD>::MATRIX;
  static constexpr int W = 0, PQ = DELTA ? MATRIX : 0, PK = PQ + MATRIX, Q = PK + MATRIX, P_LAST = Q + 3 * Q_TERM, U = P_LAST + KD * 4;
  __host__ __device__ static size_t bytes(int dv, int cols) { return (size_t)U + (size_t)((dv + cols - 1) / cols) * TOKENS * (cols + 4) * 4; }
};
__host__ __device__ inline int padded_columns(int dv) { return (dv + 31) / 32 * 32; }
// A sequence's tiles lie behind one another from this place on; the places of different sequences do not meet.
__host__ __device__ inline int first_tile(int q_start, int seq) { return q_start / TOKENS + seq; }
inline int places(int n, int num_seqs) { return n / TOKENS + num_seqs + 1; }

struct Params {
  int mode, f32;  // f32: qkv, u and a are float32, else bfloat16
  float* o;
  const void *qkv, *u, *a;  // BONUS: qkv holds the slabs r | k | v, a the decays' products
  long long u_stride;
  int b_col, a_col;
  const float *dt_bias, *a_log, *bonus;  // BONUS: dt_bias is w0
  float* state;                          // [slots][heads][dv][d]
  const int *q_start, *state_slot;
  int n, num_seqs, heads, kq, d, dv;
  float unit_eps;
  int cols;  // value columns of a CTA of the second kernel: 16 or 32
  int vec;   // rows of queries, keys and decays are whole (d = KD) and aligned: a lane's channels come in one load
  int vec_v; // rows of values lie in 16-byte runs
  int pairs; // two read-outs side by side lie on an 8-byte boundary
  int one_wave;            // every (tile, head) has an SM of its own
  int place0, num_places;  // the places that this pass takes; a sequence's state waits in its slot between two passes
  unsigned char* left;     // what the first kernel leaves, from place0 on
  int* error_flag;
};

__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ void split3(float x, bf16& hi, bf16& mid, bf16& lo) {
  hi = __float2bfloat16_rn(x);
  x -= __bfloat162float(hi);
  mid = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(mid));
}
// a b with both operands in three terms
__device__ __forceinline__ void mma6(float (&large)[4], float (&small)[4], const uint32_t (&a)[3][4], uint32_t b00, uint32_t b01, uint32_t b10,
                                     uint32_t b11, uint32_t b20, uint32_t b21) {
  mma16816(small, a[2], b00, b01);
  mma16816(large, a[0], b00, b01);
  mma16816(small, a[0], b20, b21);
  mma16816(small, a[1], b10, b11);
  mma16816(small, a[1], b00, b01);
  mma16816(small, a[0], b10, b11);
}
// N (2 or 4) numbers side by side, aligned to all of them
template <int N> __device__ __forceinline__ void load_run(const float* p, float (&v)[N]) {
  if constexpr (N == 4) { const float4 x = *reinterpret_cast<const float4*>(p); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
  else { const float2 x = *reinterpret_cast<const float2*>(p); v[0] = x.x; v[1] = x.y; }
}
template <int N> __device__ __forceinline__ void load_run(const bf16* p, float (&v)[N]) {
  uint32_t w[N / 2];
  if constexpr (N == 4) { const uint2 x = *reinterpret_cast<const uint2*>(p); w[0] = x.x; w[1] = x.y; }
  else w[0] = *reinterpret_cast<const uint32_t*>(p);
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <int N> __device__ __forceinline__ void store_run(float* p, const float (&v)[N]) {
  if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
// bytes of pair c of row r of a 16 x 16 block
__device__ __forceinline__ int block_at(int r, int c) { return r * 32 + (((c >> 2) ^ ((r >> 2) & 1)) * 16) + (c & 3) * 4; }

// A lower triangular 64 x 64 matrix, value(row, column), in three terms, block by block.
template <int THREADS, typename F> __device__ __forceinline__ void split_blocks(F&& value, unsigned char* dst, int tid) {
  for (int e = tid; e < 10 * 128; e += THREADS) {
    const int b = e >> 7, r = (e >> 3) & 15, pr = e & 7;
    const int rb = b < 1 ? 0 : (b < 3 ? 1 : (b < 6 ? 2 : 3)), cb = b - rb * (rb + 1) / 2;
    const int row = rb * 16 + r, col = cb * 16 + pr * 2;
    uint32_t t[3];
    dli::split3(value(row, col), value(row, col + 1), t[0], t[1], t[2]);
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(dst + s * Q_TERM + b * Q_TILE + block_at(r, pr)) = t[s];
  }
}

// T = (I + A)^-1 for a strictly lower triangular A (rows of F_ROW floats; what lies on and above the diagonal is not read), by all threads of a
// CTA of at least 256 or (OWN_BARRIER) by the first 256, with barriers: the blocks on the diagonal a column a lane, the others block by block away from it,
// T_ba = -T_bb sum_{a <= e < b} A_be T_ea (the sum is kept above the diagonal meanwhile).
template <bool OWN_BARRIER = false> __device__ __forceinline__ void invert_unit_lower(const float* sA, float* sT, int tid) {
  auto sync = [] {
    if (OWN_BARRIER) asm volatile("bar.sync 1, 256;" ::: "memory");
    else __syncthreads();
  };
  const int warp = tid >> 5, lane = tid & 31;
  if (warp < 4) {
    const int b0 = warp * 16;
    if (lane < 16) {
      float x[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        float s = t == lane ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < t; ++j) s = fmaf(-sA[(b0 + t) * F_ROW + b0 + j], x[j], s);
        x[t] = s;
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) sT[(b0 + t) * F_ROW + b0 + lane] = x[t];
    }
  }
  sync();
  for (int away = 1; away < 4; ++away) {  // a thread takes four columns of a row
    const int a = tid >> 6, b = a + away, r = (tid >> 2) & 15, cc = (tid & 3) * 4;
    if (b < 4) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int j = a * 16; j < b * 16; ++j) {
        const float x = sA[(b * 16 + r) * F_ROW + j];
        const float4 y = *reinterpret_cast<const float4*>(sT + j * F_ROW + a * 16 + cc);
        s[0] = fmaf(x, y.x, s[0]); s[1] = fmaf(x, y.y, s[1]); s[2] = fmaf(x, y.z, s[2]); s[3] = fmaf(x, y.w, s[3]);
      }
      *reinterpret_cast<float4*>(sT + (a * 16 + r) * F_ROW + b * 16 + cc) = make_float4(s[0], s[1], s[2], s[3]);
    }
    sync();
    if (b < 4) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float x = sT[(b * 16 + r) * F_ROW + b * 16 + j];
        const float4 y = *reinterpret_cast<const float4*>(sT + (a * 16 + j) * F_ROW + b * 16 + cc);
        s[0] = fmaf(x, y.x, s[0]); s[1] = fmaf(x, y.y, s[1]); s[2] = fmaf(x, y.z, s[2]); s[3] = fmaf(x, y.w, s[3]);
      }
      *reinterpret_cast<float4*>(sT + (b * 16 + r) * F_ROW + a * 16 + cc) = make_float4(-s[0], -s[1], -s[2], -s[3]);
    }
    sync();
  }
}

// ---------------------------------------------------------------- (1) what does not depend on the state

template <typename T, int MODE, int KD> struct Prep {
  static constexpr int THREADS = KD * 4, WARPS = THREADS / 32;
  static constexpr bool DELTA = MODE != BONUS;
  static constexpr int ROW = Rows<KD>::ROW, TERM = Rows<KD>::TERM, MATRIX = Rows<KD>::MATRIX;
  static constexpr int V_TERMS = sizeof(T) == 2 ? 1 : 3, V_ROW = 128 * 2 + 16, V_TERM = TOKENS * V_ROW;
  static constexpr int RAW = 3 * TOKENS * KD * 4;  // k, q, decays as float32
  static constexpr int LATER = DELTA ? 2 * MATRIX + V_TERMS * V_TERM : 0;  // P o K | V | W on its way out
  static constexpr int REGION = 3 * MATRIX > LATER ? 3 * MATRIX : LATER;  // (RAW is smaller than three matrices)
  static constexpr int SQUARE = TOKENS * F_ROW * 4;
  static constexpr int SMEM = REGION + (DELTA ? 3 : 1) * SQUARE + (DELTA ? 3 * Q_TERM : 0) + 8 * KD * 4 + TOKENS * 4;
  static_assert(RAW <= REGION && SMEM <= 227 * 1024, "shared memory");
};

template <typename T, int MODE, int KD>
__global__ void __launch_bounds__(KD * 4, KD == 64 && MODE == BONUS ? 2 : 1) tile_prep_kernel(const Params p) {
  // The walk's CTAs may come from the start on where all tiles have an SM each (their launch then costs nothing: 2 to 3 us of 26 in short steps), otherwise
  // at the end: waiting on SMs that the last wave of tiles leaves free, they slow that wave by 12 us (16 heads of 128, 2,048 tokens: both kernels
  // 220 us with them there from the start, 199 so).
  if (p.one_wave) pdl_launch_dependents();
  pdl_wait();
  using Z = Prep<T, MODE, KD>;
  using L = Left<KD, Prep<T, MODE, KD>::DELTA>;
  constexpr bool DELTA = Z::DELTA;
  constexpr int PER = KD / 32;
  extern __shared__ __align__(128) unsigned char smem[];
  float* sK = reinterpret_cast<float*>(smem);
  float* sQ = sK + TOKENS * KD;
  float* sG = sQ + TOKENS * KD;
  float* sQm = reinterpret_cast<float*>(smem + Z::REGION);
  float* sA = sQm + TOKENS * F_ROW;                              // (DELTA)
  float* sT = sA + TOKENS * F_ROW;                               // (DELTA)
  unsigned char* sTt = smem + Z::REGION + 3 * Z::SQUARE;         // (DELTA)
  float* sB = reinterpret_cast<float*>(smem + Z::REGION + (DELTA ? 3 * Z::SQUARE + 3 * Q_TERM : Z::SQUARE));  // [8][KD]: products of the decays of eight tokens
  float* sBeta = sB + 8 * KD;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, head = blockIdx.y, place = p.place0 + blockIdx.x;

  // ---- which sequence's tile this is: the last one that begins at or in front of this place
  int seq = -1;
  for (int s0 = 0; s0 < p.num_seqs; s0 += Z::THREADS) {
    const int s = s0 + tid;
    seq += __syncthreads_count(s < p.num_seqs && first_tile(p.q_start[s < p.num_seqs ? s : 0], s) <= place);
  }
  if (seq < 0) return;
  const int first = p.q_start[seq] + (place - first_tile(p.q_start[seq], seq)) * TOKENS, len = min(TOKENS, p.q_start[seq + 1] - first);
  if (len <= 0) return;
  const int d = p.d, dv = p.dv, kqh = head / (p.heads / p.kq), dvp = padded_columns(dv);
  unsigned char* left = p.left + ((size_t)blockIdx.x * p.heads + head) * L::bytes(dv, p.cols);
  float* left_u = reinterpret_cast<float*>(left + L::U);
  auto u_at = [&](int r, int col) { return left_u + (col / p.cols) * TOKENS * (p.cols + 4) + r * (p.cols + 4) + col % p.cols; };
  const T* qkv = (const T*)p.qkv;
  const size_t slab = (size_t)p.n * p.heads * d;  // BONUS
  const int width = 2 * p.kq * d + p.heads * dv;

  // ---- queries, keys, decays; the tokens a last tile does not have change nothing: zeros, decays of 1
  for (int i = tid; i < TOKENS * F_ROW; i += Z::THREADS) {
    sQm[i] = 0.f;
    if (DELTA) sA[i] = 0.f;
  }
  // V's rows come now, into the place of T, when they lie in 16-byte runs (p.vec_v): asked for behind the stores of the decays' products
  // they took 5,000 clocks.
  constexpr bool V_AHEAD = DELTA && sizeof(T) == 2;
  if constexpr (V_AHEAD) {
    if (p.vec_v) {
      for (int i = tid; i < TOKENS * (dv / 8); i += Z::THREADS) {
        const int r = i / (dv / 8), part = i % (dv / 8);
        const uint32_t dst = smem_u32(sT) + (r * 128 + part * 8) * 2;
        const T* src = qkv + (size_t)(first + (r < len ? r : 0)) * width + 2 * p.kq * d + head * dv + part * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(r < len ? 16 : 0) : "memory");
      }
    }
  }
  const float rate = MODE == BONUS ? 0.f : expf(p.a_log[head]);
  // A lane has PER channels side by side, which come in one load each where rows are whole and aligned (p.vec).  A warp's eight norms share five
  // rounds of shuffles and one root and division (with a load per number and these per row this part took 16,700 clocks, now 13,900).
  constexpr int ROWS = TOKENS / Z::WARPS, GROUP = 4;  // rows of a warp; those whose loads are under way together
  static_assert(ROWS % GROUP == 0, "rows");
  const int c0 = lane * PER;
  float bias[PER];
#pragma unroll
  for (int m = 0; m < PER; ++m) bias[m] = MODE != HEAD_DELTA && c0 + m < d ? p.dt_bias[head * d + c0 + m] : 0.f;
#pragma unroll 1
  for (int r0 = 0; r0 < ROWS; r0 += GROUP) {
    float qv[GROUP][PER], kv[GROUP][PER], gv[GROUP][PER];
    const int own = warp + (r0 + (lane & (GROUP - 1))) * Z::WARPS;  // the row whose beta this lane makes (all lanes load: a branch would wait for its load)
    T beta = T(0.f);
    if (DELTA) beta = ((const T*)p.u)[(size_t)(first + (own < len ? own : 0)) * p.u_stride + p.b_col + head];
#pragma unroll
    for (int e = 0; e < GROUP; ++e) {
      const int r = warp + (r0 + e) * Z::WARPS;
      const bool ok = r < len;
      const size_t t = first + (ok ? r : 0);
      const T* q = MODE == BONUS ? qkv + t * p.heads * d + head * d : qkv + t * width + kqh * d;
      const T* k = MODE == BONUS ? q + slab : q + p.kq * d;
      const T* a = (const T*)p.a + t * p.heads * d + head * d;
      if (p.vec) {
        load_run<PER>(q + c0, qv[e]);
        load_run<PER>(k + c0, kv[e]);
        if (MODE != HEAD_DELTA) load_run<PER>(a + c0, gv[e]);
      } else {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          const bool in = c0 + m < d;
          qv[e][m] = in ? to_float(q[c0 + m]) : 0.f;
          kv[e][m] = in ? to_float(k[c0 + m]) : 0.f;
          if (MODE != HEAD_DELTA) gv[e][m] = in ? to_float(a[c0 + m]) : 0.f;
        }
      }
      if (MODE == HEAD_DELTA) gv[e][0] = to_float(((const T*)p.u)[t * p.u_stride + p.a_col + head]);
      if (!DELTA) {
        const T* v = qkv + 2 * slab + t * p.heads * d + head * d;
        for (int i = lane; i < (dv + p.cols - 1) / p.cols * p.cols; i += 32) *u_at(r, i) = ok && i < dv ? to_float(v[i]) : 0.f;
      }
    }
    float factor = 0.f;  // lane 8 e + i: row e's factor, of the query (i < 4) or of the key
    if (DELTA) {
      float sum[2 * GROUP];  // eight sums over the lanes: a lane keeps the half of its numbers that its bit names
#pragma unroll
      for (int e = 0; e < GROUP; ++e) {
        sum[2 * e] = sum[2 * e + 1] = 0.f;
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          sum[2 * e] = fmaf(qv[e][m], qv[e][m], sum[2 * e]);
          sum[2 * e + 1] = fmaf(kv[e][m], kv[e][m], sum[2 * e + 1]);
        }
      }
#pragma unroll
      for (int half = 4, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
        const bool upper = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float give = upper ? sum[i] : sum[i + half], keep = upper ? sum[i + half] : sum[i];
          sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
        }
      }
      sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 2);
      sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 1);
      factor = ((lane & 4) ? 1.f : 1.f / sqrtf((float)d)) / sqrtf(sum[0] + p.unit_eps);
      if (lane < GROUP) sBeta[own] = own < len ? 1.f / (1.f + expf(-to_float(beta))) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < GROUP; ++e) {
      const int r = warp + (r0 + e) * Z::WARPS;
      const bool ok = r < len;
      if (MODE == HEAD_DELTA) {
        const float g = expf(-rate * softplus(gv[e][0] + p.dt_bias[head]));
#pragma unroll
        for (int m = 0; m < PER; ++m) gv[e][m] = g;
      } else {
#pragma unroll
        for (int m = 0; m < PER; ++m) gv[e][m] = MODE == BONUS ? expf(-expf(gv[e][m] + bias[m])) : expf(-rate * softplus(gv[e][m] + bias[m]));
      }
      const float fq = DELTA ? __shfl_sync(0xffffffffu, factor, 8 * e) : 1.f, fk = DELTA ? __shfl_sync(0xffffffffu, factor, 8 * e + 4) : 1.f;
#pragma unroll
      for (int m = 0; m < PER; ++m) {  // (0 / sqrt(0 + 0) of a row that is not there must not get through)
        qv[e][m] = ok ? qv[e][m] * fq : 0.f;
        kv[e][m] = ok ? kv[e][m] * fk : 0.f;
        gv[e][m] = ok ? gv[e][m] : 1.f;
      }
      store_run<PER>(sQ + r * KD + c0, qv[e]);
      store_run<PER>(sK + r * KD + c0, kv[e]);
      store_run<PER>(sG + r * KD + c0, gv[e]);
    }
  }
  __syncthreads();

  // ---- the blocks of 16 on the diagonal, on the CUDA cores.  A task is 64 sums over the channels, a lane adds its channels' shares and a
  // warp the lanes'.  Tasks 0..7: the pairs inside eight tokens; 8..15: four tokens of a block's second half with the first half's eight.
  for (int task = warp; task < 16; task += Z::WARPS) {
    const int base = task < 8 ? task * 8 : (task - 8) / 2 * 16, rows = base + 8 + (task & 1) * 4;
    if (base >= len || (task >= 8 && rows >= len)) continue;
    float v[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = 0.f;
#pragma unroll 1
    for (int m = 0; m < PER; ++m) {
      const int c = lane + 32 * m;
      if (task < 8) {
        float k[8], q[8], g[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          k[t] = sK[(base + t) * KD + c];
          q[t] = sQ[(base + t) * KD + c];
          g[t] = sG[(base + t) * KD + c];
        }
        const float own = MODE == BONUS && c < d ? p.bonus[head * d + c] : 1.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float run = k[j];
          v[28 + j * (j + 1) / 2 + j] = fmaf(q[j], run * own, v[28 + j * (j + 1) / 2 + j]);
#pragma unroll
          for (int t = j + 1; t < 8; ++t) {
            if (MODE == BONUS) v[28 + t * (t + 1) / 2 + j] = fmaf(q[t], run, v[28 + t * (t + 1) / 2 + j]);
            run *= g[t];
            if (DELTA) {
              v[28 + t * (t + 1) / 2 + j] = fmaf(q[t], run, v[28 + t * (t + 1) / 2 + j]);
              v[t * (t - 1) / 2 + j] = fmaf(k[t], run, v[t * (t - 1) / 2 + j]);
            }
          }
        }
      } else {
        float kc[8], kr[4], qr[4], run = 1.f;
#pragma unroll
        for (int j = 7; j >= 0; --j) {
          kc[j] = sK[(base + j) * KD + c] * run;
          run *= sG[(base + j) * KD + c];
        }
        run = 1.f;
        if (task & 1) {
#pragma unroll
          for (int t = 0; t < 4; ++t) run *= sG[(base + 8 + t) * KD + c];
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (MODE == BONUS) qr[t] = sQ[(rows + t) * KD + c] * run;
          run *= sG[(rows + t) * KD + c];
          if (DELTA) qr[t] = sQ[(rows + t) * KD + c] * run;
          kr[t] = sK[(rows + t) * KD + c] * run;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (DELTA) v[t * 8 + j] = fmaf(kr[t], kc[j], v[t * 8 + j]);
            v[32 + t * 8 + j] = fmaf(qr[t], kc[j], v[32 + t * 8 + j]);
          }
      }
    }
    // sums over the lanes: a lane keeps the half of its numbers that its bit names; after five rounds it holds two of the 64
#pragma unroll
    for (int half = 32, bit = 16; bit >= 1; half >>= 1, bit >>= 1) {
      const bool upper = (lane & bit) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int at = 2 * lane + i;  // bit 16 chose 32 numbers, bit 8 sixteen, .. bit 1 two
      int t, j;
      bool is_q;
      if (task < 8) {
        is_q = at >= 28;
        int rest = is_q ? at - 28 : at;
        t = is_q ? 0 : 1;
        while (rest >= t + (is_q ? 1 : 0)) { rest -= t + (is_q ? 1 : 0); ++t; }
        j = base + rest;
        t += base;
      } else {
        is_q = at >= 32;
        t = rows + ((at >> 3) & 3);
        j = base + (at & 7);
      }
      if (is_q) sQm[t * F_ROW + j] = v[i];
      else if (DELTA) sA[t * F_ROW + j] = v[i] * sBeta[t];
    }
  }

  // ---- products of decays: a thread per two channels and eight tokens
  const int c = tid % (KD / 2) * 2, grp = tid / (KD / 2), blk = grp >> 1;
  float2 kg[8];
  auto put = [&](unsigned char* matrix, int row, float2 x) {
    uint32_t t[3];
    dli::split3(x.x, x.y, t[0], t[1], t[2]);
    unsigned char* at = matrix + row * Z::ROW + c * 2;
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(at + s * Z::TERM) = t[s];
  };
  {
    auto mul = [](float2 x, float2 y) { return make_float2(x.x * y.x, x.y * y.y); };
    auto at = [&](const float* m, int row) { return *reinterpret_cast<const float2*>(m + row * KD + c); };
    const float2 one = make_float2(1.f, 1.f);
    float2 kk[8], qq[8], gg[8], all = one;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      kk[t] = at(sK, grp * 8 + t);
      qq[t] = at(sQ, grp * 8 + t);
      gg[t] = at(sG, grp * 8 + t);
      all = mul(all, gg[t]);
    }
    *reinterpret_cast<float2*>(sB + grp * KD + c) = all;
    __syncthreads();  // the products are there, and the float32 rows have been read: their place is taken by operands in three terms
    float2 pre[8], b16[4];  // products of the eights in front of each; of the blocks
    pre[0] = one;
#pragma unroll
    for (int g = 1; g < 8; ++g) pre[g] = mul(pre[g - 1], at(sB, g - 1));
#pragma unroll
    for (int g = 0; g < 4; ++g) b16[g] = mul(at(sB, 2 * g), at(sB, 2 * g + 1));
    float2 before = one, behind = one;
#pragma unroll
    for (int g = 0; g < 4; ++g)
      if (g == blk) before = pre[2 * g];
    if (blk <= 2) behind = b16[3];
    if (blk <= 1) behind = mul(b16[2], behind);
    if (blk == 0) behind = mul(b16[1], behind);
    if (grp == 0) *reinterpret_cast<float2*>(left + L::P_LAST + c * 4) = mul(pre[7], at(sB, 7));
    unsigned char* kh = smem;                   // rows of A: blocks 1, 2, 3 from their own starts, block 3 from the tile's middle
    unsigned char* qh = smem + Z::MATRIX;       // rows of Q: the same
    unsigned char* kc = smem + 2 * Z::MATRIX;   // columns: blocks 0 and 2 up to their own ends, blocks 0 and 1 up to the tile's middle
    const int r0 = (grp & 1) * 8;
    float2 run = (grp & 1) ? at(sB, grp - 1) : one;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float2 seen = run;  // BONUS: up to the token in front
      run = mul(run, gg[t]);
      const float2 pqt = DELTA ? run : seen;
      if (blk > 0) {
        if (DELTA) put(kh, (blk - 1) * 16 + r0 + t, mul(kk[t], run));
        put(qh, (blk - 1) * 16 + r0 + t, mul(qq[t], pqt));
      }
      if (blk == 3) {
        if (DELTA) put(kh, 48 + r0 + t, mul(kk[t], mul(run, b16[2])));
        put(qh, 48 + r0 + t, mul(qq[t], mul(pqt, b16[2])));
      }
      put(left + L::PQ, grp * 8 + t, mul(qq[t], mul(pqt, before)));
      kg[t] = mul(kk[t], mul(run, before));
    }
    run = (grp & 1) ? one : at(sB, grp + 1);
#pragma unroll
    for (int t = 7; t >= 0; --t) {
      if (blk == 0) {
        put(kc, r0 + t, mul(kk[t], run));
        put(kc, 32 + r0 + t, mul(kk[t], mul(run, b16[1])));
      } else if (blk == 1) {
        put(kc, 48 + r0 + t, mul(kk[t], run));
      } else if (blk == 2) {
        put(kc, 16 + r0 + t, mul(kk[t], run));
      }
      put(left + L::PK, grp * 8 + t, mul(kk[t], mul(run, behind)));
      run = mul(run, gg[t]);
    }
  }
  __syncthreads();

  if (V_AHEAD) asm volatile("cp.async.wait_all;" ::: "memory");  // (seen by everybody behind the barrier below)
  // ---- the six blocks below the diagonal: (1, 0) and (3, 2) across their common border, (2, 0), (2, 1), (3, 0), (3, 1) across the tile's middle
  const int kcol = (lane & 3) * 2;
  for (int task = warp; task < (DELTA ? 12 : 6); task += Z::WARPS) {
    const int pair = task >> (DELTA ? 1 : 0), is_a = DELTA ? task & 1 : 0;
    const int rb = pair == 0 ? 1 : (pair == 2 || pair == 3 ? 2 : 3), cb = pair == 1 ? 2 : (pair == 0 || pair == 2 || pair == 4 ? 0 : 1);
    if (rb * 16 >= len) continue;
    const int rs = pair == 0 ? 0 : (pair == 1 ? 2 : (pair < 4 ? 1 : 3)), cs = pair == 0 ? 0 : (pair == 1 ? 1 : (cb == 0 ? 2 : 3));
    const uint32_t a_addr = smem_u32(smem + (is_a ? 0 : Z::MATRIX)) + (rs * 16 + (lane & 15)) * Z::ROW + (lane >> 4) * 16;
    const uint32_t b_addr = smem_u32(smem + 2 * Z::MATRIX) + (cs * 16 + (lane & 7) + (lane >> 4) * 8) * Z::ROW + ((lane >> 3) & 1) * 16;
    float large[2][2][4], small[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) large[0][0][e] = large[0][1][e] = large[1][0][e] = large[1][1][e] = small[0][e] = small[1][e] = 0.f;
#pragma unroll
    for (int k16 = 0; k16 < KD / 16; ++k16) {
      uint32_t a[3][4], b[3][4];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        ldsm_x4(a[s], a_addr + s * Z::TERM + k16 * 32);
        ldsm_x4(b[s], b_addr + s * Z::TERM + k16 * 32);
      }
      mma6(large[k16 & 1][0], small[0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
      mma6(large[k16 & 1][1], small[1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
    }
    float* dst = is_a ? sA : sQm;
    const int r_lo = rb * 16 + (lane >> 2), r_hi = r_lo + 8;
    const float f_lo = is_a ? sBeta[r_lo] : 1.f, f_hi = is_a ? sBeta[r_hi] : 1.f;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int col = cb * 16 + nt * 8 + kcol;
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = (small[nt][e] + large[1][nt][e]) + large[0][nt][e];
      *reinterpret_cast<float2*>(dst + r_lo * F_ROW + col) = make_float2(x[0] * f_lo, x[1] * f_lo);
      *reinterpret_cast<float2*>(dst + r_hi * F_ROW + col) = make_float2(x[2] * f_hi, x[3] * f_hi);
    }
  }
  __syncthreads();

  auto q_leaves = [&](auto threads, int id) {  // Q in three terms, block by block
    split_blocks<decltype(threads)::value>([&](int r, int cc) { return sQm[r * F_ROW + cc]; }, left + L::Q, id);
  };
  if constexpr (!DELTA) {
    if (!p.one_wave) pdl_launch_dependents();
    q_leaves(std::integral_constant<int, Z::THREADS>(), tid);
  }
  if constexpr (DELTA) {
    // ---- P o K and V as operands, in the place of the blocks' operands.  With sixteen warps, eight make the inverse, a chain of short steps,
    // while the others see to V and Q (one after the other 14,700 of the 61,300 clocks).
    constexpr bool APART = Z::WARPS == 16;
    constexpr int V_WARPS = APART ? Z::WARPS / 2 : Z::WARPS, V_ROWS = TOKENS / V_WARPS;
    unsigned char* sKg = smem;
    unsigned char* sV = smem + Z::MATRIX;
#pragma unroll
    for (int t = 0; t < 8; ++t) put(sKg, grp * 8 + t, kg[t]);
    if (V_AHEAD && p.vec_v) {
      for (int i = tid; i < TOKENS * (dvp / 8); i += Z::THREADS) {
        const int r = i / (dvp / 8), part = i % (dvp / 8);
        *reinterpret_cast<uint4*>(sV + r * Z::V_ROW + part * 16) = part * 8 < dv ? reinterpret_cast<const uint4*>(sT)[r * 16 + part] : make_uint4(0, 0, 0, 0);
      }
      __syncthreads();  // the place is T's from here on
    }
    if (APART && warp < 8) {
      invert_unit_lower<true>(sA, sT, tid);
    } else {
      const int w0 = APART ? warp - 8 : warp;
      const bool from_rows = !(V_AHEAD && p.vec_v);
      float vv[V_ROWS][4];
#pragma unroll
      for (int e = 0; e < V_ROWS; ++e) {
        const int r = w0 + e * V_WARPS;
        const T* v = qkv + (size_t)(first + (r < len ? r : 0)) * width + 2 * p.kq * d + head * dv;
#pragma unroll
        for (int m = 0; m < 4; ++m) vv[e][m] = from_rows && r < len && lane + 32 * m < dv ? to_float(v[lane + 32 * m]) : 0.f;
      }
      q_leaves(std::integral_constant<int, V_WARPS * 32>(), w0 * 32 + lane);
#pragma unroll
      for (int e = 0; e < V_ROWS; ++e) {
        if (!from_rows) break;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (lane + 32 * m < dvp) {
            unsigned char* at = sV + (w0 + e * V_WARPS) * Z::V_ROW + (lane + 32 * m) * 2;
            if (Z::V_TERMS == 1) {
              *reinterpret_cast<bf16*>(at) = __float2bfloat16_rn(vv[e][m]);
            } else {
              bf16 h, mid, l;
              split3(vv[e][m], h, mid, l);
              *reinterpret_cast<bf16*>(at) = h;
              *reinterpret_cast<bf16*>(at + Z::V_TERM) = mid;
              *reinterpret_cast<bf16*>(at + 2 * Z::V_TERM) = l;
            }
          }
        }
      }
      if (!APART) invert_unit_lower(sA, sT, tid);
    }
    if (APART) __syncthreads();
    split_blocks<Z::THREADS>([&](int r, int cc) { return cc <= r ? sT[r * F_ROW + cc] * sBeta[cc] : 0.f; }, sTt, tid);
    __syncthreads();
    // ---- W = T (P o K) and U = T V: a warp takes sixteen columns and two of the four blocks of rows (0 and 3, or 1 and 2)
    unsigned char* sW = sV + Z::V_TERMS * Z::V_TERM;
    const uint32_t t_addr = smem_u32(sTt) + (lane & 15) * 32 + ((lane >> 4) ^ ((lane >> 2) & 1)) * 16;
    const int w_tasks = KD / 16 * 2, tasks = w_tasks + dvp / 16 * 2;
    auto columns16 = [&](auto is_w_, auto mt0_, auto mt1_, int col0) {
      constexpr bool is_w = decltype(is_w_)::value;
      constexpr int mts[2] = {decltype(mt0_)::value, decltype(mt1_)::value}, row = is_w ? Z::ROW : Z::V_ROW, term = is_w ? Z::TERM : Z::V_TERM;
      constexpr int terms = is_w ? 3 : Z::V_TERMS;
      const uint32_t b_addr = smem_u32(is_w ? sKg : sV) + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * row) + (col0 + (lane >> 4) * 8) * 2;
      float large[2][2][4], small[2][2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) large[i][0][e] = large[i][1][e] = small[i][0][e] = small[i][1][e] = 0.f;
#pragma unroll
      for (int k16 = 0; k16 <= mts[1]; ++k16) {
        uint32_t b[3][4];
#pragma unroll
        for (int s = 0; s < terms; ++s) ldsm_x4_trans(b[s], b_addr + k16 * 16 * row + s * term);
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (k16 <= mts[i]) {
            uint32_t a[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s) ldsm_x4(a[s], t_addr + s * Q_TERM + (mts[i] * (mts[i] + 1) / 2 + k16) * Q_TILE);
            if constexpr (terms == 3) {
              mma6(large[i][0], small[i][0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
              mma6(large[i][1], small[i][1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
            } else {
#pragma unroll
              for (int s = 2; s >= 0; --s) {
                mma16816(s ? small[i][0] : large[i][0], a[s], b[0][0], b[0][1]);
                mma16816(s ? small[i][1] : large[i][1], a[s], b[0][2], b[0][3]);
              }
            }
          }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const int r = mts[i] * 16 + (lane >> 2) + hf * 8, col = col0 + nt * 8 + kcol;
            const float x = large[i][nt][2 * hf] + small[i][nt][2 * hf], y = large[i][nt][2 * hf + 1] + small[i][nt][2 * hf + 1];
            if (is_w) {
              uint32_t t[3];
              dli::split3(x, y, t[0], t[1], t[2]);
#pragma unroll
              for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(sW + s * Z::TERM + r * Z::ROW + col * 2) = t[s];
            } else if (col < (dv + p.cols - 1) / p.cols * p.cols) {
              *reinterpret_cast<float2*>(u_at(r, col)) = make_float2(x, y);
            }
          }
    };
    using std::integral_constant;
    for (int task = warp; task < tasks; task += Z::WARPS) {
      const bool is_w = task < w_tasks;
      const int col0 = (is_w ? task : task - w_tasks) / 2 * 16;
      const integral_constant<bool, true> w;
      const integral_constant<bool, false> v;
      const integral_constant<int, 0> m0;
      const integral_constant<int, 1> m1;
      const integral_constant<int, 2> m2;
      const integral_constant<int, 3> m3;
      if (is_w) {
        if (task & 1) columns16(w, m1, m2, col0); else columns16(w, m0, m3, col0);
      } else {
        if (task & 1) columns16(v, m1, m2, col0); else columns16(v, m0, m3, col0);
      }
    }
    if (!p.one_wave) pdl_launch_dependents();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {  // W leaves in one piece
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(left + L::W), "r"(smem_u32(sW)), "r"(Z::MATRIX) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
}

// ---------------------------------------------------------------- (2) the walk over the tiles

// Tokens first .. last - 1 of a head token after token, for 4 columns a warp from col0 on, from and to the state in memory.  A lane holds every
// 32nd channel.
__device__ __forceinline__ void walk_again(const Params& p, int head, int col0, int first, int last, float* S0) {
  const int lane = threadIdx.x & 31, d = p.d, dv = p.dv, kqh = head / (p.heads / p.kq), width = 2 * p.kq * d + p.heads * dv;
  const size_t slab = (size_t)p.n * p.heads * d;  // BONUS
  auto number = [&](const void* base, size_t i) { return p.f32 ? static_cast<const float*>(base)[i] : to_float(static_cast<const bf16*>(base)[i]); };
  const int c0 = col0 + (threadIdx.x >> 5) * 4;
  if (c0 >= dv) return;
  float S[4][4], bias[4], own[4];
  bool in[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int i = lane + 32 * m;
    in[m] = i < d;
    bias[m] = in[m] && p.mode != HEAD_DELTA ? p.dt_bias[head * d + i] : 0.f;
    own[m] = in[m] && p.mode == BONUS ? p.bonus[head * d + i] : 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) S[c][m] = in[m] && c0 + c < dv ? S0[(size_t)(c0 + c) * d + i] : 0.f;
  }
  const float rate = p.mode == BONUS ? 0.f : expf(p.a_log[head]);
  for (size_t t = first; t < (size_t)last; ++t) {
    const size_t q_at = p.mode == BONUS ? (t * p.heads + head) * d : t * width + kqh * d, k_at = p.mode == BONUS ? q_at + slab : q_at + p.kq * d;
    const size_t v_at = p.mode == BONUS ? q_at + 2 * slab : t * width + 2 * p.kq * d + head * dv;
    float q[4], k[4], g[4], beta = 0.f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int i = lane + 32 * m;
      q[m] = in[m] ? number(p.qkv, q_at + i) : 0.f;
      k[m] = in[m] ? number(p.qkv, k_at + i) : 0.f;
      if (p.mode != HEAD_DELTA) {
        const float a = in[m] ? number(p.a, (t * p.heads + head) * d + i) + bias[m] : 0.f;
        g[m] = p.mode == BONUS ? expf(-expf(a)) : expf(-rate * softplus(a));
      }
    }
    if (p.mode != BONUS) {
      float sq = 0.f, sk = 0.f;
#pragma unroll
      for (int m = 0; m < 4; ++m) { sq = fmaf(q[m], q[m], sq); sk = fmaf(k[m], k[m], sk); }
      const float fq = (1.f / sqrtf((float)d)) / sqrtf(warp_sum(sq) + p.unit_eps), fk = 1.f / sqrtf(warp_sum(sk) + p.unit_eps);
#pragma unroll
      for (int m = 0; m < 4; ++m) { q[m] *= fq; k[m] *= fk; }
      beta = 1.f / (1.f + expf(-number(p.u, t * p.u_stride + p.b_col + head)));
      if (p.mode == HEAD_DELTA) g[0] = g[1] = g[2] = g[3] = expf(-rate * softplus(number(p.u, t * p.u_stride + p.a_col + head) + p.dt_bias[head]));
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float v = c0 + c < dv ? number(p.qkv, v_at + c0 + c) : 0.f;
      float out = 0.f;
      if (p.mode == BONUS) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (in[m]) {  // (0 times an infinity of a number that is not there must not get through)
            const float kv = k[m] * v;
            out = fmaf(q[m], fmaf(own[m], kv, S[c][m]), out);
            S[c][m] = fmaf(g[m], S[c][m], kv);
          }
      } else {
        float sum = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (in[m]) {
            S[c][m] *= g[m];
            sum = fmaf(k[m], S[c][m], sum);
          }
        const float w = beta * (v - warp_sum(sum));
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (in[m]) {
            S[c][m] = fmaf(k[m], w, S[c][m]);
            out = fmaf(q[m], S[c][m], out);
          }
      }
      out = warp_sum(out);
      if (lane == 0 && c0 + c < dv) p.o[t * p.heads * dv + (size_t)head * dv + c0 + c] = out;
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (in[m] && c0 + c < dv) S0[(size_t)(c0 + c) * d + lane + 32 * m] = S[c][m];
}

template <int KD, int COLS> struct Walk {
  static constexpr int THREADS = COLS * 8;  // warps: (block of 16 tokens, 16 of the columns) of the products with S0; (quarter of the channels, 16 columns) of S
  static constexpr int ROW = Rows<KD>::ROW, TERM = Rows<KD>::TERM, MATRIX = Rows<KD>::MATRIX;
  static constexpr int S_TERM = COLS * ROW;
  static constexpr int W_ROW = COLS * 2 + 16, W_TERM = TOKENS * W_ROW;
  static constexpr int U_ROW = COLS + 4, U_BYTES = TOKENS * U_ROW * 4;
  static constexpr int AT_W = 0, AT_PQ = MATRIX, AT_PK = 2 * MATRIX, AT_Q = 3 * MATRIX, AT_P = AT_Q + 3 * Q_TERM, AT_U = AT_P + KD * 4, AT_S = AT_U + U_BYTES,
                       AT_w = AT_S + 3 * S_TERM, AT_BAR = AT_w + 3 * W_TERM, SMEM = AT_BAR + 32;
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

// The tokens of a sequence's tiles that lie in this pass; false: none.
__device__ __forceinline__ bool tokens_of_pass(const Params& p, int seq, int& first, int& last) {
  const int begin = p.q_start[seq], end = p.q_start[seq + 1], at = first_tile(begin, seq);
  first = begin + max(0, p.place0 - at) * TOKENS;
  last = min(end, begin + (p.place0 + p.num_places - at) * TOKENS);
  return first < last;
}
// .. and where in p.left they begin
__device__ __forceinline__ int place_of_pass(const Params& p, int seq) { return max(0, first_tile(p.q_start[seq], seq) - p.place0); }

constexpr unsigned WAIT_LIMIT = 1u << 24;
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, int bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void expect_bytes(uint32_t bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool copies_arrived(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
// Waits for copies, WAIT_LIMIT polls at most; false: they did not arrive, here or for another thread, and *error_flag says so.
__device__ __forceinline__ bool wait_copies(uint32_t bar, uint32_t parity, volatile int* failed, int* error_flag) {
  for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
    if (copies_arrived(bar, parity)) return true;
    if ((i & 1023) == 1023 && *failed) return false;
  }
  *failed = 1;
  atomicExch(error_flag, 1);
  return false;
}
// For a CTA that gives up: the copies that it still has under way (`issued` so far on this barrier) may not land in shared memory that is no longer its own.
__device__ __forceinline__ void wait_for_last(uint32_t bar, int issued) {
  for (unsigned i = 0; issued > 0 && i < WAIT_LIMIT; ++i)
    if (copies_arrived(bar, (issued - 1) & 1)) return;
}

template <int KD, int COLS, bool DELTA>
__global__ void __launch_bounds__(COLS * 8, 1) tile_walk_kernel(const __grid_constant__ Params p) {
  pdl_launch_dependents();
  pdl_wait();
  using Z = Walk<KD, COLS>;
  using L = Left<KD, DELTA>;
  constexpr int SLICE = KD / 4, NT = SLICE / 8;  // channels of S of a warp, in accumulators of 16 x 8
  extern __shared__ __align__(128) unsigned char smem[];
  const int seq = p.num_seqs - 1 - blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * COLS;  // (single tokens come first in a step: long portions start first)
  int first, last;
  if (!tokens_of_pass(p, seq, first, last)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mt = warp & 3, half = warp >> 2;
  const int d = p.d, dv = p.dv, inner = p.heads * dv;
  const size_t bytes = L::bytes(dv, COLS);
  const unsigned char* left = p.left + ((size_t)place_of_pass(p, seq) * p.heads + head) * bytes;
  const float* sU = reinterpret_cast<const float*>(smem + Z::AT_U);
  const float* sP = reinterpret_cast<const float*>(smem + Z::AT_P);
  const uint32_t bar_before = smem_u32(smem + Z::AT_BAR), bar_behind = bar_before + 8;
  volatile int* failed = reinterpret_cast<volatile int*>(smem + Z::AT_BAR + 16);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_before));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_behind));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *failed = 0;
  }
  __syncthreads();
  auto load_before = [&](const unsigned char* src) {  // what the products with S0 need
    if (tid == 0) {
      expect_bytes(bar_before, (DELTA ? 2 : 1) * Z::MATRIX + Z::U_BYTES);
      if (DELTA) bulk_load(smem_u32(smem + Z::AT_W), src + L::W, Z::MATRIX, bar_before);
      bulk_load(smem_u32(smem + Z::AT_PQ), src + L::PQ, Z::MATRIX, bar_before);
      bulk_load(smem_u32(smem + Z::AT_U), src + L::U + (size_t)blockIdx.x * Z::U_BYTES, Z::U_BYTES, bar_before);
    }
  };
  auto load_behind = [&](const unsigned char* src) {  // what comes behind them: (P_last / P) o K, Q and P_last lie behind one another
    if (tid == 0) {
      expect_bytes(bar_behind, Z::MATRIX + 3 * Q_TERM + KD * 4);
      bulk_load(smem_u32(smem + Z::AT_PK), src + L::PK, Z::MATRIX + 3 * Q_TERM + KD * 4, bar_behind);
    }
  };
  load_before(left);

  // ---- S: rows = value columns of this warp's half, columns = its quarter of the channels
  const int kcol = (lane & 3) * 2, c_lo = half * 16 + (lane >> 2), slice0 = mt * SLICE;
  float S[NT][4];
  float* S0 = p.state + ((size_t)p.state_slot[seq] * p.heads + head) * dv * d;
  auto each = [&](auto&& fn) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = col0 + c_lo + (e >> 1) * 8, i = slice0 + j * 8 + kcol + (e & 1);
        fn(S[j][e], col < dv && i < d, (size_t)col * d + i);
      }
  };
  each([&](float& x, bool in, size_t at) { x = in ? S0[at] : 0.f; });

  const uint32_t row_a = (mt * 16 + (lane & 15)) * Z::ROW + (lane >> 4) * 16;
  const uint32_t w_addr = smem_u32(smem + Z::AT_W) + row_a, pq_addr = smem_u32(smem + Z::AT_PQ) + row_a;
  const uint32_t s_addr = smem_u32(smem + Z::AT_S) + (half * 16 + (lane & 7) + (lane >> 4) * 8) * Z::ROW + ((lane >> 3) & 1) * 16;
  const uint32_t q_addr = smem_u32(smem + Z::AT_Q) + (lane & 15) * 32 + ((lane >> 4) ^ ((lane >> 2) & 1)) * 16;
  const uint32_t wb_addr = smem_u32(smem + Z::AT_w) + ((lane & 7) + ((lane >> 3) & 1) * 8) * Z::W_ROW + (half * 16 + (lane >> 4) * 8) * 2;  // k = token, n = column
  const uint32_t wa_addr = smem_u32(smem + Z::AT_w) + ((lane & 7) + (lane >> 4) * 8) * Z::W_ROW + (half * 16 + ((lane >> 3) & 1) * 8) * 2;  // m = column, k = token
  const uint32_t pk_addr = smem_u32(smem + Z::AT_PK) + ((lane & 7) + ((lane >> 3) & 1) * 8) * Z::ROW + (slice0 + (lane >> 4) * 8) * 2;

  float finite = 0.f;  // 0 while every result was finite, NaN from the first one on that was not
  bool ok = true;      // every copy has arrived
  int before = 1, behind = 0;  // loads so far
  uint32_t parity = 0;
  for (int base = first; base < last; base += TOKENS, parity ^= 1) {
    const int len = min(TOKENS, last - base);
    const bool active = mt * 16 < len;
    // ---- S0 in three terms, for everybody
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t t[3];
        dli::split3(S[j][2 * hf], S[j][2 * hf + 1], t[0], t[1], t[2]);
#pragma unroll
        for (int s = 0; s < 3; ++s)
          *reinterpret_cast<uint32_t*>(smem + Z::AT_S + s * Z::S_TERM + (c_lo + hf * 8) * Z::ROW + (slice0 + j * 8 + kcol) * 2) = t[s];
      }
    __syncthreads();  // S0 is there; the operands behind (of the tile before) have been read
    if (ok) {         // (the thread that asks for copies asks again on a barrier only when it has seen the last ones arrive)
      load_behind(left);
      ++behind;
    }
    ok = wait_copies(bar_before, parity, failed, p.error_flag) && ok;
    float O[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) O[0][e] = O[1][e] = 0.f;
    if (active) {
      float yl[2][2][4], ys[2][4], ol[2][2][4], os[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        yl[0][0][e] = yl[0][1][e] = yl[1][0][e] = yl[1][1][e] = ys[0][e] = ys[1][e] = 0.f;
        ol[0][0][e] = ol[0][1][e] = ol[1][0][e] = ol[1][1][e] = os[0][e] = os[1][e] = 0.f;
      }
#pragma unroll
      for (int k16 = 0; k16 < KD / 16; ++k16) {
        uint32_t b[3][4], a[3][4], q[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          ldsm_x4(b[s], s_addr + s * Z::S_TERM + k16 * 32);
          if (DELTA) ldsm_x4(a[s], w_addr + s * Z::TERM + k16 * 32);
          ldsm_x4(q[s], pq_addr + s * Z::TERM + k16 * 32);
        }
        if (DELTA) {
          mma6(yl[k16 & 1][0], ys[0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
          mma6(yl[k16 & 1][1], ys[1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
        }
        mma6(ol[k16 & 1][0], os[0], q, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
        mma6(ol[k16 & 1][1], os[1], q, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) O[nt][e] = (os[nt][e] + ol[1][nt][e]) + ol[0][nt][e];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int r = mt * 16 + (lane >> 2) + hf * 8, col = half * 16 + nt * 8 + kcol;
          float2 w = *reinterpret_cast<const float2*>(sU + r * Z::U_ROW + col);
          if (DELTA) {
            w.x -= (ys[nt][2 * hf] + yl[1][nt][2 * hf]) + yl[0][nt][2 * hf];
            w.y -= (ys[nt][2 * hf + 1] + yl[1][nt][2 * hf + 1]) + yl[0][nt][2 * hf + 1];
          }
          uint32_t t[3];
          dli::split3(w.x, w.y, t[0], t[1], t[2]);
#pragma unroll
          for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(smem + Z::AT_w + s * Z::W_TERM + r * Z::W_ROW + col * 2) = t[s];
        }
      }
    }
    __syncthreads();  // w is there; S0 and the operands in front have been read
    if (*failed) break;
    left += (size_t)p.heads * bytes;
    if (base + TOKENS < last) { load_before(left); ++before; }
    ok = wait_copies(bar_behind, parity, failed, p.error_flag);
    // ---- the read-outs
    if (active) {
      float ql[2][4], qs[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) ql[0][e] = ql[1][e] = qs[0][e] = qs[1][e] = 0.f;
      for (int k16 = 0; k16 <= mt; ++k16) {
        uint32_t a[3][4], b[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          ldsm_x4(a[s], q_addr + s * Q_TERM + (mt * (mt + 1) / 2 + k16) * Q_TILE);
          ldsm_x4_trans(b[s], wb_addr + s * Z::W_TERM + k16 * 16 * Z::W_ROW);
        }
        mma6(ql[0], qs[0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
        mma6(ql[1], qs[1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int r = mt * 16 + (lane >> 2) + hf * 8, col = col0 + half * 16 + nt * 8 + kcol;
          if (r < len) {
            float* dst = p.o + (size_t)(base + r) * inner + (size_t)head * dv + col;
            const float x = O[nt][2 * hf] + (qs[nt][2 * hf] + ql[nt][2 * hf]), y = O[nt][2 * hf + 1] + (qs[nt][2 * hf + 1] + ql[nt][2 * hf + 1]);
            finite = fmaf(x, 0.f, fmaf(y, 0.f, finite));
            if (p.pairs) {
              if (col < dv) *reinterpret_cast<float2*>(dst) = make_float2(x, y);
            } else {
              if (col < dv) dst[0] = x;
              if (col + 1 < dv) dst[1] = y;
            }
          }
        }
    }
    // ---- the state at the tile's end
    float dl[NT][4], ds[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) dl[j][e] = ds[j][e] = 0.f;
#pragma unroll
    for (int k16 = 0; k16 < TOKENS / 16; ++k16) {
      if (k16 * 16 < len) {
        uint32_t a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) ldsm_x4_trans(a[s], wa_addr + s * Z::W_TERM + k16 * 16 * Z::W_ROW);
#pragma unroll
        for (int jp = 0; jp < NT / 2; ++jp) {
          uint32_t b[3][4];
#pragma unroll
          for (int s = 0; s < 3; ++s) ldsm_x4_trans(b[s], pk_addr + s * Z::TERM + k16 * 16 * Z::ROW + jp * 32);
          mma6(dl[2 * jp], ds[2 * jp], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
          mma6(dl[2 * jp + 1], ds[2 * jp + 1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const float2 g = *reinterpret_cast<const float2*>(sP + slice0 + j * 8 + kcol);
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf((e & 1) ? g.y : g.x, S[j][e], ds[j][e] + dl[j][e]);
    }
  }
  each([&](float& x, bool, size_t) { finite = fmaf(x, 0.f, finite); });
  if (__syncthreads_or(!ok || finite != 0.f)) {  // (also: nobody writes a read-out behind this)
    if (!__syncthreads_or(!ok)) {
      walk_again(p, head, col0, first, last, S0);
    } else if (tid == 0) {  // (the state stays as it was)
      wait_for_last(bar_before, before);
      wait_for_last(bar_behind, behind);
    }
    return;
  }
  each([&](float& x, bool in, size_t at) { if (in) S0[at] = x; });
}

// ---------------------------------------------------------------- a decay per head, bfloat16
// Here queries and keys are bfloat16 numbers times a float32 factor of their token (the unit vector's, the decays'), so they go into products as they
// came, in one term, and the factors move to the other operand's rows or to the sums: A and Q are plain products of bfloat16 rows times
// factors, W = T diag(P fk) K, (P fq) o (Q S0), S = P_last S + ((P_last / P) fk o w)^T K.  222 mma.sync a tile and warp instead of 318, 87 KB of operands
// instead of 157, and no operand is split in the first kernel but T and Q.  Decays between two tokens are powers of differences of sums of
// logarithms, the sums in double and kept as two floats.  Measured against the general kernels, 16 heads of 128, one prompt of 2,048 tokens: 202 -> 135 us (300
// tokens 36, 64 tokens 25; 32 heads 233); errors against 64 bits o 1.8e-7 and S 1.3e-7 (the tiles of sixteen tokens on the CUDA cores 3.2e-7 and 3.5e-7).
template <int KD> struct HeadLeft {
  static constexpr int TERM = Rows<KD>::TERM, MATRIX = Rows<KD>::MATRIX;
  static constexpr int FACTORS = 576;  // bytes: P fq [64] | (P_last / P) fk [64] | P_last, rounded up
  static constexpr int W = 0, QB = MATRIX, KB = QB + TERM, Q = KB + TERM, F = Q + 3 * Q_TERM, U = F + FACTORS;
  __host__ __device__ static size_t bytes(int dv, int cols) { return (size_t)U + (size_t)((dv + cols - 1) / cols) * TOKENS * (cols + 4) * 4; }
};

template <int KD> struct HeadPrep {
  static constexpr int THREADS = 256, WARPS = 8;
  static constexpr int ROW = Rows<KD>::ROW, TERM = Rows<KD>::TERM, V_ROW = 128 * 2 + 16, SQUARE = TOKENS * F_ROW * 4;
  static constexpr int SECOND = TERM > TOKENS * V_ROW ? TERM : TOKENS * V_ROW;  // queries, then values
  static constexpr int AT_Q = TERM, AT_A = AT_Q + SECOND, AT_QM = AT_A + SQUARE, AT_T = AT_QM + SQUARE, AT_TT = AT_T + SQUARE, AT_F = AT_TT + 3 * Q_TERM,
                       SMEM = AT_F + 8 * TOKENS * 4;
  static_assert(3 * Q_TERM <= SQUARE && 2 * (SMEM + 1024) <= 227 * 1024, "two CTAs an SM");
};

template <int KD>
__global__ void __launch_bounds__(256, 2) head_prep_kernel(const Params p, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  using Z = HeadPrep<KD>;
  using L = HeadLeft<KD>;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* sK = smem;
  unsigned char* sQ = smem + Z::AT_Q;
  float* sA = reinterpret_cast<float*>(smem + Z::AT_A);
  float* sQm = reinterpret_cast<float*>(smem + Z::AT_QM);
  float* sT = reinterpret_cast<float*>(smem + Z::AT_T);
  unsigned char* sTt = smem + Z::AT_TT;       // T diag(beta), in three terms
  unsigned char* sTk = smem + Z::AT_QM;       // T diag(beta P fk), in the place of Q
  float* fk = reinterpret_cast<float*>(smem + Z::AT_F);  // per token: factor of the key, of the query, beta, sums of log decays (two terms), P, P_last / P, a scratch
  float *fq = fk + TOKENS, *beta = fq + TOKENS, *lh = beta + TOKENS, *lm = lh + TOKENS, *up = lm + TOKENS, *behind = up + TOKENS, *raw = behind + TOKENS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, head = blockIdx.y, place = p.place0 + blockIdx.x;
  int seq = -1;
  for (int s0 = 0; s0 < p.num_seqs; s0 += Z::THREADS) {
    const int s = s0 + tid;
    seq += __syncthreads_count(s < p.num_seqs && first_tile(p.q_start[s < p.num_seqs ? s : 0], s) <= place);
  }
  if (seq < 0) return;
  const int first = p.q_start[seq] + (place - first_tile(p.q_start[seq], seq)) * TOKENS, len = min(TOKENS, p.q_start[seq + 1] - first);
  if (len <= 0) return;
  const int d = p.d, dv = p.dv, kqh = head / (p.heads / p.kq), dvp = padded_columns(dv), width = 2 * p.kq * d + p.heads * dv;
  unsigned char* left = p.left + ((size_t)blockIdx.x * p.heads + head) * L::bytes(dv, p.cols);
  float* left_u = reinterpret_cast<float*>(left + L::U);
  float* left_f = reinterpret_cast<float*>(left + L::F);
  const bf16* rows = (const bf16*)p.qkv + (size_t)first * width;
  const bf16* u = (const bf16*)p.u + (size_t)first * p.u_stride + head;

  auto load_rows = [&](unsigned char* dst, const bf16* src, int size, int row, int columns) {  // 64 rows of `columns` numbers, zeros where there is nothing
    if (vec) {
      const int runs = columns >> 3;
      for (int e = tid; e < TOKENS * runs; e += Z::THREADS) {
        const int r = e / runs, c = e - r * runs;
        const bool ok = r < len && c * 8 < size;
        cp_async16(smem_u32(dst + r * row + c * 16), ok ? src + (size_t)r * width + c * 8 : src, ok ? 16 : 0);
      }
    } else {
      for (int e = tid; e < TOKENS * columns; e += Z::THREADS) {
        const int r = e / columns, c = e - r * columns;
        *reinterpret_cast<bf16*>(dst + r * row + c * 2) = r < len && c < size ? src[(size_t)r * width + c] : __float2bfloat16_rn(0.f);
      }
    }
    cp_async_commit();
  };
  load_rows(sQ, rows + kqh * d, d, Z::ROW, KD);
  load_rows(sK, rows + (p.kq + kqh) * d, d, Z::ROW, KD);
  if (tid < TOKENS) {
    const bool ok = tid < len;
    beta[tid] = ok ? 1.f / (1.f + expf(-to_float(u[(size_t)(ok ? tid : 0) * p.u_stride + p.b_col]))) : 0.f;
    raw[tid] = ok ? -expf(p.a_log[head]) * softplus(to_float(u[(size_t)(ok ? tid : 0) * p.u_stride + p.a_col]) + p.dt_bias[head]) : 0.f;
  }
  cp_async_wait<0>();
  __syncthreads();

  // ---- the tokens' factors: four threads a row for the unit vectors, a warp for the sums of log decays
  {
    const int r = tid >> 2, part = tid & 3;
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int c = 0; c < KD / 8; c += 4) {
      float q[8], k[8];
      load8(reinterpret_cast<const bf16*>(sQ + r * Z::ROW + (c + part) * 16), q);
      load8(reinterpret_cast<const bf16*>(sK + r * Z::ROW + (c + part) * 16), k);
#pragma unroll
      for (int i = 0; i < 8; ++i) { sq = fmaf(q[i], q[i], sq); sk = fmaf(k[i], k[i], sk); }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) { sq += __shfl_xor_sync(0xffffffffu, sq, o); sk += __shfl_xor_sync(0xffffffffu, sk, o); }
    if (part == 0) {
      fk[r] = r < len ? 1.f / sqrtf(sk + p.unit_eps) : 0.f;
      fq[r] = r < len ? (1.f / sqrtf((float)d)) / sqrtf(sq + p.unit_eps) : 0.f;
    }
  }
  if (warp == 0) {
    double l[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) l[k] = (double)log_decay(raw[2 * lane + k], -1e4f);
    l[1] += l[0];
    double incl = l[1];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double other = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += other;
    }
    const double before = incl - l[1], end = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double lt = before + l[k], l2 = lt * 1.4426950408889634074;
      const float hi = (float)l2;
      lh[2 * lane + k] = hi;
      lm[2 * lane + k] = (float)(l2 - (double)hi);
      up[2 * lane + k] = expf((float)lt);
      behind[2 * lane + k] = expf((float)(end - lt));
    }
    if (lane == 0) left_f[2 * TOKENS] = expf((float)end);
  }
  for (int e = tid; e < TOKENS * (KD / 8); e += Z::THREADS) {  // queries and keys as the second kernel wants them
    const int at = e / (KD / 8) * Z::ROW + e % (KD / 8) * 16;
    *reinterpret_cast<uint4*>(left + L::QB + at) = *reinterpret_cast<const uint4*>(sQ + at);
    *reinterpret_cast<uint4*>(left + L::KB + at) = *reinterpret_cast<const uint4*>(sK + at);
  }
  __syncthreads();
  if (tid < TOKENS) {
    left_f[tid] = up[tid] * fq[tid];
    left_f[TOKENS + tid] = behind[tid] * fk[tid];
  }

  // ---- A and Q: a warp takes sixteen rows of one of them
  const int kcol = (lane & 3) * 2;
  {
    const int is_q = warp >> 2, mt = warp & 3;
    if (mt * 16 < len) {
      float sum[2][8][4];  // the two halves of k apart: an mma.sync addition cuts off, a plain one rounds
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[0][j][e] = sum[1][j][e] = 0.f;
      const uint32_t a_addr = smem_u32(is_q ? sQ : sK) + (mt * 16 + (lane & 15)) * Z::ROW + (lane >> 4) * 16;
      const uint32_t b_addr = smem_u32(sK) + ((lane & 7) + (lane >> 4) * 8) * Z::ROW + ((lane >> 3) & 1) * 16;
#pragma unroll
      for (int k16 = 0; k16 < KD / 16; ++k16) {
        uint32_t a[4];
        ldsm_x4(a, a_addr + k16 * 32);
#pragma unroll
        for (int jp = 0; jp < 4; ++jp)
          if (jp <= mt) {
            uint32_t b[4];
            ldsm_x4(b, b_addr + jp * 16 * Z::ROW + k16 * 32);
            mma16816(sum[k16 & 1][2 * jp], a, b[0], b[1]);
            mma16816(sum[k16 & 1][2 * jp + 1], a, b[2], b[3]);
          }
      }
      float* dst = is_q ? sQm : sA;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int r = mt * 16 + (lane >> 2) + hf * 8;
        const float h = lh[r], m = lm[r], f = is_q ? fq[r] : fk[r] * beta[r];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < 2 * (mt + 1)) {
            const int col = j * 8 + kcol;
            const float2 ch = *reinterpret_cast<const float2*>(lh + col), cm = *reinterpret_cast<const float2*>(lm + col), cf = *reinterpret_cast<const float2*>(fk + col);
            const float x = (sum[0][j][2 * hf] + sum[1][j][2 * hf]) * f * cf.x * ex2((h - ch.x) + (m - cm.x));
            const float y = (sum[0][j][2 * hf + 1] + sum[1][j][2 * hf + 1]) * f * cf.y * ex2((h - ch.y) + (m - cm.y));
            *reinterpret_cast<float2*>(dst + r * F_ROW + col) = make_float2(col <= r ? x : 0.f, col + 1 <= r ? y : 0.f);
          }
      }
    } else {
      float* dst = is_q ? sQm : sA;
      for (int e = lane; e < 16 * (mt + 1) * 16; e += 32) dst[(mt * 16 + e / ((mt + 1) * 16)) * F_ROW + e % ((mt + 1) * 16)] = 0.f;
    }
  }
  __syncthreads();
  load_rows(sQ, rows + 2 * p.kq * d + head * dv, dv, Z::V_ROW, dvp);  // the values, in the queries' place
  split_blocks<Z::THREADS>([&](int r, int c) { return c <= r ? sQm[r * F_ROW + c] : 0.f; }, left + L::Q, tid);
  invert_unit_lower(sA, sT, tid);
  split_blocks<Z::THREADS>([&](int r, int c) { return c <= r ? sT[r * F_ROW + c] * beta[c] : 0.f; }, sTt, tid);
  split_blocks<Z::THREADS>([&](int r, int c) { return c <= r ? sT[r * F_ROW + c] * (beta[c] * up[c] * fk[c]) : 0.f; }, sTk, tid);
  cp_async_wait<0>();
  __syncthreads();

  // ---- W = T diag(beta P fk) K and U = T diag(beta) V: a warp takes sixteen columns and two of the four blocks of rows (0 and 3, or 1 and 2)
  const int w_tasks = KD / 16 * 2, tasks = w_tasks + dvp / 16 * 2;
  auto columns16 = [&](auto mt0_, auto mt1_, bool is_w, int col0) {
    constexpr int mts[2] = {decltype(mt0_)::value, decltype(mt1_)::value};
    const int row = is_w ? Z::ROW : Z::V_ROW;
    const uint32_t b_addr = smem_u32(is_w ? sK : sQ) + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * row) + (col0 + (lane >> 4) * 8) * 2;
    const uint32_t t_addr = smem_u32(is_w ? sTk : sTt) + (lane & 15) * 32 + ((lane >> 4) ^ ((lane >> 2) & 1)) * 16;
    float large[2][2][4], small[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) large[i][0][e] = large[i][1][e] = small[i][0][e] = small[i][1][e] = 0.f;
#pragma unroll
    for (int k16 = 0; k16 <= mts[1]; ++k16) {
      uint32_t b[4];
      ldsm_x4_trans(b, b_addr + k16 * 16 * row);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (k16 <= mts[i]) {
#pragma unroll
          for (int s = 2; s >= 0; --s) {
            uint32_t a[4];
            ldsm_x4(a, t_addr + s * Q_TERM + (mts[i] * (mts[i] + 1) / 2 + k16) * Q_TILE);
            mma16816(s ? small[i][0] : large[i][0], a, b[0], b[1]);
            mma16816(s ? small[i][1] : large[i][1], a, b[2], b[3]);
          }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int r = mts[i] * 16 + (lane >> 2) + hf * 8, col = col0 + nt * 8 + kcol;
          const float x = large[i][nt][2 * hf] + small[i][nt][2 * hf], y = large[i][nt][2 * hf + 1] + small[i][nt][2 * hf + 1];
          if (is_w) {
            uint32_t t[3];
            dli::split3(x, y, t[0], t[1], t[2]);
#pragma unroll
            for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(left + L::W + s * Z::TERM + r * Z::ROW + col * 2) = t[s];
          } else if (col < (dv + p.cols - 1) / p.cols * p.cols) {
            *reinterpret_cast<float2*>(left_u + (col / p.cols) * TOKENS * (p.cols + 4) + r * (p.cols + 4) + col % p.cols) = make_float2(x, y);
          }
        }
  };
  for (int task = warp; task < tasks; task += Z::WARPS) {
    const bool is_w = task < w_tasks;
    const int col0 = (is_w ? task : task - w_tasks) / 2 * 16;
    if (task & 1) columns16(std::integral_constant<int, 1>(), std::integral_constant<int, 2>(), is_w, col0);
    else columns16(std::integral_constant<int, 0>(), std::integral_constant<int, 3>(), is_w, col0);
  }
}

template <int KD, int COLS> struct HeadWalk {
  static constexpr int THREADS = COLS * 8;  // warps as in the walk above
  static constexpr int ROW = Rows<KD>::ROW, TERM = Rows<KD>::TERM, MATRIX = Rows<KD>::MATRIX;
  static constexpr int S_TERM = COLS * ROW, W_ROW = COLS * 2 + 16, W_TERM = TOKENS * W_ROW, U_ROW = COLS + 4, U_BYTES = TOKENS * U_ROW * 4;
  static constexpr int BEFORE = MATRIX + TERM, BEHIND = TERM + 3 * Q_TERM + HeadLeft<KD>::FACTORS;  // bytes: W and Q rows; K rows, Q, factors
  static constexpr int AT_W = 0, AT_QB = MATRIX, AT_KB = BEFORE, AT_Q = AT_KB + TERM, AT_F = AT_Q + 3 * Q_TERM, AT_U = AT_F + HeadLeft<KD>::FACTORS,
                       AT_S = AT_U + U_BYTES, AT_w = AT_S + 3 * S_TERM, AT_BAR = AT_w + 6 * W_TERM, SMEM = AT_BAR + 32;
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

template <int KD, int COLS>
__global__ void __launch_bounds__(COLS * 8, 1) head_walk_kernel(const __grid_constant__ Params p) {
  pdl_launch_dependents();
  pdl_wait();
  using Z = HeadWalk<KD, COLS>;
  using L = HeadLeft<KD>;
  constexpr int SLICE = KD / 4, NT = SLICE / 8;
  extern __shared__ __align__(128) unsigned char smem[];
  const int seq = p.num_seqs - 1 - blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * COLS;
  int first, last;
  if (!tokens_of_pass(p, seq, first, last)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mt = warp & 3, half = warp >> 2;
  const int d = p.d, dv = p.dv, inner = p.heads * dv;
  const size_t bytes = L::bytes(dv, COLS);
  const unsigned char* left = p.left + ((size_t)place_of_pass(p, seq) * p.heads + head) * bytes;
  const float* sU = reinterpret_cast<const float*>(smem + Z::AT_U);
  const float* sF = reinterpret_cast<const float*>(smem + Z::AT_F);
  const uint32_t bar_before = smem_u32(smem + Z::AT_BAR), bar_behind = bar_before + 8;
  volatile int* failed = reinterpret_cast<volatile int*>(smem + Z::AT_BAR + 16);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_before));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_behind));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *failed = 0;
  }
  __syncthreads();
  auto load_before = [&](const unsigned char* src) {
    if (tid == 0) {
      expect_bytes(bar_before, Z::BEFORE + Z::U_BYTES);
      bulk_load(smem_u32(smem + Z::AT_W), src + L::W, Z::BEFORE, bar_before);
      bulk_load(smem_u32(smem + Z::AT_U), src + L::U + (size_t)blockIdx.x * Z::U_BYTES, Z::U_BYTES, bar_before);
    }
  };
  auto load_behind = [&](const unsigned char* src) {
    if (tid == 0) {
      expect_bytes(bar_behind, Z::BEHIND);
      bulk_load(smem_u32(smem + Z::AT_KB), src + L::KB, Z::BEHIND, bar_behind);
    }
  };
  load_before(left);

  // ---- S: rows = value columns of this warp's half, columns = its quarter of the channels
  const int kcol = (lane & 3) * 2, c_lo = half * 16 + (lane >> 2), slice0 = mt * SLICE;
  float S[NT][4];
  float* S0 = p.state + ((size_t)p.state_slot[seq] * p.heads + head) * dv * d;
  auto each = [&](auto&& fn) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = col0 + c_lo + (e >> 1) * 8, i = slice0 + j * 8 + kcol + (e & 1);
        fn(S[j][e], col < dv && i < d, (size_t)col * d + i);
      }
  };
  each([&](float& x, bool in, size_t at) { x = in ? S0[at] : 0.f; });

  const uint32_t row_a = (mt * 16 + (lane & 15)) * Z::ROW + (lane >> 4) * 16;
  const uint32_t w_addr = smem_u32(smem + Z::AT_W) + row_a, qb_addr = smem_u32(smem + Z::AT_QB) + row_a;
  const uint32_t s_addr = smem_u32(smem + Z::AT_S) + (half * 16 + (lane & 7) + (lane >> 4) * 8) * Z::ROW + ((lane >> 3) & 1) * 16;
  const uint32_t q_addr = smem_u32(smem + Z::AT_Q) + (lane & 15) * 32 + ((lane >> 4) ^ ((lane >> 2) & 1)) * 16;
  const uint32_t wb_addr = smem_u32(smem + Z::AT_w) + ((lane & 7) + ((lane >> 3) & 1) * 8) * Z::W_ROW + (half * 16 + (lane >> 4) * 8) * 2;
  const uint32_t wa_addr = smem_u32(smem + Z::AT_w) + 3 * Z::W_TERM + ((lane & 7) + (lane >> 4) * 8) * Z::W_ROW + (half * 16 + ((lane >> 3) & 1) * 8) * 2;  // with the factors
  const uint32_t kb_addr = smem_u32(smem + Z::AT_KB) + ((lane & 7) + ((lane >> 3) & 1) * 8) * Z::ROW + (slice0 + (lane >> 4) * 8) * 2;

  float finite = 0.f;  // 0 while every result was finite, NaN from the first one on that was not
  bool ok = true;      // every copy has arrived
  int before = 1, behind = 0;  // loads so far
  uint32_t parity = 0;
  for (int base = first; base < last; base += TOKENS, parity ^= 1) {
    const int len = min(TOKENS, last - base);
    const bool active = mt * 16 < len;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t t[3];
        dli::split3(S[j][2 * hf], S[j][2 * hf + 1], t[0], t[1], t[2]);
#pragma unroll
        for (int s = 0; s < 3; ++s)
          *reinterpret_cast<uint32_t*>(smem + Z::AT_S + s * Z::S_TERM + (c_lo + hf * 8) * Z::ROW + (slice0 + j * 8 + kcol) * 2) = t[s];
      }
    __syncthreads();  // S0 is there; the operands behind (of the tile before) have been read
    if (ok) {         // (the thread that asks for copies asks again on a barrier only when it has seen the last ones arrive)
      load_behind(left);
      ++behind;
    }
    ok = wait_copies(bar_before, parity, failed, p.error_flag) && ok;
    float O[2][4], w[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) O[0][e] = O[1][e] = w[0][e] = w[1][e] = 0.f;
    if (active) {
      float yl[2][2][4], ys[2][4], ol[2][2][4], os[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        yl[0][0][e] = yl[0][1][e] = yl[1][0][e] = yl[1][1][e] = ys[0][e] = ys[1][e] = 0.f;
        ol[0][0][e] = ol[0][1][e] = ol[1][0][e] = ol[1][1][e] = os[0][e] = os[1][e] = 0.f;
      }
#pragma unroll
      for (int k16 = 0; k16 < KD / 16; ++k16) {
        uint32_t b[3][4], a[3][4], q[4];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          ldsm_x4(b[s], s_addr + s * Z::S_TERM + k16 * 32);
          ldsm_x4(a[s], w_addr + s * Z::TERM + k16 * 32);
        }
        ldsm_x4(q, qb_addr + k16 * 32);
        mma6(yl[k16 & 1][0], ys[0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
        mma6(yl[k16 & 1][1], ys[1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          mma16816(s ? os[0] : ol[k16 & 1][0], q, b[s][0], b[s][1]);
          mma16816(s ? os[1] : ol[k16 & 1][1], q, b[s][2], b[s][3]);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          O[nt][e] = (os[nt][e] + ol[1][nt][e]) + ol[0][nt][e];
          w[nt][e] = sU[(mt * 16 + (lane >> 2) + (e >> 1) * 8) * Z::U_ROW + half * 16 + nt * 8 + kcol + (e & 1)] - ((ys[nt][e] + yl[1][nt][e]) + yl[0][nt][e]);
        }
      }
    }
    ok = wait_copies(bar_behind, parity, failed, p.error_flag) && ok;
    if (active) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int r = mt * 16 + (lane >> 2) + hf * 8, col = half * 16 + nt * 8 + kcol;
          const float f = sF[TOKENS + r];
          uint32_t t[3], g[3];
          dli::split3(w[nt][2 * hf], w[nt][2 * hf + 1], t[0], t[1], t[2]);
          dli::split3(w[nt][2 * hf] * f, w[nt][2 * hf + 1] * f, g[0], g[1], g[2]);
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            *reinterpret_cast<uint32_t*>(smem + Z::AT_w + s * Z::W_TERM + r * Z::W_ROW + col * 2) = t[s];
            *reinterpret_cast<uint32_t*>(smem + Z::AT_w + (3 + s) * Z::W_TERM + r * Z::W_ROW + col * 2) = g[s];
          }
        }
    }
    __syncthreads();  // w is there; S0 and the operands in front have been read
    if (*failed) break;
    left += (size_t)p.heads * bytes;
    if (base + TOKENS < last) { load_before(left); ++before; }
    // ---- the read-outs
    if (active) {
      float ql[2][4], qs[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) ql[0][e] = ql[1][e] = qs[0][e] = qs[1][e] = 0.f;
      for (int k16 = 0; k16 <= mt; ++k16) {
        uint32_t a[3][4], b[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          ldsm_x4(a[s], q_addr + s * Q_TERM + (mt * (mt + 1) / 2 + k16) * Q_TILE);
          ldsm_x4_trans(b[s], wb_addr + s * Z::W_TERM + k16 * 16 * Z::W_ROW);
        }
        mma6(ql[0], qs[0], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
        mma6(ql[1], qs[1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int r = mt * 16 + (lane >> 2) + hf * 8, col = col0 + half * 16 + nt * 8 + kcol;
          if (r < len) {
            const float f = sF[r];
            float* dst = p.o + (size_t)(base + r) * inner + (size_t)head * dv + col;
            const float x = fmaf(f, O[nt][2 * hf], qs[nt][2 * hf] + ql[nt][2 * hf]), y = fmaf(f, O[nt][2 * hf + 1], qs[nt][2 * hf + 1] + ql[nt][2 * hf + 1]);
            finite = fmaf(x, 0.f, fmaf(y, 0.f, finite));
            if (p.pairs) {
              if (col < dv) *reinterpret_cast<float2*>(dst) = make_float2(x, y);
            } else {
              if (col < dv) dst[0] = x;
              if (col + 1 < dv) dst[1] = y;
            }
          }
        }
    }
    // ---- the state at the tile's end
    float dl[NT][4], ds[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) dl[j][e] = ds[j][e] = 0.f;
#pragma unroll
    for (int k16 = 0; k16 < TOKENS / 16; ++k16) {
      if (k16 * 16 < len) {
        uint32_t a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) ldsm_x4_trans(a[s], wa_addr + s * Z::W_TERM + k16 * 16 * Z::W_ROW);
#pragma unroll
        for (int jp = 0; jp < NT / 2; ++jp) {
          uint32_t b[4];
          ldsm_x4_trans(b, kb_addr + k16 * 16 * Z::ROW + jp * 32);
#pragma unroll
          for (int s = 2; s >= 0; --s) {
            mma16816(s ? ds[2 * jp] : dl[2 * jp], a[s], b[0], b[1]);
            mma16816(s ? ds[2 * jp + 1] : dl[2 * jp + 1], a[s], b[2], b[3]);
          }
        }
      }
    }
    const float g = sF[2 * TOKENS];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(g, S[j][e], ds[j][e] + dl[j][e]);
  }
  each([&](float& x, bool, size_t) { finite = fmaf(x, 0.f, finite); });
  if (__syncthreads_or(!ok || finite != 0.f)) {  // (also: nobody writes a read-out behind this)
    if (!__syncthreads_or(!ok)) {
      walk_again(p, head, col0, first, last, S0);
    } else if (tid == 0) {  // (the state stays as it was)
      wait_for_last(bar_before, before);
      wait_for_last(bar_behind, behind);
    }
    return;
  }
  each([&](float& x, bool in, size_t at) { if (in) S0[at] = x; });
}

template <typename K> cudaError_t allow(K kernel, int smem, OncePerDevice& done) {
  if (done.here()) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) done.here() = true;
  return e;
}

int* error_flag_device = nullptr;
int* error_flag_host = nullptr;

// Value columns of a CTA of the second kernel: 16 while that leaves every CTA an SM of its own (a tile takes 3.7 us instead of 4.9 with 32), else 32
// (half the copies of the operands).
inline int columns(int heads, int num_seqs, int dv) { return (long long)heads * num_seqs * ((dv + 15) / 16) <= sm_count() ? 16 : 32; }

template <int KD, int COLS, bool DELTA> cudaError_t launch_walk(const Params& p, cudaStream_t stream) {
  using Z = Walk<KD, COLS>;
  static OncePerDevice done;
  const cudaError_t e = allow(tile_walk_kernel<KD, COLS, DELTA>, Z::SMEM, done);
  if (e != cudaSuccess) return e;
  return launch_pdl((tile_walk_kernel<KD, COLS, DELTA>), dim3((p.dv + COLS - 1) / COLS, p.heads, p.num_seqs), dim3(Z::THREADS), (size_t)Z::SMEM, stream, 1, p);
}

template <typename T, int MODE, int KD> int launch(const Params& params, cudaStream_t stream) {
  using Z = Prep<T, MODE, KD>;
  constexpr int PER = KD / 32, RUN = PER * sizeof(T);
  Params p = params;
  const int width = MODE == BONUS ? p.d : 2 * p.kq * p.d + p.heads * p.dv;  // (BONUS: every row of every head begins at a multiple of d numbers)
  p.vec = p.d == KD && width % PER == 0 && (((uintptr_t)p.qkv | (MODE == HEAD_DELTA ? 0 : (uintptr_t)p.a)) & (RUN - 1)) == 0;
  p.vec_v = width % 8 == 0 && (2 * p.kq * p.d) % 8 == 0 && p.dv % 8 == 0 && ((uintptr_t)p.qkv & 15) == 0;
  static OncePerDevice prep;
  cudaError_t e = allow(tile_prep_kernel<T, MODE, KD>, Z::SMEM, prep);
  if (e == cudaSuccess) e = launch_pdl((tile_prep_kernel<T, MODE, KD>), dim3(p.num_places, p.heads), dim3(Z::THREADS), (size_t)Z::SMEM, stream, 1, p);
  if (e == cudaSuccess) e = p.cols == 16 ? launch_walk<KD, 16, MODE != BONUS>(p, stream) : launch_walk<KD, 32, MODE != BONUS>(p, stream);
  return (int)e;
}
template <int KD, int COLS> cudaError_t launch_head_walk(const Params& p, cudaStream_t stream) {
  using Z = HeadWalk<KD, COLS>;
  static OncePerDevice done;
  const cudaError_t e = allow(head_walk_kernel<KD, COLS>, Z::SMEM, done);
  if (e != cudaSuccess) return e;
  return launch_pdl((head_walk_kernel<KD, COLS>), dim3((p.dv + COLS - 1) / COLS, p.heads, p.num_seqs), dim3(Z::THREADS), (size_t)Z::SMEM, stream, 1, p);
}
template <int KD> int launch_head(const Params& p, cudaStream_t stream) {
  using Z = HeadPrep<KD>;
  static OncePerDevice done;
  cudaError_t e = allow(head_prep_kernel<KD>, Z::SMEM, done);
  const int width = 2 * p.kq * p.d + p.heads * p.dv, vec = width % 8 == 0 && p.d % 8 == 0 && p.dv % 8 == 0 && ((uintptr_t)p.qkv & 15) == 0;  // 16-byte runs
  if (e == cudaSuccess) e = launch_pdl((head_prep_kernel<KD>), dim3(p.num_places, p.heads), dim3(Z::THREADS), (size_t)Z::SMEM, stream, 1, p, vec);
  if (e == cudaSuccess) e = p.cols == 16 ? launch_head_walk<KD, 16>(p, stream) : launch_head_walk<KD, 32>(p, stream);
  return (int)e;
}

template <typename T, int MODE> int launch_sized(const Params& p, cudaStream_t stream) {
  return p.d <= 64 ? launch<T, MODE, 64>(p, stream) : launch<T, MODE, 128>(p, stream);
}
template <typename T> int launch_mode(int mode, const Params& p, cudaStream_t stream) {
  if constexpr (sizeof(T) == 2) {
    if (mode == HEAD_DELTA) return p.d <= 64 ? launch_head<64>(p, stream) : launch_head<128>(p, stream);
  } else {
    if (mode == HEAD_DELTA) return launch_sized<T, HEAD_DELTA>(p, stream);
  }
  if (mode == CHANNEL_DELTA) return launch_sized<T, CHANNEL_DELTA>(p, stream);
  return launch_sized<T, BONUS>(p, stream);
}

}  // namespace

// Places of a step of n tokens in num_seqs sequences, and the bytes of scratch that a place takes with all heads.  A step whose places do not fit
// the caller's scratch goes in several passes, one call for each.
DLI_EXPORT int dli_recurrence_tiles_places(int n, int num_seqs) { return places(n, num_seqs); }
DLI_EXPORT long long dli_recurrence_tiles_place_bytes(int mode, int num_seqs, int heads, int d, int dv, int dtype) {
  const int cols = columns(heads, num_seqs, dv);
  size_t each;
  if (mode == HEAD_DELTA && dtype != DLI_F32) each = d <= 64 ? HeadLeft<64>::bytes(dv, cols) : HeadLeft<128>::bytes(dv, cols);
  else if (mode == BONUS) each = d <= 64 ? Left<64, false>::bytes(dv, cols) : Left<128, false>::bytes(dv, cols);
  else each = d <= 64 ? Left<64, true>::bytes(dv, cols) : Left<128, true>::bytes(dv, cols);
  return (long long)(each * heads);
}

// mode 0: gated delta rule (qkv, u with b_col and a_col, dt_bias and a_log per head); 1: a decay per channel (a [n][heads d], dt_bias [heads d]);
// 2: bonus (qkv: the slabs r | k | v, a: the decays' products, dt_bias: w0, bonus [heads][d]; kq = heads, dv = d).  Takes the tiles at places
// place0 .. place0 + num_places - 1; scratch has room for num_places.
DLI_EXPORT int dli_recurrence_tiles(int mode, float* o, const void* qkv, const void* u, long long u_stride, int b_col, int a_col, const void* a,
                                    const float* dt_bias, const float* a_log, const float* bonus, float* state, const int* q_start,
                                    const int* state_slot, void* scratch, int place0, int num_places, int n, int num_seqs, int heads, int kq, int d, int dv,
                                    float unit_eps, int dtype, cudaStream_t stream) {
  if (num_seqs == 0 || n == 0) return 0;
  if (mode < 0 || mode > 2 || heads < 1 || heads > 65535 || kq < 1 || heads % kq || d < 1 || d > 128 || dv < 1 || dv > 128 || num_seqs > 65535 || !scratch || place0 < 0 || num_places < 1 ||
      ((uintptr_t)scratch & 15) || (mode == BONUS && (dv != d || kq != heads || !bonus)))
    return DLI_ERR_UNSUPPORTED;
  if (!error_flag_host) {
    if (cudaHostAlloc((void**)&error_flag_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return (int)cudaGetLastError();
    *error_flag_host = 0;
    if (cudaHostGetDevicePointer((void**)&error_flag_device, error_flag_host, 0) != cudaSuccess) return (int)cudaGetLastError();
  }
  Params p;
  p.place0 = place0; p.num_places = num_places; p.one_wave = (long long)num_places * heads <= sm_count();
  p.mode = mode; p.f32 = dtype == DLI_F32;
  p.o = o; p.qkv = qkv; p.u = u; p.a = a; p.u_stride = u_stride; p.b_col = b_col; p.a_col = a_col; p.dt_bias = dt_bias; p.a_log = a_log; p.bonus = bonus;
  p.state = state; p.q_start = q_start; p.state_slot = state_slot; p.n = n; p.num_seqs = num_seqs; p.heads = heads; p.kq = kq; p.d = d; p.dv = dv;
  p.unit_eps = unit_eps; p.vec = p.vec_v = 0; p.pairs = dv % 2 == 0 && ((uintptr_t)o & 7) == 0; p.cols = columns(heads, num_seqs, dv); p.left = (unsigned char*)scratch; p.error_flag = error_flag_device;
  return dtype == DLI_F32 ? launch_mode<float>(mode, p, stream) : launch_mode<bf16>(mode, p, stream);
}

// 0, or 1 once a wait for copies has run out (since the library was loaded or the code was last cleared).
DLI_EXPORT int dli_recurrence_tiles_error() { return error_flag_host ? *error_flag_host : 0; }
DLI_EXPORT int dli_recurrence_tiles_clear_error() { if (error_flag_host) *error_flag_host = 0; return 0; }
