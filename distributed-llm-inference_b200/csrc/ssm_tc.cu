// The selective scan (ssm.cu says what is computed) for prompt portions in bfloat16: tiles of 64 tokens in closed form on the tensor
// cores.  Inside a tile that starts from S0 (kept transposed: P x N), with l_t the sum of the log decays -exp(A_log) dt up to t,
//   y_t = exp(l_t) S0 C_t + sum_{j <= t} exp(l_t - l_j) dt_j (C_t . B_j) x_j + D x_t,
//   S   = exp(l_last) S0 + sum_j exp(l_last - l_j) dt_j x_j B_j^T.
//
// x, B and C are bfloat16 as the convolution left them; step sizes, decays, weights, the state and every sum are float32, and nothing
// float32 is rounded on its way into a product (mma_split.cuh: three bfloat16 terms).  The sums of log decays are taken in double and
// kept as two floats, so that a difference of two of them is as exact as a token-by-token product of the decays.
//
// A CTA owns 64 columns p of one head of one sequence, a warp 16 of them: S of those columns stays in the warp's registers as the
// accumulator of mma.sync m16n8k16 over all tiles, and its layout there is that of the B operand of C S^T.  The weighted scores
// exp(l_t - l_j) dt_j (C_t . B_j) are made once per tile, a quarter by each warp, and shared as float32.  Tokens arrive by cp.async
// a tile ahead.
//
// A few long sequences leave most of the GPU idle, because a sequence's tiles follow one another.  They are cut into segments, in two
// launches: the first walks segment 0 (whose state is known) and computes what every later segment but the last adds to a state from
// zero, without read-outs; the second starts every later segment from exp(sum of its log decays) S + what was added, segment
// after segment, and walks them side by side.  A segment without read-outs costs 0.45 of one with, so segment 0 is that much shorter.
//
// A masked weight is 0, and 0 times an infinity or a NaN is a NaN; an infinity in three terms is one too.  So a CTA looks at what it
// computed: where a read-out or the state is not finite, it walks its columns again token after token (walk_again), and infinities and
// NaNs appear where ssm.cu has them.  Looking costs a multiply-add for each result.
//
// What bounds it: the latency of a warp's instructions (ncu, one prompt of 1,024 tokens, a CTA an SM: 3,500 warp instructions a tile and
// warp, an instruction every 4.3 cycles, tensor pipe active 26 %); registers and shared memory hold two CTAs an SM.  Measured, us, against
// the walk of ssm.cu (64 heads, P 64, N 128): prompts of 666, 1,000 and 1,335 tokens 772 -> 165, one of 4,096 1,409 -> 215, one
// of 600 214 -> 51; 128 heads, one of 2,048 880 -> 204; 32 heads, N 64, one of 2,048 490 -> 48.  The errors of y and S against 64 bits
// are the walk's or smaller (4,096 tokens: 1.7e-7 and 1.7e-7, the walk 2.1e-7 and 2.2e-7): a sum of mma.sync cuts off where a plain
// addition rounds, so long sums are kept apart and added by the CUDA cores.
#include "common.cuh"
#include "mma_split.cuh"

using namespace dli;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int TOKENS = 64;  // of a tile
constexpr int COLS = 64;    // columns p of a CTA
constexpr int WARPS = 4;
constexpr int X_ROW = COLS * 2 + 16;  // bytes of a staged row, padded so that ldmatrix reads different banks
constexpr int W_TILE = 16 * 32;       // bytes of a term of 16 x 16 weighted scores (two 16-byte halves a row, exchanged in rows 4..7 and 12..15)
constexpr int W_TERM = 10 * W_TILE;   // the ten 16 x 16 blocks on and below the diagonal
constexpr float LOG_FLOOR = -1e4f;    // a log decay below this is 0 as a decay, and its sums stay finite
constexpr double LOG2E = 1.4426950408889634074;

struct Params {
  float* y;
  const bf16* xbc;        // [n][heads P + 2 groups N]: x | B | C
  const bf16* u;          // dt_raw: column dt_col + head
  long long u_stride;
  int dt_col;
  const float *dt_bias, *A_log, *D;
  float* state;           // [slots][heads][P][N]
  const int *q_start, *state_slot;
  int num_seqs, heads, P, N, groups;
  int segments;           // of a sequence; with more than one:
  float* part;            // [seqs][segments - 1][heads][P][N]: the state behind segment 0, then what each segment adds
  float* part_log;        // [seqs][segments - 1][heads]: the sum of its log decays
};

template <int NK> struct Shape {  // NK: the state size in steps of 16
  static constexpr int N_ROW = NK * 32 + 16;
  static constexpr int BC_TILE = TOKENS * N_ROW, X_TILE = TOKENS * X_ROW;
  static constexpr int STAGE = 2 * BC_TILE + X_TILE;
  static constexpr int TABLE = 5 * TOKENS + 4;  // floats: l in log2 units (two terms) | exp(l) | dt | exp(l_last - l) dt | exp(l_last)
  static constexpr int SMEM = 2 * STAGE + 3 * W_TERM + 2 * TABLE * 4;
};

__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// Token range of segment `seg` of a sequence of `len` tokens, in tiles: segment 0 has what the others' even shares leave.
__device__ __forceinline__ void segment_tiles(int tiles, int segments, int seg, int& from, int& to) {
  if (segments == 1) { from = 0; to = tiles; return; }
  const int rest = segments - 1, share = (20 * tiles + 20 * rest + 8) / (20 * rest + 9);  // tiles / (rest + 0.45), rounded up
  const int head = max(1, tiles - share * rest);
  from = seg == 0 ? 0 : min(tiles, head + (seg - 1) * share);
  to = min(tiles, head + seg * share);
}

// The scan of a CTA's columns token after token: from the state `from` in front of token t_from, with read-outs of tokens t_emit .. t_end - 1, the
// state behind them to `to` (or null).  A warp takes sixteen columns, four at a time; a lane holds every 32nd number of them.
__device__ __forceinline__ void walk_again(const Params& p, int head, int col0, const float* from, int t_from, int t_emit, int t_end, float* to) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = p.N, P = p.P, inner = p.heads * P, width = inner + 2 * p.groups * N;
  const float A = expf(p.A_log[head]), bias = p.dt_bias[head], Dh = p.D[head];
  const int g = head / (p.heads / p.groups);
  for (int c0 = col0 + warp * 16; c0 < min(P, col0 + warp * 16 + 16); c0 += 4) {  // (P is a multiple of 8)
    float S[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m) S[c][m] = lane + 32 * m < N ? from[(size_t)(c0 + c) * N + lane + 32 * m] : 0.f;
    for (int t = t_from; t < t_end; ++t) {
      const bf16* row = p.xbc + (size_t)t * width;
      const float dt = softplus(to_float(p.u[(size_t)t * p.u_stride + p.dt_col + head]) + bias), decay = expf(-A * dt);
      float B[4], C[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const bool in = lane + 32 * m < N;
        B[m] = in ? to_float(row[inner + g * N + lane + 32 * m]) : 0.f;
        C[m] = in ? to_float(row[inner + (p.groups + g) * N + lane + 32 * m]) : 0.f;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float x = to_float(row[head * P + c0 + c]), dtx = dt * x;
        float sum = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (lane + 32 * m < N) {  // (0 times an infinity of a number that is not there must not get through)
            S[c][m] = fmaf(decay, S[c][m], B[m] * dtx);
            sum = fmaf(S[c][m], C[m], sum);
          }
        sum = warp_sum(sum);
        if (t >= t_emit && lane == 0) p.y[(size_t)t * inner + head * P + c0 + c] = fmaf(Dh, x, sum);
      }
    }
    if (to) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (lane + 32 * m < N) to[(size_t)(c0 + c) * N + lane + 32 * m] = S[c][m];
    }
  }
}

// SECOND: the second of the two launches over segments.
template <int NK, bool SECOND>
__global__ void __launch_bounds__(WARPS * 32, 2) ssm_chunk_kernel(const __grid_constant__ Params p) {
  pdl_launch_dependents();
  pdl_wait();
  using Z = Shape<NK>;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* sW = smem + 2 * Z::STAGE;
  float* tables = reinterpret_cast<float*>(sW + 3 * W_TERM);
  const int launched = p.segments > 1 ? p.segments - 1 : 1;
  const int z = blockIdx.z / launched, seq = p.num_seqs - 1 - z;  // single tokens come first in a step: the long portions start first
  const int seg = blockIdx.z - z * launched + (SECOND ? 1 : 0), head = blockIdx.y;
  const int first = p.q_start[seq], last = p.q_start[seq + 1];
  int from, to;
  segment_tiles((last - first + TOKENS - 1) / TOKENS, p.segments, seg, from, to);
  const int t0 = first + from * TOKENS, t1 = min(last, first + to * TOKENS);
  if (t1 <= t0) return;
  const bool emit = SECOND || seg == 0;   // with read-outs
  if (!emit && t1 == last) return;        // nothing starts behind the last segment
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, P = p.P, inner = p.heads * P, width = inner + 2 * p.groups * N;
  const int g = head / (p.heads / p.groups), col0 = blockIdx.x * COLS;
  const bf16* xsrc = p.xbc + head * P + col0;
  const bf16* bsrc = p.xbc + inner + g * N;

  auto load_tile = [&](int stage, int base) {
    unsigned char* sC = smem + stage * Z::STAGE;
    unsigned char* sB = sC + Z::BC_TILE;
    unsigned char* sX = sB + Z::BC_TILE;
    constexpr int RUNS = NK * 2, STEP = WARPS * 32 / RUNS;  // a thread keeps its 16 bytes of a row and walks down the rows
    {
      const int r0 = tid / RUNS, c = tid - r0 * RUNS;
      const bool in = c * 8 < N;
      const bf16* src = bsrc + (size_t)(base + r0) * width + c * 8;
      uint32_t dst = smem_u32(sB + r0 * Z::N_ROW + c * 16);
#pragma unroll
      for (int i = 0; i < TOKENS / STEP; ++i) {
        const bool ok = in && base + r0 + i * STEP < t1;
        const bf16* from = ok ? src : bsrc;
        cp_async16(dst, from, ok ? 16 : 0);
        cp_async16(dst - Z::BC_TILE, from + (size_t)p.groups * N, ok ? 16 : 0);
        src += (size_t)STEP * width;
        dst += STEP * Z::N_ROW;
      }
    }
    {
      constexpr int XR = COLS / 8, XS = WARPS * 32 / XR;
      const int r0 = tid / XR, c = tid - r0 * XR;
      const bool in = col0 + c * 8 < P;
      const bf16* src = xsrc + (size_t)(base + r0) * width + c * 8;
      uint32_t dst = smem_u32(sX + r0 * X_ROW + c * 16);
#pragma unroll
      for (int i = 0; i < TOKENS / XS; ++i) {
        const bool ok = in && base + r0 + i * XS < t1;
        cp_async16(dst, ok ? src : p.xbc, ok ? 16 : 0);
        src += (size_t)XS * width;
        dst += XS * X_ROW;
      }
    }
    cp_async_commit();
  };
  // step sizes and decays of a tile, by one warp: two tokens a lane
  const float A = expf(p.A_log[head]), bias = p.dt_bias[head], Dh = p.D[head];
  double total = 0.0;  // log decays so far (of the warp that makes the tables)
  float raw[2];
  auto load_dt = [&](int base) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = base + 2 * lane + k;
      raw[k] = t < t1 ? to_float(p.u[(size_t)t * p.u_stride + p.dt_col + head]) : 0.f;
    }
  };
  auto make_table = [&](float* tab, int base) {
    float dt[2];
    double l[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bool ok = base + 2 * lane + k < t1;
      dt[k] = ok ? softplus(raw[k] + bias) : 0.f;
      l[k] = ok ? (double)log_decay(-A * dt[k], LOG_FLOOR) : 0.0;
    }
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
      const double lt = before + l[k], l2 = lt * LOG2E;
      const float hi = (float)l2;
      const int i = 2 * lane + k;
      tab[i] = hi;
      tab[TOKENS + i] = (float)(l2 - (double)hi);
      tab[2 * TOKENS + i] = expf((float)lt);
      tab[3 * TOKENS + i] = dt[k];
      tab[4 * TOKENS + i] = expf((float)(end - lt)) * dt[k];
    }
    if (lane == 0) tab[5 * TOKENS] = expf((float)end);
    total += end;
  };

  load_tile(0, t0);
  if (warp == 0) {
    load_dt(t0);
    make_table(tables, t0);
    load_dt(t0 + TOKENS);
  }

  // ---- the state: rows = this warp's columns p, columns = n, in accumulators of 16 x 8
  const int row_lo = col0 + warp * 16 + (lane >> 2), row_hi = row_lo + 8, kcol = (lane & 3) * 2;
  const size_t block = (size_t)P * N;
  float S[2 * NK][4];
  auto each = [&](auto&& fn) {  // fn(accumulator j, elements e and e + 1, offset in a [P][N] block) for the pairs that exist (N is even)
#pragma unroll
    for (int j = 0; j < 2 * NK; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int col = e ? row_hi : row_lo, i = j * 8 + kcol;
        if (col < P && i < N) fn(j, e, (size_t)col * N + i);
      }
  };
  auto pbase = [&](int slot) { return (((size_t)seq * launched + slot) * p.heads + head); };
  float* slot_state = p.state + ((size_t)p.state_slot[seq] * p.heads + head) * block;
#pragma unroll
  for (int j = 0; j < 2 * NK; ++j) S[j][0] = S[j][1] = S[j][2] = S[j][3] = 0.f;
  if (emit) {
    const float* src = SECOND ? p.part + pbase(0) * block : slot_state;
    each([&](int j, int e, size_t at) {
      const float2 v = *reinterpret_cast<const float2*>(src + at);
      S[j][e] = v.x; S[j][e + 1] = v.y;
    });
    if (SECOND) {
      for (int s = 1; s < seg; ++s) {
        const float keep = expf(p.part_log[pbase(s)]);
        const float* add = p.part + pbase(s) * block;
        each([&](int j, int e, size_t at) {
          const float2 v = *reinterpret_cast<const float2*>(add + at);
          S[j][e] = fmaf(keep, S[j][e], v.x); S[j][e + 1] = fmaf(keep, S[j][e + 1], v.y);
        });
      }
    }
  }

  float finite = 0.f;  // 0 while every result was finite, NaN from the first one on that was not
  int stage = 0;
  for (int base = t0; base < t1; base += TOKENS, stage ^= 1) {
    const int len = min(TOKENS, t1 - base);
    const bool more = base + TOKENS < t1;
    cp_async_wait<0>();
    __syncthreads();  // this tile and its table have arrived; everybody is done with the tile before, its table and its scores
    if (more) load_tile(stage ^ 1, base + TOKENS);
    const unsigned char* sC = smem + stage * Z::STAGE;
    const unsigned char* sB = sC + Z::BC_TILE;
    const unsigned char* sX = sB + Z::BC_TILE;
    const float* tab = tables + stage * Z::TABLE;

    if (emit) {
      const uint32_t c_addr = smem_u32(sC) + (lane & 15) * Z::N_ROW + (lane >> 4) * 16;
      // ---- this warp's sixteen rows of the weighted scores
      if (warp * 16 < len) {
        float G[8][4], G1[8][4];  // the two halves of k apart: an mma.sync addition cuts off, a plain one rounds
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) G[j][e] = G1[j][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
          float (&sum)[8][4] = kk < NK / 2 ? G : G1;
          uint32_t a[4];
          ldsm_x4(a, c_addr + warp * 16 * Z::N_ROW + kk * 32);
#pragma unroll
          for (int jp = 0; jp < 4; ++jp) {
            if (jp <= warp) {
              uint32_t b[4];
              ldsm_x4(b, smem_u32(sB) + (jp * 16 + (lane & 7) + (lane >> 4) * 8) * Z::N_ROW + (kk * 16 + ((lane >> 3) & 1) * 8) * 2);
              mma16816(sum[2 * jp], a, b[0], b[1]);
              mma16816(sum[2 * jp + 1], a, b[2], b[3]);
            }
          }
        }
        const int r_lo = warp * 16 + (lane >> 2), r_hi = r_lo + 8;
        const float h_lo = tab[r_lo], m_lo = tab[TOKENS + r_lo], h_hi = tab[r_hi], m_hi = tab[TOKENS + r_hi];
        unsigned char* dst = sW + warp * (warp + 1) / 2 * W_TILE + (lane >> 2) * 32 + (lane & 3) * 4;
        const int swap = ((lane >> 4) & 1) * 16;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (j < 2 * (warp + 1)) {
            float v[4];
            const float2 h = *reinterpret_cast<const float2*>(tab + j * 8 + kcol), m = *reinterpret_cast<const float2*>(tab + TOKENS + j * 8 + kcol);
            const float2 d = *reinterpret_cast<const float2*>(tab + 3 * TOKENS + j * 8 + kcol);
            v[0] = (G[j][0] + G1[j][0]) * (ex2((h_lo - h.x) + (m_lo - m.x)) * d.x);
            v[1] = (G[j][1] + G1[j][1]) * (ex2((h_lo - h.y) + (m_lo - m.y)) * d.y);
            v[2] = (G[j][2] + G1[j][2]) * (ex2((h_hi - h.x) + (m_hi - m.x)) * d.x);
            v[3] = (G[j][3] + G1[j][3]) * (ex2((h_hi - h.y) + (m_hi - m.y)) * d.y);
            if (j >= 2 * warp) {  // the block on the diagonal
              const int tok = j * 8 + kcol;
              if (tok > r_lo) v[0] = 0.f;
              if (tok + 1 > r_lo) v[1] = 0.f;
              if (tok > r_hi) v[2] = 0.f;
              if (tok + 1 > r_hi) v[3] = 0.f;
            }
            uint32_t lo[3], hi[3];
            split3(v[0], v[1], lo[0], lo[1], lo[2]);
            split3(v[2], v[3], hi[0], hi[1], hi[2]);
            unsigned char* at = dst + (j >> 1) * W_TILE + (((j & 1) * 16) ^ swap);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
              *reinterpret_cast<uint32_t*>(at + s * W_TERM) = lo[s];
              *reinterpret_cast<uint32_t*>(at + s * W_TERM + 256) = hi[s];
            }
          }
        }
      }
      // ---- what the state at the tile's start gives: 64 tokens x 16 columns
      float O[TOKENS / 16][2][4], O1[TOKENS / 16][2][4];
#pragma unroll
      for (int mt = 0; mt < TOKENS / 16; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[mt][0][e] = O[mt][1][e] = O1[mt][0][e] = O1[mt][1][e] = 0.f;
#pragma unroll
      for (int pass = 0; pass < 2; ++pass) {  // the small terms of all k first: the sums then lose at the size of the large ones' few additions only
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
          uint32_t B[3][4];  // three terms: columns 0..7 (k 0..7, k 8..15), columns 8..15
          split3(S[2 * kk][0], S[2 * kk][1], B[0][0], B[1][0], B[2][0]);
          split3(S[2 * kk + 1][0], S[2 * kk + 1][1], B[0][1], B[1][1], B[2][1]);
          split3(S[2 * kk][2], S[2 * kk][3], B[0][2], B[1][2], B[2][2]);
          split3(S[2 * kk + 1][2], S[2 * kk + 1][3], B[0][3], B[1][3], B[2][3]);
          uint32_t a[TOKENS / 16][4];
#pragma unroll
          for (int mt = 0; mt < TOKENS / 16; ++mt)
            if (mt * 16 < len) ldsm_x4(a[mt], c_addr + mt * 16 * Z::N_ROW + kk * 32);
#pragma unroll
          for (int s = pass ? 0 : 2; s >= (pass ? 0 : 1); --s)  // eight accumulators in turn, so that no product waits for the one before
#pragma unroll
            for (int mt = 0; mt < TOKENS / 16; ++mt)
              if (mt * 16 < len) {
                float (&sum)[2][4] = pass && kk >= NK / 2 ? O1[mt] : O[mt];
                mma16816(sum[0], a[mt], B[s][0], B[s][1]);
                mma16816(sum[1], a[mt], B[s][2], B[s][3]);
              }
        }
      }
#pragma unroll
      for (int mt = 0; mt < TOKENS / 16; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) { O[mt][0][e] += O1[mt][0][e]; O[mt][1][e] += O1[mt][1][e]; }
      __syncthreads();  // the scores are complete
      const uint32_t w_addr = smem_u32(sW) + (lane & 15) * 32 + ((lane >> 4) ^ ((lane >> 2) & 1)) * 16;
      // ---- what the tile's own tokens give, and the read-outs
#pragma unroll
      for (int mt = 0; mt < TOKENS / 16; ++mt) {
        if (mt * 16 < len) {
          const int r_lo = mt * 16 + (lane >> 2), r_hi = r_lo + 8;
          float T[3][2][4];  // the three terms' sums apart: six accumulators in turn
#pragma unroll
          for (int s = 0; s < 3; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) T[s][0][e] = T[s][1][e] = 0.f;
#pragma unroll
          for (int kk = 0; kk <= mt; ++kk) {
            uint32_t w[3][4], b[4];
#pragma unroll
            for (int s = 0; s < 3; ++s) ldsm_x4(w[s], w_addr + s * W_TERM + (mt * (mt + 1) / 2 + kk) * W_TILE);
            ldsm_x4_trans(b, smem_u32(sX) + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * X_ROW + warp * 32 + (lane >> 4) * 16);
#pragma unroll
            for (int s = 2; s >= 0; --s) {
              mma16816(T[s][0], w[s], b[0], b[1]);
              mma16816(T[s][1], w[s], b[2], b[3]);
            }
          }
          const float e_lo = tab[2 * TOKENS + r_lo], e_hi = tab[2 * TOKENS + r_hi];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int col = warp * 16 + nt * 8 + kcol;
            if (col0 + col < P) {
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                const int r = hf ? r_hi : r_lo;
                if (r < len) {
                  const float2 x = unpack2(*reinterpret_cast<const uint32_t*>(sX + r * X_ROW + col * 2));
                  const float e = hf ? e_hi : e_lo;
                  float2 v;
                  v.x = fmaf(O[mt][nt][2 * hf], e, (T[2][nt][2 * hf] + T[1][nt][2 * hf]) + T[0][nt][2 * hf]);
                  v.y = fmaf(O[mt][nt][2 * hf + 1], e, (T[2][nt][2 * hf + 1] + T[1][nt][2 * hf + 1]) + T[0][nt][2 * hf + 1]);
                  v.x = fmaf(Dh, x.x, v.x);
                  v.y = fmaf(Dh, x.y, v.y);
                  finite = fmaf(v.x, 0.f, fmaf(v.y, 0.f, finite));
                  *reinterpret_cast<float2*>(p.y + (size_t)(base + r) * inner + head * P + col0 + col) = v;
                }
              }
            }
          }
        }
      }
    }
    if (more && warp == 0) {  // the next tile's table, while the other warps are at their products
      make_table(tables + (stage ^ 1) * Z::TABLE, base + TOKENS);
      load_dt(base + 2 * TOKENS);
    }
    // ---- the state at the tile's end
    const float eC = tab[5 * TOKENS];
#pragma unroll
    for (int j = 0; j < 2 * NK; ++j) { S[j][0] *= eC; S[j][1] *= eC; S[j][2] *= eC; S[j][3] *= eC; }
#pragma unroll
    for (int kk = 0; kk < TOKENS / 16; ++kk) {
      if (kk * 16 < len) {
        uint32_t v[4], w[3][4];
        ldsm_x4_trans(v, smem_u32(sX) + (kk * 16 + (lane & 7) + (lane >> 4) * 8) * X_ROW + warp * 32 + ((lane >> 3) & 1) * 16);
        const float* wl = tab + 4 * TOKENS + kk * 16 + kcol;
        const float2 w0 = make_float2(wl[0], wl[1]), w8 = make_float2(wl[8], wl[9]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = unpack2(v[e]);
          split3(x.x * (e < 2 ? w0.x : w8.x), x.y * (e < 2 ? w0.y : w8.y), w[0][e], w[1][e], w[2][e]);
        }
        constexpr int GROUP = NK % 4 == 0 ? 4 : 2;
#pragma unroll
        for (int j0 = 0; j0 < NK; j0 += GROUP) {  // 2 GROUP accumulators in turn
          uint32_t b[GROUP][4];
#pragma unroll
          for (int q = 0; q < GROUP; ++q)
            ldsm_x4_trans(b[q], smem_u32(sB) + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * Z::N_ROW + ((j0 + q) * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
          for (int s = 2; s >= 0; --s)
#pragma unroll
            for (int q = 0; q < GROUP; ++q) {
              mma16816(S[2 * (j0 + q)], w[s], b[q][0], b[q][1]);
              mma16816(S[2 * (j0 + q) + 1], w[s], b[q][2], b[q][3]);
            }
        }
      }
    }
  }
  float* dst = t1 == last ? slot_state : (SECOND ? nullptr : p.part + pbase(seg) * block);
  if (emit) {
    if (dst) each([&](int j, int e, size_t) { finite = fmaf(S[j][e], 0.f, fmaf(S[j][e + 1], 0.f, finite)); });
    if (__syncthreads_or(finite != 0.f)) {  // (also: nobody writes a read-out behind this)
      int second = 0, end = 0;              // segments behind the first start again from the state behind it, the last one that was walked from the slot's
      if (SECOND) segment_tiles((last - first + TOKENS - 1) / TOKENS, p.segments, 1, second, end);
      walk_again(p, head, col0, SECOND ? p.part + pbase(0) * block : slot_state, first + second * TOKENS, t0, t1, dst);
      dst = nullptr;
    }
  }
  if (dst) each([&](int j, int e, size_t at) { *reinterpret_cast<float2*>(dst + at) = make_float2(S[j][e], S[j][e + 1]); });
  if (!SECOND && t1 != last && tid == 0 && blockIdx.x == 0) p.part_log[pbase(seg)] = (float)total;
}

inline int column_blocks(int P) { return (P + COLS - 1) / COLS; }

template <int NK>
int launch(const Params& p, cudaStream_t stream) {
  static OncePerDevice configured;
  if (!configured.here()) {
    cudaError_t e = cudaFuncSetAttribute(ssm_chunk_kernel<NK, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NK>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ssm_chunk_kernel<NK, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NK>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.here() = true;
  }
  const dim3 grid(column_blocks(p.P), p.heads, p.num_seqs * (p.segments > 1 ? p.segments - 1 : 1)), block(WARPS * 32);
  cudaError_t e = launch_pdl((ssm_chunk_kernel<NK, false>), grid, block, (size_t)Shape<NK>::SMEM, stream, 1, p);
  if (e == cudaSuccess && p.segments > 1) e = launch_pdl((ssm_chunk_kernel<NK, true>), grid, block, (size_t)Shape<NK>::SMEM, stream, 1, p);
  return (int)e;
}

}  // namespace

// Into how many segments the sequences of a step are cut: a launch (of one segment fewer) gives every SM two CTAs, and no segment
// is shorter than three tiles.  Two segments would follow one another: three is the fewest that gain.  Measured (us at segments 1 / 3 / 4 /
// 5 / 6, 64 heads): one prompt of 4,096 459 / - / 260 / 214 / 306 (six: more CTAs than places), of 600 70 / 66 / 54 / 54 / -, of 300
// 37 / 43 / 39 / - / -; three prompts (192 CTAs of one segment) 187 / 157 / 156 / 178 / -; 256 CTAs of one segment 217 / 239.
DLI_EXPORT int dli_ssm_segments(int num_seqs, int heads, int P, int max_len) {
  const long long units = (long long)column_blocks(P) * heads * (num_seqs > 0 ? num_seqs : 1);
  long long fill = 2LL * sm_count() / (units > 0 ? units : 1);
  if (fill < 2 && 3 * units <= 4LL * sm_count()) fill = 2;
  const int most = (max_len + TOKENS - 1) / TOKENS / 3;
  if (fill > most) fill = most;
  return fill < 2 ? 1 : (fill > 32 ? 33 : (int)fill + 1);
}

// segments > 1: part [num_seqs (segments - 1) heads P N] and part_log [num_seqs (segments - 1) heads] are scratch.
DLI_EXPORT int dli_ssm_chunk(float* y, const void* xbc, const void* u, long long u_stride, int dt_col, const float* dt_bias, const float* A_log,
                             const float* D, float* state, const int* q_start, const int* state_slot, int num_seqs, int heads, int P, int N,
                             int groups, int segments, float* part, float* part_log, cudaStream_t stream) {
  if (num_seqs == 0) return 0;
  if (heads < 1 || heads > 65535 || groups < 1 || heads % groups || P < 8 || P % 8 || N < 8 || N % 8 || N > 128 || segments < 1 ||
      (long long)num_seqs * segments > 65535 || ((uintptr_t)xbc & 15) || ((uintptr_t)y & 7) || ((uintptr_t)state & 7) || (segments > 1 && (!part || !part_log)))
    return DLI_ERR_UNSUPPORTED;
  Params p;
  p.y = y; p.xbc = (const bf16*)xbc; p.u = (const bf16*)u; p.u_stride = u_stride; p.dt_col = dt_col; p.dt_bias = dt_bias; p.A_log = A_log; p.D = D;
  p.state = state; p.q_start = q_start; p.state_slot = state_slot; p.num_seqs = num_seqs; p.heads = heads; p.P = P; p.N = N; p.groups = groups;
  p.segments = segments; p.part = part; p.part_log = part_log;
  if (N <= 32) return launch<2>(p, stream);
  if (N <= 64) return launch<4>(p, stream);
  return launch<8>(p, stream);
}
