// out[b][t, f] = sum over k of x[b][t, k] * W[b][f, k], everything float32, on the tensor cores (tcgen05).
//
// A float32 number is cut into three bfloat16 numbers whose sum it is (8 bits of mantissa each: high, middle, low), and a product of two
// float32 numbers is the six products of terms that reach its last bit: hh + (hm + mh) + (hl + mm + lh).  Products of two bfloat16
// numbers are exact in float32.  An addition into a tensor-core accumulator cuts off where a plain one rounds, so the large products hh
// are summed there over 64 or 128 k only (accumulators in turn) and the CUDA cores add those sums; the others, 2^-8 of them and less,
// stay in accumulators of their own.  The three terms are the number down to 2^-110: the third one of a smaller number lies among the smallest bfloat16 numbers, multiples
// of 2^-133, and loses up to 2^-134 (an error of 1.1e-6 for operands around 2^-115, 9e-6 around 2^-118, where the library's product keeps 3e-7).  Operands scaled
// by 2^24 before they are cut would keep it; that took 4 % longer.
//
//   * Features take the 128-row side of the instruction, tokens its columns: a column of the accumulator is a token, whose 32
//     neighbouring features a warp stores side by side; a step of few tokens is a narrow instruction.
//   * Eight warps fetch float32 rows of W and x a step or two of 64 k ahead into registers, cut them and write the terms to shared memory in
//     the layout that the instruction reads (rows of 64 k, 128-byte swizzle).  The terms of x lie behind one another, so that one
//     instruction takes two of them as its columns: h [m l] and m [h m] into the sums s1 | s2, l [h] into s1, h [h] into the large one.
//   * A ninth warp issues the products.
//   * Few tiles are cut along k between the CTAs of a cluster, which add their sums through distributed shared memory, always in the
//     same order.
//
//   full[s]      the terms of stage s are written (one arrival a warp)
//   empty[s]     the products have read stage s
//   sum_full[b]  large accumulator b holds its chunk of the steps
//   sum_empty[b] the eight warps have read it
//
// Three terms of an infinity are infinity, NaN, NaN, and a number within 2^-9 of the largest has an infinite first term; so an output that is
// not finite is computed again by plain multiply-adds (plain_dot), as the product without terms has it.
//
// What bounds it: a step's own chain (fetch, cut, write, fence, products, 1.2 to 1.8 us; its shared memory traffic, 96 KB of terms and 160 KB of
// operands with tiles of 128 tokens, is 2,000 clocks, its products 1,536).  Measured, us, against the library's products on the CUDA cores (weights not in
// L2, launch included): 4 x 1,024 features, K 2,048, 16 / 100 / 501 tokens 41 / 68 / 167 -> 21 / 31 / 72; 2,048 features, K 8,192 92 / 211 / 338 -> 54 / 64 /
// 127; 10,304 features, K 2,048 77 / 156 / 420 -> 48 / 74 / 194.  Errors against 64 bits 0.7e-7 to 1.5e-7 of the result (the library 0.9e-7 to 1.6e-6, larger at each of
// these sizes; with 256 k in one accumulator 2.4e-7).
//
// Every wait is bounded: after `wait_limit` polls a code goes to *error_flag and the CTA ends early (it has no copies in flight).  A warp stores only sums that it has seen
// finished; in a cluster none of the CTAs stores anything (the others hear of it in front of the barrier behind which sums are added).
#include "common.cuh"
#include "mma_split.cuh"

using namespace dli;

namespace {

constexpr int BF = 128;  // features of a tile
constexpr int BK = 64;   // k of a step: 128 bytes of bfloat16, one swizzle row
constexpr int CONVERTERS = 256;  // threads
constexpr int THREADS = CONVERTERS + 32;
constexpr int MAX_SPLITS = 8;
constexpr unsigned WAIT_LIMIT = 1u << 24;

struct FloatParams {
  const float *x, *w;
  float* out;
  long long x_row, w_row, out_row, x_batch, w_batch, out_batch;  // in numbers
  int tokens, features, K, splits, token_tiles;
  int* error_flag;
  unsigned wait_limit;
  int skip_step;  // -1 in every launch of the engine: the step whose terms a test does not hand in (dli_float_gemm_wait_test)
};

template <int NT> struct Shape {  // NT: tokens of a tile
  static constexpr int STAGES = NT == 128 ? 2 : 3;
  static constexpr int AHEAD = NT == 128 ? 1 : 2;  // steps in registers
  static constexpr int CHUNK = NT == 128 ? 2 : 1, LARGE = NT == 128 ? 2 : 4;  // steps whose large products go to one accumulator; how many of those in turn
  static constexpr int A_TERM = BF * 128, B_TERM = NT * 128, STAGE = 3 * (A_TERM + B_TERM);
  static constexpr int SMALL = LARGE * NT, COLUMNS = NT == 32 ? 256 : 512;  // of tensor memory: large sums | s1 | s2
  static constexpr int PART = NT * BF * 4;  // a CTA's sums, handed round in a cluster in the stages' place
  static constexpr int SMEM = STAGES * STAGE + 256 + 1024;
  static_assert(SMEM <= 227 * 1024 && PART <= STAGES * STAGE && STAGES - 1 < (LARGE - 1) * CHUNK && SMALL + 2 * NT <= COLUMNS, "shared memory, and the order of the waits");
};

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, const FloatParams& p, volatile int* failed, int code) {
  for (unsigned i = 0; i < p.wait_limit; ++i) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((i & 1023) == 1023 && *failed) return false;
  }
  if (!*failed) { *failed = code; atomicCAS(p.error_flag, 0, code); }
  return false;
}
// Descriptor of a K-major operand whose rows are 128 bytes, swizzled in 128-byte mode: 1,024 bytes between groups of eight rows.
__device__ __forceinline__ uint64_t operand(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// kind::f16: float32 accumulator, bfloat16 operands, both K-major, M = 128
__device__ __forceinline__ uint32_t instruction(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }
// Products are issued by one lane of a warp that runs together, so that descriptors stay in uniform registers: by a thread in a branch of its own an
// instruction took 100 to 180 clocks, more than the tensor cores need for it.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one;
}
__device__ __forceinline__ void product(uint32_t one, uint32_t sum, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %5, 0;\n\tsetp.ne.b32 p, %4, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(sum), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add), "r"(one) : "memory");
}
__device__ __forceinline__ void commit(uint32_t one, uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(one) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(addr));
}
// (Pinned: the loads of a step stay in front of the wait that hides them.  Plain loads: .nc wants memory that nobody writes while the kernel runs, but with a
// programmatic launch the kernel in front, which writes x, may still run when this one starts, and the wait for it orders ordinary loads only.)
__device__ __forceinline__ float4 load4(const float* p, bool in) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in) asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float plain_dot(const float* a, const float* b, int K) {
  float s = 0.f;
#pragma unroll 1
  for (int k = 0; k < K; ++k) s = fmaf(a[k], b[k], s);
  return s;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

template <int NT>
__global__ void __launch_bounds__(THREADS, 1) float_gemm_kernel(const __grid_constant__ FloatParams p) {
  using Z = Shape<NT>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Z::STAGES * Z::STAGE);  // full[STAGES], empty[STAGES], sum_full[LARGE], sum_empty[LARGE]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * Z::STAGES + 2 * Z::LARGE);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * Z::STAGES, sum_full0 = empty0 + 8 * Z::STAGES, sum_empty0 = sum_full0 + 8 * Z::LARGE;
  if (tid == 0) {
    for (int s = 0; s < Z::STAGES; ++s) {
      bar_init(full0 + 8 * s, CONVERTERS / 32);
      bar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < Z::LARGE; ++b) {
      bar_init(sum_full0 + 8 * b, 1);
      bar_init(sum_empty0 + 8 * b, CONVERTERS / 32);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == CONVERTERS / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Z::COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // this CTA's tile and its share of the steps
  const int f0 = blockIdx.x * BF, batch = blockIdx.z / p.token_tiles, t0 = (blockIdx.z - batch * p.token_tiles) * NT, split = blockIdx.y;
  const int all = (p.K + BK - 1) / BK, share = (all + p.splits - 1) / p.splits;
  const int first = min(all, split * share), steps = min(all, first + share) - first;  // (a last split may be empty)
  const int chunks = (steps + Z::CHUNK - 1) / Z::CHUNK;
  const float* x = p.x + batch * p.x_batch;
  const float* w = p.w + batch * p.w_batch;
  float* out = p.out + batch * p.out_batch;
  bool ok = true;
  pdl_wait();

  if (warp == CONVERTERS / 32) {
    // ---- products
    const uint32_t one = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0), small = tm + Z::SMALL;
    const uint64_t stages = operand(smem_u32(smem));  // (a descriptor counts 16 bytes)
    auto wait = [&](uint32_t bar, uint32_t parity, int code) { ok = __all_sync(0xffffffffu, ok && bar_wait(bar, parity, p, failed, code)); };
    for (int s = 0; s < steps; ++s) {
      const int stage = s % Z::STAGES, chunk = s / Z::CHUNK, buf = chunk % Z::LARGE;
      if (s % Z::CHUNK == 0 && chunk >= Z::LARGE) wait(sum_empty0 + 8 * buf, (chunk / Z::LARGE - 1) & 1, 1);
      wait(full0 + 8 * stage, (s / Z::STAGES) & 1, 2);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t a = stages + (uint32_t)((stage * Z::STAGE) >> 4), b = a + ((3 * Z::A_TERM) >> 4);
      const uint32_t large = tm + buf * NT;
#pragma unroll
      for (int k = 0; k < BK / 16; ++k) {
        const uint64_t ak = a + ((k * 32) >> 4), bk = b + ((k * 32) >> 4);
        const bool add = s > 0 || k > 0;
        product(one, small, ak, bk + (Z::B_TERM >> 4), instruction(2 * NT), add);          // h [m l]
        product(one, small, ak + ((2 * Z::A_TERM) >> 4), bk, instruction(NT), true);       // l [h]
        product(one, small, ak + (Z::A_TERM >> 4), bk, instruction(2 * NT), true);         // m [h m]
        product(one, large, ak, bk, instruction(NT), s % Z::CHUNK != 0 || k > 0);          // h [h]
      }
      commit(one, empty0 + 8 * stage);
      if (s % Z::CHUNK == Z::CHUNK - 1 || s == steps - 1) commit(one, sum_full0 + 8 * buf);
    }
    __syncwarp();
  } else {
    // ---- terms.  A thread takes eight neighbouring k of every 32nd row: rows of W, then of x
    constexpr int RUNS = (BF + NT) / 32, WR = BF / 32;
    const int r0 = tid >> 3, c = tid & 7;
    const float* wp = w + (size_t)(f0 + r0) * p.w_row + c * 8;
    const float* xp = x + (size_t)(t0 + r0) * p.x_row + c * 8;
    float4 lo[Z::AHEAD][RUNS], hi[Z::AHEAD][RUNS];
    auto fetch = [&](int step, float4 (&lo)[RUNS], float4 (&hi)[RUNS]) {
      const int k = step * BK;
#pragma unroll
      for (int i = 0; i < RUNS; ++i) {
        const bool ok = i < WR ? f0 + r0 + i * 32 < p.features : t0 + r0 + (i - WR) * 32 < p.tokens;
        const float* src = i < WR ? wp + (size_t)(i * 32) * p.w_row + k : xp + (size_t)((i - WR) * 32) * p.x_row + k;
        lo[i] = load4(src, ok && k + c * 8 < p.K);  // (K is a multiple of 4)
        hi[i] = load4(src + 4, ok && k + c * 8 + 4 < p.K);
      }
    };
    const int quad = warp & 3, col0 = (warp >> 2) * (NT / 2);  // this warp's lanes (features) and columns (tokens) of the sums
    const uint32_t sums = tmem + ((uint32_t)(quad * 32) << 16) + col0;
    float acc[NT / 2];
#pragma unroll
    for (int j = 0; j < NT / 2; ++j) acc[j] = 0.f;
    auto add_columns = [&](uint32_t from) {
#pragma unroll
      for (int j = 0; j < NT / 2; j += 16) {
        uint32_t v[16];
        tmem_ld16(from + j, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[j + e] += __uint_as_float(v[e]);
      }
    };
    auto take_chunk = [&](int chunk) {
      const int buf = chunk % Z::LARGE;
      ok = __all_sync(0xffffffffu, ok && bar_wait(sum_full0 + 8 * buf, (chunk / Z::LARGE) & 1, p, failed, 3));
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      add_columns(sums + buf * NT);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(sum_empty0 + 8 * buf);
    };
    int taken = 0;
    auto one_step = [&](int s, float4 (&lo)[RUNS], float4 (&hi)[RUNS]) {
      const int stage = s % Z::STAGES;
      if (s >= Z::STAGES) ok = __all_sync(0xffffffffu, bar_wait(empty0 + 8 * stage, (s / Z::STAGES - 1) & 1, p, failed, 4));
      if (ok && s == (taken + 1) * Z::CHUNK + Z::STAGES - 1) take_chunk(taken++);  // (its products have just been seen to end)
      if (!ok) return;
      const uint32_t a = smem_u32(smem + stage * Z::STAGE), at = r0 * 128 + ((c ^ (r0 & 7)) << 4);
#pragma unroll
      for (int i = 0; i < RUNS; ++i) {
        uint32_t t[3][4];
        dli::split3(lo[i].x, lo[i].y, t[0][0], t[1][0], t[2][0]);
        dli::split3(lo[i].z, lo[i].w, t[0][1], t[1][1], t[2][1]);
        dli::split3(hi[i].x, hi[i].y, t[0][2], t[1][2], t[2][2]);
        dli::split3(hi[i].z, hi[i].w, t[0][3], t[1][3], t[2][3]);
        const uint32_t dst = i < WR ? a + i * 32 * 128 + at : a + 3 * Z::A_TERM + (i - WR) * 32 * 128 + at;
#pragma unroll
        for (int e = 0; e < 3; ++e)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + e * (i < WR ? Z::A_TERM : Z::B_TERM)), "r"(t[e][0]), "r"(t[e][1]), "r"(t[e][2]), "r"(t[e][3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (in front of the loads: it waits for those under way)
      __syncwarp();
      if (lane == 0 && first + s != p.skip_step) bar_arrive(full0 + 8 * stage);
      if (s + Z::AHEAD < steps) fetch(first + s + Z::AHEAD, lo, hi);
    };
#pragma unroll
    for (int i = 0; i < Z::AHEAD; ++i)
      if (i < steps) fetch(first + i, lo[i], hi[i]);
    for (int s = 0; s < steps && ok; s += Z::AHEAD) {
#pragma unroll
      for (int i = 0; i < Z::AHEAD; ++i)
        if (s + i < steps && ok) one_step(s + i, lo[i], hi[i]);
    }
    while (ok && taken < chunks) take_chunk(taken++);
    if (ok && steps > 0) {  // (the last chunk's commit covers the small products as well)
#pragma unroll
      for (int j = 0; j < NT / 2; j += 16) {
        uint32_t v[16], u[16];
        tmem_ld16(sums + Z::SMALL + j, v);
        tmem_ld16(sums + Z::SMALL + NT + j, u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[j + e] += __uint_as_float(v[e]) + __uint_as_float(u[e]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (p.splits == 1) {
      const int f = f0 + quad * 32 + lane;
      bool again = false;
      if (ok && f < p.features) {
        float* dst = out + (size_t)(t0 + col0) * p.out_row + f;
#pragma unroll
        for (int j = 0; j < NT / 2; ++j)
          if (t0 + col0 + j < p.tokens) {
            dst[(size_t)j * p.out_row] = acc[j];
            again |= !finite(acc[j]);
          }
        if (again) {
#pragma unroll 1
          for (int t = t0 + col0; t < min(p.tokens, t0 + col0 + NT / 2); ++t) {
            float* at = out + (size_t)t * p.out_row + f;
            if (!finite(*at)) *at = plain_dot(x + (size_t)t * p.x_row, w + (size_t)f * p.w_row, p.K);
          }
        }
      }
    } else {
      asm volatile("bar.sync 1, 256;" ::: "memory");  // every warp has seen all products end: the stages are free
      float* part = reinterpret_cast<float*>(smem) + col0 * BF + quad * 32 + lane;  // [tokens][features]
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) part[j * BF] = acc[j];
    }
  }
  if (!ok && p.splits > 1 && lane < p.splits)
    asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %0, %1;\n\tst.shared::cluster.u32 [remote], %2;\n\t}"
                 ::"r"(smem_u32(tmem_slot + 1)), "r"(lane), "r"(*failed) : "memory");
  __syncthreads();
  if (p.splits > 1) {
    // ---- every CTA of the cluster adds all sums of its share of the tile's tokens
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int per = NT / p.splits;
    if (!*failed && tid < CONVERTERS) {
      const int f = f0 + lane * 4;
      for (int j = split * per + warp; j < (split + 1) * per; j += CONVERTERS / 32) {
        const uint32_t at = smem_u32(smem) + (j * BF + lane * 4) * 4;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < MAX_SPLITS; ++r)
          if (r < p.splits) {
            float4 v;
            asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %4, %5;\n\tld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [remote];\n\t}"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at), "r"(r) : "memory");
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
        const int t = t0 + j;
        if (t < p.tokens) {
          const float v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (f + e < p.features) {
              float y = v[e];
              if (!finite(y)) y = plain_dot(x + (size_t)t * p.x_row, w + (size_t)(f + e) * p.w_row, p.K);
              out[(size_t)t * p.out_row + f + e] = y;
            }
        }
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its sums are read
  }
  // Not before: a CTA has an SM's shared memory, and what is launched meanwhile, such as the attention behind the rotary embedding, which only waits, would all
  // lie on the SMs that have none (81 tokens with 16 heads: the attention 58 us, 122 with the kernels behind this one launched at its start).
  pdl_launch_dependents();
  if (warp == CONVERTERS / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Z::COLUMNS) : "memory");
  }
}

int* error_flag_device = nullptr;
int* error_flag_host = nullptr;

template <int NT> int launch(const FloatParams& p, int batches, cudaStream_t stream) {
  static OncePerDevice configured;
  if (!configured.here()) {
    const cudaError_t e = cudaFuncSetAttribute(float_gemm_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NT>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.here() = true;
  }
  return (int)launch_pdl((float_gemm_kernel<NT>), dim3((p.features + BF - 1) / BF, p.splits, p.token_tiles * batches), dim3(THREADS), (size_t)Shape<NT>::SMEM,
                         stream, p.splits, p);
}

// Tokens of a tile and splits of k (0: to be chosen), by estimates in us: a step of 64 k takes 1.2 / 1.5 / 1.8 with 32 / 64 / 128 tokens, a tile 4.5 / 6 / 7.5
// besides, 1.5 more where sums are exchanged.  Clusters of four fill 132 of 148 SMs, clusters of eight 112.  Measured against it (cold weights, launch
// included): 4 x 1,024 features, K 2,048, 16 tokens 47 / 31 / 20 / 35 at 1 / 2 / 4 / 8 splits; 2,048 features, K 4,096, 100 tokens in tiles of 32 / 64 / 128,
// 4 splits: 51 / 39 / 43.
void choose(int tokens, int features, int batches, int steps, int& tile, int& splits) {
  const long long feature_tiles = (features + BF - 1) / BF;
  const int fixed_tile = tile, fixed_splits = splits;
  double best = -1.;
  for (int nt = 32; nt <= 128; nt *= 2)
    for (int s = 1; s <= MAX_SPLITS && s <= steps; s *= 2) {
      if ((fixed_tile && nt != fixed_tile) || (fixed_splits && s != fixed_splits)) continue;
      if (!fixed_tile && (long long)((tokens + nt - 1) / nt) * batches > 65535) continue;  // (the grid's z)
      const long long ctas = feature_tiles * ((tokens + nt - 1) / nt) * batches * s, places = s == 8 ? 112 : s == 4 ? 132 : sm_count();
      const double step = nt == 128 ? 1.8 : nt == 64 ? 1.5 : 1.2, around = (nt == 128 ? 7.5 : nt == 64 ? 6. : 4.5) + (s > 1 ? 1.5 : 0.);
      const double us = (double)((ctas + places - 1) / places) * ((steps + s - 1) / s * step + around);
      if (best < 0. || us < best) { best = us; tile = nt; splits = s; }
    }
  if (best < 0.) { tile = fixed_tile ? fixed_tile : 128; splits = 1; }  // (more splits asked for than steps: one)
}

}  // namespace

static int run(float* out, const float* x, const float* w, int batches, int tokens, int features, int K, long long x_row, long long w_row, long long out_row,
               long long x_batch, long long w_batch, long long out_batch, int tile, int splits, unsigned wait_limit, int skip_step, cudaStream_t stream) {
  if (batches == 0 || tokens == 0 || features == 0) return 0;
  if (batches < 0 || tokens < 0 || features < 0 || K < 4 || K % 4 || x_row % 4 || w_row % 4 || x_batch % 4 || w_batch % 4 || (((uintptr_t)x | (uintptr_t)w) & 15) ||
      (tile != 0 && tile != 32 && tile != 64 && tile != 128) || (splits != 0 && splits != 1 && splits != 2 && splits != 4 && splits != 8))
    return DLI_ERR_UNSUPPORTED;
  if (!error_flag_host) {
    if (cudaHostAlloc((void**)&error_flag_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return (int)cudaGetLastError();
    *error_flag_host = 0;
    if (cudaHostGetDevicePointer((void**)&error_flag_device, error_flag_host, 0) != cudaSuccess) return (int)cudaGetLastError();
  }
  if (!tile || !splits) choose(tokens, features, batches, (K + BK - 1) / BK, tile, splits);
  FloatParams p;
  p.x = x; p.w = w; p.out = out; p.x_row = x_row; p.w_row = w_row; p.out_row = out_row; p.x_batch = x_batch; p.w_batch = w_batch; p.out_batch = out_batch;
  p.tokens = tokens; p.features = features; p.K = K; p.splits = splits; p.token_tiles = (tokens + tile - 1) / tile;
  p.error_flag = error_flag_device; p.wait_limit = wait_limit; p.skip_step = skip_step;
  if ((long long)p.token_tiles * batches > 65535) return DLI_ERR_UNSUPPORTED;
  if (tile == 32) return launch<32>(p, batches, stream);
  return tile == 64 ? launch<64>(p, batches, stream) : launch<128>(p, batches, stream);
}

// tile: tokens of a tile (32, 64 or 128), splits: CTAs that share a tile's k (1, 2, 4 or 8); 0 and 0: chosen here.
DLI_EXPORT int dli_float_gemm(float* out, const float* x, const float* w, int batches, int tokens, int features, int K, long long x_row, long long w_row,
                              long long out_row, long long x_batch, long long w_batch, long long out_batch, int tile, int splits, cudaStream_t stream) {
  return run(out, x, w, batches, tokens, features, K, x_row, w_row, out_row, x_batch, w_batch, out_batch, tile, splits, WAIT_LIMIT, -1, stream);
}

// For tests: the terms of step `skip_step` (of 64 k) are never handed in and every wait gives up after `wait_limit` polls: the products' wait for them runs out (code 2),
// and those for sums and stages that depend on it (3, 4).
DLI_EXPORT int dli_float_gemm_wait_test(float* out, const float* x, const float* w, int tokens, int features, int K, int tile, int splits, unsigned wait_limit, int skip_step,
                                        cudaStream_t stream) {
  if (wait_limit < 1 || wait_limit > WAIT_LIMIT || tile == 0 || splits == 0 || skip_step < 0 || skip_step >= (K + BK - 1) / BK) return DLI_ERR_UNSUPPORTED;
  return run(out, x, w, 1, tokens, features, K, K, K, features, 0, 0, 0, tile, splits, wait_limit, skip_step, stream);
}

// 0, or the code of the first wait that ran out (1 accumulators, 2 terms, 3 sums, 4 stages)
DLI_EXPORT int dli_float_gemm_error() { return error_flag_host ? *error_flag_host : 0; }
DLI_EXPORT int dli_float_gemm_clear_error() { if (error_flag_host) *error_flag_host = 0; return 0; }
