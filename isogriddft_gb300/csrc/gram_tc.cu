// K6 on the tensor pipe: tall-skinny weighted Gram G = A W B^T with tcgen05.
//
// Reference: _weighted_overlap_columns (ks/eigensolver_jax.py:105) and
// weighted_overlap_matrix (ks/eigensolver.py:246-272): G[i][j] = sum_p A_i[p] w[p] B_j[p].
//
// The contraction dimension is the grid (millions of points) and the outputs
// are small (a, b <= 64), so a plain M = a, N = b MMA would leave most of a
// 128-row tensor-core tile empty and read it from shared memory every step.
// Instead each pipeline stage stacks s = 128 / a_pad point chunks of 32 points:
// the M = 128 operand is [A_c0; A_c1; ...] (chunk c's a rows at rows c*a_pad)
// and the N = s*b_pad operand is [B_c0; B_c1; ...].  The s diagonal blocks of
// the accumulator are the chunk Grams A_c B_c^T; the off-diagonal blocks are
// ignored.  Tensor work grows s-fold but the operand bytes read per point stay
// close to the bytes that arrive from HBM, and the kernel remains HBM-bound.
//
// Precision (3xTF32): x = hi + lo with hi = x rounded to the nearest TF32
// value and lo = x - hi (exact in FP32, |lo| <= 2^-11 |x|); A_c B_c^T ~
// A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T, about 2^-21 relative per product.
// The tensor core's FP32 accumulation does not round to nearest: each step
// into an accumulator can lose a fraction of an ulp of the running sum, and on
// sums of one sign (a self-Gram's diagonal) these losses add up instead of
// averaging out.  The hi*hi products therefore go to their own accumulator
// (4 MMAs per stage, FLUSH stages per window) and the much smaller cross terms
// to a second one, whose losses are 2^-11 smaller; both are read out every
// FLUSH stages into compensated (Kahan) FP32 sums in registers (GB300's FP64
// pipe is too slow to take one FP64 add per value and window), which become
// FP64 once per CTA and are summed in FP64 across blocks (deterministic
// per-block partials reduced by gram_reduce_kernel).
//
// Roles (384 threads, one CTA per SM, persistent over stages):
//   warp 0 lane 0: TMA producer (FP32 tiles of A and B with 128-byte swizzle)
//                  into a ring of raw slots;
//   warp 1       : TMEM allocation; lane 0 issues the MMAs (8 per stage: hi*hi and
//                  hi*lo in one of twice the width, since B's lo tile follows its
//                  hi tile, and lo*hi);
//   warps 4-11   : two groups of four warps that take the stages in turn: raw slot
//                  -> (B *= w) -> hi and lo tiles of the group's split buffer, proxy
//                  fence.  Two per TMEM lane quarter, they also run the epilogue
//                  (TMEM -> compensated sums), each for half of the columns.
// The weights come straight from memory, one stage ahead, in the splitting
// threads' registers: in the ring they would cost it its third slot.
// Two TMEM accumulator pairs alternate between windows so MMAs continue while
// the previous window is read out.  Every wait is bounded: on a timeout the error
// word is set, all roles leave their loops, TMEM is freed.
//
// What bounds it: shared memory.  A stage of 128 rows moves 32 KB in by TMA, 32 KB
// out and 64 KB back for the split and 80 KB to the tensor core, 0.9 us at 128 bytes
// a clock; it takes 1.1.  One group that split in place in a raw slot took 1.3 for
// narrow blocks and 1.7 for wide ones (four worker warps: the epilogue held all 64
// columns of a row in one thread).  Over 192^3 points, before and after: 47 x 47
// 1261 and 796 us (memory floor 400), 32 x 32 482 and 421, 16 x 16 256 and 231,
// 4 x 4 181 and 172; 64 x 64 over 10^6 203 and 147.
#include "gram_tc.cuh"
#include "tc.cuh"

namespace igd {
namespace {

constexpr int TC_ROLES = 128;  // warps 0-3: producer, MMA issuer, two idle
constexpr int TC_FLUSH = 4;    // stages per accumulation window (see the precision note)
constexpr int TC_MAX_SLOTS = 6;  // raw tiles in flight
// Two groups of workers take the stages in turn, each with its own split buffer: a group then waits only
// for products of its own previous stage, so its parity waits cannot fall a phase behind.
constexpr int TC_GROUPS = 2;
constexpr int TC_WORKERS = 256;  // 384 are slower: 929 us for 819, 47 x 47 over 192^3 points
constexpr int TC_THREADS = TC_ROLES + TC_WORKERS, TC_GROUP_THREADS = TC_WORKERS / TC_GROUPS;

struct GramTcPlan {
  int a, b, a_pad, a_rows, b_pad, s, N, slots, tmem_cols;
  size_t slot_bytes, split_bytes, smem;
};

__host__ __device__ inline int pad_rows(int r) { return r <= 8 ? 8 : r <= 16 ? 16 : r <= 32 ? 32 : 64; }

bool plan_gram_tc(int a, int b, GramTcPlan* p) {
  if (a < 1 || b < 1 || a > 64 || b > 64) return false;
  p->a = a;
  p->b = b;
  p->a_pad = pad_rows(a);
  p->s = std::min(128 / p->a_pad, 128 / pad_rows(b));  // N <= 128: two accumulator pairs fit 512 columns
  p->a_rows = (a + 7) & ~7;  // rows copied per chunk (whole swizzle atoms); the rest of a_pad stays zero
  p->b_pad = (b + 7) & ~7;
  p->N = p->s * p->b_pad;
  if (p->N % 16 != 0 || p->N > 128) return false;
  p->slot_bytes = (size_t)p->s * (p->a_rows + p->b_pad) * 128;  // whole 1024-byte swizzle atoms
  p->split_bytes = 2 * 128 * 128 + 2 * (size_t)p->N * 128;  // A hi, A lo, B hi, B lo; rows of 32 points
  const size_t budget = 225 * 1024;
  p->slots = (int)std::min<size_t>(TC_MAX_SLOTS, (budget - TC_GROUPS * p->split_bytes) / p->slot_bytes);
  if (p->slots < 2) return false;
  p->smem = p->slots * p->slot_bytes + TC_GROUPS * p->split_bytes + 1024;  // + alignment slack
  int cols = 32;
  while (cols < 4 * p->N) cols <<= 1;
  p->tmem_cols = cols;
  return true;
}

struct GramTcArgs {
  long long n;
  int a, b, a_pad, a_rows, b_pad, s, N, slots;
  unsigned slot_bytes, split_bytes;
  const double* w;
  long long stages;
  double* part;
  unsigned* err;
};

template <int BMAX>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gram_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                   const GramTcArgs g, uint32_t tmem_cols) {
  constexpr int NG = TC_GROUP_THREADS;
  extern __shared__ unsigned char tc_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[TC_MAX_SLOTS], free_bar[TC_MAX_SLOTS];
  __shared__ __align__(8) uint64_t ready_bar[TC_GROUPS], empty_bar[TC_GROUPS];
  __shared__ __align__(8) uint64_t accf_bar[2], acce_bar[2], done_bar;
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int LS = TC_GROUPS;
  const int S = g.slots;
  const long long G = gridDim.x;
  const long long J = g.stages > blockIdx.x ? (g.stages - blockIdx.x + G - 1) / G : 0;  // stages of this CTA

  // raw tile of ring slot q: A chunks, B chunks; split buffer: A hi, A lo, B hi, B lo
  auto slotA = [&](int q) { return base + (size_t)LS * g.split_bytes + (size_t)q * g.slot_bytes; };
  auto slotB = [&](int q) { return slotA(q) + (size_t)g.s * g.a_rows * 128; };
  auto splitA = [&](int u) { return base + (size_t)u * g.split_bytes; };
  auto splitB = [&](int u) { return splitA(u) + 2 * 128 * 128; };

  if (tid == 0) {
    for (int q = 0; q < S; ++q) {
      mbar_init(&full_bar[q], 1);
      mbar_init(&free_bar[q], NG / 32);
    }
    for (int u = 0; u < LS; ++u) {
      mbar_init(&ready_bar[u], NG / 32);
      mbar_init(&empty_bar[u], 1);
    }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&accf_bar[k], 1);
      mbar_init(&acce_bar[k], 8);  // the epilogue warps
    }
    mbar_init(&done_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  // zero the split buffers once: rows past the operands' own are never written and must read as zero
  for (size_t e = tid; e < (size_t)LS * g.split_bytes / 16; e += TC_THREADS)
    reinterpret_cast<uint4*>(base)[e] = make_uint4(0u, 0u, 0u, 0u);
  if (warp == 1) tmem_alloc(&tmem_holder, tmem_cols);
  fence_proxy_async();  // the zero fill is visible to the tensor core and to later copies
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_holder;
  const unsigned tx_bytes = (unsigned)(g.s * (g.a_rows + g.b_pad) * 128);

  if (warp == 0 && lane == 0) {
    // ------------------------------------------------ producer
    long long issued = 0;
    for (long long j = 0; j < J; ++j) {
      const int q = (int)(j % S);
      if (j >= S && !mbar_wait_or_abort(&free_bar[q], (unsigned)((j / S - 1) & 1), g.err, &abort_flag)) break;
      const long long t = blockIdx.x + j * G;
      const int p0 = (int)(t * 32 * g.s);
      mbar_arrive_expect_tx(&full_bar[q], tx_bytes);
      for (int c = 0; c < g.s; ++c) {
        tma_load_2d(slotA(q) + (size_t)c * g.a_rows * 128, &mapA, p0 + 32 * c, 0, &full_bar[q]);
        tma_load_2d(slotB(q) + (size_t)c * g.b_pad * 128, &mapB, p0 + 32 * c, 0, &full_bar[q]);
      }
      issued = j + 1;
    }
    // copies still in flight (after an abort) land before the CTA leaves
    for (long long j = std::max(0LL, issued - S); j < issued; ++j)
      mbar_wait(&full_bar[j % S], (unsigned)((j / S) & 1), g.err);
  } else if (warp == 1 && lane == 0) {
    // ------------------------------------------------ MMA issuer
    const uint32_t idesc = umma_idesc_tf32(128, g.N), idesc2 = umma_idesc_tf32(128, 2 * g.N);
    for (long long j = 0; j < J; ++j) {
      const int u = (int)(j % LS);
      const long long win = j / TC_FLUSH;
      const int buf = (int)(win & 1);
      if (j % TC_FLUSH == 0 && win >= 2) {
        if (!mbar_wait_or_abort(&acce_bar[buf], (unsigned)((win / 2 - 1) & 1), g.err, &abort_flag)) break;
      }
      if (!mbar_wait_or_abort(&ready_bar[u], (unsigned)((j / LS) & 1), g.err, &abort_flag)) break;
      tc_fence_after();
      const uint32_t d0 = tmem + (uint32_t)(2 * buf * g.N), d1 = d0 + (uint32_t)g.N;  // hi*hi, cross terms
      const uint32_t aH = smem_u32(splitA(u)), aL = aH + 128 * 128;
      const uint32_t bH = smem_u32(splitB(u));
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint32_t off = kk * 32;  // 8 TF32 values along K
        const uint32_t first = (j % TC_FLUSH == 0 && kk == 0) ? 0u : 1u;
        // [hi*hi | hi*lo] in one product of twice the width: B's lo tile follows its hi tile
        umma_tf32(d0, umma_desc_sw128(aH + off), umma_desc_sw128(bH + off), idesc2, first);
        umma_tf32(d1, umma_desc_sw128(aL + off), umma_desc_sw128(bH + off), idesc, 1u);
      }
      umma_commit(&empty_bar[u]);
      if (j % TC_FLUSH == TC_FLUSH - 1 || j == J - 1) umma_commit(&accf_bar[buf]);
    }
    // every MMA issued has completed before TMEM is released
    umma_commit(&done_bar);
    mbar_wait(&done_bar, 0u, g.err);
  } else if (warp >= 4) {
    // ------------------------------------------------ split pass + epilogue
    const int wt = tid - TC_ROLES;         // 0 .. TC_WORKERS - 1
    // warps 4-11: two per TMEM lane quarter, each reads half of a block's columns
    const bool epi = warp < 12;
    const int hg = (g.b_pad / 8 + 1) / 2;                       // column groups of 8 of the first half
    const int jb = warp < 8 ? 0 : 8 * hg;                       // first column of this warp
    const int jn = warp < 8 ? 8 * hg : g.b_pad - 8 * hg;        // and their number, at most BMAX
    const int m = (warp & 3) * 32 + lane;  // TMEM lane = accumulator row of this thread
    const int my_c = m / g.a_pad, my_i = m % g.a_pad;
    const bool owns_row = epi && my_c < g.s && my_i < g.a;
    float acc[BMAX], cmp[BMAX];  // Kahan sum and compensation per output column
#pragma unroll
    for (int j = 0; j < BMAX; ++j) acc[j] = cmp[j] = 0.f;
    auto kahan = [&](int j, float x) {
      const float y = x - cmp[j], t = acc[j] + y;
      cmp[j] = (t - acc[j]) - y;
      acc[j] = t;
    };
    // Worker group grp splits stages grp, grp + TC_GROUPS, ...  A thread of it takes one column group
    // (stack chunk bc, logical 16-byte chunk bjl: 4 points) and every rstep-th row of it, so each
    // weight is converted once per thread
    const int grp = wt / NG, gt = wt % NG;
    const int G = 8 * g.s;
    const int rstep = NG / G, r0 = gt / G;  // powers of two: G <= 128 = NG, rstep <= 8
    const int bc = (gt % G) >> 3, bjl = gt & 7;
    // weights of the thread's four points of a stage; zero past the grid, like the copied rows.  Read one
    // stage ahead, straight from memory (in the ring they would cost it a slot), and converted when used
    struct W4 {
      double2 lo, hi;
    };
    auto weights = [&](long long j) {
      const long long p = ((blockIdx.x + j * gridDim.x) * g.s + bc) * 32 + bjl * 4;
      W4 v = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
      if (g.w && j < J) {
        if (p + 4 <= g.n) {
          v.lo = __ldg(reinterpret_cast<const double2*>(g.w + p));
          v.hi = __ldg(reinterpret_cast<const double2*>(g.w + p) + 1);
        } else {
          if (p < g.n) v.lo.x = g.w[p];
          if (p + 1 < g.n) v.lo.y = g.w[p + 1];
          if (p + 2 < g.n) v.hi.x = g.w[p + 2];
        }
      }
      return v;
    };
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    // epilogue of window `win`: TMEM diagonal blocks -> compensated FP32 sums in registers
    auto flush = [&](long long win) -> bool {
      const int buf = (int)(win & 1);
      // lanes agree before the warp-collective TMEM loads (an abort may reach them unevenly)
      if (!__all_sync(0xffffffffu, mbar_wait_or_abort(&accf_bar[buf], (unsigned)((win / 2) & 1), g.err, &abort_flag)))
        return false;
      tc_fence_after();
      // the warp covers chunks c0 .. c0 + 32/a_pad - 1 (or one chunk when a_pad >= 32)
      const int wc0 = ((warp & 3) * 32) / g.a_pad;
      const int wcn = g.a_pad >= 32 ? 1 : 32 / g.a_pad;
      for (int cc = 0; cc < wcn; ++cc) {
        const int c = wc0 + cc;
        if (c >= g.s) break;  // warp-uniform
#pragma unroll
        for (int j0 = 0; j0 < BMAX; j0 += 8) {  // compile-time indices keep acc in registers
          if (j0 < jn) {
            float v0[8], v1[8];
            const uint32_t col = lane_base + (uint32_t)(2 * buf * g.N + c * g.b_pad + jb + j0);
            tmem_ld8(tmem + col, v0);
            tmem_ld8(tmem + col + (uint32_t)g.N, v1);
            tmem_ld_wait();
            if (owns_row && my_c == c) {
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                kahan(j0 + u, v0[u]);
                kahan(j0 + u, v1[u]);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acce_bar[buf]);
      return true;
    };
    // hi = x rounded to the nearest TF32 value (low 13 mantissa bits cleared), lo = x - hi
    auto split4 = [](float4 x, float4& h, float4& l) {
      h.x = __uint_as_float((__float_as_uint(x.x) + 0x1000u) & 0xFFFFE000u);
      h.y = __uint_as_float((__float_as_uint(x.y) + 0x1000u) & 0xFFFFE000u);
      h.z = __uint_as_float((__float_as_uint(x.z) + 0x1000u) & 0xFFFFE000u);
      h.w = __uint_as_float((__float_as_uint(x.w) + 0x1000u) & 0xFFFFE000u);
      l.x = x.x - h.x;
      l.y = x.y - h.y;
      l.z = x.z - h.z;
      l.w = x.w - h.w;
    };
    bool ok = true;
    long long fw = 0;  // windows read out so far
    W4 wnext = weights(grp);
    for (long long j = grp; j < J && ok; j += TC_GROUPS) {
      const int q = (int)(j % S), u = (int)(j % LS);
      // warp-uniform: every lane of a worker warp leaves the loop in the same stage
      bool go = j < LS || mbar_wait_or_abort(&empty_bar[u], (unsigned)((j / LS - 1) & 1), g.err, &abort_flag);
      go = go && mbar_wait_or_abort(&full_bar[q], (unsigned)((j / S) & 1), g.err, &abort_flag);
      if (!__all_sync(0xffffffffu, go)) {
        ok = false;
        break;
      }
      const float4 wv = g.w ? make_float4((float)wnext.lo.x, (float)wnext.lo.y, (float)wnext.hi.x, (float)wnext.hi.y)
                            : make_float4(1.f, 1.f, 1.f, 1.f);
      wnext = weights(j + TC_GROUPS);
      const float4* A4 = reinterpret_cast<const float4*>(slotA(q)) + bc * g.a_rows * 8;
      const float4* B4 = reinterpret_cast<const float4*>(slotB(q)) + bc * g.b_pad * 8;
      float4* A2 = reinterpret_cast<float4*>(splitA(u)) + bc * g.a_pad * 8;
      float4* B2 = reinterpret_cast<float4*>(splitB(u)) + bc * g.b_pad * 8;
#pragma unroll 4
      for (int r = r0; r < g.a_rows; r += rstep) {
        const int e = r * 8 + (bjl ^ (r & 7));  // physical 16-byte chunk (128-byte swizzle)
        float4 h, l;
        split4(A4[e], h, l);
        A2[e] = h;
        A2[128 * 8 + e] = l;
      }
#pragma unroll 4
      for (int r = r0; r < g.b_pad; r += rstep) {
        const int e = r * 8 + (bjl ^ (r & 7));
        float4 x = B4[e];
        x.x *= wv.x;
        x.y *= wv.y;
        x.z *= wv.z;
        x.w *= wv.w;
        float4 h, l;
        split4(x, h, l);
        B2[e] = h;
        B2[g.N * 8 + e] = l;
      }
      fence_proxy_async();  // generic-proxy writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&free_bar[q]);
        mbar_arrive(&ready_bar[u]);
      }
      // read out the finished windows once this group's first stage of the next one is handed over
      if (epi)
        for (; ok && fw < j / TC_FLUSH; ++fw) ok = flush(fw);
    }
    if (epi)
      for (; ok && J > 0 && fw <= (J - 1) / TC_FLUSH; ++fw) ok = flush(fw);
    // cross-chunk sum in shared memory (reuses the slots; every MMA has completed)
    named_bar_sync(1, TC_WORKERS);
    double* red = reinterpret_cast<double*>(base);
    if (owns_row) {
      double* row = red + ((size_t)my_c * g.a + my_i) * g.b;
#pragma unroll
      for (int x = 0; x < BMAX; ++x)
        if (x < jn && jb + x < g.b) row[jb + x] = (double)acc[x] - (double)cmp[x];
    }
    named_bar_sync(1, TC_WORKERS);
    double* pb = g.part + (long long)blockIdx.x * g.a * g.b;
    for (int e = wt; e < g.a * g.b; e += TC_WORKERS) {
      double v = 0.0;
      for (int c = 0; c < g.s; ++c) v += red[(size_t)c * g.a * g.b + e];
      pb[e] = abort_flag ? 0.0 : v;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

}  // namespace

int gram_tc_launch(long long n, int a, int b, const float* A, long long sa, const float* B, long long sb,
                   const double* w, double* part, int max_blocks, unsigned* err, cudaStream_t st) {
  GramTcPlan p;
  if (!plan_gram_tc(a, b, &p)) return -1;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (!al16(A) || !al16(B) || (w && !al16(w)) || (sa * 4) % 16 != 0 || (sb * 4) % 16 != 0) return -1;
  if (n < 32 || n >= (1LL << 31) - 4096) return -1;
  if (!err) return IGD_ERR_CUDA;
  CUtensorMap mA, mB;
  {
    const unsigned long long dims[2] = {(unsigned long long)n, (unsigned long long)a};
    const unsigned long long strides[1] = {(unsigned long long)sa * 4};
    const unsigned box[2] = {32, (unsigned)p.a_rows};
    if (!encode_tensor_map_ex(&mA, false, 2, A, dims, strides, box, true)) return -1;
  }
  {
    const unsigned long long dims[2] = {(unsigned long long)n, (unsigned long long)b};
    const unsigned long long strides[1] = {(unsigned long long)sb * 4};
    const unsigned box[2] = {32, (unsigned)p.b_pad};
    if (!encode_tensor_map_ex(&mB, false, 2, B, dims, strides, box, true)) return -1;
  }
  const int sms = device_sm_count();
  auto kern = p.b_pad > 32 ? gram_tc_kernel<32> : gram_tc_kernel<16>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), p.smem) != IGD_OK) return IGD_ERR_CUDA;
  GramTcArgs g;
  g.n = n;
  g.a = a;
  g.b = b;
  g.a_pad = p.a_pad;
  g.a_rows = p.a_rows;
  g.b_pad = p.b_pad;
  g.s = p.s;
  g.N = p.N;
  g.slots = p.slots;
  g.slot_bytes = (unsigned)p.slot_bytes;
  g.split_bytes = (unsigned)p.split_bytes;
  g.w = w;
  g.stages = (n + 32LL * p.s - 1) / (32LL * p.s);
  g.part = part;
  g.err = err;
  const int grid = (int)std::max<long long>(1, std::min<long long>({(long long)sms, g.stages, (long long)max_blocks}));
  kern<<<grid, TC_THREADS, p.smem, st>>>(mA, mB, g, (uint32_t)p.tmem_cols);
  return grid;
}

}  // namespace igd
