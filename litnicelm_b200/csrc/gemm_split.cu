// fp32-grade matrix products on the tensor cores for operands of any strides (sm_100a, tcgen05 + TMEM + TMA):
//     C[b] = A[b] B[b] (+ bias) (+ residual) (ReLU),    or C = sum over p of A[p] B[p]
// the products of the plugin table (litnicelm src/model/backend/device_backend.cpp:1096-1235) and of the 32-bit form of the
// registered designs, where they are large enough (gemm_f32_scratch_bytes).
//
// Two kernels. split_operands_kernel writes both operands in three bfloat16 parts, x = x0 + 2^-8 x1 + 2^-16 x2, each the part
// before it left over, rounded to nearest: all 24 bits of any finite x, since no part is smaller than bfloat16 can hold. The rows
// are K-major, which TMA can address whatever the operands' strides were. gemm_split_kernel adds the products of the parts,
// (1,2) (2,1) | (0,2) (1,1) (2,0) | (0,1) (1,0) in one accumulator, scaled by 2^-8 from one group to the next by the
// instruction that starts it, and (0,0) in another. What is left out, (2,2), is below 2^-32 of a product. The tensor pipe
// truncates when it accumulates, so a chain in tensor memory is one block of 64 k; the two accumulators are added, and the chains,
// in registers with rounding to nearest. A sum of one term is therefore rounded to within 2^-24 of itself as a fused multiply-add
// is, and exact where that is. Where an operand holds a value that is infinite, NaN or 2^63 and more the product is computed with
// plain fused multiply-adds in the order of k instead, so such values come out as they do there.
//
// gemm_split_kernel: persistent, one CTA of 10 warps per SM, tiles of 128 x BN:
//   warp 0      one lane issues the TMA loads (a ring of 2 or 3 stages of six operand tiles)
//   warp 1      owns tensor memory; one lane issues tcgen05.mma
//   warps 2-9   add finished chains (lane = row, half of the columns) and store the tile while the next one is multiplied
// Few tiles: k is cut into ranges, the CTAs of a tile form a cluster and each stores a share of the rows from the sums of all,
// read over distributed shared memory in rank order. Every wait is bounded.
//
// Bound: shared memory (a block of 64 k of a 128 x 128 tile is read 32 x 8 KB and written 96 KB, 2816 clocks at 128 bytes; 2930
// measured) and, for short k, the first loads and the last store of a CTA. 4096^3: 742 us, 185 TFLOP/s (41 on the tile kernel;
// 191 with operands as TF32 pairs, three products and 22 bits; 153 with blocks of 32 k in 64-byte rows). A training step of
// 8 x 250 tokens (width 512, two layers) takes 2.80 ms, 2.79 with pairs. Splitting inside the product's own loading warps instead
// of a kernel in front (one launch less) was slower with pairs, 52 us against 39 at 2000 x 1536 x 512: two loading warps per
// scheduler do not hide their latency, four leave too few registers.
#include "gemm_tc.cuh"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

namespace lb {

namespace {

constexpr int GS_BM = 128, GS_BK = 64, GS_SMS = 148;
constexpr int GS_ADDERS = 8;
constexpr int GS_THREADS = 64 + 32 * GS_ADDERS;

template <int BN>
struct GsSmem {
  static constexpr int STAGES = BN == 128 ? 2 : 3;
  static constexpr int CHAINS = 512 / (2 * BN);  // in flight, two accumulators each
  static constexpr int A_BYTES = GS_BM * 128;
  static constexpr int B_BYTES = BN * 128;
  static constexpr int STAGE = 3 * (A_BYTES + B_BYTES);
  static constexpr int LD = BN + 4;  // floats per row of a finished range of k, which overlays the stages
  static constexpr int PATCH_OFF = STAGES * STAGE;
  static constexpr int PIECES = BN / 32;  // 32 rows of as many float4s per adding warp
  static constexpr int BAR_OFF = PATCH_OFF + GS_ADDERS * 512 * PIECES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
  static_assert(GS_BM * LD * 4 <= STAGES * STAGE, "the finished range lies over the stages");
  static_assert(TOTAL <= 227 * 1024 && 8 * (2 * STAGES + 2 * CHAINS + 1) <= 192, "");
};

struct GsOperand {
  const float *p;
  long long outer, k;  // element strides
  int n;               // outer extent
  int vec;             // rows of k on 16-byte boundaries
  __nv_bfloat16 *part;  // [3][batch or 1][n][ld]
  long long each;       // elements of a part
  MatView view;        // batch axes
  int batch;
};

struct GsArgs {
  GsOperand a, b;
  float *c;
  const float *residual, *bias;
  long long c_rs, c_cs;
  int m, n, k, kp, sums;  // k of one summand, padded to a multiple of 64, and the number of summands
  int kblocks, relu, c_vec, splits, m_tiles, n_tiles, tiles;
  MatView cv;
  int *bad;  // [0] nonzero: an operand of this product holds a value that three parts cannot; [1] blocks that know. At rest zero
};

// x = x0 + 2^-8 x1 + 2^-16 x2, exactly: what a part leaves has at most 15, then 7 bits.
__device__ __forceinline__ void gs_split(float x, __nv_bfloat16 (&part)[3]) {
  part[0] = __float2bfloat16_rn(x);
  const float r = (x - __bfloat162float(part[0])) * 256.f;
  part[1] = __float2bfloat16_rn(r);
  part[2] = __float2bfloat16_rn((r - __bfloat162float(part[1])) * 256.f);
}

// Infinite, not a number, or from 2^63 on: products of lesser ones leave the accumulator of the scaled parts, which reaches twice
// the product, in range.
__device__ __forceinline__ bool gs_no_parts(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x5f000000u; }

// One tile of 32 rows x 64 k of one operand: read along whichever axis is contiguous, written as rows of k, 16 bytes of a part at a
// time (a thread: eight k of one row).
constexpr int GS_SPLIT_ROWS = 32;
__global__ void __launch_bounds__(256) split_operands_kernel(const __grid_constant__ GsArgs g, int a_blocks) {
  __shared__ float tile[GS_SPLIT_ROWS][65];
  pdl_launch_dependents();
  pdl_wait();
  const bool first = (int)blockIdx.x < a_blocks;
  const GsOperand &o = first ? g.a : g.b;
  const int k_tiles = (g.kp + 63) / 64, r_tiles = (o.n + GS_SPLIT_ROWS - 1) / GS_SPLIT_ROWS;
  int at = (int)blockIdx.x - (first ? 0 : a_blocks);
  const int k0 = at % k_tiles * 64;
  at /= k_tiles;
  const int r0 = at % r_tiles * GS_SPLIT_ROWS, batch = at / r_tiles, tid = threadIdx.x;
  const float *src = reinterpret_cast<const float *>(reinterpret_cast<const char *>(o.p) + batch_offset(o.view, batch));
  const long long ld = (long long)g.kp * g.sums;
  const long long to0 = g.sums > 1 ? (long long)batch * g.kp : (long long)batch * o.n * ld;
  float x[8];
  const int row = tid >> 3, k = k0 + (tid & 7) * 8, r = r0 + row;
  if (o.vec && o.k == 1) {
    const float *p = src + (long long)r * o.outer + k;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < o.n) {
        if (k + h + 4 <= g.k) {
          v = *reinterpret_cast<const float4 *>(p + h);
        } else {
          if (k + h < g.k) v.x = p[h];
          if (k + h + 1 < g.k) v.y = p[h + 1];
          if (k + h + 2 < g.k) v.z = p[h + 2];
        }
      }
      x[h] = v.x; x[h + 1] = v.y; x[h + 2] = v.z; x[h + 3] = v.w;
    }
  } else {
    const bool along_k = o.k == 1;
    float t[GS_SPLIT_ROWS / 4];
#pragma unroll
    for (int i = 0; i < GS_SPLIT_ROWS / 4; ++i) {
      const int e = tid + i * 256;
      const int rr = along_k ? e >> 6 : e % GS_SPLIT_ROWS, kk = along_k ? e & 63 : e / GS_SPLIT_ROWS;
      t[i] = r0 + rr < o.n && k0 + kk < g.k ? src[(long long)(r0 + rr) * o.outer + (long long)(k0 + kk) * o.k] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < GS_SPLIT_ROWS / 4; ++i) {
      const int e = tid + i * 256;
      tile[along_k ? e >> 6 : e % GS_SPLIT_ROWS][along_k ? e & 63 : e / GS_SPLIT_ROWS] = t[i];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = tile[row][(tid & 7) * 8 + j];
  }
  bool bad = false;
  if (r < o.n) {
    __nv_bfloat16 part[8][3];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      bad |= gs_no_parts(x[j]);
      gs_split(x[j], part[j]);
    }
    const long long to = to0 + (long long)r * ld + k;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      unsigned w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 two{part[2 * j][q], part[2 * j + 1][q]};
        w[j] = *reinterpret_cast<const unsigned *>(&two);
      }
      *reinterpret_cast<uint4 *>(o.part + q * o.each + to) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  if (bad) *g.bad = 1;
}

// Four results of a row, from column col on, through the epilogue to C.
__device__ __forceinline__ void gs_store4(const GsArgs &g, float *C, const float *R, int row, int col, float4 x) {
  float v[4] = {x.x, x.y, x.z, x.w};
  const long long at = (long long)row * g.c_rs;
  if (g.c_vec && col + 3 < g.n) {
    if (g.bias) {
      const float4 t = *reinterpret_cast<const float4 *>(g.bias + col);
      v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
    }
    if (R) {
      const float4 t = *reinterpret_cast<const float4 *>(R + at + col);
      v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
    }
    if (g.relu) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
    }
    *reinterpret_cast<float4 *>(C + at + col) = make_float4(v[0], v[1], v[2], v[3]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (col + j >= g.n) break;
    const long long to = at + (long long)(col + j) * g.c_cs;
    float o = v[j];
    if (g.bias) o += g.bias[col + j];
    if (R) o += R[to];
    if (g.relu) o = o > 0.f ? o : 0.f;
    C[to] = o;
  }
}

// D = A B, D += A B, or D = 2^-8 D + A B.
constexpr int GS_NEW = 0, GS_ADD = 1, GS_SCALED = 2;
__device__ __forceinline__ void gs_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, int how) {
  if (how == GS_SCALED)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 8;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc)
        : "memory");
  else
    tc_mma_f16(d, a, b, idesc, how == GS_ADD ? 1u : 0u);
}

struct GsMaps {
  CUtensorMap a[3], b[3];
};

// A tile of the product without parts, rows m0 .. m_end - 1: fused multiply-adds in the order of k, as in gemm_simt.cu. 256
// threads with 4 H x BN / 16 elements each (H = 1: up to 64 rows), 16 of k at a time through two buffers of shared memory, the next
// 16 on their way in registers. All threads of the block come here. A value the parts cannot hold may be in all operands of a step that
// has diverged, so this is about as fast as gemm_simt.cu (2000 x 512 x 2048: 187 us, there 175; 300 x 200 x 512: 34 and 33; 4096 x
// 4096 x 1024: 1270 and 865).
template <int BN, int H>
__device__ __noinline__ void gs_plain_tile(const GsArgs &g, float *sm, int batch, int m0, int m_end, int n0) {
  constexpr int PK = 16, BM = 64 * H, LDA = BM + 4, LDB = BN + 4, TM = 4 * H, TN = BN / 16;
  constexpr int NA = BM * PK / 256, NB = BN * PK / 256;
  float *as = sm, *bs = sm + 2 * PK * LDA;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const bool on = tid < 256;
  const int per = (g.k + PK - 1) / PK, trips = per * g.sums;
  // A thread's share: elements i of a column of places one step apart, lanes along whichever axis is contiguous
  const bool a_k = g.a.k == 1, b_k = g.b.k == 1;
  const int ar = a_k ? tid / PK : tid % BM, ak = a_k ? tid % PK : tid / BM, ar1 = a_k ? 256 / PK : 0, ak1 = a_k ? 0 : 256 / BM;
  const int br = b_k ? tid / PK : tid % BN, bk = b_k ? tid % PK : tid / BN, br1 = b_k ? 256 / PK : 0, bk1 = b_k ? 0 : 256 / BN;
  const long long a_step = ar1 * g.a.outer + ak1 * g.a.k, b_step = br1 * g.b.outer + bk1 * g.b.k;
  const long long a_at = (long long)(m0 + ar) * g.a.outer + ak * g.a.k, b_at = (long long)(n0 + br) * g.b.outer + bk * g.b.k;
  const float *x = nullptr, *y = nullptr;
  int left = 0, of = 0;  // of k in this summand
  float ra[NA], rb[NB];
  auto load = [&]() {
    if (left <= 0) {  // the next summand
      const long long at = g.sums > 1 ? of++ : batch;
      x = reinterpret_cast<const float *>(reinterpret_cast<const char *>(g.a.p) + batch_offset(g.a.view, at)) + a_at;
      y = reinterpret_cast<const float *>(reinterpret_cast<const char *>(g.b.p) + batch_offset(g.b.view, at)) + b_at;
      left = g.k;
    }
#pragma unroll
    for (int i = 0; i < NA; ++i) ra[i] = m0 + ar + i * ar1 < m_end && ak + i * ak1 < left ? x[i * a_step] : 0.f;
#pragma unroll
    for (int i = 0; i < NB; ++i) rb[i] = n0 + br + i * br1 < g.n && bk + i * bk1 < left ? y[i * b_step] : 0.f;
    x += PK * g.a.k;
    y += PK * g.b.k;
    left -= PK;
  };
  float acc[TM][TN] = {};
  if (on) load();
  for (int t = 0; t < trips; ++t) {
    float *at = as + (t & 1) * PK * LDA, *bt = bs + (t & 1) * PK * LDB;
    if (on) {
#pragma unroll
      for (int i = 0; i < NA; ++i) at[(ak + i * ak1) * LDA + ar + i * ar1] = ra[i];
#pragma unroll
      for (int i = 0; i < NB; ++i) bt[(bk + i * bk1) * LDB + br + i * br1] = rb[i];
    }
    __syncthreads();  // (a buffer is written again only behind the barrier of the trip after)
    if (!on) continue;
    if (t + 1 < trips) load();
#pragma unroll
    for (int kk = 0; kk < PK; ++kk) {
      float u[TM], v[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 f = *reinterpret_cast<const float4 *>(at + kk * LDA + i / 4 * 64 + ty * 4);
        u[i] = f.x; u[i + 1] = f.y; u[i + 2] = f.z; u[i + 3] = f.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 f = *reinterpret_cast<const float4 *>(bt + kk * LDB + j / 4 * 64 + tx * 4);
        v[j] = f.x; v[j + 1] = f.y; v[j + 2] = f.z; v[j + 3] = f.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(u[i], v[j], acc[i][j]);
    }
  }
  if (on) {
    const long long c_off = batch_offset(g.cv, batch);
    float *C = reinterpret_cast<float *>(reinterpret_cast<char *>(g.c) + c_off);
    const float *R = g.residual ? reinterpret_cast<const float *>(reinterpret_cast<const char *>(g.residual) + c_off) : nullptr;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const int row = m0 + i / 4 * 64 + ty * 4 + (i & 3), col = n0 + j / 4 * 64 + tx * 4;
        if (row < m_end && col < g.n)
          gs_store4(g, C, R, row, col, make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]));
      }
  }
  __syncthreads();  // the buffers are free for the next tile
}

template <int BN>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_split_kernel(const __grid_constant__ GsMaps maps, const __grid_constant__ GsArgs g, DevErr *err) {
  using L = GsSmem<BN>;
  constexpr int S = L::STAGES, CHAINS = L::CHAINS, CW = BN / 2;  // columns of an adding warp
  extern __shared__ unsigned char smem_raw[];
  const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const unsigned bars = base + L::BAR_OFF;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (S + s); };
  auto chain_full = [&](int b) { return bars + 8u * (2 * S + b); };
  auto chain_empty = [&](int b) { return bars + 8u * (2 * S + CHAINS + b); };
  const unsigned done = bars + 8u * (2 * S + 2 * CHAINS);
  volatile unsigned *tmem_holder = reinterpret_cast<volatile unsigned *>(base_ptr + L::BAR_OFF + 192);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(base_ptr + L::BAR_OFF + 196);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)blockIdx.x % g.splits, cta = (int)blockIdx.x / g.splits, ctas = (int)gridDim.x / g.splits;
  const int each = (g.kblocks + g.splits - 1) / g.splits;
  const int first = min(g.kblocks, rank * each), count = min(g.kblocks, first + each) - first;
  auto place = [&](int tile, int &batch, int &m0, int &n0) {
    const int per = g.m_tiles * g.n_tiles, rest = tile % per;
    batch = tile / per;
    m0 = rest % g.m_tiles * GS_BM;
    n0 = rest / g.m_tiles * BN;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < CHAINS; ++b) {
      mbar_init(chain_full(b), 1);
      mbar_init(chain_empty(b), GS_ADDERS);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_holder)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_holder;
  pdl_launch_dependents();
  pdl_wait();
  const bool plain = *static_cast<const volatile int *>(g.bad) != 0;

  if (plain) {  // the CTAs of a tile take a share of its rows each
    __syncthreads();
    if (threadIdx.x == 0) {  // the last block to have seen the mark takes it away: the next product, or replay, starts without
      __threadfence();
      if (atomicInc(reinterpret_cast<unsigned *>(g.bad) + 1, gridDim.x - 1) == gridDim.x - 1) *static_cast<volatile int *>(g.bad) = 0;
    }
    const int share = (GS_BM + g.splits - 1) / g.splits;
    for (int tile = cta; tile < g.tiles; tile += ctas) {
      int batch, m0, n0;
      place(tile, batch, m0, n0);
      const int row = m0 + rank * share;
      const int end = min(g.m, min(m0 + GS_BM, row + share));
      float *sm = reinterpret_cast<float *>(base_ptr);
      if (end - row <= 64) gs_plain_tile<BN, 1>(g, sm, batch, row, end, n0);
      else gs_plain_tile<BN, 2>(g, sm, batch, row, end, n0);
    }
  } else if (warp == 0) {
    int it = 0;
    bool ok = true;
    for (int tile = cta; tile < g.tiles && ok; tile += ctas) {
      int batch, m0, n0;
      place(tile, batch, m0, n0);
      if (g.sums == 1) {
        m0 += batch * g.m;
        if (g.b.batch > 1) n0 += batch * g.n;
      }
      for (int kb = first; kb < first + count; ++kb, ++it) {
        const int s = it % S;
        ok = mbar_wait_warp(empty(s), ((unsigned)(it / S) & 1u) ^ 1u, abort_flag, err, 51);
        if (!ok) break;
        if (lane == 0) {
          const unsigned st = base + (unsigned)(s * L::STAGE);
          mbar_expect_tx(full(s), (unsigned)L::STAGE);
#pragma unroll
          for (int q = 2; q >= 0; --q) {
            tma_load_2d(st + q * L::A_BYTES, &maps.a[q], kb * GS_BK, m0, full(s));
            tma_load_2d(st + 3 * L::A_BYTES + q * L::B_BYTES, &maps.b[q], kb * GS_BK, n0, full(s));
          }
        }
        __syncwarp();
      }
    }
    if (*abort_flag) {  // copies in flight must land before the shared memory goes away
      for (int j = it > S ? it - S : 0; j < it; ++j) {
        const unsigned long long t0 = global_timer();
        while (!mbar_try_wait(full(j % S), (unsigned)(j / S) & 1u))
          if (global_timer() - t0 > WAIT_LIMIT_NS) break;
      }
    }
  } else if (warp == 1) {
    constexpr unsigned idesc = umma_idesc_bf16(BN);
    int it = 0;
    bool ok = true;
    for (int tile = cta; tile < g.tiles && ok; tile += ctas) {
      for (int kb = 0; kb < count; ++kb, ++it) {
        const int s = it % S, buf = it % CHAINS;
        ok = mbar_wait_warp(chain_empty(buf), ((unsigned)(it / CHAINS) & 1u) ^ 1u, abort_flag, err, 52) &&
             mbar_wait_warp(full(s), (unsigned)(it / S) & 1u, abort_flag, err, 53);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lane == 0) {
          const unsigned st = base + (unsigned)(s * L::STAGE), d = tmem + (unsigned)(buf * 2 * BN);
          auto times = [&](unsigned to, int i, int j, int start) {  // 64 k of parts i and j; start: see gs_mma
            const unsigned long long a = umma_desc_k128(st + i * L::A_BYTES),
                                     b = umma_desc_k128(st + 3 * L::A_BYTES + j * L::B_BYTES);
            gs_mma(to, a, b, idesc, start);
#pragma unroll
            for (unsigned ks = 2; ks < 8; ks += 2) gs_mma(to, a + ks, b + ks, idesc, GS_ADD);
          };
          times(d + BN, 1, 2, GS_NEW);
          times(d + BN, 2, 1, GS_ADD);
          times(d + BN, 0, 2, GS_SCALED);
          times(d + BN, 1, 1, GS_ADD);
          times(d + BN, 2, 0, GS_ADD);
          times(d + BN, 0, 1, GS_SCALED);
          times(d + BN, 1, 0, GS_ADD);
          times(d, 0, 0, GS_NEW);
          tc_commit(empty(s));
          tc_commit(chain_full(buf));
        }
        __syncwarp();
      }
    }
    if (!ok) {  // what was issued ends, within the limit, before the shared memory goes away
      if (lane == 0) tc_commit(done);
      __syncwarp();
      const unsigned long long t0 = global_timer();
      while (!mbar_try_wait(done, 0u))
        if (global_timer() - t0 > WAIT_LIMIT_NS) break;
    }
  } else {
    constexpr int PIECES = L::PIECES, ROWS = 32 / PIECES;  // a warp stores ROWS rows at a time
    const int q = warp & 3, half = (warp - 2) >> 2, piece = lane % PIECES;
    auto turned = [](int row) { return PIECES == 4 ? (row >> 1) & 3 : (row >> 2) & 1; };  // distinct banks
    float4 *patch = reinterpret_cast<float4 *>(base_ptr + L::PATCH_OFF) + (warp - 2) * (32 * PIECES);
    int it = 0;
    bool ok = true;
    for (int tile = cta; tile < g.tiles && ok; tile += ctas) {
      float acc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) acc[j] = 0.f;
      for (int kb = 0; kb < count; ++kb, ++it) {
        const int buf = it % CHAINS;
        ok = mbar_wait_warp(chain_full(buf), (unsigned)(it / CHAINS) & 1u, abort_flag, err, 54);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < CW; c0 += 32) {
          unsigned r[32], t[32];
          tc_ld32(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(buf * 2 * BN + half * CW + c0), r);
          tc_ld32(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(buf * 2 * BN + BN + half * CW + c0), t);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j)
            acc[c0 + j] = __fadd_rn(acc[c0 + j], __fmaf_rn(__uint_as_float(t[j]), 0x1p-8f, __uint_as_float(r[j])));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(chain_empty(buf));
      }
      if (g.splits > 1) {  // every product has been read: the range's sums may lie over the stages
        float *sums = reinterpret_cast<float *>(base_ptr) + (q * 32 + lane) * L::LD + half * CW;
#pragma unroll
        for (int j = 0; j < CW; j += 4)
          *reinterpret_cast<float4 *>(sums + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        break;
      }
      int batch, m0, n0;
      place(tile, batch, m0, n0);
      const long long c_off = batch_offset(g.cv, batch);
      float *C = reinterpret_cast<float *>(reinterpret_cast<char *>(g.c) + c_off);
      const float *R = g.residual ? reinterpret_cast<const float *>(reinterpret_cast<const char *>(g.residual) + c_off) : nullptr;
#pragma unroll
      for (int c0 = 0; c0 < CW; c0 += 4 * PIECES) {  // turned so that PIECES lanes store a row's bytes
#pragma unroll
        for (int j = 0; j < PIECES; ++j)
          patch[lane * PIECES + (j ^ turned(lane))] =
              make_float4(acc[c0 + 4 * j], acc[c0 + 4 * j + 1], acc[c0 + 4 * j + 2], acc[c0 + 4 * j + 3]);
        __syncwarp();
        const int col = n0 + half * CW + c0 + piece * 4;
#pragma unroll 1
        for (int pass = 0; pass < PIECES; ++pass) {
          const int rr = pass * ROWS + lane / PIECES, row = m0 + q * 32 + rr;
          if (row >= g.m || col >= g.n) continue;
          gs_store4(g, C, R, row, col, patch[rr * PIECES + (piece ^ turned(rr))]);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if (g.splits > 1 && !plain) {  // one tile, its ranges of k over the CTAs of the cluster
    cluster_sync_all();
    int batch, m0, n0;
    place(cta, batch, m0, n0);
    const long long c_off = batch_offset(g.cv, batch);
    float *C = reinterpret_cast<float *>(reinterpret_cast<char *>(g.c) + c_off);
    const float *R = g.residual ? reinterpret_cast<const float *>(reinterpret_cast<const char *>(g.residual) + c_off) : nullptr;
    const int rows_each = (GS_BM + g.splits - 1) / g.splits;
    const int row_end = min(min(GS_BM, (rank + 1) * rows_each), g.m - m0);
    constexpr int LANES = BN / 4;  // threads to a row
    const int c4 = ((int)threadIdx.x % LANES) * 4, col = n0 + c4;
    for (int row = rank * rows_each + (int)threadIdx.x / LANES; row < row_end && col < g.n; row += GS_THREADS / LANES) {
      const unsigned at = base + (unsigned)(row * L::LD + c4) * 4u;
      float4 x = ld_cluster_f4(cluster_map(at, 0u));
      for (int r = 1; r < g.splits; ++r) {
        const float4 y = ld_cluster_f4(cluster_map(at, (unsigned)r));
        x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
      }
      gs_store4(g, C, R, m0 + row, col, x);
    }
    __syncwarp();
    cluster_sync_all();  // no peer reads these sums any more
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

bool on16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

bool batch_on16(const MatView &v) {
  for (int i = 0; i < v.nb; ++i)
    if ((v.bs[i] & 15) != 0) return false;
  return true;
}

GsOperand operand(const MatView &v, long long outer, long long k, int n) {
  GsOperand o{};
  o.p = reinterpret_cast<const float *>(v.data);
  o.outer = outer / 4;
  o.k = k / 4;
  o.n = n;
  o.vec = on16(v.data) && batch_on16(v) && (o.outer & 3) == 0;
  o.view = v;
  o.batch = (int)v.batch;
  return o;
}

// The innermost batch axis becomes rows where it continues them in both operands.
void fold(MatView &a, MatView &c) {
  while (a.nb > 0 && a.nb == c.nb && a.bd[a.nb - 1] == c.bd[c.nb - 1] && a.bs[a.nb - 1] == a.rows * a.rs &&
         c.bs[c.nb - 1] == c.rows * c.rs && a.rows * a.bd[a.nb - 1] < (1ll << 30)) {
    const long long n = a.bd[a.nb - 1];
    for (MatView *v : {&a, &c}) {
      v->rows *= n;
      v->batch /= n;
      --v->nb;
    }
  }
}

void turn(MatView &v) {
  std::swap(v.rows, v.cols);
  std::swap(v.rs, v.cs);
}

// Tile width and ranges of k by the time of the longest CTA: blocks of 64 k at what they were measured to take (in clocks: 2930
// at 128 columns, 2450 at 64), the store of the last tile, and for ranges the exchange of their sums. The clusters of a tile's
// ranges sit inside a GPC each; more of them than fit at once take a second wave (512 x 1536 x 2000: 48 clusters of three 55.8 us,
// of two 40.4; 613 x 512 x 2048: 20 of six 23.2, of eight 35.5).
struct Plan {
  int bn, splits, tiles;
};
Plan make_plan(long long batch, int m, int n, int kblocks) {
  Plan best{64, 1, 0};
  double least = 1e30;
  const long long mt = (m + GS_BM - 1) / GS_BM;
  const int *fit = tc_cluster_capacity();
  for (int bn : {64, 128}) {
    if (bn == 128 && n <= 64) continue;
    const long long tiles = batch * mt * ((n + bn - 1) / bn);
    if (tiles > (1 << 30)) throw std::invalid_argument("litnice_b200: product too large");
    const double block = bn == 128 ? 2930 : 2450;
    for (int s = 1; s <= 8; ++s) {
      if (s > 1 && (tiles * s > GS_SMS || kblocks < 2 * s)) break;
      if (s > 1 && fit[s] <= 0) continue;
      const int each = (kblocks + s - 1) / s;
      if ((kblocks + each - 1) / each != s) continue;  // no empty range
      const double waves = (double)(s > 1 ? (tiles + fit[s] - 1) / fit[s] : (tiles + GS_SMS - 1) / GS_SMS);
      const double t = waves * each * block + 3000 + (s > 1 ? 2500 + 500 * s : 0);
      if (t < least) {
        least = t;
        best = Plan{bn, s, (int)tiles};
      }
    }
  }
  return best;
}

template <int BN>
void launch_tile(const GsArgs &g, bool pdl, cudaStream_t st, DevErr *err) {
  GsMaps maps;
  const unsigned long long ld = (unsigned long long)g.kp * g.sums;
  const unsigned long long ra = (unsigned long long)g.m * (g.sums > 1 ? 1 : g.a.batch), rb = (unsigned long long)g.n * (g.sums > 1 ? 1 : g.b.batch);
  for (int q = 0; q < 3; ++q) {
    tc_make_map_bf16(&maps.a[q], g.a.part + q * g.a.each, ra, ld, ld, GS_BM);
    tc_make_map_bf16(&maps.b[q], g.b.part + q * g.b.each, rb, ld, ld, BN);
  }
  LB_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, GsSmem<BN>::TOTAL));
  const int ctas = g.splits > 1 || g.tiles < GS_SMS ? g.tiles : GS_SMS;
  launch_pdl_cluster_x(gemm_split_kernel<BN>, dim3((unsigned)(ctas * g.splits)), dim3(GS_THREADS), (size_t)GsSmem<BN>::TOTAL,
                       st, pdl, (unsigned)g.splits, maps, g, err);
}

// Rows of each A that one launch takes, by which the parts' memory is sized too: of a single matrix at most GS_ROWS, which
// bounds that memory; of batches and sums all.
constexpr long long GS_ROWS = 16384;
long long rows_at_once(long long m, long long a_batch, bool sum_batches) {
  return a_batch > 1 || sum_batches || m < GS_ROWS ? m : GS_ROWS;
}

void launch_gemm_split(MatView a, MatView b, MatView c, bool sum_batches, const GemmEpilogue &ep, void *scratch,
                       bool pdl, cudaStream_t st, DevErr *err) {
  GsArgs g{};
  g.m = (int)a.rows;
  g.n = (int)b.cols;
  g.k = (int)a.cols;
  g.kp = (g.k + GS_BK - 1) / GS_BK * GS_BK;
  g.sums = sum_batches ? (int)a.batch : 1;
  g.a = operand(a, a.rs, a.cs, g.m);
  g.b = operand(b, b.cs, b.rs, g.n);
  g.bad = static_cast<int *>(scratch);
  g.a.each = (long long)g.m * g.kp * g.a.batch;
  g.b.each = (long long)g.n * g.kp * g.b.batch;
  g.a.part = reinterpret_cast<__nv_bfloat16 *>(static_cast<char *>(scratch) + 256);
  g.b.part = g.a.part + 3 * g.a.each;
  g.c = reinterpret_cast<float *>(c.data);
  g.residual = ep.residual;
  g.bias = ep.bias;
  g.relu = ep.relu;
  g.c_rs = c.rs / 4;
  g.c_cs = c.cs / 4;
  g.cv = c;
  g.c_vec = g.c_cs == 1 && (g.c_rs & 3) == 0 && on16(c.data) && batch_on16(c) && (!ep.residual || on16(ep.residual)) &&
            (!ep.bias || on16(ep.bias));
  g.kblocks = g.kp / GS_BK * g.sums;
  const Plan plan = make_plan(c.batch, g.m, g.n, g.kblocks);
  g.splits = plan.splits;
  g.tiles = plan.tiles;
  g.m_tiles = (g.m + GS_BM - 1) / GS_BM;
  g.n_tiles = (g.n + plan.bn - 1) / plan.bn;
  const long long k_tiles = (g.kp + 63) / 64;
  const long long a_blocks = (g.m + GS_SPLIT_ROWS - 1) / GS_SPLIT_ROWS * k_tiles * g.a.batch;
  const long long b_blocks = (g.n + GS_SPLIT_ROWS - 1) / GS_SPLIT_ROWS * k_tiles * g.b.batch;
  launch_pdl(split_operands_kernel, dim3((unsigned)(a_blocks + b_blocks)), dim3(256), 0, st, pdl, g, (int)a_blocks);
  if (plan.bn == 128) launch_tile<128>(g, pdl, st, err);
  else launch_tile<64>(g, pdl, st, err);
}

}  // namespace

SplitScratch::~SplitScratch() { give_back(); }

void SplitScratch::give_back() {
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

bool SplitScratch::ensure(size_t need, cudaStream_t st) {
  if (need <= bytes) return true;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone) return false;
  // Products come in all sizes: with room for the largest so far alone, a first training step stopped for a new allocation a
  // dozen times (each waits for the stream). So the first is generous and the others double, up to a gigabyte.
  size_t grown = need + need / 4;
  const size_t room = bytes ? (bytes < (size_t)512 << 20 ? 2 * bytes : (size_t)1 << 30) : least;
  if (grown < room) grown = room;
  if (p) {
    LB_CUDA(cudaStreamSynchronize(st));
    give_back();
  }
  while (cudaMalloc(&p, grown) != cudaSuccess) {
    p = nullptr;
    (void)cudaGetLastError();
    if (grown == need) return false;
    grown = need;
  }
  bytes = grown;
  LB_CUDA(cudaMemsetAsync(p, 0, 256, st));
  return true;
}

// Measured on one B200, both ways, calls back to back in us (tile kernel -> two launches here): 128 x 128 x 128 10 -> 10,
// 256 x 256 x 256 17 -> 10.5, 250 x 250 x 250 of 8 batches 19.5 -> 17, 64 x 512 x 512 31 -> 11, 613 x 3072 x 512 83 -> 25,
// 2000 x 512 x 2048 174 -> 40, 4096^3 3352 -> 742. The tile kernel is bound by the latency of its k loop (0.05 us a k) where there
// are few tiles and by the FMA pipe where there are many; here the two launches cost about 8 us where they are short (the split
// alone takes 14 us on average in a training step, of which it writes a third more than it reads) and a block of 64 k 1.5 us. Few
// rows against a large matrix: splitting the matrix costs more than reading it (16 x 32000 x 1024 would write 196 MB). Errors
// against 64-bit sums, 2-norm (tile kernel, here): k = 256 2.9e-7, 8.0e-8; k = 2048 8.1e-7, 9.9e-8, on operands of one sign 7.0e-7,
// 9.2e-8, on factors over twelve decades 3.5e-7, 1.3e-7. Below 128 k the tile kernel is near enough and faster.
size_t gemm_f32_scratch_bytes(long long m, long long n, long long k, long long a_batch, long long b_batch, bool sum_batches) {
  const long long batch = a_batch, total_k = sum_batches ? k * a_batch : k;
  if (m <= 0 || n <= 0 || k <= 0 || batch <= 0) return 0;
  const double work = (double)m * n * k * batch;
  if (total_k < 128) return 0;
  if (work < 1 << 24 && !(total_k >= 256 && work >= 1 << 21)) return 0;
  const double small = (double)(m < n ? m : n);
  if (small < 64 && (double)(m < n ? n : m) * k > 4e6) return 0;
  const long long kp = (k + GS_BK - 1) / GS_BK * GS_BK;
  if ((double)m * a_batch > 1e9 || (double)n * b_batch > 1e9 || (double)kp * (sum_batches ? a_batch : 1) > 1e9) return 0;
  const double parts = 3.0 * kp * ((double)rows_at_once(m, a_batch, sum_batches) * a_batch + (double)n * b_batch);
  if (parts * 2 > 4e9) return 0;
  return (size_t)parts * 2 + 256;
}

size_t gemm_f32_scratch_bytes(MatView a, const MatView &b, MatView c) {
  if (b.batch == 1) fold(a, c);
  return gemm_f32_scratch_bytes(a.rows, b.cols, a.cols, a.batch, b.batch, false);
}

int launch_gemm_f32(const MatView &a, const MatView &b, const MatView &c, bool sum_batches, const GemmEpilogue &ep,
                    SplitScratch &scratch, cudaStream_t st, DevErr *err) {
  if (a.rows <= 0 || b.cols <= 0) return 0;
  MatView fa = a, fb = b, fc = c;
  if (sum_batches) {  // summands may lie one behind another along k
    turn(fa);
    fold(fa, fb);
    turn(fa);
  } else if (b.batch == 1) {
    fold(fa, fc);
  }
  const size_t need = gemm_f32_scratch_bytes(fa.rows, fb.cols, fa.cols, fa.batch, fb.batch, sum_batches);
  if (need > 0 && scratch.ensure(need, st)) {
    int launched = 0;
    const long long part = rows_at_once(fa.rows, fa.batch, sum_batches);
    for (long long r = 0; r < fa.rows; r += part) {
      MatView pa = fa, pc = fc;
      pa.rows = pc.rows = fa.rows - r < part ? fa.rows - r : part;
      pa.data += r * fa.rs;
      pc.data += r * fc.rs;
      GemmEpilogue pe = ep;
      if (pe.residual) pe.residual = reinterpret_cast<const float *>(reinterpret_cast<const char *>(pe.residual) + r * fc.rs);
      launch_gemm_split(pa, fb, pc, sum_batches, pe, scratch.p, scratch.pdl || g_pdl_enabled, st, err);
      launched += 2;
    }
    return launched;
  }
  if (!sum_batches) {
    launch_gemm_simt(a, b, c, c.rows, c.cols, a.cols, ep, st);
    return 1;
  }
  for (long long p = 0; p < a.batch; ++p) {  // each summand added to the sum of those before it
    MatView ap = a, bp = b;
    ap.data += batch_offset(a, p);
    bp.data += batch_offset(b, p);
    ap.nb = bp.nb = 0;
    ap.batch = bp.batch = 1;
    GemmEpilogue pe = ep;
    if (p > 0) pe.residual = reinterpret_cast<const float *>(c.data);  // in place: every element by one thread
    launch_gemm_simt(ap, bp, c, c.rows, c.cols, a.cols, pe, st);
  }
  return (int)a.batch;
}

}  // namespace lb
