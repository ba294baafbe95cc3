// Matrix products on bfloat16 operands for sm_100a (tcgen05 + TMEM + TMA): C[m, n] = A[m, k] W[n, k]^T
// with 32-bit accumulation. The many-row counterpart of few_row_bf16.cu.
//
// Persistent kernel, one CTA per SM, tiles of 128 x BN taken round robin:
//   warp 0      one lane issues the TMA loads of the A and W tiles (64 k per stage, 128-byte swizzle)
//   warp 1      owns tensor memory (two accumulators of BN columns); one lane issues tcgen05.mma
//   warps 2-9   read a finished accumulator and store the tile while the next one is multiplied: two warps
//               to each 32 rows, 32 columns at a time through a swizzled shared-memory patch that a TMA store
//               (or, for results that are added, a TMA reduction) carries out, clipped at the result's edges
// Bound: the tensor pipe for long k (an instruction of 128 x 256 x 16 takes about 160 clocks), the store for short k and
// for GELU (erff: about 35 instructions an element). The store used to be four warps with whole-row global accesses behind a
// padded patch, residuals read back inside it: about 12 us a tile of 128 x 256 whatever the activation, against 1 us of
// products at k = 256 and 4 us at k = 1024. Prompts of 4 x 2048 tokens through six Mitilix layers of width 1024, 30 of these
// products: 3.06 ms a pass before, 1.97 ms with eight warps and TMA stores.
// Long k is bound by shared memory too: an instruction of 128 x 256 reads 384 operand rows of its SM for 128 x 256 products a k.
// A pair of CTAs (cta_group::2) takes tiles of 256 x 256 instead, each CTA loading its 128 rows of A and 128 of W's 256, two
// thirds of the operand bytes, with six stages in place of four; each stores its own 128 rows. The even CTA issues the
// instructions of both and owns the barriers they wait on; commits arrive in both. Where activations make the store the longer
// part, sixteen warps store. Mitilix 4 x 2048 (above) 1.897 -> 1.801 ms, Gobesun 4 x 2047 2.571 -> 2.471 ms.
// A launch may begin while its predecessor ends (its dependents are let go behind the allocation of tensor memory, so a CTA
// never waits for tensor memory that a later launch holds).
// Rows and columns outside the operands load as zeros (k need not be a multiple of 64) and are not
// stored. Every mbarrier wait is bounded; a wait that runs out sets the error word and ends the kernel
// after its copies have landed and tensor memory is freed. No load is multicast.
#include "activation.cuh"
#include "model.cuh"
#include "gemm_tc.cuh"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

#include <mutex>

namespace lb {

namespace {

typedef __nv_bfloat16 bf16;

constexpr int GB_PATCH = 32 * 32 * 4;  // a warp's staging patch: 32 rows of 32 floats, or two buffers of 32 rows of 32 bfloat16
constexpr int GB_GROUP = 16;     // row tiles that share a sweep over the columns (W tiles stay in L2)

template <int BN, bool PAIR, int WARPS>
struct GbSmem {
  static constexpr int THREADS = 64 + 32 * WARPS;
  static constexpr int STAGES = PAIR ? (WARPS == 8 ? 6 : 5) : BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int A_BYTES = TC_BM * 128;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * 128;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int PATCH_OFF = STAGES * STAGE;
  static constexpr int BAR_OFF = PATCH_OFF + WARPS * GB_PATCH;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

// Instructions of a pair of CTAs (cta_group::2): the even one's thread issues them for both, operands at the same places of both
// shared memories, rows 128 .. 255 of the result in the odd one's tensor memory.
__device__ __forceinline__ void gb_pair_load(unsigned dst, const CUtensorMap *map, int x, int y, unsigned leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void gb_pair_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc,
                                            unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void gb_pair_commit(unsigned bar) {  // the barrier at this place in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((unsigned short)3)
               : "memory");
}
__device__ __forceinline__ void gb_arrive_cluster(unsigned cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

template <int BN, int GATED, bool PAIR, int WARPS>
__global__ void __launch_bounds__(64 + 32 * WARPS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_half, const __grid_constant__ CUtensorMap map_float, int half_tma,
                 int float_tma, const __grid_constant__ Bf16Product p, int m, int m_tiles, int n_tiles, DevErr *err) {
  using L = GbSmem<BN, PAIR, WARPS>;
  constexpr int S = L::STAGES, CTAS = PAIR ? 2 : 1, GROUP = GB_GROUP / CTAS;  // m_tiles counts tiles of CTAS * 128 rows
  const int rank = PAIR ? (int)blockIdx.x & 1 : 0, cta = (int)blockIdx.x / CTAS, ctas = (int)gridDim.x / CTAS;
  extern __shared__ unsigned char smem_raw[];
  const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const unsigned bars = base + L::BAR_OFF;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (S + s); };
  auto tfull = [&](int b) { return bars + 8u * (2 * S + b); };
  auto tempty = [&](int b) { return bars + 8u * (2 * S + 2 + b); };
  volatile unsigned *tmem_holder = reinterpret_cast<volatile unsigned *>(base_ptr + L::BAR_OFF + 192);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(base_ptr + L::BAR_OFF + 196);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = m_tiles * n_tiles, kblocks = (p.k + 63) / 64;
  auto place = [&](int tile, int &m0, int &n0) {
    const int per = GROUP * n_tiles, grp = tile / per, rest = tile - grp * per;
    const int gm = min(GROUP, m_tiles - grp * GROUP);
    n0 = rest / gm * BN;
    m0 = ((grp * GROUP + rest % gm) * CTAS + rank) * TC_BM;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull(b), 1);
      mbar_init(tempty(b), CTAS * WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_holder)),
                   "r"((unsigned)(2 * BN))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_holder)),
                   "r"((unsigned)(2 * BN))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // both CTAs' barriers are there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_holder;
  pdl_launch_dependents();  // behind the allocation: a dependent's CTA must not take tensor memory first
  pdl_wait();

  auto commit = [](unsigned bar) {
    if constexpr (PAIR) gb_pair_commit(bar);
    else tc_commit(bar);
  };
  if (warp == 0) {
    int it = 0;
    bool ok = true;
    for (int tile = cta; tile < tiles && ok; tile += ctas) {
      int m0, n0;
      place(tile, m0, n0);
      for (int kb = 0; kb < kblocks; ++kb, ++it) {
        const int s = it % S;
        ok = mbar_wait(empty(s), ((unsigned)(it / S) & 1u) ^ 1u, abort_flag, err, 11);
        __syncwarp();
        if (!ok) break;
        if (lane == 0) {
          const unsigned st = base + (unsigned)(s * L::STAGE);
          if constexpr (PAIR) {  // this CTA's rows of A and half of W's; the even one's barrier counts both CTAs' bytes
            if (rank == 0) mbar_expect_tx(full(s), 2u * (unsigned)L::STAGE);
            const unsigned bar = cluster_map(full(s), 0);
            gb_pair_load(st, &map_a, kb * 64, m0, bar);
            gb_pair_load(st + L::A_BYTES, &map_w, kb * 64, n0 + rank * (BN / 2), bar);
          } else {
            mbar_expect_tx(full(s), (unsigned)L::STAGE);
            tma_load_2d(st, &map_a, kb * 64, m0, full(s));
            tma_load_2d(st + L::A_BYTES, &map_w, kb * 64, n0, full(s));
          }
        }
        __syncwarp();
      }
    }
    if (PAIR && *abort_flag) {  // copies in flight must land (only the even CTA's barriers know: a millisecond is ample)
      const unsigned long long t0 = global_timer();
      while (global_timer() - t0 < 1000000ull) {
      }
    } else if (*abort_flag) {  // copies in flight must land before the shared memory goes away
      for (int j = it > S ? it - S : 0; j < it; ++j) {
        const unsigned long long t0 = global_timer();
        while (!mbar_try_wait(full(j % S), (unsigned)(j / S) & 1u))
          if (global_timer() - t0 > WAIT_LIMIT_NS) break;
      }
    }
  } else if (warp == 1) {
    constexpr unsigned idesc = umma_idesc_bf16(BN) + (PAIR ? (unsigned)(TC_BM >> 4) << 24 : 0u);  // 256 rows of a pair
    int it = 0, use = 0;
    bool ok = true;
    for (int tile = rank == 0 ? cta : tiles; tile < tiles && ok; tile += ctas, ++use) {
      const int buf = use & 1;
      ok = mbar_wait(tempty(buf), ((unsigned)(use >> 1) & 1u) ^ 1u, abort_flag, err, 12);
      __syncwarp();
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int kb = 0; kb < kblocks; ++kb, ++it) {
        const int s = it % S;
        ok = mbar_wait(full(s), (unsigned)(it / S) & 1u, abort_flag, err, 13);
        __syncwarp();
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lane == 0) {
          const unsigned st = base + (unsigned)(s * L::STAGE);
          const unsigned long long da = umma_desc_k128(st), db = umma_desc_k128(st + L::A_BYTES);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const unsigned d = tmem + (unsigned)(buf * BN), more = (kb | ks) ? 1u : 0u;
            if constexpr (PAIR) gb_pair_mma(d, da + (unsigned long long)(ks * 2), db + (unsigned long long)(ks * 2), idesc, more);
            else tc_mma_f16(d, da + (unsigned long long)(ks * 2), db + (unsigned long long)(ks * 2), idesc, more);
          }
          commit(empty(s));
        }
        __syncwarp();
      }
      if (ok && lane == 0) commit(tfull(buf));
      __syncwarp();
    }
    if (!ok) {  // give the tensor pipe a bounded chance to finish before tensor memory is freed
      const unsigned long long t0 = global_timer();
      if (lane == 0) commit(tfull(use & 1));
      __syncwarp();
      while (!mbar_try_wait(tfull(use & 1), (unsigned)(use >> 1) & 1u))
        if (global_timer() - t0 > WAIT_LIMIT_NS) break;
    }
  } else {
    constexpr int COLS = BN / (WARPS / 4);
    const int q = warp & 3, part = (warp - 2) >> 2;  // lanes of tensor memory, share of the columns
    unsigned char *patch = base_ptr + L::PATCH_OFF + (warp - 2) * GB_PATCH;
    const unsigned patch_u = base + (unsigned)(L::PATCH_OFF + (warp - 2) * GB_PATCH);
    int use = 0, turn = 0;
    bool wide = false;  // the last store read the whole patch
    for (int tile = cta; tile < tiles; tile += ctas, ++use) {
      const int buf = use & 1;
      if (!mbar_wait_warp(tfull(buf), (unsigned)(use >> 1) & 1u, abort_flag, err, 14)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int m0, n0;
      place(tile, m0, n0);
      const int row0 = m0 + q * 32;
#pragma unroll 1
      for (int c0 = part * COLS; c0 < (part + 1) * COLS; c0 += 32) {
        unsigned r[32];
        tc_ld32(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(buf * BN + c0), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 == (part + 1) * COLS) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if constexpr (PAIR) gb_arrive_cluster(cluster_map(tempty(buf), 0));
            else mbar_arrive(tempty(buf));
          }
        }
        const int col = n0 + c0;
        if (col >= p.n || row0 >= m) continue;
        const bool to_half = col + 32 <= p.n_half || (col < p.n_half && p.n_half == p.n);
        if (to_half && half_tma) {
          if (p.act == ACT_GELU_ERF) {
#pragma unroll
            for (int j = 0; j < 32; j += 1 + GATED) r[j] = __float_as_uint(activate(__uint_as_float(r[j]), ACT_GELU_ERF));
          } else if (p.act == ACT_GELU_TANH) {
#pragma unroll
            for (int j = 0; j < 32; j += 1 + GATED) r[j] = __float_as_uint(activate(__uint_as_float(r[j]), ACT_GELU_TANH));
          }
          constexpr int PIECES = GATED ? 2 : 4;  // 16-byte pieces of a row
          unsigned h[4 * PIECES];
#pragma unroll
          for (int j = 0; j < 4 * PIECES; ++j) {
            __nv_bfloat162 v;
            if (GATED)
              v = __floats2bfloat162_rn(__uint_as_float(r[4 * j]) * __uint_as_float(r[4 * j + 1]),
                                        __uint_as_float(r[4 * j + 2]) * __uint_as_float(r[4 * j + 3]));
            else
              v = __floats2bfloat162_rn(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
            h[j] = *reinterpret_cast<const unsigned *>(&v);
          }
          if (lane == 0) {
            if (wide) bulk_wait_read<0>();
            else bulk_wait_read<1>();
          }
          __syncwarp();
          const unsigned at = (unsigned)(turn * (GB_PATCH / 2));
          const int turned = GATED ? (lane >> 2) & 1 : (lane >> 1) & 3;
#pragma unroll
          for (int j = 0; j < PIECES; ++j)
            *reinterpret_cast<uint4 *>(patch + at + lane * (16 * PIECES) + ((j ^ turned) << 4)) =
                make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) tma_store_2d(&map_half, patch_u + at, GATED ? col >> 1 : col, row0);
          turn ^= 1;
          wide = false;
          continue;
        }
        if (lane == 0) bulk_wait_read<0>();
        __syncwarp();
        if (col >= p.n_half && float_tma) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4 *>(patch + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if (p.accumulate) tma_add_2d(&map_float, patch_u, col - p.n_half, row0);
            else tma_store_2d(&map_float, patch_u, col - p.n_half, row0);
          }
          wide = true;
          continue;
        }
        // columns on both sides of n_half, or a result no tensor map can address: a row at a time, lane = column
        float *plain = reinterpret_cast<float *>(patch);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4 *>(patch + lane * 128 + ((j ^ (lane & 7)) << 4)) =
              make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        __syncwarp();
        const int mine = col + lane, rows = min(32, m - row0);
        if (mine < p.n) {
          for (int rr = 0; rr < rows; ++rr) {
            const float v = plain[rr * 32 + ((((lane >> 2) ^ (rr & 7)) << 2) | (lane & 3))];
            const long long row = row0 + rr;
            if (mine >= p.n_half) {
              float *o = p.float_out + row * p.float_ld + (mine - p.n_half);
              *o = p.accumulate ? *o + v : v;
            } else if (!GATED) {
              static_cast<bf16 *>(p.half_out)[row * p.half_ld + mine] = __float2bfloat16_rn(activate(v, p.act));
            } else if ((lane & 1) == 0) {  // n_half is even
              const float f = plain[rr * 32 + ((((lane >> 2) ^ (rr & 7)) << 2) | ((lane & 3) + 1))];
              static_cast<bf16 *>(p.half_out)[row * p.half_ld + (mine >> 1)] = __float2bfloat16_rn(activate(v, p.act) * f);
            }
          }
        }
        __syncwarp();
        wide = false;
      }
    }
    if (lane == 0) bulk_wait_all();  // the stores are part of the grid's results
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // nothing of the pair's is on its way to the other CTA
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)(2 * BN)));
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)(2 * BN)));
  }
}

int device_sms() {
  static int n = 0;
  static std::once_flag once;
  std::call_once(once, [] {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  });
  return n;
}

template <int BN, int GATED, bool PAIR, int WARPS>
void launch_bn(const Bf16Product &p, int m, cudaStream_t st, DevErr *err) {
  using L = GbSmem<BN, PAIR, WARPS>;
  CUtensorMap ma, mw, mh{}, mf{};
  tc_make_map_bf16(&ma, p.a, (unsigned long long)m, (unsigned long long)p.k, (unsigned long long)p.a_ld, TC_BM);
  tc_make_map_bf16(&mw, p.w, (unsigned long long)p.n, (unsigned long long)p.k, (unsigned long long)p.w_ld, PAIR ? BN / 2 : BN);
  const int halves = GATED ? p.n_half / 2 : p.n_half, floats = p.n - p.n_half;
  const bool half_tma = halves > 0 && p.half_ld % 8 == 0 && (reinterpret_cast<uintptr_t>(p.half_out) & 15) == 0;
  const bool float_tma = floats > 0 && p.float_ld % 4 == 0 && p.n_half % 4 == 0 &&
                         (reinterpret_cast<uintptr_t>(p.float_out) & 15) == 0;
  if (half_tma) tc_make_store_map(&mh, p.half_out, true, (unsigned long long)m, (unsigned long long)halves,
                                  (unsigned long long)p.half_ld, GATED ? 16 : 32);
  if (float_tma) tc_make_store_map(&mf, p.float_out, false, (unsigned long long)m, (unsigned long long)floats,
                                   (unsigned long long)p.float_ld, 32);
  LB_CUDA(cudaFuncSetAttribute(gemm_bf16_kernel<BN, GATED, PAIR, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
  constexpr int CTAS = PAIR ? 2 : 1;
  const int mt = (m + CTAS * TC_BM - 1) / (CTAS * TC_BM), nt = (p.n + BN - 1) / BN;
  const long long tiles = (long long)mt * nt;
  const unsigned grid = CTAS * (unsigned)(tiles < device_sms() / CTAS ? tiles : device_sms() / CTAS);
  launch_pdl_cluster_x(gemm_bf16_kernel<BN, GATED, PAIR, WARPS>, dim3(grid), dim3(L::THREADS), L::TOTAL, st, g_pdl_enabled,
                       (unsigned)CTAS, ma, mw, mh, mf, half_tma ? 1 : 0, float_tma ? 1 : 0, p, m, mt, nt, err);
}

template <int BN, bool PAIR = false, int WARPS = 8>
void launch_form(const Bf16Product &p, int m, cudaStream_t st, DevErr *err) {
  if (p.gated) launch_bn<BN, 1, PAIR, WARPS>(p, m, st, err);
  else launch_bn<BN, 0, PAIR, WARPS>(p, m, st, err);
}

}  // namespace

void launch_gemm_bf16(const Bf16Product &p, int m, cudaStream_t st, DevErr *err) {
  if (m < 1 || p.n < 1 || p.k < 1) throw std::invalid_argument("launch_gemm_bf16: empty product");
  if (p.gated && ((p.n_half | p.half_ld) & 1) != 0) throw std::invalid_argument("launch_gemm_bf16: a gated product needs pairs");
  // The widest tile of which the next narrower would need a second turn: a turn costs about what its tile's k loop does, 1 : 0.8 :
  // 0.7 from 256 to 64 columns. 2368 x 1024 (76 tiles of 256 columns), by 64, 128 and 256: k 512 11.7, 9.4, 8.0 us, k 5120 74, 51, 29;
  // 613 x 2048 (80 of 128): k 512 9.1, 6.9, 7.8, k 5120 51, 29, 28; 613 x 1600 (65 of 128, 125 of 64): k 512 6.4, 6.9, 7.8, with GELU 7.5,
  // 8.9, 11.9. Mitilix, 8 streams of 256 + 96 tokens: 31.51 ms with 256 columns from 111 tiles on (and so 128), 31.24.
  const long long mt = (m + TC_BM - 1) / TC_BM;
  const long long sms = device_sms();
  const long long nt = (p.n + 255) / 256, turns = (mt * nt + sms - 1) / sms;
  const long long pair_turns = ((mt + 1) / 2 * nt + sms / 2 - 1) / (sms / 2);
  if (p.n > 128 && mt * ((p.n + 127) / 128) > sms) {
    // A pair starts 1.5 to 2 us later (its CTAs meet before and after) and then gains a share of each 64 k of each tile: 6 % at 7
    // tiles of 1024 k a CTA, 6 to 9 % at 2 of 5120, 9 to 12 % at 4 and 7 of 5120, against 1 to 4 % lost at 2 of 2048 and more below.
    // With an activation, sixteen storing warps: with eight a pair gains nothing (gated 8192 x 4096 x 1024: 64 us alone, 69 a
    // pair with eight, 57 with sixteen; plain results prefer the sixth operand stage, 8192 x 4096 x 1024 60.5, 56.9 and 58.8).
    const bool pair = turns >= 2 && turns * p.k >= 5120 && pair_turns <= turns;
    if (pair && p.act != ACT_NONE && p.n_half > 0) launch_form<256, true, 16>(p, m, st, err);
    else if (pair) launch_form<256, true>(p, m, st, err);
    else launch_form<256>(p, m, st, err);
  } else if (p.n > 64 && mt * ((p.n + 63) / 64) > sms) launch_form<128>(p, m, st, err);
  else launch_form<64>(p, m, st, err);
}

}  // namespace lb
