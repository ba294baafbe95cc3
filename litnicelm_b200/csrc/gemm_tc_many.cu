// Tensor-core projections of the token loop for many rows: the product of gemm_tc.cu on fp16 pairs
// (three kind::f16 products per k-step, one accumulation chain per 64 of k, chains added in fp32
// registers under the operands' block scales) with resident CTAs that walk 128 x 256 tiles.
//
// What bounds such a product is the tensor pipe (12 instructions of 128 x 256 x 16 per chain, 1.05 us)
// as long as nothing else stands in line with it. In gemm_tc.cu a tile's start (tensor memory,
// barriers, first loads) and its store phase do: at k = 512 a 128 x 256 tile took 27 us of which the
// chains are 8. Here
//   * one CTA per SM takes tile after tile; the TMA and MMA warps run ahead into the next tile while
//     the eight drain warps still store the last one (two chains deep: the tensor-memory ring),
//   * a drain thread finishes its row's 128 columns in its own registers (a block scale or a slot of
//     row statistics is 64 columns of one row: no exchange between threads) and the results leave as
//     32-row boxes, swizzled in shared memory and stored by TMA, and
//   * two otherwise idle warps form the folded LayerNorm's row statistics a tile ahead (3.3 us of a
//     drain warp's time per tile).
// Measured in the loop of 64 streams (contexts 128 .. 160, width 512, per launch): QKV and W1 105 -> 61 us,
// out-projection and W2 79 -> 55 us, of which the rows left out of a bucket's bound are a quarter. At 9216
// rows W1 (2048 columns, k 512) takes 61 us, W2 (512, 2048) 60 us. A tile's store phase still takes 4 us
// (W1) to 9 us (residual, fp32 result, statistics): a box may be overwritten only once TMA has read it,
// and there is room for one box of 4 KB per warp beside two stages of operands.
// Every value is formed by the same operations in the same order as in gemm_tc_epilogue.cuh.
//
// Warps: 0 TMA loads, 1 tensor memory + MMA issue, 2 and 3 the folded LayerNorm's row statistics, 4..11
// drain (lane quarter w % 4, columns half). Every wait is bounded; a wait that runs out sets the error
// word and all roles leave.
#include "gemm_tc.cuh"
#include "tc_ptx.cuh"
#include "gemm_tc_epilogue.cuh"

#include <mutex>

namespace lb {

namespace {

constexpr int GM_BN = 256, GM_STAGES = 2, GM_DRAIN = 8, GM_ROLES = 4, GM_THREADS = 32 * (GM_ROLES + GM_DRAIN);
// 384 threads start with 168 registers each (64512); the drain warps hold 128 accumulators, so the warpgroup of the
// roles gives its share up: 128 * 72 + 256 * 216 = 64512.
constexpr int GM_REGS_ROLE = 72, GM_REGS_DRAIN = 216;
constexpr int GM_A_BYTES = TC_BM * 128, GM_B_BYTES = GM_BN * 128;
constexpr int GM_STAGE_BYTES = 2 * (GM_A_BYTES + GM_B_BYTES);
constexpr int GM_PATCH = 4096;  // a box of 32 rows x 128 bytes per drain warp
constexpr int GM_PATCH_OFF = GM_STAGES * GM_STAGE_BYTES;
constexpr int GM_BAR_OFF = GM_PATCH_OFF + GM_DRAIN * GM_PATCH;
constexpr int GM_STATS_OFF = GM_BAR_OFF + 128;  // float2 (mean, 1/std) per tile row
constexpr int GM_SMEM = GM_STATS_OFF + TC_BM * 8 + 1024;  // + alignment slack

struct GmShape {
  int m, n, kblocks, n_tiles;
};

// Columns first: the CTAs at work at one time share few row tiles, and the column tile a CTA starts with does not
// depend on how many row tiles there are (its weights are requested before that is known).
__device__ __forceinline__ void gm_place(const GmShape &p, int tile, int &m0, int &n0) {
  m0 = tile / p.n_tiles * TC_BM;
  n0 = tile % p.n_tiles * GM_BN;
}
// Row tiles that hold rows: a launch sized for a bound of the context length (graph replay) leaves out the tiles
// behind the last stream's last row. After the wait for the predecessor.
__device__ __forceinline__ int gm_tiles(const GmShape &p, const TcEpilogue &ep) {
  const int rows = ep.state != nullptr ? min(p.m, ep.vt_streams * ep.state->s) : p.m;
  return (rows + TC_BM - 1) / TC_BM * p.n_tiles;
}

// The last box has been read, the next may be written / the box is written, send it.
__device__ __forceinline__ void gm_box_free(int lane) {
  if (lane == 0) bulk_wait_read<0>();
  __syncwarp();
}
__device__ __forceinline__ void gm_box_send(const CUtensorMap *map, unsigned patch, int x, int y, int lane) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) tma_store_2d(map, patch, x, y);
}

// 64 columns of the thread's row, v * scale, as pair words of two columns each.
__device__ __forceinline__ void gm_pair(const float *v, float scale, unsigned *hi, unsigned *lo) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    uint2 h, l;
    f16_pair4(make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]), scale, h, l);
    hi[2 * j] = h.x;
    hi[2 * j + 1] = h.y;
    lo[2 * j] = l.x;
    lo[2 * j + 1] = l.y;
  }
}
// 128 bytes of the thread's row into its box row (the 128-byte swizzle of the store maps).
__device__ __forceinline__ void gm_write_row(unsigned char *patch, int lane, const unsigned *w) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4 *>(patch + lane * 128 + ((j ^ (lane & 7)) << 4)) =
        make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
}
// A box of the residual, 32 rows x 32 columns, as whole 128-byte row segments: 8 lanes a row, 4 rows per load (a
// lane per row would cost a cache line per lane and load).
__device__ __forceinline__ void gm_residual_load(float4 (&r)[8], const TcEpilogue &ep, const GmShape &p, int row0, int col,
                                                 int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = row0 + 4 * i + (lane >> 3);
    r[i] = row < p.m ? __ldg(reinterpret_cast<const float4 *>(ep.residual + (long long)row * p.n + col) + (lane & 7))
                     : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// One 64-column block of the thread's row: the epilogue terms F names, then every output. res: the
// residual's box at col, loaded; replaced by the one at next_col (negative: none).
template <unsigned F>
__device__ __forceinline__ void gm_finish_block(float *v, const TcEpilogue &ep, const GmShape &p, int row, int row0, int col,
                                                float2 ln_st, float4 (&res)[8], int next_col, unsigned char *patch,
                                                unsigned patch_u, int lane, const CUtensorMap *map_c,
                                                const CUtensorMap *map_hi, const CUtensorMap *map_lo) {
  const bool act = row < p.m;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (F & TC_EP_RESIDUAL) {  // through the box, to the lane that holds the row
      gm_box_free(lane);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (lane >> 3);
        *reinterpret_cast<float4 *>(patch + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) = res[i];
      }
      __syncwarp();
      if (h == 0) gm_residual_load(res, ep, p, row0, col + 32, lane);
      else if (next_col >= 0) gm_residual_load(res, ep, p, row0, next_col, lane);
    }
#pragma unroll
    for (int jj = 0; jj < 32; jj += 4) {
      const int j = 32 * h + jj;
      const float4 bb = __ldg(reinterpret_cast<const float4 *>(ep.bias + col + j));
      float4 rr = make_float4(0.f, 0.f, 0.f, 0.f);
      if (F & TC_EP_RESIDUAL) rr = *reinterpret_cast<const float4 *>(patch + lane * 128 + (((jj >> 2) ^ (lane & 7)) << 4));
      if (F & TC_EP_FOLD) {  // inv_std * (x W' - mean * u); v comes in as the bias
        const float4 uu = __ldg(reinterpret_cast<const float4 *>(ep.ln_u + col + j));
        v[j] = __fmul_rn(ln_st.y, __fmaf_rn(-ln_st.x, uu.x, v[j]));
        v[j + 1] = __fmul_rn(ln_st.y, __fmaf_rn(-ln_st.x, uu.y, v[j + 1]));
        v[j + 2] = __fmul_rn(ln_st.y, __fmaf_rn(-ln_st.x, uu.z, v[j + 2]));
        v[j + 3] = __fmul_rn(ln_st.y, __fmaf_rn(-ln_st.x, uu.w, v[j + 3]));
      }
      v[j] += bb.x + rr.x;
      v[j + 1] += bb.y + rr.y;
      v[j + 2] += bb.z + rr.z;
      v[j + 3] += bb.w + rr.w;
      if (F & TC_EP_RELU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[j + e] = fmaxf(v[j + e], 0.f);
      }
      if (F & TC_EP_C)  // over the residual the lane has just read
        *reinterpret_cast<float4 *>(patch + lane * 128 + (((jj >> 2) ^ (lane & 7)) << 4)) =
            make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
    if (F & TC_EP_C) gm_box_send(map_c, patch_u, col + 32 * h, row0, lane);
  }
  if (F & TC_EP_STATS) {  // (sum x, sum x^2) of the slot: four sums of 16 columns, added in order
    double tx = 0.0, txx = 0.0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      double sx = 0.0, sxx = 0.0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const double t = (double)v[16 * g + j];
        sx += t;
        sxx += t * t;
      }
      tx = g ? tx + sx : sx;
      txx = g ? txx + sxx : sxx;
    }
    if (act) ep.stats_out[(long long)row * TC_STAT_SLOTS + col / 64] = make_double2(tx, txx);
  }
  unsigned hi[32], lo[32];
  if (F & TC_EP_F16) {
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 64; ++j) am = fmaxf(am, fabsf(v[j]));
    float inv;
    gm_pair(v, f16_block_scale(am, &inv), hi, lo);
    if (act) ep.c_f16.inv_scale[(long long)row * (p.n / TC_F16_SLOT) + col / TC_F16_SLOT] = inv;
  }
  bool boxes = true;
  if (F & TC_EP_QK16) {  // Q, K or V of one head: pairs under the head's fixed scale, V transposed
    const bool is_v = col >= ep.vt_col0;
    const int sl = ep.state ? ep.state->s : ep.vt_s;
    const int stream = row / sl, tok = row - stream * sl;
    const bool mine = act && stream < ep.vt_streams;
    float *cache = is_v ? ep.vcache : col >= ep.vt_col0 - ep.vt_rows ? ep.kcache : nullptr;
    if (cache != nullptr && mine) {
      float4 *cp = reinterpret_cast<float4 *>(cache + ((long long)stream * ep.kv_cap + tok) * ep.vt_rows + col % ep.vt_rows);
#pragma unroll
      for (int j = 0; j < 16; ++j) cp[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    gm_pair(v, __ldg(ep.col_scale + col / 64), hi, lo);
    boxes = !is_v;
    if (is_v && mine) {  // the warp's 32 rows are consecutive positions: 64 bytes of one V^T row per store
      const long long at0 = ((long long)stream * ep.vt_rows + (col - ep.vt_col0)) * ep.vt_pitch + tok;
      unsigned short *hp = reinterpret_cast<unsigned short *>(ep.vt16_hi) + at0;
      unsigned short *lp = reinterpret_cast<unsigned short *>(ep.vt16_lo) + at0;
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        hp[(long long)j * ep.vt_pitch] = (unsigned short)(j & 1 ? hi[j >> 1] >> 16 : hi[j >> 1]);
        lp[(long long)j * ep.vt_pitch] = (unsigned short)(j & 1 ? lo[j >> 1] >> 16 : lo[j >> 1]);
      }
    }
  }
  if (boxes) {
    gm_box_free(lane);
    gm_write_row(patch, lane, hi);
    gm_box_send(map_hi, patch_u, col, row0, lane);
    gm_box_free(lane);
    gm_write_row(patch, lane, lo);
    gm_box_send(map_lo, patch_u, col, row0, lane);
  }
}

template <unsigned F>
__global__ void __launch_bounds__(GM_THREADS, 1)
gemm_tc_many_kernel(const __grid_constant__ CUtensorMap map_a_hi, const __grid_constant__ CUtensorMap map_a_lo,
                    const __grid_constant__ CUtensorMap map_b_hi, const __grid_constant__ CUtensorMap map_b_lo,
                    const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_hi,
                    const __grid_constant__ CUtensorMap map_lo, TcEpilogue ep, GmShape p, DevErr *err,
                    const float *__restrict__ a_inv_scale, const float *__restrict__ b_inv_scale) {
  constexpr int S = GM_STAGES;
  extern __shared__ unsigned char smem_raw[];
  const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const unsigned bars = base + GM_BAR_OFF;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (S + s); };
  auto tfull = [&](int b) { return bars + 8u * (2 * S + b); };
  auto tempty = [&](int b) { return bars + 8u * (2 * S + 2 + b); };
  const unsigned sfull = bars + 8u * (2 * S + 4), sempty = bars + 8u * (2 * S + 5);  // the tile's row statistics
  float2 *row_stats = reinterpret_cast<float2 *>(base_ptr + GM_STATS_OFF);
  volatile unsigned *tmem_holder = reinterpret_cast<volatile unsigned *>(base_ptr + GM_BAR_OFF + 96);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(base_ptr + GM_BAR_OFF + 100);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  pdl_launch_dependents();
  if (ep.timeline != nullptr && threadIdx.x == 0) {
    const unsigned long long t = global_timer();
    atomicMin(ep.timeline + 8, t);
    atomicMax(ep.timeline + 10, t);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull(b), 1);
      mbar_init(tempty(b), GM_DRAIN);
    }
    mbar_init(sfull, 2);
    mbar_init(sempty, GM_DRAIN);
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

  if (warp < GM_ROLES) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GM_REGS_ROLE));
    if (warp == 0) {
      // ---- TMA loads; the weights of the first stages before the wait for the predecessor ----
      int it = 0, pre = 0;
      bool ok = true;
      {
        int m0, n0;
        gm_place(p, blockIdx.x, m0, n0);
        pre = min(S, p.kblocks);
        if (lane == 0) {
          tma_prefetch_map(&map_a_hi);
          tma_prefetch_map(&map_a_lo);
          for (int kb = 0; kb < pre; ++kb) {
            const unsigned st = base + (unsigned)(kb * GM_STAGE_BYTES);
            mbar_expect_tx(full(kb), (unsigned)GM_STAGE_BYTES);
            tma_load_2d(st + 2 * GM_A_BYTES, &map_b_hi, kb * TC_F16_SLOT, n0, full(kb));
            tma_load_2d(st + 2 * GM_A_BYTES + GM_B_BYTES, &map_b_lo, kb * TC_F16_SLOT, n0, full(kb));
          }
        }
      }
      pdl_wait();
      if (ep.timeline != nullptr && lane == 0) atomicMin(ep.timeline + 14, global_timer());
      const int tiles = gm_tiles(p, ep);
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        int m0, n0;
        gm_place(p, tile, m0, n0);
        for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
          const int s = it % S;
          const bool b_sent = it < pre;
          if (!b_sent) {
            ok = mbar_wait_inline(empty(s), ((unsigned)(it / S) & 1u) ^ 1u, abort_flag, err, 21);
            __syncwarp();
            if (!ok) break;
          }
          if (lane == 0) {
            const unsigned st = base + (unsigned)(s * GM_STAGE_BYTES);
            const int kx = kb * TC_F16_SLOT;
            if (!b_sent) mbar_expect_tx(full(s), (unsigned)GM_STAGE_BYTES);
            tma_load_2d(st, &map_a_hi, kx, m0, full(s));
            tma_load_2d(st + GM_A_BYTES, &map_a_lo, kx, m0, full(s));
            if (!b_sent) {
              tma_load_2d(st + 2 * GM_A_BYTES, &map_b_hi, kx, n0, full(s));
              tma_load_2d(st + 2 * GM_A_BYTES + GM_B_BYTES, &map_b_lo, kx, n0, full(s));
            }
          }
          __syncwarp();
        }
      }
      if ((int)blockIdx.x >= tiles) {  // no tile after all: the weights requested ahead, with the rest of their stages
        if (lane == 0) {
          for (int kb = 0; kb < pre; ++kb) {
            const unsigned st = base + (unsigned)(kb * GM_STAGE_BYTES);
            tma_load_2d(st, &map_a_hi, kb * TC_F16_SLOT, 0, full(kb));
            tma_load_2d(st + GM_A_BYTES, &map_a_lo, kb * TC_F16_SLOT, 0, full(kb));
          }
        }
        it = pre;
        __syncwarp();
      }
      if (*abort_flag || (int)blockIdx.x >= tiles) {  // copies in flight must land before the shared memory goes away
        for (int j = it > S ? it - S : 0; j < it; ++j) {
          const unsigned long long t0 = global_timer();
          while (!mbar_try_wait(full(j % S), (unsigned)(j / S) & 1u))
            if (global_timer() - t0 > WAIT_LIMIT_NS) break;
        }
      }
    } else if (warp != 1) {
      // ---- the folded LayerNorm's row statistics, a tile ahead of the drain warps' use: two rows per lane ----
      pdl_wait();
      if (F & TC_EP_FOLD) {
        const int tiles = gm_tiles(p, ep);
        int nth = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++nth) {
          int m0, n0;
          gm_place(p, tile, m0, n0);
          float2 st[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int row = min(m0 + (warp - 2) * 64 + h * 32 + lane, p.m - 1);
            st[h] = ln_row_stats(ep.ln_stats + (long long)row * TC_STAT_SLOTS, ep.ln_slots, p.kblocks * TC_F16_SLOT);
          }
          if (!__all_sync(0xffffffffu, mbar_wait_inline(sempty, ((unsigned)nth & 1u) ^ 1u, abort_flag, err, 25))) break;
#pragma unroll
          for (int h = 0; h < 2; ++h) row_stats[(warp - 2) * 64 + h * 32 + lane] = st[h];
          __syncwarp();
          if (lane == 0) mbar_arrive(sfull);
        }
      }
    } else {
      // ---- MMA issue: one chain per 64 of k, small products first ----
      pdl_wait();
      const int tiles = gm_tiles(p, ep);
      const unsigned idesc = umma_idesc_f16(GM_BN);
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
          const int s = it % S, buf = it & 1;
          ok = mbar_wait_inline(tempty(buf), ((unsigned)(it >> 1) & 1u) ^ 1u, abort_flag, err, 24) &&
               mbar_wait_inline(full(s), (unsigned)(it / S) & 1u, abort_flag, err, 22);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (lane == 0) {
            const unsigned st = base + (unsigned)(s * GM_STAGE_BYTES), d = tmem + (unsigned)(buf * GM_BN);
            const unsigned long long a_hi = umma_desc_k128(st), a_lo = umma_desc_k128(st + GM_A_BYTES);
            const unsigned long long b_hi = umma_desc_k128(st + 2 * GM_A_BYTES);
            const unsigned long long b_lo = umma_desc_k128(st + 2 * GM_A_BYTES + GM_B_BYTES);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              tc_mma_f16(d, a_lo + 2 * ks, b_hi + 2 * ks, idesc, ks ? 1u : 0u);
              tc_mma_f16(d, a_hi + 2 * ks, b_lo + 2 * ks, idesc, 1u);
            }
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) tc_mma_f16(d, a_hi + 2 * ks, b_hi + 2 * ks, idesc, 1u);
            tc_commit(empty(s));
            tc_commit(tfull(buf));
          }
          __syncwarp();
        }
      }
      if (!ok) {  // give the tensor pipe a bounded chance to finish before tensor memory is freed
        if (lane == 0) tc_commit(tfull(it & 1));
        __syncwarp();
        const unsigned long long t0 = global_timer();
        while (!mbar_try_wait(tfull(it & 1), (unsigned)(it >> 1) & 1u))
          if (global_timer() - t0 > WAIT_LIMIT_NS) break;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(GM_REGS_DRAIN));
    // ---- drain: 32 rows x 128 columns per warp ----
    pdl_wait();
    const int tiles = gm_tiles(p, ep);
    const int q = warp & 3, half = (warp - GM_ROLES) >> 2;
    unsigned char *patch = base_ptr + GM_PATCH_OFF + (warp - GM_ROLES) * GM_PATCH;
    const unsigned patch_u = base + (unsigned)(GM_PATCH_OFF + (warp - GM_ROLES) * GM_PATCH);
    const float b_inv = *b_inv_scale;
    auto scales_of = [&](int tile) {  // the thread's row of a tile's block scales
      int m0, n0;
      gm_place(p, tile, m0, n0);
      return a_inv_scale + (long long)min(m0 + q * 32 + lane, p.m - 1) * p.kblocks;
    };
    int it = 0, nth = 0;
    float chain_scale = (int)blockIdx.x < tiles ? *scales_of(blockIdx.x) * b_inv : 0.f;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++nth) {
      int m0, n0;
      gm_place(p, tile, m0, n0);
      const int row0 = m0 + q * 32, row = row0 + lane;
      const float *scales = scales_of(tile);
      float2 ln_st = make_float2(0.f, 1.f);
      float acc[128];
#pragma unroll
      for (int j = 0; j < 128; ++j) acc[j] = 0.f;
#pragma unroll 1
      for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
        const int buf = it & 1;
        ok = __all_sync(0xffffffffu, mbar_wait_inline(tfull(buf), (unsigned)(it >> 1) & 1u, abort_flag, err, 23));
        if (!ok) break;
        const float sc = chain_scale;
        if (kb + 1 < p.kblocks) chain_scale = scales[kb + 1] * b_inv;  // in flight during this chain's adds
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < 128; c0 += 64) {
          unsigned r[32], t[32];
          tc_ld32(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(buf * GM_BN + half * 128 + c0), r);
          tc_ld32(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(buf * GM_BN + half * 128 + c0 + 32), t);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[c0 + j] = __fmaf_rn(__uint_as_float(r[j]), sc, acc[c0 + j]);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[c0 + 32 + j] = __fmaf_rn(__uint_as_float(t[j]), sc, acc[c0 + 32 + j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty(buf));
      }
      if (!ok) break;
      if (tile + (int)gridDim.x < tiles) chain_scale = *scales_of(tile + gridDim.x) * b_inv;
      if (F & TC_EP_FOLD) {
        ok = __all_sync(0xffffffffu, mbar_wait_inline(sfull, (unsigned)nth & 1u, abort_flag, err, 26));
        if (!ok) break;
        ln_st = row_stats[q * 32 + lane];
        __syncwarp();
        if (lane == 0) mbar_arrive(sempty);
      }
      if (row0 >= p.m) continue;
      float4 res[8];
      const int col = n0 + half * 128;
      if (F & TC_EP_RESIDUAL) gm_residual_load(res, ep, p, row0, col, lane);
      // one body for both blocks (the second moves down): as straight-line code twice as long it ran at the speed of
      // instruction fetch
#pragma unroll 1
      for (int b = 0; b < 2; ++b) {
        gm_finish_block<F>(acc, ep, p, row, row0, col + 64 * b, ln_st, res, b ? -1 : col + 64, patch, patch_u, lane, &map_c,
                           &map_hi, &map_lo);
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = acc[64 + j];
      }
    }
    if (lane == 0) bulk_wait_all();  // the stores are part of the grid's results
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (ep.timeline != nullptr && threadIdx.x == 0) atomicMax(ep.timeline + 9, global_timer());
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

int gm_device_sms() {
  static int sms[64] = {};
  static std::mutex mu;
  int dev = 0;
  LB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 64 && sms[dev] > 0) return sms[dev];
  int v = 0;
  LB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
  if (dev < 64) sms[dev] = v;
  return v;
}

template <unsigned F>
void gm_launch(const TcMatrix &a, const float *a_inv_scale, const TcMatrix &b, const float *b_inv_scale, int m, int n, int k,
               const TcEpilogue &ep, DevErr *err, cudaStream_t st) {
  const GmShape p{m, n, k / TC_F16_SLOT, n / GM_BN};
  CUtensorMap mc{}, mh{}, ml{};
  const unsigned long long rows = (unsigned long long)m, cols = (unsigned long long)n;
  if (F & TC_EP_C) tc_make_store_map(&mc, ep.c, false, rows, cols, cols, 32);
  tc_make_store_map(&mh, (F & TC_EP_QK16) ? ep.qk16_hi : ep.c_f16.hi, true, rows, cols, cols, 64);
  tc_make_store_map(&ml, (F & TC_EP_QK16) ? ep.qk16_lo : ep.c_f16.lo, true, rows, cols, cols, 64);
  LB_CUDA(cudaFuncSetAttribute(gemm_tc_many_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM));
  const long long tiles = (long long)((m + TC_BM - 1) / TC_BM) * p.n_tiles;
  const int sms = gm_device_sms();
  launch_pdl(gemm_tc_many_kernel<F>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(GM_THREADS), (size_t)GM_SMEM, st,
             g_pdl_enabled, a.hi, a.lo, b.hi, b.lo, mc, mh, ml, ep, p, err, a_inv_scale, b_inv_scale);
}

}  // namespace

bool launch_gemm_tc_many(const TcMatrix &a, const float *a_inv_scale, const TcMatrix &b, const float *b_inv_scale, int m, int n,
                         int k, const TcEpilogue &ep, DevErr *err, cudaStream_t st) {
  const auto aligned = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const unsigned form = tc_ep_form(ep);
  if (n % GM_BN != 0 || k % TC_F16_SLOT != 0) return false;
  if (form == TC_EP_FORM_QKV) {
    // heads of 64 columns in thirds; Q and K boxes and V^T rows
    if (ep.vt16_hi == nullptr || ep.vt_rows % 64 != 0 || ep.vt_col0 != 2 * ep.vt_rows || !aligned(ep.qk16_hi) ||
        !aligned(ep.qk16_lo))
      return false;
    gm_launch<TC_EP_FORM_QKV>(a, a_inv_scale, b, b_inv_scale, m, n, k, ep, err, st);
  } else if (form == TC_EP_FORM_W1 && !ep.has_vt() && aligned(ep.c_f16.hi) && aligned(ep.c_f16.lo)) {
    gm_launch<TC_EP_FORM_W1>(a, a_inv_scale, b, b_inv_scale, m, n, k, ep, err, st);
  } else if (form == TC_EP_FORM_RES && !ep.has_vt() && aligned(ep.c) && aligned(ep.c_f16.hi) && aligned(ep.c_f16.lo)) {
    gm_launch<TC_EP_FORM_RES>(a, a_inv_scale, b, b_inv_scale, m, n, k, ep, err, st);
  } else {
    return false;
  }
  return true;
}

}  // namespace lb
