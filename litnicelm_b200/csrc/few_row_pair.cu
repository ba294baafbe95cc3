// The products of a cached step for up to 64 rows on the weights' fp16 pairs: out[m, n] = x[m, k] W (+ bias) (+ residual) (ReLU),
// or LayerNorm(x) W + b with the LayerNorm folded into W (gemm_tc_epilogue.cuh's form). Rows in and out are fp32: a kernel
// here turns its rows into pairs by itself, so that nothing between two products has to be written in a product's format.
//
// Bound by latency: a product of 64 rows has few tiles of 128 x 64, and on tcgen05 tiles each took 9.7 us, first loads, four
// blocks of k, the exchange of k ranges and the store one behind the other. Here W rows are the M side of mma.sync m16n8k16
// tiles and activation rows the N side, as in few_row_bf16.cu: a CTA owns 16 columns and NT tiles of 8 rows, its eight warps take
// interleaved spans of 64 k, a lane loads 16 consecutive bytes (8 k) of its W rows and 32 of its activation row and feeds them to
// two k-steps as they lie. A span's activations get the power-of-two scale that puts a row's largest magnitude in [2^12, 2^13),
// are split into hi + lo and multiplied three times (hi hi, and lo hi + hi lo in an accumulator of its own); spans are added
// in fp32 with their scales. Sums and sums of squares of the folded LayerNorm are taken in double: by the product that makes the
// row, a slot per 16 columns, or where none does (the embedding) from the consumer's own loads.
//
// 64 rows, us a launch in a row of them: n 1536 k 512 with LayerNorm 4.4, n 512 k 512 3.1, n 2048 k 512 with LayerNorm 5.5, n 512 k
// 2048 5.4 (9.7 on average on the tiles, alone). A cached step of 6 layers x 512, 64 streams: 320 -> 268 us.
#include "gemm_tc.cuh"
#include "tc_ptx.cuh"

namespace lb {

namespace {

constexpr int FP_WARPS = 8;
constexpr int FP_COLS = 16;  // output columns per CTA
constexpr int FP_SPAN = 64;  // k per warp and trip: one scale

__device__ __forceinline__ void fp_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct FpShape {
  const float *x;
  const __half *w_hi, *w_lo;  // [n][k]
  const float *w_inv;         // the matrix's scale, inverse
  const float *bias;          // folded: v[n]
  const float *u;             // folded LayerNorm: u[n], or null
  const float *residual;      // [rows][n], or null
  float *out;                 // [rows][n]
  const double2 *sums_in;     // [rows][k / 16]: sum and sum of squares of 16 columns of x
  double2 *sums_out;          // the same of out, or null
  int rows, n, k, relu;
};
enum { FP_PLAIN, FP_FOLD, FP_FOLD_SUMS };  // no LayerNorm; one whose sums are taken here; one whose sums there are

// MORE: k longer than one span per warp, the next span's weights come ahead. CTAs an SM with next to no spills (4 and 24 bytes in two
// of the eighteen forms).
constexpr int fp_ctas(int nt, int fold, bool more) { return more ? (nt == 1 ? 2 : 1) : nt == 1 ? (fold ? 3 : 4) : nt == 2 ? 3 : 2; }
template <int NT, int FOLD, bool MORE>
__global__ void __launch_bounds__(FP_WARPS * 32, fp_ctas(NT, FOLD, MORE)) few_row_pair_kernel(const __grid_constant__ FpShape g) {
  __shared__ __align__(16) float red[FP_WARPS][NT][FP_COLS][8];
  __shared__ double2 stat[FP_WARPS][NT * 8];
  __shared__ float2 norm[NT * 8];  // mean, 1 / standard deviation
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, r = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * FP_COLS, first = blockIdx.y * NT * 8, m = min(NT * 8, g.rows - first);
  struct Weights {
    uint4 hi[2][2], lo[2][2];  // [block of 32 k][column r, r + 8]
  };
  Weights next;
  const long long w_at = (long long)(n0 + r) * g.k + t * 8;
  auto load_w = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const long long at = w_at + (long long)c * 8 * g.k + k0 + u * 32;
        next.hi[u][c] = __ldg(reinterpret_cast<const uint4 *>(g.w_hi + at));
        next.lo[u][c] = __ldg(reinterpret_cast<const uint4 *>(g.w_lo + at));
      }
  };
  pdl_launch_dependents();
  if (wid * FP_SPAN < g.k) load_w(wid * FP_SPAN);  // the weights do not depend on the predecessor
  const float w_inv = *g.w_inv;
  pdl_wait();
  // mean and biased variance in double, inv_std = 1/sqrt(float(var) + 1e-5f) (device_backend.cpp:1247-1279)
  auto finish = [&](double s, double q) {
    const double mean = s / (double)g.k;
    double var = q / (double)g.k - mean * mean;
    if (var < 0.0) var = 0.0;
    return make_float2((float)mean, 1.0f / sqrtf((float)var + 1e-5f));
  };
  if constexpr (FOLD == FP_FOLD_SUMS) {  // sixteen lanes a row
    const int slots = g.k / FP_COLS, slot = threadIdx.x % 16;
#pragma unroll
    for (int row = threadIdx.x / 16; row < NT * 8; row += FP_WARPS * 2) {
      double s = 0.0, q = 0.0;
      if (row < m) {
        const double2 *from = g.sums_in + (long long)(first + row) * slots;
        for (int x = slot; x < slots; x += 16) {
          const double2 v = from[x];
          s += v.x;
          q += v.y;
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
      }
      if (slot == 0) norm[row] = finish(s, q);
    }
  }
  float acc[NT][4];
  double sum[NT], sq[NT];  // of row r of every tile, this lane's k
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    sum[i] = sq[i] = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  }
#pragma unroll 1
  for (int k0 = wid * FP_SPAN; k0 < g.k; k0 += MORE ? FP_WARPS * FP_SPAN : g.k) {
    const Weights w = next;
    float4 x[NT][2][2];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float *row = g.x + (long long)(first + i * 8 + r) * g.k + k0 + t * 8;
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          x[i][u][h] = i * 8 + r < m ? *reinterpret_cast<const float4 *>(row + u * 32 + h * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if constexpr (MORE) {
      if (k0 + FP_WARPS * FP_SPAN < g.k) load_w(k0 + FP_WARPS * FP_SPAN);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      float amax = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = x[i][u][h];
          amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        }
      if constexpr (FOLD == FP_FOLD) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 v = x[i][u][h];
            const double a = v.x, b = v.y, c = v.z, d = v.w;
            sum[i] += (a + b) + (c + d);
            sq[i] += (a * a + b * b) + (c * c + d * d);
          }
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      float inv;
      const float scale = f16_block_scale(amax, &inv);
      float big[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint2 hi, lo;
          f16_pair4(x[i][u][h], scale, hi, lo);
          const unsigned w0 = h ? w.hi[u][0].z : w.hi[u][0].x, w1 = h ? w.hi[u][1].z : w.hi[u][1].x;
          const unsigned w2 = h ? w.hi[u][0].w : w.hi[u][0].y, w3 = h ? w.hi[u][1].w : w.hi[u][1].y;
          const unsigned l0 = h ? w.lo[u][0].z : w.lo[u][0].x, l1 = h ? w.lo[u][1].z : w.lo[u][1].x;
          const unsigned l2 = h ? w.lo[u][0].w : w.lo[u][0].y, l3 = h ? w.lo[u][1].w : w.lo[u][1].y;
          fp_mma(small, l0, l1, l2, l3, hi.x, hi.y);
          fp_mma(small, w0, w1, w2, w3, lo.x, lo.y);
          fp_mma(big, w0, w1, w2, w3, hi.x, hi.y);
        }
      // this lane's sums are of rows 2 t and 2 t + 1, whose scales the lanes of those rows hold
      const float inv0 = __shfl_sync(0xffffffffu, inv, t * 8), inv1 = __shfl_sync(0xffffffffu, inv, t * 8 + 4);
      acc[i][0] = fmaf(big[0] + small[0], inv0, acc[i][0]);
      acc[i][1] = fmaf(big[1] + small[1], inv1, acc[i][1]);
      acc[i][2] = fmaf(big[2] + small[2], inv0, acc[i][2]);
      acc[i][3] = fmaf(big[3] + small[3], inv1, acc[i][3]);
    }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    *reinterpret_cast<float2 *>(&red[wid][i][r][t * 2]) = make_float2(acc[i][0], acc[i][1]);
    *reinterpret_cast<float2 *>(&red[wid][i][r + 8][t * 2]) = make_float2(acc[i][2], acc[i][3]);
    if constexpr (FOLD == FP_FOLD) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
        sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
      }
      if (t == 0) stat[wid][i * 8 + r] = make_double2(sum[i], sq[i]);
    }
  }
  __syncthreads();
  if constexpr (FOLD == FP_FOLD) {
    if (threadIdx.x < NT * 8) {
      double s = 0.0, q = 0.0;
#pragma unroll
      for (int w = 0; w < FP_WARPS; ++w) {
        s += stat[w][threadIdx.x].x;
        q += stat[w][threadIdx.x].y;
      }
      norm[threadIdx.x] = finish(s, q);
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < NT * 8 * FP_COLS; e += FP_WARPS * 32) {
    const int c = e % FP_COLS, row = e / FP_COLS, col = n0 + c;
    float v = 0.f;
    if (row < m) {
#pragma unroll
      for (int w = 0; w < FP_WARPS; ++w) v += red[w][row >> 3][c][row & 7];
      v *= w_inv;
      if constexpr (FOLD != FP_PLAIN) v = (v - norm[row].x * __ldg(g.u + col)) * norm[row].y;
      if (g.bias != nullptr) v += __ldg(g.bias + col);
      const long long at = (long long)(first + row) * g.n + col;
      if (g.residual != nullptr) v += g.residual[at];
      if (g.relu) v = v > 0.f ? v : 0.f;
      g.out[at] = v;
    }
    if (g.sums_out != nullptr) {  // (sixteen lanes a row, whole warps)
      double s = v, q = (double)v * (double)v;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
      }
      if (c == 0 && row < m) g.sums_out[(long long)(first + row) * (g.n / FP_COLS) + blockIdx.x] = make_double2(s, q);
    }
  }
}

}  // namespace

bool few_row_pair_supports(int rows, int n, int k) { return rows >= 1 && rows <= 64 && n % FP_COLS == 0 && k % FP_SPAN == 0; }

void launch_few_row_pair(const FewRowPairProduct &p, int rows, cudaStream_t st) {
  if (!few_row_pair_supports(rows, p.n, p.k)) throw std::invalid_argument("litnice_b200: the few-row pair product does not take this shape");
  const FpShape g{p.x, p.w_hi, p.w_lo, p.w_inv, p.bias, p.ln_u, p.residual, p.out, p.sums_in, p.sums_out, rows, p.n, p.k, p.relu};
  // as few tiles of rows per CTA as give no more than four CTAs an SM: the loads of a launch want to be spread (few_row_bf16.cu)
  const int tiles = (rows + 7) / 8;
  const long long blocks = p.n / FP_COLS;
  int nt = 1;
  while (nt < 4 && nt < tiles && blocks * ((tiles + nt - 1) / nt) > 4 * 148) nt *= 2;
  const dim3 grid((unsigned)blocks, (unsigned)((tiles + nt - 1) / nt));
  auto go = [&](auto kernel) { launch_pdl(kernel, grid, dim3(FP_WARPS * 32), 0, st, g_pdl_enabled, g); };
  auto by_k = [&](auto tiles_c, auto fold_c) {
    if (p.k > FP_WARPS * FP_SPAN) go(few_row_pair_kernel<tiles_c.value, fold_c.value, true>);
    else go(few_row_pair_kernel<tiles_c.value, fold_c.value, false>);
  };
  auto by_fold = [&](auto tiles_c) {
    if (p.ln_u == nullptr) by_k(tiles_c, std::integral_constant<int, FP_PLAIN>());
    else if (p.sums_in == nullptr) by_k(tiles_c, std::integral_constant<int, FP_FOLD>());
    else by_k(tiles_c, std::integral_constant<int, FP_FOLD_SUMS>());
  };
  if (nt == 1) by_fold(std::integral_constant<int, 1>());
  else if (nt == 2) by_fold(std::integral_constant<int, 2>());
  else by_fold(std::integral_constant<int, 4>());
}

}  // namespace lb
