// Cached mode, greedy, up to 8 streams, models whose heads fit one cluster of 8 CTAs each: the whole token loop as one
// resident kernel (transformer_layer.cpp:50-92, output_head.cpp:58-70, inference.cpp:188-198 for one row per stream).
//
// What bounds it. A token is a chain of small products with 1 to 2 microseconds of hand-over each; the weights, out of L2,
// would take 11 us a token on these CTAs (six layers of width 512). decode_persistent.cu hands over five times a layer
// through global memory behind a grid-wide barrier. Here a head's cluster does everything that is a matter of that head
// by itself: the QKV product's columns, the attention (CTA r holds the keys at positions r mod 8), the out-projection's
// rows, and a slice of the hidden units in both feed-forward products. Inside a cluster values travel by st.async into the
// readers' shared memory, whose mbarrier counts the bytes. Only the sums over heads and over hidden slices leave the
// cluster, twice a layer: as words that carry their own number (value, epoch), which the readers poll, so that arrival and
// data are one round trip; CTA r adds columns r * d/8 .. of the row and sends them, with the sums for the LayerNorm, to its
// cluster.
//
// Measured, us a token (decode_persistent.cu, here): 6 layers x 512 x 2048, 8 heads, contexts of 230, one stream 172, 56;
// eight streams 461, 124; 2 layers x 64, 2 heads, one stream 46, 18; 3 layers x 512 x 1024, vocabulary 1000, four streams 147, 40.
// A layer of the first takes 8.5 us: products 1.0 each (their weights at 64 KB a CTA come out of shared memory in 0.26),
// words polled 0.8 twice, rows sent and normalised 0.9 twice, attention 1.4, its hand-overs inside the cluster 0.2 each.
//
// Weights are laid out once per load in the order they are used (cl_pack_kernel) and come by bulk copies, a product's with one
// wait, into two buffers: the first product of each half of a layer uses one, the second the other, and a buffer is filled
// for its next use as soon as it has been read, three hand-overs ahead (a ring of 16 KB stages with a wait each: 11.1 us a
// layer, not 8.8). A warp takes four columns, a lane four rows of 128, so that a product's sums meet in shuffles and leave
// from the warp that made them, without a barrier of the CTA.
//
// Every wait is bounded: after a second it gives up, sets the error word and a flag that all CTAs look at; waits return
// at once from then on and the CTAs leave together at the next check, their copies having landed.
#include "common.cuh"
#include "tc_ptx.cuh"

#include <algorithm>

namespace lb {

namespace {

constexpr int CL_CTAS = 8;  // CTAs of a cluster
constexpr int CL_THREADS = 256;
constexpr int CL_WARPS = CL_THREADS / 32;
constexpr int CL_ROWS = 128;  // rows of a pass: four a lane
constexpr int CL_BATCH = 8;  // keys of a warp's trip; the next trip's are in flight with them
constexpr unsigned CL_NO_INDEX = 0xfffffu;

// One product of a CTA: k rows, c columns in groups of four. Layout: [group][pass of up to CL_ROWS rows][4][rows / 4][4 columns]:
// row 4 q + i of the pass at [i][q], so that a warp reads contiguous memory.
struct ClProd {
  int k, c;
};

enum { CL_QKV, CL_WO, CL_W1, CL_W2, CL_HEAD };
struct ClShape {
  int n_layers, heads, dh, d, f, vocab;
  ClProd prod[5];
  int head_tiles;
  // floats: a layer's parts from its start (vectors and QKV, out-projection, vectors and W1, W2), then its end
  unsigned part[5];
  unsigned buffer[2];  // of the first and the second products
  unsigned long long cta_floats;
};

struct ClParams {
  ClShape S;
  const float *packed;
  const char *params;
  const unsigned long long *off;
  int n_streams, cap, ids_ld, out_ld, s0, step0, steps;
  float *kcache, *vcache;
  unsigned long long layer_stride;
  int *ids, *out_tokens;
  LoopState *state;
  float *logits;
  unsigned long long *part;  // [2][heads][MB][d] words (value, epoch)
  unsigned long long *sel;   // [CTAs][MB] words (value, tag, index)
  unsigned *abort;
  DevErr *err;
  unsigned long long *timeline;
};

enum { LN1G, LN1B, QKVW, QKVB, OUTW, OUTB, LN2G, LN2B, W1, B1, W2, B2 };

__device__ __forceinline__ unsigned cl_ld_flag(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void cl_ld_words(const unsigned long long *p, unsigned long long &a, unsigned long long &b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void cl_st_words(unsigned long long *p, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ unsigned long long cl_word(float v, unsigned epoch) {
  return (unsigned long long)__float_as_uint(v) << 32 | epoch;
}
__device__ __forceinline__ void cl_send(unsigned addr, float4 v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_send2(unsigned addr, double a, double b, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];"
               ::"r"(addr), "d"(a), "d"(b), "r"(bar)
               : "memory");
}
// (Waits acquire at the scope of the CTA: its own shared memory holds both the barrier and what has arrived, the bytes ahead of
// their count.)
// A spin's slow turns: true when the run has failed or this wait has taken too long.
static __device__ __noinline__ bool cl_give_up(unsigned *flag, DevErr *err, unsigned long long t0, int where) {
  if (cl_ld_flag(flag) != 0u) return true;
  if (global_timer() - t0 <= WAIT_LIMIT_NS) return false;
  atomicExch(flag, 1u);
  err->code = DEVERR_WAIT_TIMEOUT;
  err->detail = where;
  return true;
}
static __device__ __noinline__ bool cl_wait_slow(unsigned bar, unsigned parity, unsigned *flag, DevErr *err, int where) {
  const unsigned long long t0 = global_timer();
  unsigned spins = 0;
  while (!mbar_try_wait(bar, parity))
    if ((++spins & 63u) == 0 && cl_give_up(flag, err, t0, where)) return true;
  return false;
}

// Requests the part that product ph of half layer i uses (i == 2 n_layers: tile ph of the head) into its buffer.
__device__ __forceinline__ void cl_fetch(const ClShape &S, const float *mine, unsigned dst, unsigned bar, int i, int ph) {
  unsigned floats;
  if (i < 2 * S.n_layers) {
    const int part = (i & 1) * 2 + ph;
    floats = S.part[part + 1] - S.part[part];
    mine += (unsigned long long)(i >> 1) * S.part[4] + S.part[part];
  } else {
    const ClProd &g = S.prod[CL_HEAD];
    floats = (unsigned)(g.k * g.c + (ph == 0 ? 2 * S.d : 0));
    mine += (unsigned long long)S.n_layers * S.part[4] + (ph == 0 ? 0ull : 2ull * S.d + (unsigned long long)ph * (g.k * g.c));
  }
  mbar_expect_tx(bar, floats * 4);
  bulk_load(dst, mine, floats * 4, bar);
}

// One instance of each operator in a loop over half layers: a CTA runs through its code once a layer, and the operators written
// out one after the other were twice the code.
template <int MB, int DH>
__global__ void __launch_bounds__(CL_THREADS, 1) decode_cluster_kernel(const __grid_constant__ ClParams P) {
  extern __shared__ __align__(128) char cl_smem[];
  __shared__ __align__(16) double2 s_stat[2][CL_CTAS][MB];
  __shared__ __align__(8) unsigned long long s_bar[7];
  __shared__ int s_tok[MB];
  __shared__ float s_best[MB * CL_WARPS];
  __shared__ int s_at[MB * CL_WARPS];
  constexpr int WPS = CL_WARPS / MB;  // warps per stream
  constexpr int AP = DH + 4;          // pitch of attention partials: outputs, maximum, sum
  const ClShape &S = P.S;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rank = blockIdx.x % CL_CTAS, head = blockIdx.x / CL_CTAS;
  const int D = S.d, FC = S.f / S.heads, V = S.vocab, B = P.n_streams, SL = D / CL_CTAS, LS = SL / 4;

  float *buffer[2];  // weights of the first and the second products
  buffer[0] = reinterpret_cast<float *>(cl_smem);
  buffer[1] = buffer[0] + S.buffer[0];
  float *rows = buffer[1] + S.buffer[1];  // [2][MB][D] x and y as they arrive
  float *act = rows + 2 * MB * D;                                       // [MB][D] behind the LayerNorm
  float *hid = act + MB * D;                                            // [MB][FC]
  float *qkv = hid + MB * FC;                                           // [MB][3][DH]
  float *ctx = qkv + MB * 3 * DH;                                       // [MB][DH]
  float *att = ctx + MB * DH;                                           // [MB][CL_CTAS][AP]
  float *attw = att + CL_CTAS * MB * AP;                                // [CL_WARPS][AP]
  // barriers: both buffers, x row, y row, q k v, hidden units, attention; their parities by the same index
  enum { BAR_BUFFER = 0, BAR_ROW = 2, BAR_MID = 4, BAR_ATT = 6 };
  const unsigned bars = smem_u32(s_bar);
  auto bytes_of = [&](int i) {
    return (unsigned)(i < BAR_MID ? MB * D * 4 + CL_CTAS * MB * 16 : i == BAR_MID ? MB * 3 * DH * 4 : i == BAR_ATT ? CL_CTAS * MB * AP * 4 : MB * FC * 4);
  };
  bool bad = false;  // this thread knows that the run has failed
  unsigned parities = 0;
  // Everybody waits; one thread opens the barrier's next phase.
  auto wait_exchange = [&](int i) {
    const unsigned bar = bars + 8 * i, parity = parities >> i & 1;
    if (!bad && !mbar_try_wait(bar, parity)) bad = cl_wait_slow(bar, parity, P.abort, P.err, i);
    parities ^= 1u << i;
    if (tid == 0) mbar_expect_tx(bar, bytes_of(i));
  };

  if (tid == 0) {
    for (int i = 0; i <= BAR_ATT; ++i) mbar_init(bars + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int i = BAR_ROW; i <= BAR_ATT; ++i) mbar_expect_tx(bars + 8 * i, bytes_of(i));
  }
  if (tid < MB) s_tok[tid] = 0;
  cluster_sync_all();

  // ---- the weights: requested by the last thread, read by all in the order of use ----
  const float *packed = P.packed + (unsigned long long)blockIdx.x * S.cta_floats;
  unsigned filled = 0;  // a bit per buffer: whether it has been requested an odd number of times
  auto fetch = [&](int i, int ph) {
    const int k = ph & 1;
    cl_fetch(S, packed, smem_u32(buffer[0]) + k * S.buffer[0] * 4, bars + 8 * (BAR_BUFFER + k), i, ph);
    filled ^= 1u << k;
  };
  // The buffer of product ph of half layer i has been read, by every thread of the CTA: behind a barrier, or behind a wait
  // for values that every warp of this CTA sent its part of when it was past its reads.
  auto give_back = [&](int t, int i, int ph) {
    if (tid != CL_THREADS - 1 || bad) return;
    bool again = t + 1 < P.steps;  // for the next token, unless this one still needs it
    if (i < 2 * S.n_layers) {
      ++i;
      if (i < 2 * S.n_layers || ph < S.head_tiles) again = true;
      else i = 0;
    } else if (ph + 2 < S.head_tiles) {
      ph += 2;
      again = true;
    } else {
      i = 0;
      ph &= 1;
    }
    if (again) fetch(i, ph);
  };
  auto wait_buffer = [&](int k) -> const float * {
    const unsigned bar = bars + 8 * (BAR_BUFFER + k), parity = parities >> (BAR_BUFFER + k) & 1;
    if (!bad && !mbar_try_wait(bar, parity)) bad = cl_wait_slow(bar, parity, P.abort, P.err, 80 + k);
    parities ^= 1u << (BAR_BUFFER + k);
    return k ? buffer[1] : buffer[0];
  };
  if (tid == CL_THREADS - 1) {
    fetch(0, 0);
    fetch(0, 1);
  }

  // ---- this thread's four columns of one stream's residual row: sixteen items a warp, the heads in two halves ----
  const int item = wid * 16 + (lane & 15), half = lane >> 4;
  const bool slicing = wid * 16 < LS * MB, slicer = item < LS * MB;
  const int sb = item / LS, sc = rank * SL + item % LS * 4;
  float4 res = make_float4(0.f, 0.f, 0.f, 0.f), b2 = res;

  // ---- keys and values of earlier positions, a batch per warp ----
  constexpr int LPK = DH / 8, KPP = 32 / LPK, NP = CL_BATCH / KPP, VW = DH / 32;
  const int ab = wid / WPS, wi = wid % WPS, sub = lane % LPK, grp = lane / LPK;
  const int key_step = CL_CTAS * WPS, key0 = rank + CL_CTAS * wi;  // positions of the warp's keys: key0 + key_step * i
  const size_t row0 = ((size_t)ab * P.cap + key0) * D + head * DH, key_pitch = (size_t)key_step * D;
  const float *k_at = P.kcache + row0 + grp * key_pitch + sub * 8, *v_at = P.vcache + row0 + lane * VW;
  struct Batch {
    float4 k0[NP], k1[NP];
    float v[CL_BATCH][VW];
  };
  Batch next;
  // keys q0 .. q0 + CL_BATCH of the warp in layer l, those of the first `have`
  auto load_batch = [&](int l, int q0, int have) {
    const size_t at = (size_t)l * P.layer_stride + q0 * key_pitch;
    const float *kp = k_at + at, *vp = v_at + at;
#pragma unroll
    for (int u = 0; u < NP; ++u, kp += key_pitch * KPP) {
      next.k0[u] = next.k1[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (q0 + u * KPP + grp < have) {
        next.k0[u] = __ldcg(reinterpret_cast<const float4 *>(kp));
        next.k1[u] = __ldcg(reinterpret_cast<const float4 *>(kp + 4));
      }
    }
#pragma unroll
    for (int n = 0; n < CL_BATCH; ++n, vp += key_pitch) {
#pragma unroll
      for (int c = 0; c < VW; ++c) next.v[n][c] = 0.f;
      if (q0 + n < have) {
        if constexpr (VW == 2) {
          const float2 x = __ldcg(reinterpret_cast<const float2 *>(vp));
          next.v[n][0] = x.x;
          next.v[n][1] = x.y;
        } else {
          next.v[n][0] = __ldcg(vp);
        }
      }
    }
  };

  const unsigned long long *tail = P.off + (long long)S.n_layers * 12;
  const float scale = 1.0f / sqrtf((float)DH);
  const double inv_d = 1.0 / (double)D;  // exact: D is a power of two
  const int head_c = S.prod[CL_HEAD].c;
  unsigned epoch = 0;
  int stamp_i = 0;
  for (int t = 0; t < P.steps; ++t) {
    const int p = P.s0 + t - 1;  // newest position
    const int have = ab < B && p > key0 ? (p - 1 - key0) / key_step + 1 : 0;  // keys of the warp that the caches hold
    const int mine = ab < B && rank == p % CL_CTAS && p / CL_CTAS % WPS == wi ? have : -1;  // the newest one's place, if it is the warp's
    const bool stamping = P.timeline != nullptr && blockIdx.x == 0 && tid == 0 && t == 10;
#define CL_STAMP() do { if (stamping && stamp_i < 64) P.timeline[stamp_i++] = global_timer(); } while (0)
    CL_STAMP();
    float best = -3.402823466e+38f;  // head: of this lane's stream, the columns of this warp
    unsigned best_at = CL_NO_INDEX;
    // Half layers: attention (x row, q k v, out-projection), feed-forward (y row, both products); the head at the end.
#pragma unroll 1
    for (int i = 0; i <= 2 * S.n_layers; ++i) {
      const int l = i >> 1, f = i & 1;  // f: the feed-forward half, and which of the two rows
      const bool last = i == 2 * S.n_layers;
      const float *vec = wait_buffer(0);
      // ---- this CTA's slice of the row, to the cluster: the newest token's embedding, or the row so far + what the heads
      // or hidden slices made, once every cluster's words carry this epoch ----
      if (slicing) {
        if (i == 0) {
          if (slicer) {  // (both halves alike)
            res = make_float4(0.f, 0.f, 0.f, 0.f);
            if (sb < B) {
              int id = t == 0 ? P.ids[(long long)sb * P.ids_ld + p] : s_tok[sb];
              if (id < 0 || id >= V) {
                if (head == 0 && sc == 0) {
                  P.err->code = DEVERR_BAD_TOKEN_ID;
                  P.err->detail = id;
                }
                id = 0;
              }
              const float *a = reinterpret_cast<const float *>(P.params + tail[0]) + (long long)id * D + sc;
              const float *e = reinterpret_cast<const float *>(P.params + tail[1]) + (long long)p * D + sc;
              res = make_float4(__ldg(a) + __ldg(e), __ldg(a + 1) + __ldg(e + 1), __ldg(a + 2) + __ldg(e + 2), __ldg(a + 3) + __ldg(e + 3));
            }
          }
        } else {
          float4 bias = b2;
          if (f) {  // this stage holds both of the layer's: the out-projection's, and W2's for the next row
            const float *own = vec + 2 * D + FC / CL_CTAS + (sc - rank * SL);
            bias = *reinterpret_cast<const float4 *>(own);
            b2 = *reinterpret_cast<const float4 *>(own + SL);
          }
          const int n = (S.heads + 1) / 2, h0 = half * n, h1 = min(S.heads, h0 + n);
          const unsigned long long *src = P.part + ((unsigned long long)((f ? 0 : S.heads) + h0) * MB + sb) * D + sc;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (slicer) {
            unsigned long long w[4][4], t0 = 0;
            unsigned spins = 0;
#pragma unroll 1
            while (true) {
              unsigned off = 0;
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                w[h][0] = w[h][1] = w[h][2] = w[h][3] = epoch;  // (no such head: zero)
                if (h0 + h < h1) {
                  cl_ld_words(src + (unsigned)(h * MB * D), w[h][0], w[h][1]);
                  cl_ld_words(src + (unsigned)(h * MB * D) + 2, w[h][2], w[h][3]);
                }
              }
#pragma unroll
              for (int h = 0; h < 4; ++h)
#pragma unroll
                for (int c = 0; c < 4; ++c) off |= (unsigned)w[h][c] ^ epoch;
              if (off == 0 || bad) break;
              if (t0 == 0) t0 = global_timer();
              if ((++spins & 63u) == 0) bad = cl_give_up(P.abort, P.err, t0, 81);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              v.x += __uint_as_float((unsigned)(w[h][0] >> 32));
              v.y += __uint_as_float((unsigned)(w[h][1] >> 32));
              v.z += __uint_as_float((unsigned)(w[h][2] >> 32));
              v.w += __uint_as_float((unsigned)(w[h][3] >> 32));
            }
          }
          __syncwarp();
          v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);  // (the same bits in both halves)
          v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
          v.z += __shfl_xor_sync(0xffffffffu, v.z, 16);
          v.w += __shfl_xor_sync(0xffffffffu, v.w, 16);
          if (slicer) res = make_float4((v.x + bias.x) + res.x, (v.y + bias.y) + res.y, (v.z + bias.z) + res.z, (v.w + bias.w) + res.w);
        }
        CL_STAMP();
        // the slice and its sums for the LayerNorm, each half to four of the CTAs
        const double a = res.x, b = res.y, c = res.z, e = res.w;
        double sum = (a + b) + (c + e), sq = (a * a + b * b) + (c * c + e * e);
#pragma unroll 1
        for (int o = LS >> 1; o > 0; o >>= 1) {
          sum += __shfl_xor_sync(0xffffffffu, sum, o);
          sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        if (slicer) {
          const unsigned dst = smem_u32(rows + (f * MB + sb) * D + sc), stat = smem_u32(&s_stat[f][rank][sb]), bar = bars + 8 * (BAR_ROW + f);
#pragma unroll
          for (int x = 0; x < CL_CTAS / 2; ++x) {
            const int r = half * (CL_CTAS / 2) + x;
            const unsigned rbar = cluster_map(bar, r);
            cl_send(cluster_map(dst, r), res, rbar);
            if (item % LS == 0) cl_send2(cluster_map(stat, r), sum, sq, rbar);
          }
        }
      }
      // ---- act = LayerNorm(row) (device_backend.cpp:1247-1279: mean and biased variance in double, inv_std =
      // 1/sqrt(float(var) + 1e-5f)); the stage holds scale [D], shift [D] ----
      wait_exchange(BAR_ROW + f);
      {
        const int b = wid / WPS;
        double sum = 0.0, sq = 0.0;
#pragma unroll
        for (int r = 0; r < CL_CTAS; ++r) {
          const double2 v = s_stat[f][r][b];
          sum += v.x;
          sq += v.y;
        }
        const double mean = sum * inv_d;
        double var = sq * inv_d - mean * mean;
        if (var < 0.0) var = 0.0;
        const float inv_std = 1.0f / sqrtf((float)var + 1e-5f), fmean = (float)mean;
#pragma unroll 1
        for (int c = tid % (WPS * 32); c < D; c += WPS * 32)
          act[b * D + c] = __fadd_rn(__fmul_rn((rows[(f * MB + b) * D + c] - fmean) * inv_std, vec[c]), vec[D + c]);
      }
      if (__syncthreads_or(bad)) goto out;
      if (i > 0) give_back(t, i - 1, 1);
      if (!f && !last) load_batch(l, 0, have);  // (on their way during the product)
      CL_STAMP();
      // ---- the half's two products; of the head, its tiles ----
      const int products = last ? S.head_tiles : 2;
#pragma unroll 1
      for (int ph = 0; ph < products; ++ph) {
        const bool second = ph == 1 && !last;
        const float *in = act;
        int pitch = D;
        if (second) {
          wait_exchange(BAR_MID + f);
          give_back(t, i, 0);
          CL_STAMP();
          in = f ? hid : ctx;
          pitch = f ? FC : DH;
        }
        if (second && !f) {
          // ---- attention: CTA r has the keys at positions r mod 8, a warp every WPS-th of them ----
          if (rank == p % CL_CTAS)
            for (int e = tid; e < B * 2 * DH; e += CL_THREADS) {
              const int b = e / (2 * DH), c = e % (2 * DH);
              float *dst = (c < DH ? P.kcache : P.vcache) + (unsigned long long)l * P.layer_stride;
              dst[((long long)b * P.cap + p) * D + head * DH + c % DH] = qkv[b * 3 * DH + DH + c];
            }
          {
            const float *q = qkv + ab * 3 * DH;
            const float4 q0 = *reinterpret_cast<const float4 *>(q + sub * 8), q1 = *reinterpret_cast<const float4 *>(q + sub * 8 + 4);
            float m = -INFINITY, o[VW];
            double lsum = 0.0;
#pragma unroll
            for (int c = 0; c < VW; ++c) o[c] = 0.f;
            const int keys = mine >= 0 ? have + 1 : have;
#pragma unroll 1
            for (int base = 0; base < keys; base += CL_BATCH) {
              Batch now = next;
              if (base + CL_BATCH < keys) load_batch(l, base + CL_BATCH, have);
              if (mine >= base && mine < base + CL_BATCH) {  // the newest position's key and value are this step's own
#pragma unroll
                for (int u = 0; u < NP; ++u)
                  if (base + u * KPP + grp == mine) {
                    now.k0[u] = *reinterpret_cast<const float4 *>(q + DH + sub * 8);
                    now.k1[u] = *reinterpret_cast<const float4 *>(q + DH + sub * 8 + 4);
                  }
#pragma unroll
                for (int n = 0; n < CL_BATCH; ++n)
                  if (base + n == mine)
#pragma unroll
                    for (int c = 0; c < VW; ++c) now.v[n][c] = q[2 * DH + lane * VW + c];
              }
              float sco[NP], bm = -INFINITY;
#pragma unroll
              for (int u = 0; u < NP; ++u) {
                float dot = q0.x * now.k0[u].x;
                dot = fmaf(q0.y, now.k0[u].y, dot);
                dot = fmaf(q0.z, now.k0[u].z, dot);
                dot = fmaf(q0.w, now.k0[u].w, dot);
                dot = fmaf(q1.x, now.k1[u].x, dot);
                dot = fmaf(q1.y, now.k1[u].y, dot);
                dot = fmaf(q1.z, now.k1[u].z, dot);
                dot = fmaf(q1.w, now.k1[u].w, dot);
#pragma unroll
                for (int x = LPK >> 1; x > 0; x >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, x);
                sco[u] = base + u * KPP + grp < keys ? dot * scale : -INFINITY;
                bm = fmaxf(bm, sco[u]);
              }
#pragma unroll
              for (int x = LPK; x < 32; x <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, x));
              const float mn = fmaxf(m, bm);
              if (base > 0) {
                const float keep = m == -INFINITY ? 0.f : expf(m - mn);
                lsum *= (double)keep;
#pragma unroll
                for (int c = 0; c < VW; ++c) o[c] *= keep;
              }
              m = mn;
#pragma unroll
              for (int u = 0; u < NP; ++u) {
                sco[u] = sco[u] == -INFINITY ? 0.f : expf(sco[u] - m);
                lsum += (double)sco[u];
              }
#pragma unroll
              for (int n = 0; n < CL_BATCH; ++n) {
                const float w = __shfl_sync(0xffffffffu, sco[n / KPP], n % KPP * LPK);
#pragma unroll
                for (int c = 0; c < VW; ++c) o[c] = fmaf(w, now.v[n][c], o[c]);
              }
            }
#pragma unroll
            for (int x = LPK; x < 32; x <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, x);
#pragma unroll
            for (int c = 0; c < VW; ++c) attw[wid * AP + lane * VW + c] = o[c];
            if (lane == 0) {
              attw[wid * AP + DH] = m;
              attw[wid * AP + DH + 1] = (float)lsum;
            }
          }
          __syncthreads();
          // joined over the warps of a stream and sent: outputs relative to the CTA's maximum, maximum, sum
          {
            const float *aw = attw + ab * WPS * AP;
            const float mw = aw[lane % WPS * AP + DH];
            float m = mw;
#pragma unroll
            for (int x = WPS >> 1; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
            const float fw = mw == -INFINITY ? 0.f : expf(mw - m);
            double sum = (double)aw[lane % WPS * AP + DH + 1] * (double)fw;
#pragma unroll
            for (int x = WPS >> 1; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            float fa[WPS];
#pragma unroll
            for (int w = 0; w < WPS; ++w) fa[w] = __shfl_sync(0xffffffffu, fw, w);
            // a lane per four outputs, one more for maximum and sum; the stream's warps share the receivers
            float4 v = make_float4(m, (float)sum, 0.f, 0.f);
            if (lane < DH / 4) {
              v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int w = 0; w < WPS; ++w) {
                const float4 y = *reinterpret_cast<const float4 *>(aw + w * AP + lane * 4);
                v.x = fmaf(y.x, fa[w], v.x);
                v.y = fmaf(y.y, fa[w], v.y);
                v.z = fmaf(y.z, fa[w], v.z);
                v.w = fmaf(y.w, fa[w], v.w);
              }
            }
            if (lane <= DH / 4) {
              const unsigned dst = smem_u32(att + (ab * CL_CTAS + rank) * AP + lane * 4);
#pragma unroll 1
              for (int r = wi; r < CL_CTAS; r += WPS) cl_send(cluster_map(dst, r), v, cluster_map(bars + 8 * BAR_ATT, r));
            }
          }
          CL_STAMP();
          wait_exchange(BAR_ATT);
          // joined over the CTAs
#pragma unroll 1
          for (int x = tid; x < MB * DH; x += CL_THREADS) {  // (whole warps, one stream each)
            const float *a = att + x / DH * CL_CTAS * AP;
            const float mr = a[lane % CL_CTAS * AP + DH];
            float m = mr;
#pragma unroll
            for (int y = CL_CTAS >> 1; y > 0; y >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, y));
            const float fr = mr == -INFINITY ? 0.f : expf(mr - m);
            double sum = (double)a[lane % CL_CTAS * AP + DH + 1] * (double)fr;
#pragma unroll
            for (int y = CL_CTAS >> 1; y > 0; y >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, y);
            float v = 0.f;
#pragma unroll
            for (int r = 0; r < CL_CTAS; ++r) v = fmaf(a[r * AP + x % DH], __shfl_sync(0xffffffffu, fr, r), v);
            ctx[x] = x / DH < B ? v / (float)sum : 0.f;
          }
          __syncthreads();
          CL_STAMP();
        }
        const int k = second ? (f ? FC : DH) : D;
        const int c = last ? head_c : second ? SL : f ? FC / CL_CTAS : 3 * DH / CL_CTAS;
        if (second) ++epoch;
        // in[MB][pitch] (shared) times the buffer's weights. G: groups of a warp that go together
        const float4 *weights = reinterpret_cast<const float4 *>(last ? (ph == 0 ? vec + 2 * D : wait_buffer(ph & 1))
                                                                      : second ? wait_buffer(1) : vec + 2 * D + c + (f ? 2 * SL : 0));
        const int groups = c >> 2;
        auto multiply = [&](auto gc) {
          constexpr int G = gc.value, AHEAD = (MB >= 4 ? 2 : 4) / G;  // passes whose loads are in flight together
          constexpr int LANES = 32 / (MB * G);                       // lanes that have one stream's sums of one group
#pragma unroll 1
          for (int tile = wid; tile < groups; tile += CL_WARPS * G) {
            float v[4 * MB * G];
#pragma unroll
            for (int x = 0; x < 4 * MB * G; ++x) v[x] = 0.f;
#pragma unroll 1
            for (int r0 = 0; r0 < k; r0 += CL_ROWS * AHEAD) {
              float4 wv[G][AHEAD][4];
#pragma unroll
              for (int e = 0; e < G; ++e)
#pragma unroll
                for (int a = 0; a < AHEAD; ++a) {
                  const int at = r0 + a * CL_ROWS, nq = min(CL_ROWS, k - at) >> 2, group = tile + e * CL_WARPS;
                  const float4 *w = weights + group * k + at + lane;
#pragma unroll
                  for (int c = 0; c < 4; ++c) wv[e][a][c] = lane < nq && group < groups ? w[c * nq] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
              for (int a = 0; a < AHEAD; ++a) {
                const int at = r0 + a * CL_ROWS + lane * 4;
#pragma unroll
                for (int b = 0; b < MB; ++b) {
                  const float4 x = at < k ? *reinterpret_cast<const float4 *>(in + b * pitch + at) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                  for (int e = 0; e < G; ++e) {
                    float *y = v + (e * MB + b) * 4;
                    const float4(&w)[4] = wv[e][a];
                    y[0] = fmaf(x.w, w[3].x, fmaf(x.z, w[2].x, fmaf(x.y, w[1].x, fmaf(x.x, w[0].x, y[0]))));
                    y[1] = fmaf(x.w, w[3].y, fmaf(x.z, w[2].y, fmaf(x.y, w[1].y, fmaf(x.x, w[0].y, y[1]))));
                    y[2] = fmaf(x.w, w[3].z, fmaf(x.z, w[2].z, fmaf(x.y, w[1].z, fmaf(x.x, w[0].z, y[2]))));
                    y[3] = fmaf(x.w, w[3].w, fmaf(x.z, w[2].w, fmaf(x.y, w[1].w, fmaf(x.x, w[0].w, y[3]))));
                  }
                }
              }
            }
            // Sums over the lanes: as long as a lane has several, it passes half of them on and keeps the other half's sums;
            // value (group * MB + stream) * 4 + column ends in lanes value * LANES / 4 ..
            int held = 4 * MB * G;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              if (held > 1) {
                held >>= 1;
                const bool up = lane & o;
#pragma unroll
                for (int c = 0; c < 2 * MB * G; ++c)
                  if (c < held) {
                    const float pass_on = up ? v[c] : v[c + held], keep = up ? v[c + held] : v[c];
                    v[c] = keep + __shfl_xor_sync(0xffffffffu, pass_on, o);
                  }
              } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
              }
            }
            const int from = lane & ~(LANES - 1), b = lane / LANES % MB, j = lane % LANES, group = tile + lane / (LANES * MB) * CL_WARPS;
            float4 sum;
            sum.x = __shfl_sync(0xffffffffu, v[0], from);
            sum.y = __shfl_sync(0xffffffffu, v[0], from + LANES / 4);
            sum.z = __shfl_sync(0xffffffffu, v[0], from + LANES / 2);
            sum.w = __shfl_sync(0xffffffffu, v[0], from + LANES / 4 * 3);
            // four columns of stream b, in lanes j = 0 .. LANES - 1
            if (group >= groups) {
            } else if (last) {
              const int col = (blockIdx.x * S.head_tiles + ph) * c + group * 4;
              const float x[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
              for (int y = 0; y < 4; ++y)
                if (col + y < V) {
                  if (x[y] > best || (x[y] == best && best_at == CL_NO_INDEX)) {
                    best = x[y];
                    best_at = (unsigned)(col + y);
                  }
                  if (j == 0 && t + 1 == P.steps && b < B) P.logits[(long long)b * V + col + y] = x[y];
                }
            } else if (second) {  // this head's, or slice's, part of columns rank * SL ..
              if (j == 0) {
                unsigned long long *dst = P.part + ((unsigned long long)(f * S.heads + head) * MB + b) * D + rank * SL + group * 4;
                cl_st_words(dst, cl_word(sum.x, epoch), cl_word(sum.y, epoch));
                cl_st_words(dst + 2, cl_word(sum.z, epoch), cl_word(sum.w, epoch));
              }
            } else {  // to the cluster, with bias (and ReLU)
              const float4 bias = *reinterpret_cast<const float4 *>(vec + 2 * D + group * 4);
              sum = make_float4(sum.x + bias.x, sum.y + bias.y, sum.z + bias.z, sum.w + bias.w);
              constexpr int PER = DH / 32;  // groups of q, of k, of v
              const float *dst = f ? hid + b * FC + rank * c + group * 4
                                   : qkv + (b * 3 + group / PER) * DH + rank * (DH / CL_CTAS) + group % PER * 4;
              if (f)
                sum = make_float4(sum.x > 0.f ? sum.x : 0.f, sum.y > 0.f ? sum.y : 0.f, sum.z > 0.f ? sum.z : 0.f, sum.w > 0.f ? sum.w : 0.f);
              const unsigned local = smem_u32(dst), bar = bars + 8 * (BAR_MID + f);
#pragma unroll
              for (int r = j; r < CL_CTAS; r += LANES) cl_send(cluster_map(local, r), sum, cluster_map(bar, r));
            }
          }
        };
        // Two groups at once where a warp has two: one chain of loads and shuffles instead of two. (The head has at most one,
        // whose maxima its lanes keep by stream.)
        if (MB <= 2 && groups > CL_WARPS) multiply(std::integral_constant<int, MB <= 2 ? 2 : 1>());
        else multiply(std::integral_constant<int, 1>());
        if (last) {
          __syncthreads();
          give_back(t, i, ph);
        }
        CL_STAMP();
      }
    }
    // ---- the first maximum of all logits (inference.cpp:188-198: strict '>' from index 0) ----
    {
      constexpr int LANES = 32 / MB;
      if (lane % LANES == 0) {
        s_best[lane / LANES * CL_WARPS + wid] = best;
        s_at[lane / LANES * CL_WARPS + wid] = (int)best_at;
      }
      __syncthreads();
      const unsigned tag = (unsigned)(t + 1) & 0xfffu;
      if (wid < MB) {  // a warp per stream: this CTA's, then all CTAs'
        best = lane < CL_WARPS ? s_best[wid * CL_WARPS + lane] : -3.402823466e+38f;
        best_at = lane < CL_WARPS ? (unsigned)s_at[wid * CL_WARPS + lane] : CL_NO_INDEX;
#pragma unroll 1
        for (int round = 0; round < 2; ++round) {
          if (round == 1) {
            best = -3.402823466e+38f;
            best_at = CL_NO_INDEX;
#pragma unroll 1
            for (int c = lane; c < S.heads * CL_CTAS; c += 32) {
              unsigned long long word, t0 = 0;
              unsigned spins = 0;
              while (true) {
                asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(word) : "l"(P.sel + (long long)c * MB + wid) : "memory");
                if (((unsigned)word >> 20) == tag || bad) break;
                if (t0 == 0) t0 = global_timer();
                if ((++spins & 63u) == 0) bad = cl_give_up(P.abort, P.err, t0, 82);
              }
              const float ov = __uint_as_float((unsigned)(word >> 32));
              const unsigned oi = (unsigned)word & CL_NO_INDEX;
              if (ov > best || (ov == best && oi < best_at)) {
                best = ov;
                best_at = oi;
              }
            }
            __syncwarp();
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const unsigned oi = __shfl_xor_sync(0xffffffffu, best_at, o);
            if (ov > best || (ov == best && oi < best_at)) {
              best = ov;
              best_at = oi;
            }
          }
          if (round == 0 && lane == 0) {
            const unsigned long long word = (unsigned long long)__float_as_uint(best) << 32 | tag << 20 | best_at;
            asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(P.sel + (long long)blockIdx.x * MB + wid), "l"(word) : "memory");
          }
        }
        if (lane == 0) {
          const int token = best_at == CL_NO_INDEX ? 0 : (int)best_at;
          s_tok[wid] = token;
          if (blockIdx.x == 0 && wid < B) {
            P.ids[(long long)wid * P.ids_ld + p + 1] = token;
            P.out_tokens[(long long)wid * P.out_ld + P.step0 + t] = token;
          }
        }
      }
    }
    if (__syncthreads_or(bad)) goto out;
    CL_STAMP();
  }
  if (blockIdx.x == 0 && tid == 0) {
    P.state->s = P.s0 + P.steps;
    P.state->step = P.step0 + P.steps;
  }
out:
  // A run that ends early has copies in flight: they land before the CTA leaves.
  if (tid == CL_THREADS - 1) {
    const unsigned long long t0 = global_timer();
    for (int k = 0; k < 2; ++k) {
      while (!mbar_try_wait(bars + 8 * (BAR_BUFFER + k), (filled >> k & 1) ^ 1) && global_timer() - t0 < WAIT_LIMIT_NS) {
      }
    }
  }
  __syncthreads();
  cluster_sync_all();
  // Nobody's shared memory goes away under a peer's stores: in a run that ended well all that was sent has been waited for; in
  // one that failed what is on its way has a millisecond to land.
  if (cl_ld_flag(P.abort) != 0u) {
    const unsigned long long t0 = global_timer();
    while (global_timer() - t0 < 1000000ull) {
    }
  }
}

// ---- the weights of every CTA in the order it uses them ----
struct ClPack {
  ClShape S;
  const char *params;
  const unsigned long long *off;
  float *packed;
};

// One product's rows r and columns c of src(r, c).
template <class Src>
__device__ float *cl_pack_product(float *dst, const ClProd &g, Src src) {
  for (int i = threadIdx.x; i < g.k * g.c; i += CL_THREADS) {
    const int group = i / (g.k * 4), in_group = i - group * g.k * 4, pass = in_group / (CL_ROWS * 4), at = in_group - pass * CL_ROWS * 4;
    const int nq = min(CL_ROWS, g.k - pass * CL_ROWS) >> 2;
    const int col = at & 3, q = (at >> 2) % nq, row = (at >> 2) / nq;
    dst[i] = src(pass * CL_ROWS + q * 4 + row, group * 4 + col);
  }
  return dst + g.k * g.c;
}
template <class Src>
__device__ float *cl_pack_row(float *dst, int n, Src src) {
  for (int i = threadIdx.x; i < n; i += CL_THREADS) dst[i] = src(i);
  return dst + n;
}

// blockIdx.x: the CTA whose weights they are; blockIdx.y: layer, or behind the last one the head
__global__ void __launch_bounds__(CL_THREADS) cl_pack_kernel(const __grid_constant__ ClPack P) {
  const ClShape &S = P.S;
  const int rank = blockIdx.x % CL_CTAS, head = blockIdx.x / CL_CTAS, l = blockIdx.y;
  const int D = S.d, F = S.f, FC = F / S.heads, SL = D / CL_CTAS, QD = S.dh / CL_CTAS, C1 = S.prod[CL_W1].c;
  float *dst = P.packed + (unsigned long long)blockIdx.x * S.cta_floats + (unsigned long long)l * S.part[4];
  if (l == S.n_layers) {
    const unsigned long long *tail = P.off + (long long)l * 12;
    const float *g = reinterpret_cast<const float *>(P.params + tail[2]), *b = reinterpret_cast<const float *>(P.params + tail[3]),
                *w = reinterpret_cast<const float *>(P.params + tail[4]);
    dst = cl_pack_row(dst, D, [&](int i) { return g[i]; });
    dst = cl_pack_row(dst, D, [&](int i) { return b[i]; });
    for (int t = 0; t < S.head_tiles; ++t) {
      const int c0 = (blockIdx.x * S.head_tiles + t) * S.prod[CL_HEAD].c;
      dst = cl_pack_product(dst, S.prod[CL_HEAD], [&](int r, int c) { return c0 + c < S.vocab ? w[(long long)r * S.vocab + c0 + c] : 0.f; });
    }
    return;
  }
  auto off = [&](int which) { return reinterpret_cast<const float *>(P.params + P.off[l * 12 + which]); };
  const float *g1 = off(LN1G), *s1 = off(LN1B), *wq = off(QKVW), *bq = off(QKVB), *wo = off(OUTW), *bo = off(OUTB), *g2 = off(LN2G),
              *s2 = off(LN2B), *w1 = off(W1), *b1 = off(B1), *w2 = off(W2), *b2 = off(B2);
  auto qkv_col = [&](int c) { return c / QD * D + head * S.dh + rank * QD + c % QD; };  // QD columns of q, of k, of v
  dst = cl_pack_row(dst, D, [&](int i) { return g1[i]; });
  dst = cl_pack_row(dst, D, [&](int i) { return s1[i]; });
  dst = cl_pack_row(dst, S.prod[CL_QKV].c, [&](int i) { return bq[qkv_col(i)]; });
  dst = cl_pack_product(dst, S.prod[CL_QKV], [&](int r, int c) { return wq[(long long)r * 3 * D + qkv_col(c)]; });
  dst = cl_pack_product(dst, S.prod[CL_WO], [&](int r, int c) { return wo[(long long)(head * S.dh + r) * D + rank * SL + c]; });
  dst = cl_pack_row(dst, D, [&](int i) { return g2[i]; });
  dst = cl_pack_row(dst, D, [&](int i) { return s2[i]; });
  dst = cl_pack_row(dst, C1, [&](int i) { return b1[head * FC + rank * C1 + i]; });
  dst = cl_pack_row(dst, SL, [&](int i) { return bo[rank * SL + i]; });
  dst = cl_pack_row(dst, SL, [&](int i) { return b2[rank * SL + i]; });
  dst = cl_pack_product(dst, S.prod[CL_W1], [&](int r, int c) { return w1[(long long)r * F + head * FC + rank * C1 + c]; });
  cl_pack_product(dst, S.prod[CL_W2], [&](int r, int c) { return w2[(long long)(head * FC + r) * D + rank * SL + c]; });
}

int cl_rows(int n_streams) { return n_streams <= 1 ? 1 : n_streams <= 2 ? 2 : n_streams <= 4 ? 4 : 8; }

// False: this kernel does not take the model.
bool cl_shape(int n_layers, int heads, int d, int f, int vocab, ClShape &S) {
  if (heads != 1 && heads != 2 && heads != 4 && heads != 8) return false;  // a cluster each, all resident; rows are powers of two
  if (d != heads * 32 && d != heads * 64) return false;
  if (f < heads * 32 || f % (heads * 32) != 0 || f > heads * CL_CTAS * 128) return false;  // 4 .. 128 hidden units a CTA
  if (n_layers < 1 || vocab < 1 || vocab >= (int)CL_NO_INDEX) return false;
  S = ClShape{};
  S.n_layers = n_layers;
  S.heads = heads;
  S.dh = d / heads;
  S.d = d;
  S.f = f;
  S.vocab = vocab;
  const int fc = f / heads, sl = d / CL_CTAS, ctas = heads * CL_CTAS;
  S.prod[CL_QKV] = ClProd{d, 3 * S.dh / CL_CTAS};
  S.prod[CL_WO] = ClProd{S.dh, sl};
  S.prod[CL_W1] = ClProd{d, fc / CL_CTAS};
  S.prod[CL_W2] = ClProd{fc, sl};
  const int groups = (vocab + 4 * ctas - 1) / (4 * ctas);  // columns of the head a CTA has, by four
  S.head_tiles = (groups + CL_WARPS - 1) / CL_WARPS;
  S.prod[CL_HEAD] = ClProd{d, (groups + S.head_tiles - 1) / S.head_tiles * 4};
  auto floats = [&](int i) { return (unsigned)(S.prod[i].k * S.prod[i].c); };
  S.part[1] = 2 * d + S.prod[CL_QKV].c + floats(CL_QKV);
  S.part[2] = S.part[1] + floats(CL_WO);
  S.part[3] = S.part[2] + 2 * d + S.prod[CL_W1].c + 2 * sl + floats(CL_W1);
  S.part[4] = S.part[3] + floats(CL_W2);
  S.buffer[0] = std::max({S.part[1], S.part[3] - S.part[2], 2 * d + floats(CL_HEAD)});
  S.buffer[1] = std::max({floats(CL_WO), floats(CL_W2), S.head_tiles > 1 ? floats(CL_HEAD) : 0u});
  S.cta_floats = (unsigned long long)n_layers * S.part[4] + 2ull * d + (unsigned long long)S.head_tiles * floats(CL_HEAD);
  return true;
}

size_t cl_smem_bytes(const ClShape &S, int mb) {
  return 4 * ((size_t)S.buffer[0] + S.buffer[1] + (size_t)3 * mb * S.d + (size_t)mb * (S.f / S.heads) + (size_t)mb * 4 * S.dh +
              (size_t)CL_CTAS * mb * (S.dh + 4) + (size_t)CL_WARPS * (S.dh + 4));
}
constexpr size_t CL_SMEM = 227 * 1024 - 4096;  // (static shared memory: up to 2 KB)

template <int MB, int DH>
cudaLaunchConfig_t cl_config(const ClShape &S, cudaLaunchAttribute (&attr)[2], cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(S.heads * CL_CTAS));
  cfg.blockDim = dim3(CL_THREADS);
  cfg.dynamicSmemBytes = cl_smem_bytes(S, MB);
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL_CTAS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  LB_CUDA(cudaFuncSetAttribute(decode_cluster_kernel<MB, DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM));
  return cfg;
}

template <int MB, int DH>
void cl_launch(const ClParams &P, cudaStream_t st) {
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = cl_config<MB, DH>(P.S, attr, st);
  LB_CUDA(cudaLaunchKernelEx(&cfg, decode_cluster_kernel<MB, DH>, P));
}

// Whether all clusters are resident at once on an otherwise empty device.
template <int MB, int DH>
bool cl_fits(const ClShape &S) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = cl_config<MB, DH>(S, attr, nullptr);
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, decode_cluster_kernel<MB, DH>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n >= S.heads;
}

template <class Fn>
auto cl_dispatch(int mb, int dh, Fn fn) {
  if (dh == 64) {
    if (mb == 1) return fn(std::integral_constant<int, 1>(), std::integral_constant<int, 64>());
    if (mb == 2) return fn(std::integral_constant<int, 2>(), std::integral_constant<int, 64>());
    if (mb == 4) return fn(std::integral_constant<int, 4>(), std::integral_constant<int, 64>());
    return fn(std::integral_constant<int, 8>(), std::integral_constant<int, 64>());
  }
  if (mb == 1) return fn(std::integral_constant<int, 1>(), std::integral_constant<int, 32>());
  if (mb == 2) return fn(std::integral_constant<int, 2>(), std::integral_constant<int, 32>());
  if (mb == 4) return fn(std::integral_constant<int, 4>(), std::integral_constant<int, 32>());
  return fn(std::integral_constant<int, 8>(), std::integral_constant<int, 32>());
}

}  // namespace

bool decode_cluster_supports(int n_streams, int n_layers, int n_heads, int d_model, int d_ff, int vocab) {
  ClShape S;
  if (n_streams < 1 || n_streams > 8 || !cl_shape(n_layers, n_heads, d_model, d_ff, vocab, S)) return false;
  const int mb = cl_rows(n_streams);
  return cl_smem_bytes(S, mb) <= CL_SMEM && cl_dispatch(mb, S.dh, [&](auto m, auto h) { return cl_fits<m.value, h.value>(S); });
}

size_t decode_cluster_packed_floats(int n_layers, int n_heads, int d_model, int d_ff, int vocab) {
  ClShape S;
  return cl_shape(n_layers, n_heads, d_model, d_ff, vocab, S) ? (size_t)S.cta_floats * n_heads * CL_CTAS : 0;
}

size_t decode_cluster_words(int n_heads, int d_model) { return (size_t)8 * (2 * n_heads * d_model + n_heads * CL_CTAS); }

void launch_decode_cluster_pack(const DecodePersistentArgs &a, float *packed, cudaStream_t st) {
  ClPack P{};
  if (!cl_shape(a.n_layers, a.n_heads, a.d_model, a.d_ff, a.vocab, P.S))
    throw std::invalid_argument("litnice_b200: the cluster decode kernel does not take this shape");
  P.params = a.params;
  P.off = a.offsets;
  P.packed = packed;
  cl_pack_kernel<<<dim3((unsigned)(a.n_heads * CL_CTAS), (unsigned)(a.n_layers + 1)), CL_THREADS, 0, st>>>(P);
  LB_LAUNCH_CHECK();
}

void launch_decode_cluster(const DecodePersistentArgs &a, const float *packed, unsigned long long *words, cudaStream_t st) {
  ClParams P{};
  const int mb = cl_rows(a.n_streams);
  if (!cl_shape(a.n_layers, a.n_heads, a.d_model, a.d_ff, a.vocab, P.S))
    throw std::invalid_argument("litnice_b200: the cluster decode kernel does not take this shape");
  P.packed = packed;
  P.params = a.params;
  P.off = a.offsets;
  P.n_streams = a.n_streams;
  P.cap = a.cap;
  P.ids_ld = a.ids_ld;
  P.out_ld = a.out_ld;
  P.s0 = a.s0;
  P.step0 = a.step0;
  P.steps = a.steps;
  P.kcache = a.kcache;
  P.vcache = a.vcache;
  P.layer_stride = a.layer_stride;
  P.ids = a.ids;
  P.out_tokens = a.out_tokens;
  P.state = a.state;
  P.logits = a.logits;
  P.part = words;
  P.sel = words + (size_t)2 * a.n_heads * mb * a.d_model;
  P.abort = a.barrier + 1;
  P.err = a.err;
  P.timeline = a.timeline;
  LB_CUDA(cudaMemsetAsync(a.barrier, 0, 8, st));
  LB_CUDA(cudaMemsetAsync(words, 0, decode_cluster_words(a.n_heads, a.d_model) * 8, st));
  cl_dispatch(mb, P.S.dh, [&](auto m, auto h) { cl_launch<m.value, h.value>(P, st); });
}

}  // namespace lb
