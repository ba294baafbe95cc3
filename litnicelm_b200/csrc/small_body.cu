// Transformer::forward over all rows up to the last layer's output for small models (width up to 128):
// embedding and every layer (transformer.cpp:70-114, transformer_layer.cpp:50-92, self_attention.cpp:52-103,
// ffn.cpp:50-62) in one launch, where the operators one by one are eleven launches of 6 to 7 us that
// compute next to nothing each.
//
// A stream belongs to a cluster of eight CTAs; row block j (eight rows) to CTA j mod 8, so that the causal
// attention's work is even. Only keys and values cross CTAs, through global memory with one cluster
// barrier per layer (two buffers in turn: a CTA overwrites one only after a barrier that every CTA reaches
// past its last read). Everything else of a row stays in its CTA's shared memory.
//
// Bound by latency, not by bytes or products: a product of eight rows is cut into (four columns) x (a range
// of k) per thread, so that the 256 threads hold all of its weights in flight at once; the first weights of
// the next product, and the vectors of the next layer, are requested before the work in front of them; all
// loads of a phase are in flight together. The ranges' sums meet in shared memory, in range order.
// 32-bit products and sums; LayerNorm sums and the softmax's sum in double, expf, as in the host code.
//
// Greedy runs of small vocabularies go through all their tokens in one launch (small_loop_supports): the CTA that has the last row
// finishes it (final norm, head out of shared memory, first maximum; output_head.cpp:58-70, inference.cpp:188-198) and a barrier
// of the stream's cluster hands the token on; every token still computes its whole context. Two layers of width 64, one
// stream, contexts of 6 to 63: 47 us a token with a launch for the body and one for the tail, replayed from a graph, 37 in
// one launch. (RUN: such a run; the body of one step is compiled without what only a run needs, which cost it 1 %.)
#include "common.cuh"
#include "tc_ptx.cuh"

namespace lb {

namespace {

constexpr int SB_THREADS = 256, SB_WARPS = 8, SB_ROWS = 8, SB_CTAS = 8;
constexpr int SB_FLIGHT = 16;  // weight loads (16 bytes each) a thread has in flight
constexpr int SB_MAX_D = 128, SB_MAX_F = 512;
constexpr int SB_VECTORS = (9 * SB_MAX_D + SB_MAX_F + SB_THREADS - 1) / SB_THREADS;  // of a layer's vectors, per thread
constexpr int SB_PARTIALS = SB_THREADS * 4 * SB_ROWS;  // floats: every thread's sums

struct SmallShape {
  int layers, heads, d, f, vocab, streams, s_cap;
};

// A run of `steps` tokens behind contexts of s0 positions; steps == 0: the body of one step, rows to x_out.
struct SmallRun {
  int s0, steps, step0, out_ld;
  int *ids, *out_tokens;
  float *logits;  // [streams][vocab] of the last step
  LoopState *state;
};

// One product's cut: groups of four columns, ranges of k; a thread's range and group.
struct SbCut {
  int k, n, groups, ranges, per, q, c4;
  __device__ __forceinline__ void make(int k_, int n_) {
    k = k_;
    n = n_;
    groups = n >> 2;
    ranges = 1;
    while (ranges * 2 * groups <= SB_THREADS && ranges * 2 <= k) ranges *= 2;
    per = (k + ranges - 1) / ranges;
    q = threadIdx.x / groups;
    c4 = threadIdx.x - q * groups;
  }
};

struct SbWeights {
  float4 w[SB_FLIGHT];
  __device__ __forceinline__ void load(const float *__restrict__ base, int n, int c4, int k0, int k1) {
#pragma unroll
    for (int i = 0; i < SB_FLIGHT; ++i)
      w[i] = k0 + i < k1 ? __ldg(reinterpret_cast<const float4 *>(base + (long long)(k0 + i) * n) + c4)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the first loads of a product, ahead of its input
  __device__ __forceinline__ void request(const float *__restrict__ base, const SbCut &c) {
    if (c.q < c.ranges) load(base, c.n, c.c4, c.q * c.per, min(c.k, (c.q + 1) * c.per));
  }
};

__device__ __forceinline__ double sb_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// LayerNorm of eight rows [SB_ROWS][d], a warp each, to out [d][SB_ROWS] (device_backend.cpp:1247-1279). Both sums in one
// pass, in double, of the values less one of the row's own: its distance from the mean squared is at most d variances, so the
// variance loses d * 2^-52 of itself however far the row lies from zero.
__device__ __forceinline__ void sb_layernorm(const float *rows, const float *gamma, const float *beta, int d, double inv_d,
                                             float *out) {
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
  const float *x = rows + r * d;
  const double at = (double)x[0];
  double sum = 0.0, sq = 0.0;
  for (int c = lane; c < d; c += 32) {
    const double v = (double)x[c] - at;
    sum += v;
    sq = fma(v, v, sq);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  const double off = sum * inv_d, mean = at + off, spread = fma(-off, off, sq * inv_d), var = spread < 0.0 ? 0.0 : spread;
  const float inv_std = 1.0f / sqrtf((float)var + 1e-5f), fmean = (float)mean;  // (not a number where a value is not finite)
  for (int c = lane; c < d; c += 32) out[c * SB_ROWS + r] = __fadd_rn(__fmul_rn((x[c] - fmean) * inv_std, gamma[c]), beta[c]);
  __syncthreads();
}

// Attention of one row (position t, a warp) over keys 0 .. t, the heads in turn: out[column * SB_ROWS]. p: room for the scores.
__device__ __forceinline__ void sb_attention(const float *qr, const float *ks, int kp, const float *vs, int D, int H, int dh, int t,
                                             int s, float scale, float *p, float *out) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int h = 0; h < H; ++h) {
    if (t >= s) {  // the warp's row lies behind the text
      for (int c = lane; c < dh; c += 32) out[(h * dh + c) * SB_ROWS] = 0.f;
      continue;
    }
    const float4 *q = reinterpret_cast<const float4 *>(qr + h * dh);
    float m = -INFINITY;
#pragma unroll 1
    for (int k = lane; k <= t; k += 32) {
      const float4 *kr = reinterpret_cast<const float4 *>(ks + k * kp + h * dh);
      float d0 = 0.f, d1 = 0.f;
#pragma unroll 4
      for (int i = 0; i < dh / 4; i += 2) {
        const float4 qa = q[i], ka = kr[i], qb = q[i + 1], kb = kr[i + 1];
        d0 = fmaf(qa.x, ka.x, fmaf(qa.y, ka.y, fmaf(qa.z, ka.z, fmaf(qa.w, ka.w, d0))));
        d1 = fmaf(qb.x, kb.x, fmaf(qb.y, kb.y, fmaf(qb.z, kb.z, fmaf(qb.w, kb.w, d1))));
      }
      const float v = (d0 + d1) * scale;
      p[k] = v;
      m = fmaxf(m, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    double sum = 0.0;
#pragma unroll 1
    for (int k = lane; k <= t; k += 32) {
      const float e = expf(p[k] - m);
      p[k] = e;
      sum += (double)e;
    }
    const float inv = (float)(1.0 / sb_warp_sum(sum));
    __syncwarp();
#pragma unroll 1
    for (int c = lane; c < dh; c += 32) {
      float o[4] = {};
      const float *v = vs + h * dh + c;
      int k = 0;
#pragma unroll 1
      for (; k + 8 <= t + 1; k += 8) {
        const float4 e = *reinterpret_cast<const float4 *>(p + k), f = *reinterpret_cast<const float4 *>(p + k + 4);
        o[0] = fmaf(e.x, v[k * D], o[0]);
        o[1] = fmaf(e.y, v[(k + 1) * D], o[1]);
        o[2] = fmaf(e.z, v[(k + 2) * D], o[2]);
        o[3] = fmaf(e.w, v[(k + 3) * D], o[3]);
        o[0] = fmaf(f.x, v[(k + 4) * D], o[0]);
        o[1] = fmaf(f.y, v[(k + 5) * D], o[1]);
        o[2] = fmaf(f.z, v[(k + 6) * D], o[2]);
        o[3] = fmaf(f.w, v[(k + 7) * D], o[3]);
      }
#pragma unroll 1
      for (; k <= t; ++k) o[0] = fmaf(p[k], v[k * D], o[0]);
      out[(h * dh + c) * SB_ROWS] = ((o[0] + o[1]) + (o[2] + o[3])) * inv;
    }
    __syncwarp();
  }
}

// offsets: [layers][12] byte offsets into params: ln1_g, ln1_b, qkv_w, qkv_b, out_w, out_b, ln2_g, ln2_b, w1, b1, w2,
// b2; then tok_emb, pos_emb. kv: [2][streams][s_cap][2 d]. x: [streams * s][d], rows as the other kernels pack them.
template <bool RUN>
__global__ void __launch_bounds__(SB_THREADS)
small_body_kernel(SmallShape g, SmallRun run, const char *__restrict__ params, const unsigned long long *__restrict__ offsets, const int *ids,
                  int ids_ld, const LoopState *state, float *kv, float *x_out, DevErr *err) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_best[SB_WARPS];
  __shared__ int s_at[SB_WARPS];
  const int tid = threadIdx.x, wid = tid >> 5;
  const int b = blockIdx.y, me = blockIdx.x, D = g.d, F = g.f, H = g.heads, dh = D / H;
  const int blocks_max = ((g.s_cap + SB_ROWS - 1) / SB_ROWS + SB_CTAS - 1) / SB_CTAS;
  const int kp = D + 4;  // pitch of keys: 16-byte reads of consecutive rows hit all banks
  float *part = sm;                                 // [SB_PARTIALS]
  float *in = part + SB_PARTIALS;                   // [max(D, F)][SB_ROWS] input of the product at hand
  float *y = in + max(D, F) * SB_ROWS;              // [SB_ROWS][D]
  float *x = y + SB_ROWS * D;                       // [blocks][SB_ROWS][D]
  float *qs = x + blocks_max * SB_ROWS * D;         // the same of the queries
  float *pr = qs + blocks_max * SB_ROWS * D;        // [SB_WARPS][s_cap rounded up to 4] scores, then weights
  const int pp = (g.s_cap + 3) & ~3;
  float *ks = pr + SB_WARPS * pp;                   // [s][kp]
  float *vs = ks + g.s_cap * kp;                    // [s][D]
  float *vecs = vs + g.s_cap * D;                   // [2][9 D + F] a layer's vectors: LayerNorms and biases
  const int nvec = 9 * D + F;
  float *tail = vecs + 2 * nvec;                    // of a run: final norm [2][D], head [D][vocab]
  unsigned long long *offs = reinterpret_cast<unsigned long long *>(tail + (RUN ? D * (g.vocab + 2) : 0));  // the table of offsets
  auto P = [&](int l, int i) { return reinterpret_cast<const float *>(params + offs[l * 12 + i]); };
  enum { LN1G, LN1B, QKVW, QKVB, OUTW, OUTB, LN2G, LN2B, W1, B1, W2, B2 };
  auto weight_of = [](int op) { return op == 0 ? (int)QKVW : op == 1 ? (int)OUTW : op == 2 ? (int)W1 : (int)W2; };
  // places of a layer's vectors: ln1 gamma 0, ln1 beta D, ln2 gamma 2D, ln2 beta 3D, out bias 4D, W2 bias 5D, QKV bias 6D, W1 bias 9D
  float vr[SB_VECTORS];  // a layer's vectors on their way
  auto request_vectors = [&](int l) {
#pragma unroll
    for (int i = 0; i < SB_VECTORS; ++i) {
      const int e = tid + i * SB_THREADS;
      const int at = min(e / D, 9), which = at == 9 ? (int)B1 : at >= 6 ? (int)QKVB : at == 5 ? (int)B2 : at == 4 ? (int)OUTB
                                            : at == 3 ? (int)LN2B : at == 2 ? (int)LN2G : at;
      vr[i] = e < nvec ? __ldg(P(l, which) + e - (at >= 6 && at < 9 ? 6 : at) * D) : 0.f;
    }
  };
  auto store_vectors = [&](int turn) {
#pragma unroll
    for (int i = 0; i < SB_VECTORS; ++i)
      if (tid + i * SB_THREADS < nvec) vecs[turn * nvec + tid + i * SB_THREADS] = vr[i];
  };
  pdl_launch_dependents();
  for (int i = tid; i < g.layers * 12 + 5; i += SB_THREADS) offs[i] = offsets[i];
  __syncthreads();
  SbWeights wt;
  SbCut cut[4];  // QKV, out-projection, W1, W2
  cut[0].make(D, 3 * D);
  cut[1].make(D, D);
  cut[2].make(D, F);
  cut[3].make(F, D);
  auto cut_of = [&](int op) { return op == 0 ? cut[0] : op == 1 ? cut[1] : op == 2 ? cut[2] : cut[3]; };
  const double inv_d = 1.0 / (double)D;
  wt.request(P(0, QKVW), cut[0]);
  request_vectors(0);  // (all of this never changes: before the wait)
  store_vectors(0);
  if constexpr (RUN) {
    const float *gamma = P(g.layers, 2), *beta = P(g.layers, 3), *w = P(g.layers, 4);
    for (int c = tid; c < D; c += SB_THREADS) {
      tail[c] = __ldg(gamma + c);
      tail[D + c] = __ldg(beta + c);
    }
    for (int e = tid; e < D * g.vocab; e += SB_THREADS) tail[2 * D + e] = __ldg(w + e);
  }
  pdl_wait();
  int turn = 0;  // of the two buffers, for keys and values and for a layer's vectors
#pragma unroll 1
  for (int step = 0; step < (RUN ? run.steps : 1); ++step) {
  const bool another = RUN && step + 1 < run.steps;
  const int s = RUN ? run.s0 + step : state ? state->s : g.s_cap;
  const int blocks = (s + SB_ROWS - 1) / SB_ROWS;
  const int mine = blocks > me ? (blocks - me + SB_CTAS - 1) / SB_CTAS : 0;
  auto row_of = [&](int j, int r) { return (j * SB_CTAS + me) * SB_ROWS + r; };
  const float *tok = P(g.layers, 0), *pos = P(g.layers, 1);
#pragma unroll 2
  for (int e = tid; e < mine * SB_ROWS * D; e += SB_THREADS) {
    const int i = e / D, c = e - i * D, t = row_of(i / SB_ROWS, i % SB_ROWS);
    float v = 0.f;
    if (t < s) {
      int id = RUN ? __ldcg(ids + (long long)b * ids_ld + t) : ids[(long long)b * ids_ld + t];
      if (id < 0 || id >= g.vocab) {
        if (c == 0) {
          err->code = DEVERR_BAD_TOKEN_ID;
          err->detail = id;
        }
        id = 0;
      }
      v = __ldg(tok + (long long)id * D + c) + __ldg(pos + (long long)t * D + c);
    }
    x[e] = v;
  }
  __syncthreads();
  const float scale = 1.0f / sqrtf((float)dh);
  const int last = mine > 0 ? min(s, row_of(mine - 1, SB_ROWS)) : 0;  // keys this CTA's rows see
  enum { QKV = 0, WO, FF1, FF2 };
  for (int l = 0; l < g.layers; ++l, turn ^= 1) {
    const float *vec = vecs + turn * nvec;
    float *kvl = kv + ((long long)turn * g.streams + b) * g.s_cap * 2 * D;
    const bool more = l + 1 < g.layers || another;  // a layer follows: nl
    const int nl = l + 1 < g.layers ? l + 1 : 0;
    if (mine == 0) {
      __syncwarp();
      cluster_sync_all();
      if (more) {  // this CTA may have rows in the next step
        request_vectors(nl);
        store_vectors(turn ^ 1);
      }
      continue;
    }
    if (more) request_vectors(nl);
    // the operators as steps of one loop, with one instance of the product, the LayerNorm and the attention
#pragma unroll 1
    for (int at = 0; at < 4 * mine; ++at) {
      const int op = at < mine ? QKV : WO + (at - mine) % 3, j = at < mine ? at : (at - mine) / 3;
      const float *xj = x + j * SB_ROWS * D;
      if (at == mine) {  // every CTA's keys and values of this layer
        __syncwarp();
        cluster_sync_all();
        const int pieces = last * (D / 2);  // float4s: a position's keys, then its values
#pragma unroll 1
        for (int e0 = tid; e0 < pieces; e0 += 8 * SB_THREADS) {
          float4 v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (e0 + i * SB_THREADS < pieces) v[i] = __ldcg(reinterpret_cast<const float4 *>(kvl) + e0 + i * SB_THREADS);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = e0 + i * SB_THREADS, t = e / (D / 2), c = (e - t * (D / 2)) * 4;
            if (e < pieces) *reinterpret_cast<float4 *>(c < D ? ks + t * kp + c : vs + t * D + c - D) = v[i];
          }
        }
        if (more) store_vectors(turn ^ 1);
        __syncthreads();
      }
      if (op == QKV || op == FF1) {
        sb_layernorm(op == QKV ? xj : y, vec + (op == QKV ? 0 : 2 * D), vec + (op == QKV ? D : 3 * D), D, inv_d, in);
      } else if (op == WO) {
        sb_attention(qs + (j * SB_ROWS + wid) * D, ks, kp, vs, D, H, dh, row_of(j, wid), s, scale, pr + wid * pp, in + wid);
        __syncthreads();
      }
      // ---- sums[range][row][column] over the range's k of in [k][SB_ROWS] times the weights requested before ----
      const SbCut c = cut_of(op);
      float acc[SB_ROWS][4] = {};
      if (c.q < c.ranges) {
        const int k0 = c.q * c.per, k1 = min(c.k, k0 + c.per);
        auto add = [&](int i, int at) {
          const float4 a = *reinterpret_cast<const float4 *>(in + at * SB_ROWS);
          const float4 b = *reinterpret_cast<const float4 *>(in + at * SB_ROWS + 4);
          const float xv[SB_ROWS] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
          for (int r = 0; r < SB_ROWS; ++r) {
            acc[r][0] = fmaf(xv[r], wt.w[i].x, acc[r][0]);
            acc[r][1] = fmaf(xv[r], wt.w[i].y, acc[r][1]);
            acc[r][2] = fmaf(xv[r], wt.w[i].z, acc[r][2]);
            acc[r][3] = fmaf(xv[r], wt.w[i].w, acc[r][3]);
          }
        };
#pragma unroll 1
        for (int kk = k0; kk < k1; kk += SB_FLIGHT) {
          if (kk > k0) wt.load(P(l, weight_of(op)), c.n, c.c4, kk, k1);
#pragma unroll
          for (int i4 = 0; i4 < SB_FLIGHT; i4 += 4) {
            if (kk + i4 + 4 <= k1) {
#pragma unroll
              for (int i = 0; i < 4; ++i) add(i4 + i, kk + i4 + i);
            } else {
#pragma unroll
              for (int i = 0; i < 3; ++i)
                if (kk + i4 + i < k1) add(i4 + i, kk + i4 + i);
            }
          }
        }
      }
      {  // the first weights of the step that follows
        const int after = at + 1;
        const bool over = after == 4 * mine;
        if (!over || more) {
          const int nop = over || after < mine ? QKV : WO + (after - mine) % 3;
          wt.request(P(over ? nl : l, weight_of(nop)), cut_of(nop));
        }
      }
      if (c.q < c.ranges) {
#pragma unroll
        for (int r = 0; r < SB_ROWS; ++r)
          *reinterpret_cast<float4 *>(part + ((c.q * SB_ROWS + r) * c.groups + c.c4) * 4) =
              make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      }
      __syncthreads();
      // ---- the ranges' sums in order, and where the values go ----
      const int bias = op == QKV ? 6 * D : op == WO ? 4 * D : op == FF1 ? 9 * D : 5 * D;
#pragma unroll 1
      for (int e = tid; e < SB_ROWS * c.groups; e += SB_THREADS) {
        const float4 *sums = reinterpret_cast<const float4 *>(part) + e;
        const int stride = SB_ROWS * c.groups;
        float4 v = sums[0];
#pragma unroll 4
        for (int z = 1; z < c.ranges; ++z) {
          const float4 p = sums[z * stride];
          v = make_float4(v.x + p.x, v.y + p.y, v.z + p.z, v.w + p.w);
        }
        const int r = e / c.groups, col = (e - r * c.groups) * 4;
        const float4 bv = *reinterpret_cast<const float4 *>(vec + bias + col);
        v = make_float4(v.x + bv.x, v.y + bv.y, v.z + bv.z, v.w + bv.w);
        if (op == QKV) {
          const int t = row_of(j, r);
          if (col < D) *reinterpret_cast<float4 *>(qs + (j * SB_ROWS + r) * D + col) = v;
          else if (t < s) *reinterpret_cast<float4 *>(kvl + (long long)t * 2 * D + col - D) = v;
        } else if (op == FF1) {
          in[col * SB_ROWS + r] = fmaxf(v.x, 0.f);
          in[(col + 1) * SB_ROWS + r] = fmaxf(v.y, 0.f);
          in[(col + 2) * SB_ROWS + r] = fmaxf(v.z, 0.f);
          in[(col + 3) * SB_ROWS + r] = fmaxf(v.w, 0.f);
        } else {
          const float4 rest = *reinterpret_cast<const float4 *>((op == WO ? xj : y) + r * D + col);
          *reinterpret_cast<float4 *>((op == WO ? y : x + j * SB_ROWS * D) + r * D + col) =
              make_float4(v.x + rest.x, v.y + rest.y, v.z + rest.z, v.w + rest.w);
        }
      }
      __syncthreads();
    }
  }
  if constexpr (!RUN) {
    for (int e = tid; e < mine * SB_ROWS * D; e += SB_THREADS) {
      const int i = e / D, t = row_of(i / SB_ROWS, i % SB_ROWS);
      if (t < s) x_out[((long long)b * s + t) * D + (e - i * D)] = x[e];
    }
  }
  if constexpr (RUN) {
  // ---- the last row's token: a strict '>' scan from index 0 ----
  if (me == (blocks - 1) % SB_CTAS) {
    const int V = g.vocab, r = (s - 1) % SB_ROWS;
    sb_layernorm(x + (mine - 1) * SB_ROWS * D, tail, tail + D, D, inv_d, in);
    int wide = 1;  // columns side by side, the threads left over share k
    while (wide < V && wide < SB_THREADS) wide *= 2;
    const int ranges = SB_THREADS / wide, q = tid / wide;
#pragma unroll 1
    for (int c = tid % wide; c < V; c += wide) {
      const float *w = tail + 2 * D + c;
      float v = 0.f;
#pragma unroll 4
      for (int k = q; k < D; k += ranges) v = fmaf(in[k * SB_ROWS + r], w[k * V], v);
      part[q * V + c] = v;
    }
    __syncthreads();
    float best = -3.402823466e+38f;
    int best_at = 0x7fffffff;
#pragma unroll 1
    for (int c = tid; c < V; c += SB_THREADS) {
      float v = 0.f;
      for (int z = 0; z < ranges; ++z) v += part[z * V + c];
      if (!another) run.logits[(long long)b * V + c] = v;
      if (v > best || (v == best && c < best_at)) {
        best = v;
        best_at = c;
      }
    }
    auto first = [&]() {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_at, o);
        if (ov > best || (ov == best && oi < best_at)) {
          best = ov;
          best_at = oi;
        }
      }
    };
    first();
    if ((tid & 31) == 0) {
      s_best[wid] = best;
      s_at[wid] = best_at;
    }
    __syncthreads();
    if (wid == 0) {
      best = tid < SB_WARPS ? s_best[tid] : -3.402823466e+38f;
      best_at = tid < SB_WARPS ? s_at[tid] : 0x7fffffff;
      first();
      if (tid == 0) {
        const int token = best_at == 0x7fffffff ? 0 : best_at;  // every entry NaN or below the sentinel
        run.ids[(long long)b * ids_ld + s] = token;
        run.out_tokens[(long long)b * run.out_ld + run.step0 + step] = token;
      }
    }
  }
  __syncthreads();
  cluster_sync_all();  // the token is there for every CTA of the stream
  }
  }
  if (RUN && b == 0 && me == 0 && tid == 0) {
    run.state->s = run.s0 + run.steps;
    run.state->step = run.step0 + run.steps;
  }
}

size_t small_smem(int layers, int d, int f, int s) {
  const size_t blocks = ((size_t)(s + SB_ROWS - 1) / SB_ROWS + SB_CTAS - 1) / SB_CTAS;
  return 4 * (SB_PARTIALS + (size_t)(d > f ? d : f) * SB_ROWS + SB_ROWS * (size_t)d + 2 * blocks * SB_ROWS * d +
              (size_t)SB_WARPS * ((s + 3) & ~3) + (size_t)s * (2 * d + 4) + 2 * (9 * (size_t)d + f)) +
         8 * ((size_t)layers * 12 + 5);
}

void small_launch(const SmallShape &g, const SmallRun &run, const char *params, const unsigned long long *offsets, const int *ids,
                  int ids_ld, const LoopState *state, float *kv, float *x, DevErr *err, cudaStream_t st) {
  const size_t smem = small_smem(g.layers, g.d, g.f, g.s_cap) + (run.steps ? (size_t)4 * g.d * (g.vocab + 2) : 0);
  auto kernel = run.steps ? small_body_kernel<true> : small_body_kernel<false>;
  if (smem > 48 * 1024) LB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_pdl_cluster_x(kernel, dim3(SB_CTAS, (unsigned)g.streams), dim3(SB_THREADS), smem, st, g_pdl_enabled,
                       (unsigned)SB_CTAS, g, run, params, offsets, ids, ids_ld, state, kv, x, err);
}

}  // namespace

bool small_body_supports(int streams, int s, int layers, int n_heads, int d, int f) {
  if (d > SB_MAX_D || f > SB_MAX_F || d % 8 != 0 || f % 4 != 0 || d % n_heads != 0 || (d / n_heads) % 8 != 0) return false;
  return streams >= 1 && streams <= 65535 && small_smem(layers, d, f, s) <= 220 * 1024;
}

size_t small_body_kv_floats(int streams, int s, int d) { return (size_t)2 * streams * s * 2 * d; }

void launch_small_body(const char *params, const unsigned long long *offsets, int layers, int n_heads, int d, int f, int vocab,
                       const int *ids, int ids_ld, int streams, int s, const LoopState *state, float *kv, float *x, DevErr *err,
                       cudaStream_t st) {
  small_launch(SmallShape{layers, n_heads, d, f, vocab, streams, s}, SmallRun{}, params, offsets, ids, ids_ld, state, kv, x, err, st);
}

// The head stays in shared memory for the run: vocabularies beyond what is left there go token by token.
bool small_loop_supports(int streams, int s, int layers, int n_heads, int d, int f, int vocab) {
  return small_body_supports(streams, s, layers, n_heads, d, f) && vocab >= 1 && vocab <= 1024 &&
         small_smem(layers, d, f, s) + (size_t)4 * d * (vocab + 2) <= 220 * 1024;
}

void launch_small_loop(const char *params, const unsigned long long *offsets, int layers, int n_heads, int d, int f, int vocab,
                       int *ids, int ids_ld, int *out_tokens, int out_ld, int streams, int s0, int step0, int steps, LoopState *state,
                       float *logits, float *kv, DevErr *err, cudaStream_t st) {
  const SmallShape g{layers, n_heads, d, f, vocab, streams, s0 + steps - 1};
  small_launch(g, SmallRun{s0, steps, step0, out_ld, ids, out_tokens, logits, state}, params, offsets, ids, ids_ld, nullptr, kv, nullptr, err, st);
}

}  // namespace lb
