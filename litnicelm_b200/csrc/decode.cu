// Kernels of the opt-in cached mode (LITNICE_B200_KV_CACHE=1): one new row per
// stream and step. The reference keeps no key/value cache (inference.cpp:278-284
// runs Transformer::forward over the whole context for every token), so this mode
// is an extension: the same arithmetic per row (transformer_layer.cpp:50-92,
// self_attention_fused_inplace.cpp:82-97), with the keys and values of earlier
// positions read back from HBM instead of being recomputed.
//
// Layout: kcache, vcache [n_layers][n_streams][cap][d_model] fp32, a position's
// row as the QKV projection produced it (heads side by side). The step's rows
// live in [n_streams, ...] buffers: x (residual stream), ln, qkv [.., 3 d_model],
// ctx, h [.., d_ff].
#include "common.cuh"
#include "gemm_tc.cuh"

namespace lb {

namespace {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// x[b, :] = tok_emb[ids[b, s-1]] + pos_emb[s-1] (transformer.cpp:91-94 for the newest row) and
// ln[b, :] = LayerNorm(x[b, :]) with the first layer's gamma / beta (device_backend.cpp:1247-1279:
// mean and biased variance in double, inv_std = 1/sqrt(float(var) + 1e-5f)). One warp per stream.
__global__ void embed_last_ln_kernel(const float *__restrict__ tok_emb, const float *__restrict__ pos_emb,
                                     const int *__restrict__ ids, int ids_ld, const LoopState *state, int s_host,
                                     int n_streams, int d, int vocab, const float *__restrict__ gamma,
                                     const float *__restrict__ beta, float *__restrict__ x, float *__restrict__ ln,
                                     DevErr *err) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = state ? state->s : s_host;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= n_streams) return;
  const int lane = threadIdx.x & 31, t = s - 1;
  int id = ids[(long long)b * ids_ld + t];
  if (id < 0 || id >= vocab) {
    if (lane == 0) {
      err->code = DEVERR_BAD_TOKEN_ID;
      err->detail = id;
    }
    id = 0;
  }
  const float *tp = tok_emb + (long long)id * d, *pp = pos_emb + (long long)t * d;
  float *xp = x + (long long)b * d;
  double sum = 0.0;
  for (int c = lane; c < d; c += 32) {
    const float v = tp[c] + pp[c];
    xp[c] = v;
    sum += (double)v;
  }
  if (ln == nullptr) return;  // the consumer normalises the row itself
  const double mean = warp_sum_d(sum) / (double)d;
  double var = 0.0;
  for (int c = lane; c < d; c += 32) {  // each lane re-reads the elements it wrote itself
    const double dd = (double)xp[c] - mean;
    var += dd * dd;
  }
  var = warp_sum_d(var) / (double)d;
  const float inv_std = 1.0f / sqrtf((float)var + 1e-5f);
  const float fmean = (float)mean;
  for (int c = lane; c < d; c += 32)
    ln[(long long)b * d + c] = __fadd_rn(__fmul_rn((xp[c] - fmean) * inv_std, gamma[c]), beta[c]);
}

// Prefill: the K and V thirds of the QKV rows of a whole-context pass, rows r = b * s + t of
// qkv [rows, 3 d], to the caches at position t of stream b.
__global__ void kv_store_kernel(const float *__restrict__ qkv, const LoopState *state, int s_host, int n_streams,
                                int d, int cap, float *__restrict__ kc, float *__restrict__ vc) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = state ? state->s : s_host;
  const long long r = blockIdx.x;
  if (r >= (long long)n_streams * s) return;
  const int b = (int)(r / s), t = (int)(r - (long long)b * s);
  const float4 *src = reinterpret_cast<const float4 *>(qkv + r * 3 * d);
  float4 *kd = reinterpret_cast<float4 *>(kc + ((long long)b * cap + t) * d);
  float4 *vd = reinterpret_cast<float4 *>(vc + ((long long)b * cap + t) * d);
  const int n4 = d >> 2;
  for (int c = threadIdx.x; c < n4; c += blockDim.x) {
    kd[c] = src[n4 + c];
    vd[c] = src[2 * n4 + c];
  }
}

// Where the context row goes: fp32 (lo == nullptr), a TF32 pair (ctx, lo), or the fp16 pair a
// projection on fp16 pairs reads (one scale per 64 columns; head dimension 64).
struct DecodeCtx {
  float *ctx, *lo;
  TcPairF16 pair;
};

// Column tid of head h of stream b's context row (threads tid < DH hold one each). All 128 threads
// call it together.
template <int DH>
__device__ __forceinline__ void store_context(const DecodeCtx &o, float v, int b, int h, int d_model, int tid, float *red) {
  const long long at = (long long)b * d_model + h * DH + tid;
  if (DH == 64 && o.pair.hi != nullptr) {
    float am = tid < DH ? fabsf(v) : 0.f;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, s));
    if ((tid & 31) == 0) red[tid >> 5] = am;
    __syncthreads();
    if (tid >= DH) return;
    float inv;
    const float a = v * f16_block_scale(fmaxf(red[0], red[1]), &inv);
    const __half hi = __float2half_rn(a);
    o.pair.hi[at] = hi;
    o.pair.lo[at] = __float2half_rn(a - __half2float(hi));
    if (tid == 0) o.pair.inv_scale[(long long)b * (d_model / TC_F16_SLOT) + h] = inv;
    return;
  }
  if (tid >= DH) return;
  if (o.lo != nullptr) {
    float hi, lo;
    split_tf32(v, hi, lo);
    o.ctx[at] = hi;
    o.lo[at] = lo;
  } else {
    o.ctx[at] = v;
  }
}

// Attention of the newest row of stream b, head h, over the keys of one chunk of positions:
// scores q.k / sqrt(dh) in fp32, their maximum, e = expf(score - max), the sum of e in double
// (scaled_causal_softmax_rows, device_backend.cpp:1554-1592, restricted to one row) and
// o = sum e_j v_j. The CTA whose chunk holds the newest position first appends that position's K
// and V (this step's QKV row) to the caches. With one chunk the normalised context row is
// written directly; otherwise (o, max, sum) go to `part` and the chunk that finishes last joins them.
//
// Bound by the cache bytes (8 * s * d_model per layer and stream), so what counts is bytes in flight: the chunk's lines are asked for
// towards L2 before the predecessor has ended, and a warp has a batch of 4 KB of keys and values in use and as much on its way, without
// a barrier before the warps' results meet. With scores, weights and values as three phases of the CTA, four loads in flight in each
// (which heads of 16 columns still do), and now, us a launch: 64 streams, 8 heads of 64, 160 positions 16.6, 9.4, 250 positions 27.1,
// 16.9; 40 streams, 8 heads of 32, 250 positions 7.9, 6.6 (9.9 with values read four bytes a lane).
// The batch on its way costs registers: five CTAs an SM, eight without. More CTAs than five an SM hold run without, and chunks that
// are one batch a warp: 40 streams, 16 heads of 64, 4 positions 3.5 in three phases, 4.6 always ahead, 3.4 so; 64 streams, 60 positions
// 8.0, 9.1, 7.2; 64 streams, 16 heads of 32, 100 positions 6.2, 8.9, 6.9.
constexpr int DEC_UNROLL = 4;
__host__ __device__ constexpr int dec_batch(int dh) { return dh <= 32 ? 16 : dh == 64 ? 8 : 4; }  // keys of a warp's batch: 2 KB, and 2 KB of values
template <int DH, bool MORE>
__global__ void __launch_bounds__(128, DH < 32 ? 0 : MORE ? 5 : 8)
attn_decode_kernel(const float *__restrict__ qkv, float *kc, float *vc, int cap, int d_model, const LoopState *state,
                   int s_host, int keys_per_chunk, float scale, float *__restrict__ part, DecodeCtx ctx,
                   int *__restrict__ counters) {
  constexpr int LPK = DH / 8;      // lanes that share one key: 8 floats of the head each
  constexpr int KPI = 128 / LPK;   // keys per trip of the CTA
  constexpr int VPR = DH / 4;      // lanes that share one row of values: 4 floats each
  constexpr int VPI = 128 / VPR;   // rows of values per trip of the CTA
  extern __shared__ float sc[];    // heads of 16 columns: scores, then e, of the chunk's keys
  __shared__ float red_f[4];
  __shared__ double red_d[4];
  __shared__ __align__(16) float o_part[512];  // [VPI][DH]
  __shared__ int is_last;
  pdl_launch_dependents();
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, chunks = gridDim.x;
  if constexpr (DH >= 32) {  // the chunk's keys and values of earlier positions, on their way to L2 while the predecessor ends and scores are formed
    const int early = min(state ? *static_cast<const volatile int *>(&state->s) : s_host, cap);  // (of the step before, perhaps)
    const int first = c * keys_per_chunk, lines = max(0, min(early, first + keys_per_chunk) - first) * (DH / 32);
    for (int i = threadIdx.x; i < 2 * lines; i += 128) {
      const int at = i < lines ? i : i - lines;
      const float *line = (i < lines ? kc : vc) + ((long long)b * cap + first + at / (DH / 32)) * d_model + h * DH + at % (DH / 32) * 32;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
    }
  }
  pdl_wait();
  const int s = state ? state->s : s_host;  // context length including the newest token
  const int p = s - 1;
  const int c0 = c * keys_per_chunk, c1 = min(s, c0 + keys_per_chunk);
  float *out = part ? part + (((long long)b * gridDim.y + h) * chunks + c) * (DH + 2) : nullptr;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (c0 >= s) {  // a launch sized for a longer context: nothing in this chunk
    if (out == nullptr) return;
    if (tid == 0) {
      out[DH] = -INFINITY;
      out[DH + 1] = 0.f;
    }
  } else {
    const float *row = qkv + (long long)b * 3 * d_model;
    float t = 0.f, m = -INFINITY;
    double l = 0.0;
    if (p >= c0 && p < c1 && tid < DH / 4) {
      const float4 k4 = *reinterpret_cast<const float4 *>(row + d_model + h * DH + tid * 4);
      const float4 v4 = *reinterpret_cast<const float4 *>(row + 2 * d_model + h * DH + tid * 4);
      *reinterpret_cast<float4 *>(kc + ((long long)b * cap + p) * d_model + h * DH + tid * 4) = k4;
      *reinterpret_cast<float4 *>(vc + ((long long)b * cap + p) * d_model + h * DH + tid * 4) = v4;
    }
    if constexpr (DH >= 32) {
      // A warp takes every fourth key, a batch at a time: their scores over LPK lanes a key, the running maximum and sum, the weighted
      // values with a lane per four columns of every KPV-th key. MORE: the next batch is on its way while one is used.
      constexpr int KB = dec_batch(DH), KPP = 32 / LPK, NP = KB / KPP;  // keys of a load of keys, such loads
      constexpr int KPV = 32 / VPR, NV = KB / KPV;                      // of a load of values: a lane has four columns of one key
      const int sub = lane % LPK, grp = lane / LPK, vq = lane % VPR, vr = lane / VPR;
      const int mine = (c1 - c0 - wid + 3) / 4;  // keys of this warp: positions c0 + wid + 4 n
      const float4 q0 = *reinterpret_cast<const float4 *>(row + h * DH + sub * 8);
      const float4 q1 = *reinterpret_cast<const float4 *>(row + h * DH + sub * 8 + 4);
      const long long at0 = ((long long)b * cap + c0 + wid) * d_model + h * DH;
      struct Batch {
        float4 k0[NP], k1[NP], v[NV];
      };
      Batch next;
      auto load = [&](int n0) {
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          const int n = n0 + u * KPP + grp;
          next.k0[u] = next.k1[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (n < mine) {  // (the newest position's key and value are this step's own)
            const float *kp = c0 + wid + 4 * n == p ? row + d_model + h * DH : kc + at0 + (long long)(4 * n) * d_model;
            next.k0[u] = *reinterpret_cast<const float4 *>(kp + sub * 8);
            next.k1[u] = *reinterpret_cast<const float4 *>(kp + sub * 8 + 4);
          }
        }
#pragma unroll
        for (int x = 0; x < NV; ++x) {
          const int n = n0 + x * KPV + vr;
          next.v[x] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (n < mine) {
            const float *vp = c0 + wid + 4 * n == p ? row + 2 * d_model + h * DH : vc + at0 + (long long)(4 * n) * d_model;
            next.v[x] = *reinterpret_cast<const float4 *>(vp + vq * 4);
          }
        }
      };
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
      load(0);
#pragma unroll 1
      for (int n0 = 0; n0 < mine; n0 += KB) {
        if (!MORE && n0 > 0) load(n0);
        const Batch now = next;
        if (MORE && n0 + KB < mine) load(n0 + KB);
        float e[NP], bm = -INFINITY;
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
          e[u] = n0 + u * KPP + grp < mine ? dot * scale : -INFINITY;
          bm = fmaxf(bm, e[u]);
        }
#pragma unroll
        for (int x = LPK; x < 32; x <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, x));
        const float mn = fmaxf(m, bm), keep = m == -INFINITY ? 0.f : expf(m - mn);
        m = mn;
        l *= (double)keep;
        o = make_float4(o.x * keep, o.y * keep, o.z * keep, o.w * keep);
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          e[u] = e[u] == -INFINITY ? 0.f : expf(e[u] - m);
          l += (double)e[u];
        }
#pragma unroll
        for (int x = 0; x < NV; ++x) {
          const float w = __shfl_sync(0xffffffffu, e[x * KPV / KPP], (x * KPV % KPP + vr) * LPK);
          o.x = fmaf(w, now.v[x].x, o.x);
          o.y = fmaf(w, now.v[x].y, o.y);
          o.z = fmaf(w, now.v[x].z, o.z);
          o.w = fmaf(w, now.v[x].w, o.w);
        }
      }
#pragma unroll
      for (int x = LPK; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
      for (int x = VPR; x < 32; x <<= 1) {
        o.x += __shfl_xor_sync(0xffffffffu, o.x, x);
        o.y += __shfl_xor_sync(0xffffffffu, o.y, x);
        o.z += __shfl_xor_sync(0xffffffffu, o.z, x);
        o.w += __shfl_xor_sync(0xffffffffu, o.w, x);
      }
      if (lane < VPR) *reinterpret_cast<float4 *>(o_part + wid * DH + lane * 4) = o;
      if (lane == 0) {
        red_f[wid] = m;
        red_d[wid] = l;
      }
      __syncthreads();
      m = fmaxf(fmaxf(red_f[0], red_f[1]), fmaxf(red_f[2], red_f[3]));
      l = 0.0;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float f = red_f[w] == -INFINITY ? 0.f : expf(red_f[w] - m);
        l += red_d[w] * (double)f;
        if (tid < DH) t = fmaf(o_part[w * DH + tid], f, t);
      }
      __syncthreads();  // (red_f is used again below)
    } else {
      __syncthreads();
      const int sub = tid % LPK;
      const float4 q0 = *reinterpret_cast<const float4 *>(row + h * DH + sub * 8);
      const float4 q1 = *reinterpret_cast<const float4 *>(row + h * DH + sub * 8 + 4);
      const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
      const float *kb = kc + (long long)b * cap * d_model + h * DH + sub * 8;
      for (int base = c0; base < c1; base += DEC_UNROLL * KPI) {  // uniform trip count: the shuffles need whole warps
        float4 k0[DEC_UNROLL], k1[DEC_UNROLL];
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
          const int j = base + u * KPI + tid / LPK;
          const float4 *kp = reinterpret_cast<const float4 *>(kb + (long long)j * d_model);
          k0[u] = j < c1 ? kp[0] : zero4;
          k1[u] = j < c1 ? kp[1] : zero4;
        }
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
          const int j = base + u * KPI + tid / LPK;
          float dot = q0.x * k0[u].x;
          dot = fmaf(q0.y, k0[u].y, dot);
          dot = fmaf(q0.z, k0[u].z, dot);
          dot = fmaf(q0.w, k0[u].w, dot);
          dot = fmaf(q1.x, k1[u].x, dot);
          dot = fmaf(q1.y, k1[u].y, dot);
          dot = fmaf(q1.z, k1[u].z, dot);
          dot = fmaf(q1.w, k1[u].w, dot);
#pragma unroll
          for (int o = LPK >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
          if (j < c1 && sub == 0) sc[j - c0] = dot * scale;
        }
      }
      __syncthreads();
      const int nk = c1 - c0;
      for (int i = tid; i < nk; i += 128) m = fmaxf(m, sc[i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) red_f[wid] = m;
      __syncthreads();
      m = fmaxf(fmaxf(red_f[0], red_f[1]), fmaxf(red_f[2], red_f[3]));
      for (int i = tid; i < nk; i += 128) {
        const float e = expf(sc[i] - m);
        sc[i] = e;
        l += (double)e;
      }
      l = warp_sum_d(l);
      if (lane == 0) red_d[wid] = l;
      __syncthreads();
      l = ((red_d[0] + red_d[1]) + red_d[2]) + red_d[3];
      // second product: thread -> (four columns of the head, every VPI-th key)
      const int vr = tid / VPR, vq = tid % VPR;
      float4 o = zero4;
      const float *vp = vc + ((long long)b * cap + c0) * d_model + h * DH + vq * 4;
      for (int i0 = vr; i0 < nk; i0 += DEC_UNROLL * VPI) {
        float4 v[DEC_UNROLL];
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
          const int i = i0 + u * VPI;
          v[u] = i < nk ? *reinterpret_cast<const float4 *>(vp + (long long)i * d_model) : zero4;
        }
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
          const int i = i0 + u * VPI;
          const float e = i < nk ? sc[i] : 0.f;
          o.x = fmaf(e, v[u].x, o.x);
          o.y = fmaf(e, v[u].y, o.y);
          o.z = fmaf(e, v[u].z, o.z);
          o.w = fmaf(e, v[u].w, o.w);
        }
      }
      *reinterpret_cast<float4 *>(o_part + vr * DH + vq * 4) = o;
      __syncthreads();
      if (tid < DH) {
        t = o_part[tid];
#pragma unroll
        for (int q = 1; q < VPI; ++q) t += o_part[q * DH + tid];
      }
    }
    if (out == nullptr) {
      store_context<DH>(ctx, t * (float)(1.0 / l), b, h, d_model, tid, red_f);
    } else if (tid < DH) {
      out[tid] = t;
      if (tid == 0) {
        out[DH] = m;
        out[DH + 1] = (float)l;
      }
    }
  }  // chunk with keys
  if (out == nullptr) return;
  // The chunk that finishes last joins all chunks of its (stream, head) in chunk order: the common
  // maximum, every chunk's sums rescaled to it, the context row normalised by the total. The
  // counter rests at zero between launches.
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    is_last = atomicAdd(&counters[b * gridDim.y + h], 1) == chunks - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  float v = 0.f;
  if (tid < DH) {
    const float *pp = part + ((long long)b * gridDim.y + h) * chunks * (DH + 2);
    float mm = -INFINITY;
    for (int q = 0; q < chunks; ++q) mm = fmaxf(mm, __ldcg(&pp[q * (DH + 2) + DH]));
    double ll = 0.0;
    float oo = 0.f;
    for (int q = 0; q < chunks; ++q) {
      const float mc = __ldcg(&pp[q * (DH + 2) + DH]);
      if (mc == -INFINITY) continue;  // an empty chunk of a launch sized for a longer context
      const float w = expf(mc - mm);
      ll += (double)__ldcg(&pp[q * (DH + 2) + DH + 1]) * (double)w;
      oo = fmaf(__ldcg(&pp[q * (DH + 2) + tid]), w, oo);
    }
    v = oo * (float)(1.0 / ll);
    if (tid == 0) counters[b * gridDim.y + h] = 0;
  }
  store_context<DH>(ctx, v, b, h, d_model, tid, red_f);
}

}  // namespace

void launch_embed_last_ln(const float *tok_emb, const float *pos_emb, const int *ids, int ids_ld,
                          const LoopState *state, int s_host, int n_streams, int d, int vocab, const float *gamma,
                          const float *beta, float *x, float *ln, DevErr *err, cudaStream_t st) {
  const int warps = 4;
  launch_pdl(embed_last_ln_kernel, dim3((n_streams + warps - 1) / warps), dim3(warps * 32), 0, st, g_pdl_enabled,
             tok_emb, pos_emb, ids, ids_ld, state, s_host, n_streams, d, vocab, gamma, beta, x, ln, err);
}

void launch_kv_store(const float *qkv, const LoopState *state, int s_host, int n_streams, int d, int cap, float *kc,
                     float *vc, cudaStream_t st) {
  const long long rows = (long long)n_streams * s_host;
  if (rows <= 0) return;
  launch_pdl(kv_store_kernel, dim3((unsigned)rows), dim3(128), 0, st, g_pdl_enabled, qkv, state, s_host, n_streams, d,
             cap, kc, vc);
}

DecodeAttnPlan attn_decode_plan(int n_streams, int s, int n_heads, int dh) {
  DecodeAttnPlan p{};
  const long long heads = (long long)n_streams * n_heads;
  // about two CTAs per SM, chunks of 32..1024 keys
  long long want = (2 * 148 + heads - 1) / heads;
  if (want < 1) want = 1;
  int keys = (int)((s + want - 1) / want);
  keys = (keys + 31) / 32 * 32;
  if (keys < 32) keys = 32;
  if (keys > 1024) keys = 1024;
  p.keys_per_chunk = keys;
  p.chunks = (s + keys - 1) / keys;
  p.scratch_floats = p.chunks > 1 ? (size_t)heads * p.chunks * (dh + 2) : 0;
  return p;
}

// The number of chunks is not monotone in the context (their length grows in steps of 32): of 48 heads, 192 positions are cut
// into 6, 224 into 7 and 256 into 4. At most as many as are wanted, or as chunks of 32 (or, where wanted chunks would be longer
// than that, of 1024) there are in the longest context.
size_t attn_decode_scratch_floats(int n_streams, int cap, int n_heads, int dh) {
  const long long heads = (long long)n_streams * n_heads, want = (2 * 148 + heads - 1) / heads;
  const long long shortest = (cap + 31) / 32, longest = (cap + 1023) / 1024;
  long long chunks = want < shortest ? want : shortest;
  if (chunks < longest) chunks = longest;
  return chunks > 1 ? (size_t)heads * chunks * (dh + 2) : 0;
}

template <int DH>
static void launch_attn_decode_dh(const float *qkv, float *kc, float *vc, int cap, int d_model, int n_heads,
                                  int n_streams, const LoopState *state, int s_host, const DecodeAttnPlan &plan,
                                  float *part, int *counters, const DecodeCtx &ctx, cudaStream_t st) {
  const float scale = 1.0f / sqrtf((float)DH);
  dim3 grid((unsigned)plan.chunks, (unsigned)n_heads, (unsigned)n_streams);
  float *pp = plan.chunks > 1 ? part : nullptr;
  const size_t smem = DH < 32 ? (size_t)plan.keys_per_chunk * sizeof(float) : 0;
  auto go = [&](auto kernel) {
    launch_pdl(kernel, grid, dim3(128), smem, st, g_pdl_enabled, qkv, kc, vc, cap, d_model, state, s_host, plan.keys_per_chunk, scale, pp, ctx,
               counters);
  };
  if constexpr (DH >= 32) {
    if (plan.keys_per_chunk <= 4 * dec_batch(DH) || (long long)plan.chunks * n_heads * n_streams > 5 * 148) return go(attn_decode_kernel<DH, false>);
  }
  go(attn_decode_kernel<DH, true>);
}

int launch_attn_decode(const float *qkv, float *kc, float *vc, int cap, int d_model, int n_heads, int n_streams,
                       const LoopState *state, int s_host, float *part, int *counters, float *ctx_out, cudaStream_t st,
                       float *ctx_lo, const TcPairF16 *ctx_f16) {
  const DecodeCtx ctx{ctx_out, ctx_lo, ctx_f16 ? *ctx_f16 : TcPairF16{}};
  const int dh = d_model / n_heads;
  const DecodeAttnPlan plan = attn_decode_plan(n_streams, s_host, n_heads, dh);
  if (plan.chunks > 1 && (part == nullptr || counters == nullptr))
    throw std::invalid_argument("litnice_b200: decode attention needs scratch");
  if (ctx_f16 != nullptr && dh != TC_F16_SLOT)
    throw std::invalid_argument("litnice_b200: decode attention stores fp16 pairs for head dimension 64 only");
  switch (dh) {
    case 16: launch_attn_decode_dh<16>(qkv, kc, vc, cap, d_model, n_heads, n_streams, state, s_host, plan, part, counters, ctx, st); break;
    case 32: launch_attn_decode_dh<32>(qkv, kc, vc, cap, d_model, n_heads, n_streams, state, s_host, plan, part, counters, ctx, st); break;
    case 64: launch_attn_decode_dh<64>(qkv, kc, vc, cap, d_model, n_heads, n_streams, state, s_host, plan, part, counters, ctx, st); break;
    case 128: launch_attn_decode_dh<128>(qkv, kc, vc, cap, d_model, n_heads, n_streams, state, s_host, plan, part, counters, ctx, st); break;
    default: throw std::invalid_argument("litnice_b200: decode attention supports head dimensions 16, 32, 64, 128");
  }
  return 1;
}

}  // namespace lb
