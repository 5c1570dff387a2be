// plain.cu -- the plain FP32 guiding step around the network kernels of
// plain_net.cu, and the optimiser both paths share:
//   query: network -> mixture sample/pdf
//   train: network forward -> KL loss/adjoint -> network backward -> Adam+EMA
// Query counts are read from device memory (d_count, clamped to n_max), so
// every launch is shape-agnostic and capturable in a CUDA graph.
#include <math.h>
#include <stdio.h>

#include "api_common.cuh"
#include "ctx.cuh"

namespace nmg {

NMG_D int dev_count(const int* d_count, int n_max) {
  if (!d_count) return n_max;
  int n = *d_count;
  return n < 0 ? 0 : (n > n_max ? n_max : n);
}

static int blocks_for(long n, int threads, int cap_per_sm = 8) {
  long b = (n + threads - 1) / threads;
  long cap = 152L * cap_per_sm;
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}

// ----------------------------------------------------------------- featurize
__global__ void k_featurize(EncodingParams e, const float* __restrict__ pos, const float* __restrict__ wo,
                            const float* __restrict__ nrm, const float* __restrict__ rough, const int* d_count,
                            int n_max, float* __restrict__ x) {
  const int n = dev_count(d_count, n_max);
  for (long q = long(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += long(gridDim.x) * blockDim.x) {
    float row[10];
    featurize(e, load3(pos, q), load3(wo, q), load3(nrm, q), rough[q], row);
    for (int d = 0; d < e.n_input; ++d) x[q * e.n_input + d] = row[d];
  }
}

// ----------------------------------------------------------------- mixture
NMG_D f3 face_forward(f3 n, f3 v) { return dot3(n, v) > 0.f ? n : f3{-n.x, -n.y, -n.z}; }

template <int K>
__global__ void __launch_bounds__(128) k_query_mixture(const float* __restrict__ raw, int stride,
                                                       const float* __restrict__ nrm, const float* __restrict__ wo,
                                                       const float* __restrict__ u4, MixOpts o, const int* d_count,
                                                       int n_max, float* __restrict__ dir, float* __restrict__ pdf,
                                                       int* __restrict__ lobe, float* __restrict__ sel, int has_sel) {
  const int n = dev_count(d_count, n_max);
  for (long q = long(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += long(gridDim.x) * blockDim.x) {
    const float* r = raw + q * stride;
    Mix<K> m;
    mix_activate<K, false>(m, r, o.kappa_softplus);
    if (o.cosine) mix_apply_cosine<K, false>(m, face_forward(load3(nrm, q), load3(wo, q)));
    float4 u = reinterpret_cast<const float4*>(u4)[q];
    int s = mix_select<K>(m, u.y);
    f3 d = mix_sample_lobe<K, false>(m, s, u.z, u.w);
    store3(dir, q, d);
    pdf[q] = mix_pdf<K, false>(m, d);
    if (lobe) lobe[q] = s;
    if (sel && has_sel) sel[q] = logistic<false>(r[4 * K]);
  }
}

template <int K>
__global__ void __launch_bounds__(128) k_pdf_mixture(const float* __restrict__ raw, int stride,
                                                     const float* __restrict__ nrm, const float* __restrict__ wo,
                                                     const float* __restrict__ wi, MixOpts o, const int* d_count,
                                                     int n_max, float* __restrict__ pdf) {
  const int n = dev_count(d_count, n_max);
  for (long q = long(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += long(gridDim.x) * blockDim.x) {
    Mix<K> m;
    mix_activate<K, false>(m, raw + q * stride, o.kappa_softplus);
    if (o.cosine) mix_apply_cosine<K, false>(m, face_forward(load3(nrm, q), load3(wo, q)));
    pdf[q] = mix_pdf<K, false>(m, load3(wi, q));
  }
}

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double s[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) s[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < int(blockDim.x >> 5); ++w) r += s[w];
  return r;
}

template <int K, bool SEL>
__global__ void __launch_bounds__(128) k_train_loss(const float* __restrict__ raw, int stride,
                                                    const float* __restrict__ rec, int rstride, MixOpts o,
                                                    float loss_scale, const int* d_count, int n_max,
                                                    float* __restrict__ draw, double* __restrict__ partials) {
  const int n = dev_count(d_count, n_max);
  const float scale = n > 0 ? loss_scale / float(n) : 0.f;
  double acc = 0.0;
  for (long q = long(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += long(gridDim.x) * blockDim.x) {
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = j < rstride ? rec[q * rstride + j] : 0.f;
    float g[4 * K + 1];
    float l = SEL ? mix_kl_loss_grad_selection<K, false>(raw + q * stride, r, scale, o, g)
                  : mix_kl_loss_grad<K, false>(raw + q * stride, r, scale, o, g);
    float* gr = draw + q * stride;
    for (int j = 0; j < stride; ++j) gr[j] = j < 4 * K + (SEL ? 1 : 0) ? g[j] : 0.f;
    acc += double(l);
  }
  double s = block_sum(acc);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// ---------------------------------------------------------------- optimiser
// A training step whose device count is zero takes no optimiser step (the
// reference's training loop stops before a batch below its minimum size,
// integrator.cpp:670-671): the step counter (k_finish_step), Adam and the EMA
// leave the parameters and the optimiser state as they are.

// adam.h:47-119 + ema.h:62-75/102-145 in one pass over four parameters per
// thread (128-bit loads and stores); also writes the reduced-precision copies
// of the training and inference weights and FP64 partial sums of the squared
// unscaled gradient. Bias corrections beta^t use exp2(t log2 beta) with the
// logarithms computed once on the host (adam.h:103 evaluates powf per
// parameter). Requires n_params and n_matrix to be multiples of 4 (layer
// widths are multiples of 16).
struct AdamArgs {
  long n4;               // n_params / 4
  long n_matrix;         // parameters that get l2 and never skip
  float loss_scale, lr, beta1, beta2, eps, l2, ema_decay;
  float log2_beta1, log2_beta2, log2_decay;
  int use_ema, fp16;
};

NMG_D uint32_t pack16(float a, float b, int fp16) {
  if (fp16) return uint32_t(__half_as_ushort(__float2half_rn(a))) | (uint32_t(__half_as_ushort(__float2half_rn(b))) << 16);
  return uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(a))) |
         (uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(b))) << 16);
}

// Bound by memory, and by the exponentials, roots and divides of the update if
// they are not kept few: parameters with the same step count share the
// bias-corrected learning rate (neighbours mostly do), and what a group of four
// needs in any case is loaded first. One wave of 4 blocks per SM (64 registers):
// the training step of 262,144 records 386 -> 373 us, of 65,536 252 -> 241 us
// (2 waves 378, 3 blocks per SM 385, 5 blocks 378, two groups of four at a time
// 391 us; evict-first loads and stores 379 us).
constexpr int kAdamBlocks = 4;
template <bool HALF16>
__global__ void __launch_bounds__(256, kAdamBlocks) k_adam_ema(AdamArgs a, const float4* __restrict__ grad,
                                                  const uint32_t* __restrict__ d_step, float4* __restrict__ w,
                                                  float4* __restrict__ m, float4* __restrict__ v,
                                                  uint4* __restrict__ psteps, float4* __restrict__ w_inf,
                                                  uint2* __restrict__ w16, uint2* __restrict__ w16_inf,
                                                  double* __restrict__ partials, const int* __restrict__ d_count) {
  if (d_count && *d_count <= 0) return;  // an empty batch takes no step
  const uint32_t step = *d_step + 1;  // d_step counts the steps taken before this one
  const float debias_old = 1.f - exp2f(float(step - 1) * a.log2_decay);
  const float debias_new = 1.f / (1.f - exp2f(float(step) * a.log2_decay));
  const bool separate_inf = w_inf != w;
  // squared-gradient sum: FP32 within each group of four (the FP64 pipe of
  // this GPU is narrow), FP64 across groups and threads
  double gn = 0.0;
  for (long j = long(blockIdx.x) * blockDim.x + threadIdx.x; j < a.n4; j += long(gridDim.x) * blockDim.x) {
    const bool matrix = 4 * j < a.n_matrix;
    const float4 g4 = grad[j], w4 = w[j];
    float4 e4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.use_ema) e4 = w_inf[j];
    const float gg[4] = {g4.x / a.loss_scale, g4.y / a.loss_scale, g4.z / a.loss_scale, g4.w / a.loss_scale};
    float ww[4] = {w4.x, w4.y, w4.z, w4.w};
    bool any = matrix;
    float g2 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      g2 = fmaf(gg[k], gg[k], g2);
      any |= gg[k] != 0.f;
    }
    gn += double(g2);
    if (any) {
      const float4 m4 = m[j], v4 = v[j];
      const uint4 t4 = psteps[j];
      float mm[4] = {m4.x, m4.y, m4.z, m4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
      uint32_t tt[4] = {t4.x, t4.y, t4.z, t4.w};
      float lr_t = 0.f;
      uint32_t t_of = 0u;  // the step count that lr_t is for
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!matrix && gg[k] == 0.f) continue;  // non-matrix parameters without gradient keep their state
        float g = gg[k];
        if (matrix) g += a.l2 * ww[k];
        mm[k] = a.beta1 * mm[k] + (1.f - a.beta1) * g;
        vv[k] = a.beta2 * vv[k] + (1.f - a.beta2) * (g * g);
        const uint32_t t = ++tt[k];
        if (t != t_of) {
          // adam.h:102: the bias-correction quotient first, then the learning rate
          lr_t = a.lr * (sqrtf(1.f - exp2f(float(t) * a.log2_beta2)) / (1.f - exp2f(float(t) * a.log2_beta1)));
          t_of = t;
        }
        ww[k] = ww[k] - lr_t / (sqrtf(vv[k]) + a.eps) * mm[k];
      }
      m[j] = make_float4(mm[0], mm[1], mm[2], mm[3]);
      v[j] = make_float4(vv[0], vv[1], vv[2], vv[3]);
      psteps[j] = make_uint4(tt[0], tt[1], tt[2], tt[3]);
      w[j] = make_float4(ww[0], ww[1], ww[2], ww[3]);
    }
    float wv[4] = {ww[0], ww[1], ww[2], ww[3]};
    if (a.use_ema) {
      const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) wv[k] = (ee[k] * a.ema_decay * debias_old + ww[k] * (1.f - a.ema_decay)) * debias_new;
      w_inf[j] = make_float4(wv[0], wv[1], wv[2], wv[3]);
    } else if (separate_inf) {
      w_inf[j] = make_float4(ww[0], ww[1], ww[2], ww[3]);
    }
    if (HALF16) {
      w16[j] = make_uint2(pack16(ww[0], ww[1], a.fp16), pack16(ww[2], ww[3], a.fp16));
      w16_inf[j] = make_uint2(pack16(wv[0], wv[1], a.fp16), pack16(wv[2], wv[3], a.fp16));
    }
  }
  double s = block_sum(gn);
  if (threadIdx.x == 0 && partials) partials[blockIdx.x] = s;
}

// Counter-based uniform in [0,1) for parameter initialisation (splitmix64).
NMG_D float hash_uniform(uint64_t seed, uint64_t i) {
  uint64_t z = seed * 0x9E3779B97F4A7C15ull + i * 0xBF58476D1CE4E5B9ull + 0x94D049BB133111EBull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return float(z >> 40) * (1.0f / 16777216.0f);
}

__global__ void k_init_params(Layout lay, uint32_t seed, float* __restrict__ w) {
  for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < lay.n_params; i += long(gridDim.x) * blockDim.x) {
    float u = hash_uniform(seed, uint64_t(i));
    float bound = 1e-4f;  // grid.h:1333-1336
    for (int l = 0; l < lay.n_layers; ++l)
      if (i >= lay.off[l] && i < lay.off[l + 1]) bound = sqrtf(6.f / float(lay.in[l] + lay.out[l]));
    w[i] = (2.f * u - 1.f) * bound;
  }
}

// ------------------------------------------------------------ host launchers
nmg_status plain_featurize(nmg_ctx* c, const nmg_shading* in, const int* d_count, int n_max, float* x,
                           cudaStream_t st) {
  k_featurize<<<blocks_for(n_max, 128, 16), 128, 0, st>>>(c->enc, in->pos, in->wo, in->normal, in->roughness,
                                                          d_count, n_max, x);
  return check_launch("k_featurize");
}

template <int K>
static void launch_query_mix(nmg_ctx* c, const float* raw, const nmg_shading* in, const float* u4, const int* d_count,
                             int n_max, const nmg_query_out* out, cudaStream_t st) {
  k_query_mixture<K><<<blocks_for(n_max, 128, 16), 128, 0, st>>>(raw, c->lay.n_out_pad, in->normal, in->wo, u4, c->mix,
                                                                 d_count, n_max, out->dir, out->pdf, out->lobe,
                                                                 out->selection, c->cfg.selection);
}

nmg_status plain_query(nmg_ctx* c, const nmg_shading* in, const float* u4, const int* d_count, int n_max,
                       const nmg_query_out* out, cudaStream_t st) {
  Workspace& w = c->ws;
  float* raw = out->raw ? out->raw : w.raw;
  NMG_TRY(plain_forward(c, in, nullptr, d_count, n_max, c->w_inf, false, raw, st));
  switch (c->lay.K) {
    case 7: launch_query_mix<7>(c, raw, in, u4, d_count, n_max, out, st); break;
    case 8: launch_query_mix<8>(c, raw, in, u4, d_count, n_max, out, st); break;
    case 16: launch_query_mix<16>(c, raw, in, u4, d_count, n_max, out, st); break;
    default: return set_error(NMG_ERR_UNSUPPORTED, "K=%d", c->lay.K);
  }
  return check_launch("k_query_mixture");
}

nmg_status pdf_from_raw(nmg_ctx* c, const float* raw, const nmg_shading* in, const float* wi, const int* d_count,
                        int n_max, float* pdf, cudaStream_t st) {
  const int b = blocks_for(n_max, 128, 16);
  const int sd = c->lay.n_out_pad;
  switch (c->lay.K) {
    case 7: k_pdf_mixture<7><<<b, 128, 0, st>>>(raw, sd, in->normal, in->wo, wi, c->mix, d_count, n_max, pdf); break;
    case 8: k_pdf_mixture<8><<<b, 128, 0, st>>>(raw, sd, in->normal, in->wo, wi, c->mix, d_count, n_max, pdf); break;
    case 16: k_pdf_mixture<16><<<b, 128, 0, st>>>(raw, sd, in->normal, in->wo, wi, c->mix, d_count, n_max, pdf); break;
    default: return set_error(NMG_ERR_UNSUPPORTED, "K=%d", c->lay.K);
  }
  return check_launch("k_pdf_mixture");
}

nmg_status plain_pdf(nmg_ctx* c, const nmg_shading* in, const float* wi, const int* d_count, int n_max, float* pdf,
                     cudaStream_t st) {
  Workspace& w = c->ws;
  NMG_TRY(plain_forward(c, in, nullptr, d_count, n_max, c->w_inf, false, w.raw, st));
  return pdf_from_raw(c, w.raw, in, wi, d_count, n_max, pdf, st);
}

nmg_status optimizer_step(nmg_ctx* c, const int* d_count, int n_max, int n_loss, double* stats, cudaStream_t st) {
  const Layout& L = c->lay;
  const nmg_config& g = c->cfg;
  const int nb = kAdamBlocks * sm_count();
  double* gp = c->ws.partials + c->ws.n_partials / 2;
  if (L.n_params % 4 || L.n_mlp % 4) return set_error(NMG_ERR_UNSUPPORTED, "parameter count not a multiple of 4");
  AdamArgs aa;
  aa.n4 = L.n_params / 4;
  aa.n_matrix = L.n_mlp;
  aa.loss_scale = g.loss_scale;
  aa.lr = g.learning_rate;
  aa.beta1 = g.beta1;
  aa.beta2 = g.beta2;
  aa.eps = g.epsilon;
  aa.l2 = g.l2_reg;
  aa.ema_decay = g.ema_decay;
  aa.log2_beta1 = log2f(g.beta1);
  aa.log2_beta2 = log2f(g.beta2);
  aa.log2_decay = log2f(g.ema_decay);
  aa.use_ema = g.use_ema;
  aa.fp16 = g.path == NMG_PATH_FP16;
  if (c->w16)
    k_adam_ema<true><<<nb, 256, 0, st>>>(aa, reinterpret_cast<const float4*>(c->grad), c->d_step,
                                         reinterpret_cast<float4*>(c->w), reinterpret_cast<float4*>(c->m),
                                         reinterpret_cast<float4*>(c->v), reinterpret_cast<uint4*>(c->psteps),
                                         reinterpret_cast<float4*>(c->w_inf), reinterpret_cast<uint2*>(c->w16),
                                         reinterpret_cast<uint2*>(c->w16_inf), gp, d_count);
  else
    k_adam_ema<false><<<nb, 256, 0, st>>>(aa, reinterpret_cast<const float4*>(c->grad), c->d_step,
                                          reinterpret_cast<float4*>(c->w), reinterpret_cast<float4*>(c->m),
                                          reinterpret_cast<float4*>(c->v), reinterpret_cast<uint4*>(c->psteps),
                                          reinterpret_cast<float4*>(c->w_inf), nullptr, nullptr, gp, d_count);
  NMG_TRY(check_launch("k_adam_ema"));
  return finish_step(c, c->ws.partials, n_loss, gp, nb, d_count, n_max, stats, c->d_step, st);
}

nmg_status plain_train_step(nmg_ctx* c, const float* x, const float* rec, const int* d_count, int n_max,
                            double* stats, cudaStream_t st) {
  const Layout& L = c->lay;
  Workspace& w = c->ws;
  NMG_TRY(plain_forward(c, nullptr, x, d_count, n_max, c->w, true, w.raw, st));
  const int lb = blocks_for(n_max, 128, 4);
  if (lb > w.n_partials / 2) return set_error(NMG_ERR_CAPACITY, "loss partials");
#define LOSS(KK)                                                                                                  \
  if (c->cfg.selection)                                                                                           \
    k_train_loss<KK, true><<<lb, 128, 0, st>>>(w.raw, L.n_out_pad, rec, L.record_floats, c->mix, c->cfg.loss_scale, \
                                               d_count, n_max, w.draw, w.partials);                              \
  else                                                                                                            \
    k_train_loss<KK, false><<<lb, 128, 0, st>>>(w.raw, L.n_out_pad, rec, L.record_floats, c->mix,                  \
                                                c->cfg.loss_scale, d_count, n_max, w.draw, w.partials);
  switch (L.K) {
    case 7: LOSS(7) break;
    case 8: LOSS(8) break;
    case 16: LOSS(16) break;
    default: return set_error(NMG_ERR_UNSUPPORTED, "K=%d", L.K);
  }
#undef LOSS
  NMG_TRY(check_launch("k_train_loss"));
  NMG_CUDA_TRY(cudaMemsetAsync(c->grad, 0, sizeof(float) * L.n_params, st));
  NMG_TRY(plain_backward(c, x, d_count, n_max, c->w, c->grad, st));
  return optimizer_step(c, d_count, n_max, lb, stats, st);
}

// Network VJP at the training weights: draw given, accumulate unscaled
// dL/dparams.
nmg_status plain_vjp(nmg_ctx* c, const float* x, const float* draw, int n, float* raw, float* dparams,
                     cudaStream_t st) {
  const Layout& L = c->lay;
  Workspace& w = c->ws;
  NMG_TRY(plain_forward(c, nullptr, x, nullptr, n, c->w, true, raw ? raw : w.raw, st));
  NMG_CUDA_TRY(cudaMemcpyAsync(w.draw, draw, sizeof(float) * size_t(n) * L.n_out_pad, cudaMemcpyDeviceToDevice, st));
  return plain_backward(c, x, nullptr, n, c->w, dparams, st);
}

nmg_status init_params(nmg_ctx* c, uint32_t seed, cudaStream_t st) {
  k_init_params<<<152 * 8, 256, 0, st>>>(c->lay, seed, c->w);
  return check_launch("k_init_params");
}

__global__ void k_sync_copies(long n, const float* __restrict__ w, const float* __restrict__ wi,
                              uint16_t* __restrict__ w16, uint16_t* __restrict__ w16i, int fp16) {
  for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) {
    w16[i] = fp16 ? __half_as_ushort(__float2half_rn(w[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(w[i]));
    w16i[i] = fp16 ? __half_as_ushort(__float2half_rn(wi[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(wi[i]));
  }
}

// Refreshes the reduced-precision weight copies from the FP32 ones.
nmg_status sync_copies(nmg_ctx* c, cudaStream_t st) {
  if (!c->w16) return NMG_OK;
  k_sync_copies<<<152 * 8, 256, 0, st>>>(c->lay.n_params, c->w, c->w_inf, c->w16, c->w16_inf,
                                         c->cfg.path == NMG_PATH_FP16);
  NMG_TRY(check_launch("k_sync_copies"));
  return pack_images(c, st);
}

}  // namespace nmg
