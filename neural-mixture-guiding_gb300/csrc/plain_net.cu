// plain_net.cu -- the plain FP32 network: encoding, MLP forward, backward
// through the MLP and the grid, weight gradients.
//
// FP32 FMAs on the CUDA cores, every sum in the order of one input after
// another. What bounds it is those FMAs (13,312 a row for the reference
// network, 16,384 for the hash-grid one: 72 TFLOP/s measured for plain FMAs on
// this GPU), so nothing else may be in the way: one kernel per direction keeps
// a tile of 64 rows in shared memory from the first layer to the last, next to
// all of the weights. Four warps of a block do the matrix products of one tile
// while the other four gather the next tile's table entries (forward) or
// scatter the last tile's grid gradient (backward). Two blocks fit an SM at
// three hidden layers and up to 8 lobes (92 KB forward for the reference
// network, 104 KB backward for the hash-grid one); 16 lobes (119 and 118 KB) and
// deeper networks run one. A product thread holds 4 rows x 8 columns, three
// 16-byte shared loads per 32 FMAs. The forward kernel takes 410 us for 524,288
// queries of the reference network, bound by issue slots that FMAs (48% of them
// busy) share with the products' shared loads (472 us with 4 x 4 per thread on all eight warps and
// the roles one after the other, the shared-memory pipe 80% busy; 493 us at 2
// rows x 16 columns, 444 us with eight gathering warps, 430 us on 128-row
// tiles at 8 x 4).
//
// For the backward pass the forward kernel leaves the encoded rows and the
// hidden activations in global memory as tiles of [column][64 rows], the order
// they have in shared memory; the backward kernel does the same with the
// deltas, and the weight-gradient kernel reads both.
#include <string.h>

#include "api_common.cuh"
#include "ctx.cuh"

namespace nmg {

constexpr int kProduct = 128, kMovers = 128;  // threads of a block's two roles, the product warps first
constexpr int kPlainThreads = kProduct + kMovers;

struct PlainNet {
  EncodingParams enc;
  int n_layers, n_grid;           // n_grid = levels * feats
  int in[kMaxLayers], out[kMaxLayers];
  const float* w[kMaxLayers];     // row-major [out][in]
  const float* table;
  uint32_t T[kMaxLevels], sy[kMaxLevels], sz[kMaxLevels];  // entries; dense strides of y and z
  uint32_t hashed;                // bit l: level l is hashed
  uint32_t pow2;                  // bit l: T is a power of two
  const int* d_count;
  int n_max;
};

struct PlainFwd {
  PlainNet net;
  nmg_shading in;                 // pos non-NULL: featurise these
  const float* x;                 // else network input rows
  float* enc_t;                   // NULL, or the tiles kept for the backward pass
  float* h_t[kMaxLayers];
  float* raw;                     // [n][ld_raw]
  int ld_raw;
  int raw_wide;                   // raw is 16-byte aligned
};

struct PlainBwd {
  PlainNet net;
  const float* x;                 // network input rows
  const float* draw;              // [n][out of the last layer]
  const float* h_t[kMaxLayers];
  float* d_t[kMaxLayers];         // delta tiles of every layer
  float* gtable;
  int wide;                       // gtable is 16-byte aligned
};

NMG_D int plain_count(const PlainNet& p) {
  if (!p.d_count) return p.n_max;
  const int n = *p.d_count;
  return n < 0 ? 0 : (n > p.n_max ? p.n_max : n);
}

// Entry of a corner (grid.h:171-187 with the coherent-prime hash, grid.h:132-135),
// the level's strides and hashing worked out on the host (plain_net).
NMG_D uint32_t plain_index(const PlainNet& p, int l, uint32_t x, uint32_t y, uint32_t z) {
  const uint32_t T = p.T[l];
  const uint32_t i = (p.hashed >> l) & 1u ? x ^ (y * 2654435761u) ^ (z * 805459861u)
                                          : x + y * p.sy[l] + z * p.sz[l];
  if ((p.pow2 >> l) & 1u) return i & (T - 1u);
  return i < T ? i : i % T;
}

template <int F> NMG_D void plain_entry(const float* table, uint32_t e, float (&v)[F]) {
  if constexpr (F == 1) {
    v[0] = __ldg(table + e);
  } else if constexpr (F == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(table) + e);
    v[0] = t.x, v[1] = t.y;
  } else {
#pragma unroll
    for (int k = 0; k < F / 4; ++k) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(table) + size_t(e) * (F / 4) + k);
      v[4 * k] = t.x, v[4 * k + 1] = t.y, v[4 * k + 2] = t.z, v[4 * k + 3] = t.w;
    }
  }
}

// Part h of 4 of the featurisation of one query (featurize<false>'s
// expressions): position, outgoing direction, normal, roughness.
NMG_D void featurize_part(const EncodingParams& e, const nmg_shading& in, long q, int h, int r, float* xs) {
  if (h == 0) {
    const f3 pos = load3(in.pos, q);
    const float p[3] = {pos.x, pos.y, pos.z};
    const float infl = aabb_inflation(e.aabb);
#pragma unroll
    for (int d = 0; d < 3; ++d) xs[d * kPlainRows + r] = normalize_coord(e.aabb, infl, d, p[d]);
  } else if (h == 1) {
    const f3 w = normalize3(load3(in.wo, q));
    xs[3 * kPlainRows + r] = (w.x + 1.f) * 0.5f;
    xs[4 * kPlainRows + r] = (w.y + 1.f) * 0.5f;
    xs[5 * kPlainRows + r] = (w.z + 1.f) * 0.5f;
  } else if (h == 2) {
    const f3 nn = normalize3(load3(in.normal, q));
    if (e.input_mode == 0) {
      const float th = acosf(fminf(1.f, fmaxf(-1.f, nn.z)));
      float ph = atan2f(nn.y, nn.x);
      if (ph < 0.f) ph += NMG_TWO_PI;
      xs[6 * kPlainRows + r] = float(double(th) / 3.14159265358979323846);
      xs[7 * kPlainRows + r] = ph / NMG_TWO_PI;
    } else {
      xs[6 * kPlainRows + r] = (nn.x + 1.f) * 0.5f;
      xs[7 * kPlainRows + r] = (nn.y + 1.f) * 0.5f;
      xs[8 * kPlainRows + r] = (nn.z + 1.f) * 0.5f;
    }
  } else {
    xs[(e.input_mode == 0 ? 8 : 9) * kPlainRows + r] = 1.f - expf(-in.roughness[q]);
  }
}

// Direction columns of row r (encode_directional's), DIR 0: any degree and bin
// count, as part 3; 1 and 2: the hash-grid (SH 4 twice, 4 bins) and the
// reference preset (SH 2, three one-blobs of 4 bins), unrolled, in four parts.
template <int DIR>
NMG_D void plain_directional(const EncodingParams& e, const float* xs, float* act, int n_grid, int r, int h) {
  auto x = [&](int d) { return xs[d * kPlainRows + r]; };
  if constexpr (DIR == 0) {
    if (h != 3) return;
    float xr[10], rest[64];
    for (int d = 0; d < 10; ++d) xr[d] = d < e.n_input ? x(d) : 0.f;
    encode_directional(e, xr, rest);
    for (int k = n_grid; k < e.n_enc_pad; ++k) act[k * kPlainRows + r] = rest[k - n_grid];
  } else {
    constexpr int SH = DIR == 1 ? 4 : 2, SH2 = SH * SH;
    float* o = act + n_grid * kPlainRows + r;
    if (h == 0 || (DIR == 1 && h == 1)) {
      const int b = h == 0 ? 3 : 6;
      float d[16];
      sh_basis(SH, x(b) * 2.f - 1.f, x(b + 1) * 2.f - 1.f, x(b + 2) * 2.f - 1.f, d);
#pragma unroll
      for (int k = 0; k < SH2; ++k) o[(h * SH2 + k) * kPlainRows] = d[k];
    } else if (DIR == 2 || h == 2) {
      float d[4];
      oneblob(4, x(DIR == 1 ? 9 : 5 + h), d);
#pragma unroll
      for (int k = 0; k < 4; ++k) o[((DIR == 1 ? 2 * SH2 : SH2 + 4 * (h - 1)) + k) * kPlainRows] = d[k];
    }
    if (h == 3)
      for (int k = n_grid + (DIR == 1 ? 2 * SH2 + 4 : SH2 + 12); k < e.n_enc_pad; ++k) act[k * kPlainRows + r] = 1.f;
  }
}

// The product warps' thread tile: 4 rows x 8 columns, a warp 32 rows x 32
// columns, the four warps 64 x 64.
struct PlainTile {
  int row, col;
  NMG_D PlainTile() {
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    row = 32 * (wid & 1) + 4 * (lane & 7);
    col = 32 * ((wid >> 1) & 1) + 8 * (lane >> 3);
  }
};

// acc[column][row] = sum over k < n of A[k][row] B[k][col], k ascending.
NMG_D void plain_product(const float* A, const float* B, int ldb, int n, float (&acc)[8][4]) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[c][r] = 0.f;
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(A + k * kPlainRows);
    const float4 b = *reinterpret_cast<const float4*>(B + k * ldb), b2 = *reinterpret_cast<const float4*>(B + k * ldb + 4);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b.x, b.y, b.z, b.w, b2.x, b2.y, b2.z, b2.w};
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[c][r] = fmaf(av[r], bv[c], acc[c][r]);
  }
}

NMG_D void bar_product() { asm volatile("bar.sync 1, %0;" ::"n"(kProduct) : "memory"); }
NMG_D void bar_movers() { asm volatile("bar.sync 2, %0;" ::"n"(kMovers) : "memory"); }

constexpr int kPlainPad = 4;  // floats after each transposed weight row: its 16-byte stores spread over the banks

template <int F, int DIR>
__global__ void __launch_bounds__(kPlainThreads, 2) k_plain_forward(const __grid_constant__ PlainFwd a) {
  extern __shared__ __align__(16) float sm[];
  const PlainNet& p = a.net;
  const int L = p.n_layers, n_enc = p.in[0], n_grid = p.n_grid;
  float* W = sm;  // per layer [in][out + pad]
  int w_floats = 0;
  for (int l = 0; l < L; ++l) {
    const int nin = p.in[l], nout = p.out[l], ld = nout + kPlainPad, q4 = nin / 4;
    // 8 output rows x 4 groups of 4 inputs per warp: whole sectors in, two-way conflicts out
    for (int i = threadIdx.x; i < q4 * nout; i += kPlainThreads) {
      const int blk = i >> 5, ln = i & 31;
      const int j = (blk / (q4 / 4)) * 8 + (ln >> 2), k = (blk % (q4 / 4)) * 4 + (ln & 3);
      const float4 v = __ldg(reinterpret_cast<const float4*>(p.w[l] + size_t(j) * nin) + k);
      float* d = W + w_floats + 4 * k * ld + j;
      d[0] = v.x;
      d[ld] = v.y;
      d[2 * ld] = v.z;
      d[3 * ld] = v.w;
    }
    w_floats += nin * ld;
  }
  const int act_floats = (n_enc > kWidth ? n_enc : kWidth) * kPlainRows;
  float* act = sm + w_floats;          // two buffers of [max(n_enc, 64)][64]
  float* xs = act + 2 * act_floats;    // [10][64]
  const int n = plain_count(p);
  const bool encoder = threadIdx.x >= kProduct;
  const int t = int(threadIdx.x) - kProduct, r = t % kPlainRows, h = t / kPlainRows;  // of an encoder
  const PlainTile tl;
  const int tiles = (n + kPlainRows - 1) / kPlainRows;

  // One tile's rows into A (the encoder warps; two threads per row, which take
  // every second level each).
  auto encode = [&](int tile, float* A) {
    const long q0 = long(tile) * kPlainRows, q = q0 + r;
    if (a.in.pos) {
      if (q < n) {
        featurize_part(p.enc, a.in, q, 2 * h, r, xs);
        featurize_part(p.enc, a.in, q, 2 * h + 1, r, xs);
      } else if (h == 0) {
        for (int d = 0; d < p.enc.n_input; ++d) xs[d * kPlainRows + r] = 0.f;
      }
    } else {
      const int ni = p.enc.n_input;
      for (int i = t; i < kPlainRows * ni; i += kMovers) {
        const int rr = i / ni, d = i - rr * ni;
        xs[d * kPlainRows + rr] = q0 + rr < n ? a.x[q0 * ni + i] : 0.f;
      }
    }
    bar_movers();
    for (int l = h; l < p.enc.levels; l += 2) {
      float w[3];
      uint32_t g[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) pos_fract(xs[d * kPlainRows + r], p.enc.scale[l], p.enc.smoothstep, &w[d], &g[d]);
      const float* tab = p.table + size_t(p.enc.offset[l]) * F;
      float acc[F];
#pragma unroll
      for (int f = 0; f < F; ++f) acc[f] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float wt = ((k & 1 ? w[0] : 1.f - w[0]) * (k & 2 ? w[1] : 1.f - w[1])) * (k & 4 ? w[2] : 1.f - w[2]);
        float v[F];
        plain_entry<F>(tab, plain_index(p, l, g[0] + (k & 1), g[1] + ((k >> 1) & 1), g[2] + (k >> 2)), v);
#pragma unroll
        for (int f = 0; f < F; ++f) acc[f] = fmaf(wt, v[f], acc[f]);
      }
#pragma unroll
      for (int f = 0; f < F; ++f) A[(l * F + f) * kPlainRows + r] = acc[f];
    }
    plain_directional<DIR>(p.enc, xs, A, n_grid, r, 2 * h);
    plain_directional<DIR>(p.enc, xs, A, n_grid, r, 2 * h + 1);
    bar_movers();  // xs is rewritten by the next call
    if (a.enc_t) {
      float4* dst = reinterpret_cast<float4*>(a.enc_t + size_t(tile) * kPlainRows * n_enc);
      for (int i = t; i < n_enc * kPlainRows / 4; i += kMovers) dst[i] = reinterpret_cast<const float4*>(A)[i];
    }
  };

  // One tile's layers, in place in A (the product warps).
  auto layers = [&](int tile, float* A) {
    const long q0 = long(tile) * kPlainRows;
    const float* Wl = W;
    for (int l = 0; l < L; ++l) {
      const int nin = p.in[l], nout = p.out[l], ld = nout + kPlainPad;
      float acc[8][4];
      if (l == L - 1) {
        for (int c0 = tl.col; c0 < nout; c0 += kWidth) {
          plain_product(A + tl.row, Wl + c0, ld, nin, acc);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (q0 + tl.row + i < n) {
              float* dst = a.raw + (q0 + tl.row + i) * a.ld_raw + c0;
              if (a.raw_wide) {
                *reinterpret_cast<float4*>(dst) = make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]);
                *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[4][i], acc[5][i], acc[6][i], acc[7][i]);
              } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) dst[c] = acc[c][i];
              }
            }
        }
        break;
      }
      plain_product(A + tl.row, Wl + tl.col, ld, nin, acc);  // hidden layers are kWidth wide
      bar_product();
      float* keep = a.h_t[l] ? a.h_t[l] + size_t(tile) * kPlainRows * kWidth : nullptr;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 v = make_float4(fmaxf(acc[c][0], 0.f), fmaxf(acc[c][1], 0.f), fmaxf(acc[c][2], 0.f),
                                     fmaxf(acc[c][3], 0.f));
        const int at = (tl.col + c) * kPlainRows + tl.row;
        *reinterpret_cast<float4*>(A + at) = v;
        if (keep) *reinterpret_cast<float4*>(keep + at) = v;
      }
      bar_product();
      Wl += nin * ld;
    }
  };

  int buf = 0;
  if (encoder && int(blockIdx.x) < tiles) encode(blockIdx.x, act);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
    __syncthreads();
    if (!encoder)
      layers(tile, act + buf * act_floats);
    else if (tile + int(gridDim.x) < tiles)
      encode(tile + gridDim.x, act + (buf ^ 1) * act_floats);
  }
}

// Adds one record's grid-feature gradient g[F] at corner x + xb of level l's
// four (y, z) into the table gradient (grid.h:387-510). Neighbouring lanes
// take the two x corners of a record, which mostly share a 128-byte line: one
// L2 request for both.
template <int F>
NMG_D void plain_scatter(const PlainNet& p, int l, const float (&pos)[3], const float (&g)[F], uint32_t xb,
                         float* gtable, bool wide) {
  float w[3];
  uint32_t gc[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) pos_fract(pos[d], p.enc.scale[l], p.enc.smoothstep, &w[d], &gc[d]);
  const float wx = xb ? w[0] : 1.f - w[0];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float wt = (wx * (c & 1 ? w[1] : 1.f - w[1])) * (c & 2 ? w[2] : 1.f - w[2]);
    const uint32_t e = p.enc.offset[l] + plain_index(p, l, gc[0] + xb, gc[1] + (c & 1), gc[2] + (c >> 1));
    float* dst = gtable + size_t(e) * F;
    if (F == 1 || !wide) {
#pragma unroll
      for (int k = 0; k < F; ++k) atomicAdd(dst + k, wt * g[k]);
    } else if constexpr (F == 2) {
      atomicAdd(reinterpret_cast<float2*>(dst), make_float2(wt * g[0], wt * g[1]));
    } else {
#pragma unroll
      for (int k = 0; k + 3 < F; k += 4)
        atomicAdd(reinterpret_cast<float4*>(dst + k),
                  make_float4(wt * g[k], wt * g[k + 1], wt * g[k + 2], wt * g[k + 3]));
    }
  }
}

// Deltas of every layer from dL/draw, and the grid gradient. Of layer 0's
// input only the grid columns have parameters below. The product warps carry
// one tile's delta from the last layer to the first in D and leave its grid
// gradient in G; the other warps meanwhile scatter the last tile's grid
// gradient and read the next tile's dL/draw. D is double, and so is G where
// shared memory holds it beside the weights; with one G (ONE_G) the product
// warps wait for the last tile's scatter before they write theirs.
template <int F, bool ONE_G>
__global__ void __launch_bounds__(kPlainThreads, 2) k_plain_backward(const __grid_constant__ PlainBwd a) {
  extern __shared__ __align__(16) float sm[];
  const PlainNet& p = a.net;
  const int L = p.n_layers, nout = p.out[L - 1], ng = (p.n_grid + 15) / 16 * 16;
  float* W = sm;  // per layer, the last first: [out][in], layer 0: [out][ng]
  int w_floats = 0;
  for (int l = L - 1; l >= 0; --l) {
    const int ld = l == 0 ? ng : p.in[l];
    for (int i = threadIdx.x; i < p.out[l] * (ld / 4); i += kPlainThreads) {
      const int j = i / (ld / 4), k = i - j * (ld / 4);
      reinterpret_cast<float4*>(W + w_floats)[i] = __ldg(reinterpret_cast<const float4*>(p.w[l] + size_t(j) * p.in[l]) + k);
    }
    w_floats += p.out[l] * ld;
  }
  const int d_floats = (nout > kWidth ? nout : kWidth) * kPlainRows;
  float* D = sm + w_floats;              // two buffers
  float* G = D + 2 * d_floats;           // two buffers (ONE_G: one) of [ng][64]
  float* xs = G + (ONE_G ? 1 : 2) * ng * kPlainRows;  // two buffers of [3][64]
  const int n = plain_count(p), ni = p.enc.n_input;
  const bool mover = threadIdx.x >= kProduct;
  const int t = int(threadIdx.x) - kProduct;  // of a mover
  const PlainTile tl;
  const int tiles = (n + kPlainRows - 1) / kPlainRows;

  auto read = [&](int tile, int buf) {
    const long q0 = long(tile) * kPlainRows;
    float* keep = a.d_t[L - 1] + size_t(tile) * kPlainRows * nout;
    for (int i = t; i < kPlainRows * (nout / 4); i += kMovers) {
      const int r = i % kPlainRows, k = i / kPlainRows;
      const float4 v = q0 + r < n ? __ldg(reinterpret_cast<const float4*>(a.draw + (q0 + r) * nout) + k)
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        D[buf * d_floats + (4 * k + c) * kPlainRows + r] = e[c];
        keep[(4 * k + c) * kPlainRows + r] = e[c];
      }
    }
    for (int i = t; i < 3 * kPlainRows; i += kMovers) {
      const int r = i % kPlainRows, d = i / kPlainRows;
      xs[buf * 3 * kPlainRows + i] = q0 + r < n ? a.x[(q0 + r) * ni + d] : 0.f;
    }
  };
  auto scatter = [&](int tile, int buf) {  // two lanes per row, every second level
    const int r = (t >> 1) % kPlainRows;
    if (long(tile) * kPlainRows + r >= n) return;
    const float* x = xs + buf * 3 * kPlainRows + r;
    const float pos[3] = {x[0], x[kPlainRows], x[2 * kPlainRows]};
    for (int l = t / (2 * kPlainRows); l < p.enc.levels; l += kMovers / (2 * kPlainRows)) {
      float g[F];
#pragma unroll
      for (int f = 0; f < F; ++f) g[f] = G[((ONE_G ? 0 : buf * ng) + l * F + f) * kPlainRows + r];
      plain_scatter<F>(p, l, pos, g, t & 1u, a.gtable, a.wide != 0);
    }
  };
  auto deltas = [&](int tile, int buf) {
    float acc[8][4];
    float* d = D + buf * d_floats;
    const float* Wl = W;
    for (int l = L - 1; l >= 1; --l) {
      const size_t at0 = size_t(tile) * kPlainRows * kWidth;
      plain_product(d + tl.row, Wl + tl.col, kWidth, p.out[l], acc);
      bar_product();
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int at = (tl.col + c) * kPlainRows + tl.row;
        const float4 h = __ldg(reinterpret_cast<const float4*>(a.h_t[l - 1] + at0 + at));
        const float4 v = make_float4(h.x > 0.f ? acc[c][0] : 0.f, h.y > 0.f ? acc[c][1] : 0.f,
                                     h.z > 0.f ? acc[c][2] : 0.f, h.w > 0.f ? acc[c][3] : 0.f);
        *reinterpret_cast<float4*>(d + at) = v;
        *reinterpret_cast<float4*>(a.d_t[l - 1] + at0 + at) = v;
      }
      bar_product();
      Wl += p.out[l] * kWidth;
    }
    if (ONE_G) asm volatile("bar.sync 3, %0;" ::"n"(kPlainThreads) : "memory");  // the last tile's G has been read
    for (int c0 = tl.col; c0 < ng; c0 += kWidth) {
      plain_product(d + tl.row, Wl + c0, ng, kWidth, acc);
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<float4*>(G + ((ONE_G ? 0 : buf * ng) + c0 + c) * kPlainRows + tl.row) =
            make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
    }
  };

  int buf = 0, last = -1;
  if (mover && int(blockIdx.x) < tiles) read(blockIdx.x, 0);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
    __syncthreads();  // D[buf] and xs[buf], and the last tile's G, are in place
    if (!mover) {
      deltas(tile, buf);
    } else {
      if (last >= 0) scatter(last, buf ^ 1);
      if (ONE_G) asm volatile("bar.arrive 3, %0;" ::"n"(kPlainThreads) : "memory");
      bar_movers();  // xs[buf ^ 1] is rewritten only when every lane has read it
      if (tile + int(gridDim.x) < tiles) read(tile + gridDim.x, buf ^ 1);
    }
    last = tile;
  }
  __syncthreads();
  if (mover && last >= 0) scatter(last, buf ^ 1);
}

// dW[j][i] += sum over rows of delta[j][row] input[i][row] for one 64 x 64
// block of one layer's matrix (blockIdx.y), over this block's share of the
// tiles. Four groups of 64 threads take 16 rows of a tile each; a thread holds
// every 8th row and column of the 64 x 64 (8 x 8 sums, 16 shared loads per 256
// FMAs; a 16-byte load of four rows of a column is conflict-free at a pitch of
// 68 floats). The groups' sums meet in shared memory at the end.
struct PlainWgradBlock {
  const float *d_t, *x_t;  // tiles [nout][64], [nin][64]
  float* dw;
  int nout, nin, j0, i0;
};
constexpr int kMaxWgradBlocks = 4 * kMaxLayers;
struct PlainWgrad {
  PlainWgradBlock blk[kMaxWgradBlocks];
  const int* d_count;
  int n_max;
};
constexpr int kWgradPitch = kPlainRows + 4;

constexpr int kWgradThreads = 256, kWgradFloats = 2 * 64 * kWgradPitch;  // one stage: delta and input tile

// 16 bytes global -> shared, or 16 zero bytes.
NMG_D void copy16(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}

__global__ void __launch_bounds__(kWgradThreads, 2) k_plain_wgrad(const __grid_constant__ PlainWgrad a) {
  extern __shared__ __align__(16) float sh[];  // two stages
  const PlainWgradBlock& b = a.blk[blockIdx.y];
  int n = a.n_max;
  if (a.d_count) n = *a.d_count < 0 ? 0 : (*a.d_count > n ? n : *a.d_count);
  const int tiles = (n + kPlainRows - 1) / kPlainRows;
  if (int(blockIdx.x) >= tiles) return;
  const int nj = b.nout - b.j0 < 64 ? b.nout - b.j0 : 64, nx = b.nin - b.i0 < 64 ? b.nin - b.i0 : 64;
  const int grp = threadIdx.x / 64, t = threadIdx.x % 64;
  const int i = t & 7, j = t >> 3;
  float acc[8][8] = {};
  auto fetch = [&](int tile, int stage) {  // columns c / 16, rows 4 (c % 16) ..; columns beyond the matrix as zeros
    const float* d = b.d_t + (size_t(tile) * b.nout + b.j0) * kPlainRows;
    const float* x = b.x_t + (size_t(tile) * b.nin + b.i0) * kPlainRows;
    float* s = sh + stage * kWgradFloats;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = threadIdx.x + k * kWgradThreads, at = (c / 16) * kWgradPitch + 4 * (c % 16);
      copy16(s + at, c / 16 < nj ? d + 4 * c : d, c / 16 < nj);
      copy16(s + 64 * kWgradPitch + at, c / 16 < nx ? x + 4 * c : x, c / 16 < nx);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int stage = 0;
  fetch(blockIdx.x, 0);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, stage ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // this stage is in place, and the other one has been read
    if (tile + int(gridDim.x) < tiles) fetch(tile + gridDim.x, stage ^ 1);
    const float *Ds = sh + stage * kWgradFloats, *Xs = Ds + 64 * kWgradPitch;
#pragma unroll 1
    for (int r = 16 * grp; r < 16 * grp + 16; r += 4) {
      float4 d[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) d[k] = *reinterpret_cast<const float4*>(Ds + (j + 8 * k) * kWgradPitch + r);
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        if (8 * v >= nx) break;  // the block's columns beyond the matrix
        const float4 x = *reinterpret_cast<const float4*>(Xs + (i + 8 * v) * kWgradPitch + r);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          acc[u][v] = fmaf(d[u].x, x.x, acc[u][v]);
          acc[u][v] = fmaf(d[u].y, x.y, acc[u][v]);
          acc[u][v] = fmaf(d[u].z, x.z, acc[u][v]);
          acc[u][v] = fmaf(d[u].w, x.w, acc[u][v]);
        }
      }
    }
  }
  // groups 1-3 hand their sums to group 0 one after another
  for (int g = 3; g >= 1; --g) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        float& s = sh[(u * 8 + v) * 64 + t];
        if (grp == g) s = acc[u][v];
      }
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) acc[u][v] += sh[(u * 8 + v) * 64 + t];
    }
  }
  if (grp != 0) return;
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int jj = j + 8 * u, ii = i + 8 * v;
      if (jj < nj && ii < nx) atomicAdd(b.dw + size_t(b.j0 + jj) * b.nin + b.i0 + ii, acc[u][v]);
    }
}

// ------------------------------------------------------------ host launchers
static PlainNet plain_net(const nmg_ctx* c, const float* weights, const int* d_count, int n_max) {
  PlainNet p;
  memset(&p, 0, sizeof(p));
  p.enc = c->enc;
  p.n_layers = c->lay.n_layers;
  p.n_grid = c->enc.levels * c->enc.feats;
  for (int l = 0; l < p.n_layers; ++l) {
    p.in[l] = c->lay.in[l];
    p.out[l] = c->lay.out[l];
    p.w[l] = weights + c->lay.off[l];
  }
  p.table = weights + c->lay.n_mlp;
  for (int l = 0; l < c->enc.levels; ++l) {  // strides and hashing as grid.h:171-187
    const uint32_t T = c->enc.offset[l + 1] - c->enc.offset[l];
    uint32_t s[3] = {0, 0, 0}, stride = 1;
    for (int d = 0; d < 3; ++d)
      if (stride <= T) {
        s[d] = stride;
        stride *= c->enc.res[l];
      }
    p.T[l] = T;
    p.sy[l] = s[1];
    p.sz[l] = s[2];
    if (c->enc.grid_hash && T < stride) p.hashed |= 1u << l;
    if ((T & (T - 1u)) == 0u) p.pow2 |= 1u << l;
  }
  p.d_count = d_count;
  p.n_max = n_max;
  return p;
}

static int plain_grid(int n_max) {
  const long tiles = (long(n_max) + kPlainRows - 1) / kPlainRows, cap = 2L * sm_count();
  return int(tiles < 1 ? 1 : (tiles < cap ? tiles : cap));
}

template <int F, int DIR>
static nmg_status launch_forward(const PlainFwd& a, size_t smem, cudaStream_t st) {
  auto kern = k_plain_forward<F, DIR>;
  NMG_TRY(ensure_smem(reinterpret_cast<const void*>(kern), smem));
  kern<<<plain_grid(a.net.n_max), kPlainThreads, smem, st>>>(a);
  return check_launch("k_plain_forward");
}

// Encode + MLP forward of shading data (in non-NULL) or network input rows x.
// With keep_hidden the encoded rows and the activations stay in the workspace
// for the backward pass.
nmg_status plain_forward(nmg_ctx* c, const nmg_shading* in, const float* x, const int* d_count, int n_max,
                         const float* weights, bool keep_hidden, float* raw_out, cudaStream_t st) {
  Workspace& w = c->ws;
  PlainFwd a;
  memset(&a, 0, sizeof(a));
  a.net = plain_net(c, weights, d_count, n_max);
  if (in) a.in = *in;
  a.x = x;
  a.raw = raw_out;
  a.ld_raw = c->lay.n_out_pad;
  a.raw_wide = aligned16(raw_out);
  if (keep_hidden) {
    a.enc_t = w.enc;
    for (int l = 0; l < c->lay.n_layers - 1; ++l) a.h_t[l] = w.h[l];
  }
  const int ne = c->enc.n_enc_pad;
  size_t fl = 2 * size_t(ne > kWidth ? ne : kWidth) * kPlainRows + 10 * kPlainRows;
  for (int l = 0; l < c->lay.n_layers; ++l) fl += size_t(c->lay.in[l]) * (c->lay.out[l] + kPlainPad);
  const size_t smem = fl * sizeof(float);
  const EncodingParams& e = c->enc;
  const bool hash = e.input_mode == 1 && e.sh_degree == 4 && e.oneblob_bins == 4;
  const bool ref = e.input_mode == 0 && e.sh_degree == 2 && e.oneblob_bins == 4;
  switch (e.feats) {
    case 1: return launch_forward<1, 0>(a, smem, st);
    case 2: return hash ? launch_forward<2, 1>(a, smem, st) : launch_forward<2, 0>(a, smem, st);
    case 4: return ref ? launch_forward<4, 2>(a, smem, st) : launch_forward<4, 0>(a, smem, st);
    case 8: return launch_forward<8, 0>(a, smem, st);
  }
  return set_error(NMG_ERR_UNSUPPORTED, "grid_features=%d", e.feats);
}

// One grid-gradient buffer where two exceed what a block may have: 16 lobes with
// selection on seven hidden layers from 81 grid columns on, the widest of the
// others (259,584 bytes at most, the device allows 232,448; one buffer: 226,816).
template <int F, bool ONE_G = false>
static nmg_status launch_backward(const PlainBwd& a, size_t smem, size_t g_bytes, cudaStream_t st) {
  if (!ONE_G && smem > smem_optin()) return launch_backward<F, true>(a, smem - g_bytes, g_bytes, st);
  auto kern = k_plain_backward<F, ONE_G>;
  NMG_TRY(ensure_smem(reinterpret_cast<const void*>(kern), smem));
  kern<<<plain_grid(a.net.n_max), kPlainThreads, smem, st>>>(a);
  return check_launch("k_plain_backward");
}

// Backward through the MLP and the grid from dL/draw held in w.draw, after a
// forward pass that kept its activations; adds into dparams (layout of the
// parameters).
nmg_status plain_backward(nmg_ctx* c, const float* x, const int* d_count, int n_max, const float* weights,
                          float* dparams, cudaStream_t st) {
  const Layout& L = c->lay;
  Workspace& w = c->ws;
  PlainBwd a;
  memset(&a, 0, sizeof(a));
  a.net = plain_net(c, weights, d_count, n_max);
  a.x = x;
  a.draw = w.draw;
  for (int l = 0; l < L.n_layers; ++l) {
    a.h_t[l] = w.h[l];
    a.d_t[l] = w.delta[l];
  }
  a.gtable = dparams + L.n_mlp;
  a.wide = aligned16(a.gtable);
  const int ng = (a.net.n_grid + 15) / 16 * 16, dw = L.n_out_pad > kWidth ? L.n_out_pad : kWidth;
  size_t fl = 2 * size_t(dw + ng) * kPlainRows + 6 * kPlainRows + size_t(kWidth) * ng;
  for (int l = 1; l < L.n_layers; ++l) fl += size_t(L.in[l]) * L.out[l];
  const size_t smem = fl * sizeof(float), g_bytes = size_t(ng) * kPlainRows * sizeof(float);
  switch (c->enc.feats) {
    case 1: NMG_TRY(launch_backward<1>(a, smem, g_bytes, st)); break;
    case 2: NMG_TRY(launch_backward<2>(a, smem, g_bytes, st)); break;
    case 4: NMG_TRY(launch_backward<4>(a, smem, g_bytes, st)); break;
    case 8: NMG_TRY(launch_backward<8>(a, smem, g_bytes, st)); break;
    default: return set_error(NMG_ERR_UNSUPPORTED, "grid_features=%d", c->enc.feats);
  }
  PlainWgrad g;
  memset(&g, 0, sizeof(g));
  int nb = 0;
  for (int l = 0; l < L.n_layers; ++l)
    for (int j0 = 0; j0 < L.out[l]; j0 += 64)
      for (int i0 = 0; i0 < L.in[l]; i0 += 64)
        g.blk[nb++] = PlainWgradBlock{w.delta[l], l == 0 ? w.enc : w.h[l - 1], dparams + L.off[l],
                                      L.out[l], L.in[l], j0, i0};
  g.d_count = d_count;
  g.n_max = n_max;
  // two blocks per SM in all; each adds its 64 x 64 sums once
  const long tiles = (long(n_max) + kPlainRows - 1) / kPlainRows;
  long gx = 2L * sm_count() / nb;
  if (gx > tiles) gx = tiles;
  const size_t wsm = 2 * kWgradFloats * sizeof(float);
  NMG_TRY(ensure_smem(reinterpret_cast<const void*>(k_plain_wgrad), wsm));
  k_plain_wgrad<<<dim3(unsigned(gx < 1 ? 1 : gx), unsigned(nb)), kWgradThreads, wsm, st>>>(g);
  return check_launch("k_plain_wgrad");
}

}  // namespace nmg
