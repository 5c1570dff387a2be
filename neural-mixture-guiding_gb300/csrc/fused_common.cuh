// fused_common.cuh -- device helpers shared by the fused query and training
// kernels: the argument block, the row encoder that writes one input row
// into a 16-bit operand tile in core-matrix order, and warpgroup barriers.
#pragma once
#include "ctx.cuh"
#include "tcgen05.cuh"

namespace nmg {

constexpr int kRows = 128;      // rows per tile (MMA M)

struct FusedArgs {
  EncodingParams enc;
  MixOpts mix;
  const uint8_t* wimg;               // packed weight image
  uint32_t w_bytes;                  // image bytes (multiple of 16)
  uint32_t layer_off[kMaxLayers];    // byte offset of each layer in the image
  int n_layers;
  int fp16;                          // grid table and encoded features FP16 instead of BF16
  uint32_t fp16_layers;              // bit l: layer l's operands (its weights and input tile) are FP16
  uint32_t w0_lo_off;                // non-zero: byte offset of a second layer-0 image (the BF16 low
                                     // parts w - bf16(w)) whose products the first layer adds
  const uint16_t* table;             // 16-bit grid table [entries][F]
  uint32_t lvl_T[kMaxLevels];        // entries per level
  uint32_t lvl_hash;                 // bit l: level l is hashed (res^3 > T, T a power of two)
  uint32_t lvl_rec;                  // bit l: level l has cell records (CellRecords)
  uint32_t lvl_oct;                  // bit l: ... of all 8 corners (else of the 4 corners at one x)
  const uint4* cells;                // the records, in 16-byte units from cell_off[l]
  uint32_t cell_off[kMaxLevels];
  int half_levels;                   // levels of the first of two threads that share a row (even, > 0, < levels)
  int raw_mode;                      // 1: inputs are network input rows x, output raw only
  int n_out;                         // used outputs (4K [+1])
  int n_out_pad;
  int selection;
  const float* pos;
  const float* wo;
  const float* nrm;
  const float* rough;
  const float* u4;
  const float* wi;                   // non-NULL: evaluate the pdf at wi[n][3] instead of sampling
  const float* x;
  const int* d_count;
  int n_max;
  float* dir;
  float* pdf;
  int* lobe;
  float* raw;
  float* sel;
  int* err;
};

NMG_D bool layer_fp16(const FusedArgs& a, int l) { return ((a.fp16_layers >> l) & 1u) != 0; }

// Issues the MMAs of layer l (one thread): D[tmem] = A[a_addr] * W_l^T over
// the kin input columns, both operands K-major core-matrix tiles in shared
// memory (w_addr: the weight image). With a low-part image for layer 0 the
// same A also multiplies W0's low parts into the accumulator, which carries
// W0 = hi + lo to ~16 significant bits on BF16 operands.
NMG_D void issue_layer(const FusedArgs& a, int l, uint32_t tmem, uint32_t a_addr, uint32_t w_addr, int kin, int nout) {
  const uint32_t sbo = uint32_t(kin / 8) * 128u;
  const uint32_t idesc = tc::idesc_f16(kRows, nout, layer_fp16(a, l));
  const uint32_t b_addr = w_addr + a.layer_off[l];
  for (int kk = 0; kk < kin / 16; ++kk)
    tc::mma_f16(tmem, tc::smem_desc(a_addr + kk * 256u, 128u, sbo), tc::smem_desc(b_addr + kk * 256u, 128u, sbo),
                idesc, kk > 0 ? 1u : 0u);
  if (l == 0 && a.w0_lo_off) {
    const uint32_t lo_addr = w_addr + a.w0_lo_off;
    for (int kk = 0; kk < kin / 16; ++kk)
      tc::mma_f16(tmem, tc::smem_desc(a_addr + kk * 256u, 128u, sbo), tc::smem_desc(lo_addr + kk * 256u, 128u, sbo),
                  idesc, 1u);
  }
}

// D[tmem] (+)= sum over STEPS 16-deep slices of A and B whose descriptors
// advance by a_step / b_step bytes per slice. The descriptors are formed once
// and stepped by adding to their address field: one thread issues a tile's
// MMAs, and building two descriptors per MMA cost it more than the MMAs take.
template <int STEPS>
NMG_D void issue_steps(uint32_t tmem, uint64_t a, uint32_t a_step, uint64_t b, uint32_t b_step, uint32_t idesc,
                       bool accumulate) {
#pragma unroll
  for (int kk = 0; kk < STEPS; ++kk)
    tc::mma_f16(tmem, a + uint64_t(kk * (a_step >> 4)), b + uint64_t(kk * (b_step >> 4)), idesc,
                (accumulate || kk > 0) ? 1u : 0u);
}

// issue_layer on stepped descriptors, for KIN input columns.
template <int KIN>
NMG_D void issue_layer_steps(const FusedArgs& a, int l, uint32_t tmem, uint32_t a_addr, uint32_t w_addr, int nout) {
  constexpr uint32_t sbo = uint32_t(KIN / 8) * 128u;
  const uint32_t idesc = tc::idesc_f16(kRows, nout, layer_fp16(a, l));
  const uint64_t ad = tc::smem_desc(a_addr, 128u, sbo);
  issue_steps<KIN / 16>(tmem, ad, 256u, tc::smem_desc(w_addr + a.layer_off[l], 128u, sbo), 256u, idesc, false);
  if (l == 0 && a.w0_lo_off)
    issue_steps<KIN / 16>(tmem, ad, 256u, tc::smem_desc(w_addr + a.w0_lo_off, 128u, sbo), 256u, idesc, true);
}

NMG_D int fused_count(const int* d_count, int n_max) {
  if (!d_count) return n_max;
  int n = *d_count;
  return n < 0 ? 0 : (n > n_max ? n_max : n);
}

NMG_D bool bar_red_and(int id, int count, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred pin, pout;\n\t"
      "setp.ne.u32 pin, %1, 0;\n\t"
      "bar.red.and.pred pout, %2, %3, pin;\n\t"
      "selp.u32 %0, 1, 0, pout;\n\t}"
      : "=r"(r)
      : "r"(uint32_t(v)), "r"(id), "r"(count)
      : "memory");
  return r != 0;
}

NMG_D uint32_t level_index(const FusedArgs& a, int l, uint32_t x, uint32_t y, uint32_t z) {
  const uint32_t T = a.lvl_T[l];
  if ((a.lvl_hash >> l) & 1u) return (x ^ (y * 2654435761u) ^ (z * 805459861u)) & (T - 1u);
  const uint32_t res = a.enc.res[l];
  uint32_t idx = x + y * res + z * (res * res);
  return idx < T ? idx : (idx < 2u * T ? idx - T : idx % T);
}

template <int BINS>
NMG_D void oneblob_fixed(float x, float* o) {
  const float nb = float(BINS);
  float left = quartic_cdf(-x, nb) + quartic_cdf(-x - 1.f, nb) + quartic_cdf(-x + 1.f, nb);
#pragma unroll
  for (int k = 0; k < BINS; ++k) {
    const float rb = float(k + 1) / nb;
    float right = quartic_cdf(rb - x, nb) + quartic_cdf(rb - x - 1.f, nb) + quartic_cdf(rb - x + 1.f, nb);
    o[k] = right - left;
    left = right;
  }
}

// ReLU of 8 accumulator values packed straight into a 16-byte tile chunk.
NMG_D void store_chunk_relu(uint8_t* tile, int row, int chunk, int chunks, const float* f, bool fp16) {
  uint4 v;
  v.x = tc::pack2_relu(f[0], f[1], fp16);
  v.y = tc::pack2_relu(f[2], f[3], fp16);
  v.z = tc::pack2_relu(f[4], f[5], fp16);
  v.w = tc::pack2_relu(f[6], f[7], fp16);
  *reinterpret_cast<uint4*>(tile + tc::cm_offset(row, chunk, chunks)) = v;
}

NMG_D void store_chunk(uint8_t* tile, int row, int chunk, int chunks, const float* f, bool fp16) {
  uint4 v;
  v.x = tc::pack2(f[0], f[1], fp16);
  v.y = tc::pack2(f[2], f[3], fp16);
  v.z = tc::pack2(f[4], f[5], fp16);
  v.w = tc::pack2(f[6], f[7], fp16);
  *reinterpret_cast<uint4*>(tile + tc::cm_offset(row, chunk, chunks)) = v;
}

template <int F>
NMG_D void load_feats(const uint16_t* table, uint32_t entry, float* v, bool fp16) {
  if (F == 2) {
    uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(table) + entry);
    float2 p = tc::unpack2(w, fp16);
    v[0] = p.x;
    v[1] = p.y;
  } else {
    uint2 w = __ldg(reinterpret_cast<const uint2*>(table) + entry);
    float2 p = tc::unpack2(w.x, fp16), q = tc::unpack2(w.y, fp16);
    v[0] = p.x;
    v[1] = p.y;
    v[2] = q.x;
    v[3] = q.y;
  }
}

// The coarse dense levels' corners gathered into one record per entry, so
// that a cell takes one or two wide loads instead of eight corner loads: a
// query sends ~1 L2 request per cycle and SM at most, whatever its size up to
// a sector, and the eight corners of a dense cell lie in four to five
// sectors. The record of entry c holds the entries c + x + res y + res^2 z
// (wrapped like the corners they stand for) of
//   F = 2, small levels:  x, y, z in {0, 1}, x fastest: 32 bytes, one load;
//   F = 2, larger levels: y, z in {0, 1}, y fastest: 16 bytes, loaded at c and c + 1;
//   F = 4:                y, z in {0, 1}, y fastest: 32 bytes, loaded at c and c + 1.
// Levels get records from the coarsest on while they fit kCellBytes per copy
// of the table: for the hash-grid network levels 0-2 (32-byte) and 3 (16-byte)
// of its five dense levels, 3.7 MB for each of the training and the inference
// table, for the reference network six of eight (4.2 MB). The line lies where a
// context with the default table still holds less than 28 bytes a parameter and
// 8 MB. us without records / with these / with a limit of 10 MB, which takes in
// the hash grid's fifth dense level (5.5 MB more a copy; the reference network's
// seventh would be 7.3 MB): 2,073,600 queries 688 / 538 / 523, 900,000 at 16 lobes
// 348 / 320 / 315, the reference network's pdf of 550,001 134 / 110 / 110, training
// steps of 262,144 and 65,536 records 376 / 373 / 371 and 246 / 249 / 249.
constexpr size_t kCellBytes = 4608u << 10;
constexpr uint32_t kOctEntries = 1u << 16;  // F = 2 levels up to this size have 32-byte records

// 32 bytes of global memory in one load (p 32-byte aligned, constant during the kernel).
NMG_D void ld_v8(const uint4* p, uint4& a, uint4& b) {
  asm("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(p));
}

// One corner's F features (16-bit pairs) times wt into acc.
template <int F>
NMG_D void corner_fma(const uint32_t* w, float wt, float* acc, bool fp16) {
#pragma unroll
  for (int k = 0; k < F / 2; ++k) {
    const float2 v = tc::unpack2(w[k], fp16);
    acc[2 * k] = fmaf(wt, v.x, acc[2 * k]);
    acc[2 * k + 1] = fmaf(wt, v.y, acc[2 * k + 1]);
  }
}

// grid_level of a level with cell records: the same corners, weights and
// order of additions. A cell whose entry lies beyond the level (a position
// outside the box) reads its corners from the table one by one.
template <int F>
NMG_D void cell_features(const FusedArgs& a, int l, const uint32_t (&g)[3], const float (&w)[3], const float (&wxy)[4],
                         const float (&wz)[2], float* out) {
  const uint32_t T = a.lvl_T[l], res = a.enc.res[l], r2 = res * res;
  const uint32_t c0 = g[0] + g[1] * res + g[2] * r2;
  const bool fp16 = a.fp16 != 0;
  const uint4* rec = a.cells + a.cell_off[l];
  float acc[F];
#pragma unroll
  for (int k = 0; k < F; ++k) acc[k] = 0.f;
  if (c0 >= T) {
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      uint32_t idx = c0 + uint32_t(c & 1) + uint32_t((c >> 1) & 1) * res + uint32_t(c >> 2) * r2;
      if (idx >= T) idx %= T;
      const float wt = ((c & 1 ? w[0] : 1.f - w[0]) * (c & 2 ? w[1] : 1.f - w[1])) * (c & 4 ? w[2] : 1.f - w[2]);
      float v[F];
      load_feats<F>(a.table, a.enc.offset[l] + idx, v, fp16);
#pragma unroll
      for (int k = 0; k < F; ++k) acc[k] = fmaf(wt, v[k], acc[k]);
    }
  } else if (F == 2 && ((a.lvl_oct >> l) & 1u)) {
    uint4 lo, hi;
    ld_v8(rec + 2 * size_t(c0), lo, hi);
    const uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int c = 0; c < 8; ++c) corner_fma<2>(v + c, wxy[c & 3] * wz[c >> 2], acc, fp16);
  } else {
    const uint32_t c1 = c0 + 1u == T ? 0u : c0 + 1u;  // x + 1 wraps like any corner beyond the level
    uint32_t v[2][2 * F];  // [x][(y, z), y fastest][feature pair]
    if constexpr (F == 2) {
      const uint4 q0 = __ldg(rec + c0), q1 = __ldg(rec + c1);
      v[0][0] = q0.x, v[0][1] = q0.y, v[0][2] = q0.z, v[0][3] = q0.w;
      v[1][0] = q1.x, v[1][1] = q1.y, v[1][2] = q1.z, v[1][3] = q1.w;
    } else {
      uint4 q[4];
      ld_v8(rec + 2 * size_t(c0), q[0], q[1]);
      ld_v8(rec + 2 * size_t(c1), q[2], q[3]);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          v[x][4 * i] = q[2 * x + i].x, v[x][4 * i + 1] = q[2 * x + i].y;
          v[x][4 * i + 2] = q[2 * x + i].z, v[x][4 * i + 3] = q[2 * x + i].w;
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
      corner_fma<F>(&v[c & 1][(c >> 1) * (F / 2)], wxy[c & 3] * wz[c >> 2], acc, fp16);
  }
#pragma unroll
  for (int k = 0; k < F; ++k) out[k] = acc[k];
}

// Features of grid level l at position p3 (F values into out). The cell and
// weights follow grid.h:221-385; the corner indices are formed from per-axis
// terms (x, y*P1, z*P2 for hashed levels, x, y*res, z*res^2 for dense ones),
// which equal grid.h:171-187's index for every corner, and the corner weight is
// (w_x' * w_y') * w_z' as in the reference. PAIR (F = 2): the x and x+1
// corners of a (y, z) pair that share an aligned 8-byte word (every other
// cell: for dense levels e1 = e0 + 1, for hashed ones e1 = e0 ^ 1 when x is
// even) are read with one 8-byte load: a quarter fewer L1 requests, 4% of the
// query kernels' time and 1.5% of the training step's when it came in.
template <int F, bool SMOOTH, bool PAIR = false>
NMG_D void grid_level(const FusedArgs& a, int l, const float (&p3)[3], float* out) {
  float w[3];
  uint32_t g[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float pp = __fadd_rn(__fmul_rn(p3[d], a.enc.scale[l]), 0.5f);
    const float fl = floorf(pp);
    g[d] = uint32_t(int(fl));
    const float f = pp - fl;
    w[d] = SMOOTH ? f * f * (3.f - 2.f * f) : f;
  }
  const float wxy[4] = {(1.f - w[0]) * (1.f - w[1]), w[0] * (1.f - w[1]), (1.f - w[0]) * w[1], w[0] * w[1]};
  const float wz[2] = {1.f - w[2], w[2]};
  const uint32_t T = a.lvl_T[l];
  const uint32_t base = a.enc.offset[l];
  if ((a.lvl_rec >> l) & 1u) {
    cell_features<F>(a, l, g, w, wxy, wz, out);
    return;
  }
  uint32_t e[8];
  if ((a.lvl_hash >> l) & 1u) {
    const uint32_t mask = T - 1u;
    const uint32_t hy0 = g[1] * 2654435761u, hz0 = g[2] * 805459861u;
    const uint32_t hx[2] = {g[0], g[0] + 1u};
    const uint32_t hy[2] = {hy0, hy0 + 2654435761u};
    const uint32_t hz[2] = {hz0, hz0 + 805459861u};
#pragma unroll
    for (int c = 0; c < 8; ++c) e[c] = base + ((hx[c & 1] ^ hy[(c >> 1) & 1] ^ hz[c >> 2]) & mask);
  } else {
    const uint32_t res = a.enc.res[l], r2 = res * res;
    const uint32_t dy0 = g[1] * res, dz0 = g[2] * r2;
    const uint32_t dx[2] = {g[0], g[0] + 1u};
    const uint32_t dy[2] = {dy0, dy0 + res};
    const uint32_t dz[2] = {dz0, dz0 + r2};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t idx = dx[c & 1] + dy[(c >> 1) & 1] + dz[c >> 2];
      if (idx >= T) idx %= T;
      e[c] = base + idx;
    }
  }
  float acc[F];
#pragma unroll
  for (int k = 0; k < F; ++k) acc[k] = 0.f;
  if constexpr (PAIR && F == 2) {
    const bool fp16 = a.fp16 != 0;
    const uint32_t* tw = reinterpret_cast<const uint32_t*>(a.table);
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      uint32_t w0, w1;
      if ((e[c] ^ e[c + 1]) == 1u) {  // entries 2m and 2m+1
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(tw + (e[c] & ~1u)));
        const bool lo0 = e[c] < e[c + 1];
        w0 = lo0 ? w.x : w.y;
        w1 = lo0 ? w.y : w.x;
      } else {
        w0 = __ldg(tw + e[c]);
        w1 = __ldg(tw + e[c + 1]);
      }
      const float2 v0 = tc::unpack2(w0, fp16), v1 = tc::unpack2(w1, fp16);
      const float wt0 = wxy[c & 3] * wz[c >> 2], wt1 = wxy[(c + 1) & 3] * wz[c >> 2];
      acc[0] = fmaf(wt0, v0.x, acc[0]);  // same corner order as below
      acc[1] = fmaf(wt0, v0.y, acc[1]);
      acc[0] = fmaf(wt1, v1.x, acc[0]);
      acc[1] = fmaf(wt1, v1.y, acc[1]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float wt = wxy[c & 3] * wz[c >> 2];
      float v[F];
      load_feats<F>(a.table, e[c], v, a.fp16 != 0);
#pragma unroll
      for (int k = 0; k < F; ++k) acc[k] = fmaf(wt, v[k], acc[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < F; ++k) out[k] = acc[k];
}

// The two-feature levels as the kernels encode them: a level's eight corner
// words are loaded (level_load) while the level before it is blended
// (level_blend), so that a thread has two levels' gathers in flight. Same
// corners, weights and order of additions as grid_level.
struct LevelWords {
  uint32_t w[8];  // corner c = x + 2 y + 4 z
  float f[3];     // interpolation weights
  uint32_t swap;  // bit j: corners 2j and 2j + 1 are exchanged
};

// Entries e0 (corner x) and e1 (x + 1): one 8-byte load when they share an
// aligned pair (every second cell: for dense levels e1 = e0 + 1, for hashed
// ones e1 = e0 ^ 1 when x is even), else two 4-byte loads. Returns whether the
// pair came in exchanged. The loads are predicated, not branched around: the
// next pair's and the next level's are issued behind them.
NMG_D uint32_t load_pair(const uint32_t* tab, uint32_t e0, uint32_t e1, uint32_t& w0, uint32_t& w1) {
  const uint32_t single = (e0 ^ e1) ^ 1u;  // 0: one aligned pair
  asm("{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "@!p ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t"
      "@p ld.global.nc.u32 %0, [%2];\n\t"
      "@p ld.global.nc.u32 %1, [%3];\n\t}"
      : "=&r"(w0), "=&r"(w1)
      : "l"(tab + (single ? e0 : (e0 & ~1u))), "l"(tab + e1), "r"(single));
  return single == 0u ? (e0 & 1u) : 0u;
}

template <bool SMOOTH>
NMG_D void level_load(const FusedArgs& a, int l, const float (&p3)[3], LevelWords& v) {
  uint32_t g[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float pp = __fadd_rn(__fmul_rn(p3[d], a.enc.scale[l]), 0.5f);
    const float fl = floorf(pp);
    g[d] = uint32_t(int(fl));
    const float f = pp - fl;
    v.f[d] = SMOOTH ? f * f * (3.f - 2.f * f) : f;
  }
  const uint32_t T = a.lvl_T[l];
  const uint32_t* tab = reinterpret_cast<const uint32_t*>(a.table) + a.enc.offset[l];
  v.swap = 0u;
  if ((a.lvl_hash >> l) & 1u) {
    const uint32_t mask = T - 1u;
    const uint32_t hy = g[1] * 2654435761u, hz = g[2] * 805459861u;
    const uint32_t hy1 = hy + 2654435761u, hz1 = hz + 805459861u;
    const uint32_t h[4] = {hy ^ hz, hy1 ^ hz, hy ^ hz1, hy1 ^ hz1};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v.swap |= load_pair(tab, (g[0] ^ h[j]) & mask, ((g[0] + 1u) ^ h[j]) & mask, v.w[2 * j], v.w[2 * j + 1]) << j;
    return;
  }
  const uint32_t res = a.enc.res[l], r2 = res * res, c0 = g[0] + g[1] * res + g[2] * r2;
  if (((a.lvl_rec >> l) & 1u) && c0 < T) {
    const uint4* rec = a.cells + a.cell_off[l];
    uint4 p, q;
    if ((a.lvl_oct >> l) & 1u) {
      ld_v8(rec + 2 * size_t(c0), p, q);
      v.w[0] = p.x, v.w[1] = p.y, v.w[2] = p.z, v.w[3] = p.w, v.w[4] = q.x, v.w[5] = q.y, v.w[6] = q.z, v.w[7] = q.w;
    } else {
      p = __ldg(rec + c0);
      q = __ldg(rec + (c0 + 1u == T ? 0u : c0 + 1u));  // x + 1 wraps like any corner beyond the level
      v.w[0] = p.x, v.w[2] = p.y, v.w[4] = p.z, v.w[6] = p.w, v.w[1] = q.x, v.w[3] = q.y, v.w[5] = q.z, v.w[7] = q.w;
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t e0 = c0 + (j & 1 ? res : 0u) + (j & 2 ? r2 : 0u), e1 = e0 + 1u;
    if (e0 >= T) e0 %= T;
    if (e1 >= T) e1 %= T;
    v.swap |= load_pair(tab, e0, e1, v.w[2 * j], v.w[2 * j + 1]) << j;
  }
}

NMG_D float2 level_blend(const LevelWords& v, bool fp16) {
  const float wxy[4] = {(1.f - v.f[0]) * (1.f - v.f[1]), v.f[0] * (1.f - v.f[1]), (1.f - v.f[0]) * v.f[1],
                        v.f[0] * v.f[1]};
  const float wz[2] = {1.f - v.f[2], v.f[2]};
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool sw = (v.swap >> j) & 1u;
    const float2 v0 = tc::unpack2(sw ? v.w[2 * j + 1] : v.w[2 * j], fp16);
    const float2 v1 = tc::unpack2(sw ? v.w[2 * j] : v.w[2 * j + 1], fp16);
    const float wt0 = wxy[(2 * j) & 3] * wz[j >> 1], wt1 = wxy[(2 * j + 1) & 3] * wz[j >> 1];
    acc.x = fmaf(wt0, v0.x, acc.x);
    acc.y = fmaf(wt0, v0.y, acc.y);
    acc.x = fmaf(wt1, v1.x, acc.x);
    acc.y = fmaf(wt1, v1.y, acc.y);
  }
  return acc;
}

// Levels [l0, l1) of a row, both even, into its tile (KC chunks a row).
template <int KC, bool SMOOTH>
NMG_D void encode_levels2(const FusedArgs& a, int l0, int l1, const float (&p3)[3], uint8_t* tile, int row) {
  const bool fp16 = a.fp16 != 0, out16 = layer_fp16(a, 0);
  LevelWords u, v;
  level_load<SMOOTH>(a, l0, p3, u);
#pragma unroll 1
  for (int l = l0; l < l1; l += 2) {
    level_load<SMOOTH>(a, l + 1, p3, v);
    const float2 f0 = level_blend(u, fp16);
    if (l + 2 < l1) level_load<SMOOTH>(a, l + 2, p3, u);
    const float2 f1 = level_blend(v, fp16);
    *reinterpret_cast<uint2*>(tile + tc::cm_offset(row, l >> 2, KC) + (l & 2) * 4) =
        make_uint2(tc::pack2(f0.x, f0.y, out16), tc::pack2(f1.x, f1.y, out16));
  }
}

// The direction chunks of a row (spherical harmonics, one-blob, padding).
template <int F, int LEVELS, int MODE, int SHDEG, int BINS>
NMG_D void encode_direction(const float (&x)[10], uint8_t* tile, int row, bool fp16) {
  constexpr int NDIR = MODE == 0 ? SHDEG * SHDEG + 3 * BINS : 2 * SHDEG * SHDEG + BINS;
  constexpr int NGRID = LEVELS * F;
  constexpr int NPAD = (NGRID + NDIR + 15) / 16 * 16;
  float d[NPAD - NGRID];
  sh_basis(SHDEG, x[3] * 2.f - 1.f, x[4] * 2.f - 1.f, x[5] * 2.f - 1.f, d);
  if (MODE == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) oneblob_fixed<BINS>(x[6 + k], d + SHDEG * SHDEG + k * BINS);
  } else {
    sh_basis(SHDEG, x[6] * 2.f - 1.f, x[7] * 2.f - 1.f, x[8] * 2.f - 1.f, d + SHDEG * SHDEG);
    oneblob_fixed<BINS>(x[9], d + 2 * SHDEG * SHDEG);
  }
#pragma unroll
  for (int k = NDIR; k < NPAD - NGRID; ++k) d[k] = 1.f;
#pragma unroll
  for (int ch = 0; ch < (NPAD - NGRID) / 8; ++ch) store_chunk(tile, row, NGRID / 8 + ch, NPAD / 8, d + 8 * ch, fp16);
}

// Encodes one input row x into `tile` row `row` (KC 16-byte chunks).
// UNROLL = false keeps one copy of the chunk body (smaller code for kernels
// whose instruction footprint matters more than the loop overhead). With AHEAD
// and two features a level's loads run ahead of the last one's blend
// (encode_levels2), for kernels with the registers to hold both; the other
// forms gather one level at a time.
template <int F, int LEVELS, int MODE, int SHDEG, int BINS, bool SMOOTH, bool UNROLL = true, bool PAIR = false,
          bool AHEAD = PAIR>
NMG_D void encode_row(const FusedArgs& a, const float (&x)[10], uint8_t* tile, int row) {
  constexpr int NDIR = MODE == 0 ? SHDEG * SHDEG + 3 * BINS : 2 * SHDEG * SHDEG + BINS;
  constexpr int NGRID = LEVELS * F;
  constexpr int NPAD = (NGRID + NDIR + 15) / 16 * 16;
  constexpr int KC = NPAD / 8;
  constexpr int LPC = 8 / F;
  static_assert(NGRID % 8 == 0, "grid features must fill whole chunks");
  const bool fp16 = layer_fp16(a, 0);  // the tile's format is layer 0's operand format, not the table's
  const float p3[3] = {x[0], x[1], x[2]};
  if constexpr (F == 2 && AHEAD) {
    encode_levels2<KC, SMOOTH>(a, 0, LEVELS, p3, tile, row);
  } else {
#pragma unroll(UNROLL ? NGRID / 8 : 1)
    for (int ch = 0; ch < NGRID / 8; ++ch) {
      float f[8];
#pragma unroll
      for (int j = 0; j < LPC; ++j) grid_level<F, SMOOTH, PAIR>(a, ch * LPC + j, p3, f + j * F);
      store_chunk(tile, row, ch, KC, f, fp16);
    }
  }
  encode_direction<F, LEVELS, MODE, SHDEG, BINS>(x, tile, row, fp16);
}

// encode_row for one of `parts` threads that share a row: about as many levels
// each, and the direction chunks by part 0 (whose levels are the coarse ones).
// Together the calls write exactly what encode_row writes.
template <int F, int LEVELS, int MODE, int SHDEG, int BINS, bool SMOOTH, bool PAIR>
NMG_D void encode_row_part(const FusedArgs& a, const float (&x)[10], uint8_t* tile, int row, int part, int parts) {
  constexpr int NDIR = MODE == 0 ? SHDEG * SHDEG + 3 * BINS : 2 * SHDEG * SHDEG + BINS;
  constexpr int KC = (LEVELS * F + NDIR + 15) / 16 * 2;
  constexpr int LPC = 8 / F;
  const bool fp16 = layer_fp16(a, 0);
  const float p3[3] = {x[0], x[1], x[2]};
  if constexpr (F == 2 && PAIR) {
    encode_levels2<KC, SMOOTH>(a, LEVELS / 2 * part / parts * 2, LEVELS / 2 * (part + 1) / parts * 2, p3, tile, row);
  } else {
    constexpr int GCH = LEVELS * F / 8;
#pragma unroll 1
    for (int ch = GCH * part / parts; ch < GCH * (part + 1) / parts; ++ch) {
      float f[8];
#pragma unroll
      for (int j = 0; j < LPC; ++j) grid_level<F, SMOOTH, PAIR>(a, ch * LPC + j, p3, f + j * F);
      store_chunk(tile, row, ch, KC, f, fp16);
    }
  }
  if (part == 0) encode_direction<F, LEVELS, MODE, SHDEG, BINS>(x, tile, row, fp16);
}

// encode_row for one of the two threads that share a row: half h writes its
// levels (F = 2: the first a.half_levels ones or the rest, so that the halves
// gather about as many sectors; else the grid chunks ch with ch % 2 == h, each
// 8 / F consecutive levels) and its share of the direction
// chunks: for input mode 1 half 0 the SH(wo) chunks and half 1 the rest
// (SH(normal), one-blob(roughness), padding), each computing only what it
// stores; for mode 0, whose encodings share chunks, both compute the whole
// direction part and split its chunks. Together the two calls write exactly
// what encode_row writes.
template <int F, int LEVELS, int MODE, int SHDEG, int BINS, bool SMOOTH, bool PAIR = false>
NMG_D void encode_row_half(const FusedArgs& a, const float (&x)[10], uint8_t* tile, int row, int h) {
  constexpr int NDIR = MODE == 0 ? SHDEG * SHDEG + 3 * BINS : 2 * SHDEG * SHDEG + BINS;
  constexpr int NGRID = LEVELS * F;
  constexpr int NPAD = (NGRID + NDIR + 15) / 16 * 16;
  constexpr int KC = NPAD / 8;
  constexpr int LPC = 8 / F;
  constexpr int GCH = NGRID / 8, DCH = (NPAD - NGRID) / 8;
  constexpr bool SPLIT_SH = MODE == 1 && (SHDEG * SHDEG) % 8 == 0;
  constexpr int DCH0 = SPLIT_SH ? SHDEG * SHDEG / 8 : (DCH + 1) / 2;  // direction chunks of half 0
  static_assert(NGRID % 16 == 0, "grid chunks split evenly over the two halves");
  const bool fp16 = layer_fp16(a, 0);
  const float p3[3] = {x[0], x[1], x[2]};
  float d[NPAD - NGRID];
#pragma unroll
  for (int k = 0; k < NPAD - NGRID; ++k) d[k] = 1.f;
  if (MODE == 0) {
    sh_basis(SHDEG, x[3] * 2.f - 1.f, x[4] * 2.f - 1.f, x[5] * 2.f - 1.f, d);
#pragma unroll
    for (int k = 0; k < 3; ++k) oneblob_fixed<BINS>(x[6 + k], d + SHDEG * SHDEG + k * BINS);
  } else if (!SPLIT_SH || h == 0) {
    sh_basis(SHDEG, x[3] * 2.f - 1.f, x[4] * 2.f - 1.f, x[5] * 2.f - 1.f, d);
  }
  if (MODE == 1 && (!SPLIT_SH || h == 1)) {
    sh_basis(SHDEG, x[6] * 2.f - 1.f, x[7] * 2.f - 1.f, x[8] * 2.f - 1.f, d + SHDEG * SHDEG);
    oneblob_fixed<BINS>(x[9], d + 2 * SHDEG * SHDEG);
  }
#pragma unroll
  for (int ch = 0; ch < DCH; ++ch)
    if ((ch < DCH0) == (h == 0)) store_chunk(tile, row, GCH + ch, KC, d + 8 * ch, fp16);
  if constexpr (F == 2 && PAIR) {
    const bool out16 = fp16;
    const int l1 = h ? LEVELS : a.half_levels;
#pragma unroll 1
    for (int l = h ? a.half_levels : 0; l < l1; l += 2) {  // (level_load ahead of the blend would spill here)
      float f[4];
      grid_level<F, SMOOTH, PAIR>(a, l, p3, f);
      grid_level<F, SMOOTH, PAIR>(a, l + 1, p3, f + 2);
      *reinterpret_cast<uint2*>(tile + tc::cm_offset(row, l >> 2, KC) + (l & 2) * 4) =
          make_uint2(tc::pack2(f[0], f[1], out16), tc::pack2(f[2], f[3], out16));
    }
  } else {
#pragma unroll 1
    for (int ch = h; ch < GCH; ch += 2) {
      float f[8];
#pragma unroll
      for (int j = 0; j < LPC; ++j) grid_level<F, SMOOTH, PAIR>(a, ch * LPC + j, p3, f + j * F);
      store_chunk(tile, row, ch, KC, f, fp16);
    }
  }
}

// Loads network input row q (n_input <= 10 floats) with compile-time indices.
NMG_D void load_row(const float* x, long q, int n_input, float (&v)[10]) {
#pragma unroll
  for (int d = 0; d < 10; ++d) v[d] = d < n_input ? x[q * n_input + d] : 0.f;
}

NMG_D f3 face_fwd(f3 n, f3 v) { return dot3(n, v) > 0.f ? n : f3{-n.x, -n.y, -n.z}; }

// Output stage of one query from its raw network outputs r (registers):
// optional raw row, then (unless raw_mode) the mixture with the optional
// cosine lobe, and either the sampled direction with its pdf, lobe and
// selection probability, or (a.wi set) the pdf at the given direction.
// (The direction is stored per thread here, as the kernels with mixture
// warpgroups of their own do: gathering a warp's directions into whole-sector
// float4 stores, as query_epilogue_streamed does, kept three more values live
// across the pdf and made the consumers spill. To mapped host memory the scalar
// stores cost nothing that shows: nmg_query_host at 16 lobes, 500,000 queries,
// 193 us, the device call 185.)
template <int K, int NOUTMAX>
NMG_D void query_epilogue(const FusedArgs& a, long q, const float (&r)[NOUTMAX]) {
  if (a.raw) {
    float4* dst = reinterpret_cast<float4*>(a.raw + q * a.n_out_pad);
#pragma unroll
    for (int c = 0; c < NOUTMAX / 4; ++c)
      if (c * 4 < a.n_out_pad) dst[c] = make_float4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
  }
  if (a.raw_mode) return;
  Mix<K> m;
  mix_activate_regs<K, true>(m, r, a.mix.kappa_softplus);
  if (a.mix.cosine) mix_apply_cosine<K, true>(m, face_fwd(load3(a.nrm, q), load3(a.wo, q)));
  if (a.wi) {
    a.pdf[q] = mix_pdf<K, true>(m, load3(a.wi, q));
    return;
  }
  const float4 u = reinterpret_cast<const float4*>(a.u4)[q];
  const int sel = mix_select<K>(m, u.y);
  const f3 dv = mix_sample_lobe<K, true>(m, sel, u.z, u.w);
  store3(a.dir, q, dv);
  a.pdf[q] = mix_pdf<K, true>(m, dv);
  if (a.lobe) a.lobe[q] = sel;
  if (a.sel && a.selection) a.sel[q] = logistic<true>(r[4 * K < NOUTMAX ? 4 * K : 0]);
}

// query_epilogue for wide mixtures (K = 16) with the raw outputs left in
// TMEM: holding all K lobes (7 K floats) next to the 4 K raw outputs does not
// fit the registers of a 128-query warpgroup, so this variant keeps only the
// K lobe weights and derives each lobe again from its 4 raw outputs
// (tcgen05.ld of 16 columns = 4 lobes) when it is needed: once for the
// weights, once for the sampled lobe, once for the pdf. The lobe arithmetic
// is that of query_epilogue (same helpers, same order), so the results are
// the same. Warp-collective: every thread of the warpgroup calls it with its
// TMEM row address; rows past n (valid = false) compute and store nothing.
template <int K>
NMG_D void query_epilogue_streamed(const FusedArgs& a, long q, bool valid, uint32_t lane_addr) {
  static_assert(K % 4 == 0, "lobes come in groups of four (16 TMEM columns)");
  constexpr int G = K / 4;
  const bool cosine = a.mix.cosine != 0;
  f3 mb{0.f, 0.f, 1.f};
  if (cosine && valid) mb = unit3<true>(face_fwd(load3(a.nrm, q), load3(a.wo, q)));
  const float nb = prod_norm<true>(kCosineKappa);
  // lobe i of the 16-column group in v, as query_epilogue's activation (+ cosine product) makes it
  auto lobe = [&](const float (&v)[16], int j, float& lam, float& kap, f3& mu, float& nrm) {
    lobe_activate<true>(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], a.mix.kappa_softplus, lam, kap, mu);
    nrm = vmf_norm<true>(kap);
    if (cosine) lobe_cosine<true>(mb, nb, lam, kap, mu, nrm);
  };
  // pass 1: weights
  float lw[K];
  float total = 0.f;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float v[16];
    tc::tmem_load<1>(lane_addr + 16 * g, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lam, kap, nrm;
      f3 mu;
      lobe(v, j, lam, kap, mu, nrm);
      lw[4 * g + j] = lam;
      total += lam;
    }
  }
  if (cosine) total = fmaxf(total, NMG_EPS);  // distribution.h:191
  const float inv = 1.f / total;
#pragma unroll
  for (int i = 0; i < K; ++i) lw[i] *= inv;
  f3 d;
  int sel = 0;
  if (a.wi) {
    d = valid ? load3(a.wi, q) : f3{0.f, 0.f, 1.f};
  } else {
    // selection (distribution.h:132-140) and pass 2: the selected lobe, sampled
    const float4 u = valid ? reinterpret_cast<const float4*>(a.u4)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    float uu = u.y;
    sel = -1;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (sel < 0) {
        if (uu < lw[i])
          sel = i;
        else
          uu -= lw[i];
      }
    }
    sel = sel < 0 ? 0 : sel;
    // the selected lobe's four raw outputs, picked from each group as it is read (the reads are
    // warp-collective, the lobe is each thread's own), then that one lobe derived
    float rs[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) rs[k] = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float v[16];
      tc::tmem_load<1>(lane_addr + 16 * g, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool pick = 4 * g + j == sel;
#pragma unroll
        for (int k = 0; k < 4; ++k) rs[k] = pick ? v[4 * j + k] : rs[k];
      }
    }
    float lam, ks, nrm;
    f3 ms;
    lobe(rs, 0, lam, ks, ms, nrm);
    d = vmf_sample_dir<true>(ks, ms, u.z, u.w);
  }
  // pass 3: pdf at d (distribution.h:113-119)
  float p = 0.f;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float v[16];
    tc::tmem_load<1>(lane_addr + 16 * g, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lam, kap, nrm;
      f3 mu;
      lobe(v, j, lam, kap, mu, nrm);
      const float c = dot3(d, mu);
      const float vv = kap < NMG_EPS ? NMG_INV_4PI : __expf(kap * fminf(0.f, c - 1.f)) * nrm;
      p += lw[4 * g + j] * vv;
    }
  }
  float slogit = 0.f;
  if (a.sel && a.selection) {  // the selection logit follows the lobes (column 4K)
    float v[16];
    tc::tmem_load<1>(lane_addr + 4 * K, v);
    slogit = v[0];
  }
  if (a.wi) {
    if (valid) a.pdf[q] = p;
    return;
  }
  store3_warp(a.dir, q, d, valid);
  if (!valid) return;
  a.pdf[q] = p;
  if (a.lobe) a.lobe[q] = sel;
  if (a.sel && a.selection) a.sel[q] = logistic<true>(slogit);
}

// ------------------------------------------------------------ weight image
// Image 0 holds the training weights, image 1 the inference weights; each
// layer l of image i is converted to FP16 when bit l of fp16_layers[i] is
// set, else to BF16, and image i carries W0's BF16 low parts at w0_lo_off[i]
// when that is non-zero.
struct PackArgs {
  long off[kMaxLayers + 1];
  int in[kMaxLayers];
  uint32_t layer_off[kMaxLayers];
  int n_layers;
  uint32_t fp16_layers[2];
  uint32_t w0_lo_off[2];
};

// Cell records (see kCellBytes) of the levels in rec_mask, one after another:
// level i of the n_lvl packed ones has entries [first[i], first[i + 1]) of the
// running record count.
struct CellPackArgs {
  int n_lvl;
  uint32_t first[kMaxLevels + 1];
  uint32_t T[kMaxLevels], res[kMaxLevels], table_off[kMaxLevels], cell_off[kMaxLevels];
  uint32_t oct_mask;  // bit i: packed level i has 8-corner records
};

struct FusedState {
  uint8_t* img_train;
  uint8_t* img_infer;
  int* err;
  uint32_t w_bytes;      // training image
  uint32_t w_bytes_inf;  // inference image
  PackArgs pack;
  CellPackArgs cells;
  uint32_t lvl_rec, lvl_oct;  // FusedArgs' masks
  uint32_t cell_units;        // 16-byte units of one copy's records
  uint4* cell_mem[2];         // training, inference
  int preset;  // 0 none, 1 hash-grid K8, 2 hash-grid K16, 3 reference K8
};

inline FusedState* fstate(nmg_ctx* c) { return reinterpret_cast<FusedState*>(c->ws.fused); }

FusedArgs fused_make_args(nmg_ctx* c, bool infer_weights);

// Query tilings >= 8, and 7 at 16 lobes, select a warp-specialised kernel
// (fused_ws.cu): 12 (8-lobe networks) and 7 (16 lobes) = encoder, MLP and
// mixture warpgroups; 8 (8-lobe networks) = network and mixture warpgroups;
// 9 = 5 encoders + 1 consumer, 5 slots; 10 = 6 + 2, 6 slots; 11 = 4 + 2, 8
// slots; 8 at 16 lobes = 4 + 2, 4 slots.
constexpr int kTilingWarpSpecialised = 8;
constexpr int kTilingPair = 7;
nmg_status launch_query_ws(int preset, int tiling, const FusedArgs& a, cudaStream_t st);

}  // namespace nmg
