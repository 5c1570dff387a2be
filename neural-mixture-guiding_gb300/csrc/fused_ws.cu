// fused_ws.cu -- warp-specialised fused query kernel.
//
// The query pass spends most of its time on the hash-grid corner gathers: 128
// four-byte loads per query into the L2-resident table, which reach L1 as ~70
// separate 32-byte sector requests. An SM issues about one such request per
// cycle, and it only does so while enough of its threads are gathering. In
// the one-kernel-per-warpgroup design (fused.cu) every warpgroup alternates
// between gathering, the MLP chain and the mixture epilogue, so the request
// path idles whenever the groups happen to be in the other phases.
//
// Here the roles are split inside one persistent CTA per SM. Three kernels:
//   * k_fused_query_roles (the default of the hash-grid networks): encoders,
//     an MLP warpgroup, mixture warpgroups;
//   * k_fused_query_duo (the default of the reference network and of deep 8-lobe
//     ones, roles_mlp_bound): warpgroups that encode and run the MLP, mixture
//     warpgroups;
//   * k_fused_query_ws (tilings 9-11 and the 16-lobe tiling 8): E encoder
//     warpgroups, and C consumer warpgroups that run the MLP and the mixture.
// In the last, thread t of an encoder warpgroup writes row t of a 128-query
// tile into a shared-memory slot of a ring of S and arrives on the slot's
// "full" mbarrier (count 128); the consumers take the tiles in turn: one
// elected thread issues the tcgen05 MMAs of the 4 layers (weights resident in
// shared memory, accumulators in the group's TMEM columns), the group's
// threads apply the ReLU epilogues into their own hidden tile and finally run
// the mixture (activation, cosine lobe, selection, vMF sampling, pdf) on the
// output row held in registers. The layer-0 MMA's commit also arrives on the
// slot's "empty" mbarrier, which hands the slot back to the encoders as soon as
// the tensor core has read it. Tile j of a CTA lives in slot j % S, is encoded
// by warpgroup j % E and consumed by consumer j % C; the parities of round j / S
// drive the waits. The autotuner times the tiling ids against each other.
//
// Every wait is bounded; on a timeout the kernel records an error and all
// roles leave through their own (bounded) waits. Each configuration's
// register split adds up to its launch allocation, and the host launches a
// configuration only after checking that the kernel was compiled to exactly
// that many registers per thread.
#include <type_traits>

#include "api_common.cuh"
#include "ctx.cuh"
#include "fused_common.cuh"
#include "tcgen05.cuh"

namespace nmg {

// A warp-specialised configuration: E encoder and C consumer warpgroups, S
// ring slots, and the register split (launch / encoder / consumer registers
// per thread), which must add up to the launch allocation.
template <int E_, int C_, int S_, int RL_, int RE_, int RC_>
struct WsCfg {
  static constexpr int E = E_, C = C_, S = S_, RL = RL_, RE = RE_, RC = RC_;
  static constexpr int THREADS = (E + C) * kRows;
  static_assert(E * kRows * RE + C * kRows * RC == THREADS * RL, "register split must equal the launch allocation");
  static_assert(THREADS * RL <= 65536, "one CTA per SM");
  static_assert(S % E == 0, "each slot keeps one encoder warpgroup");
};
// Tiling ids of nmg_set_query_tiling.
using WsE4C2 = WsCfg<4, 2, 4, 80, 56, 128>;   // 8 (16 lobes)
using WsE5C1 = WsCfg<5, 1, 5, 80, 64, 160>;   // 9
using WsE6C2 = WsCfg<6, 2, 6, 64, 48, 112>;   // 10
using WsE4C2S8 = WsCfg<4, 2, 8, 80, 56, 128>; // 11

template <int F, int LEVELS, int MODE, int SHDEG, int BINS>
struct WsShape {
  static constexpr int NDIR = MODE == 0 ? SHDEG * SHDEG + 3 * BINS : 2 * SHDEG * SHDEG + BINS;
  static constexpr int NENC = (LEVELS * F + NDIR + 15) / 16 * 16;
  static constexpr uint32_t TILE_IN = uint32_t(kRows) * NENC * 2;
  static constexpr uint32_t TILE_H = uint32_t(kRows) * kWidth * 2;
  static constexpr uint32_t TILE_ANY = TILE_H > TILE_IN ? TILE_H : TILE_IN;  // a tile that holds either
};

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, class Cfg>
static size_t ws_smem_bytes(uint32_t w_bytes) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  return size_t((w_bytes + 1023u) & ~1023u) + Cfg::S * size_t(Sh::TILE_IN) +
         Cfg::C * size_t(Sh::TILE_H) + (2 * Cfg::S + 1 + Cfg::C) * 8 + 16;
}

// STREAM: the mixture epilogue re-reads the raw outputs from TMEM lobe group
// by lobe group (query_epilogue_streamed); 16-lobe queries without raw outputs.
template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg,
          bool STREAM = false>
__global__ void __launch_bounds__(Cfg::THREADS, 1) k_fused_query_ws(const __grid_constant__ FusedArgs a) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  constexpr int NENC = Sh::NENC;
  constexpr int S = Cfg::S;
  constexpr uint32_t SLOT = Sh::TILE_IN;
  constexpr int kWsEncoders = Cfg::E, kWsConsumers = Cfg::C;
  constexpr uint32_t COLS = NOUTMAX <= 64 ? 64 : 128;  // TMEM columns per consumer
  constexpr uint32_t TCOLS = COLS * kWsConsumers <= 64 ? 64 : (COLS * kWsConsumers <= 128 ? 128 : 256);
  static_assert(COLS * kWsConsumers <= 256, "TMEM columns");
  extern __shared__ __align__(1024) uint8_t smem[];

  const uint32_t w_region = (a.w_bytes + 1023u) & ~1023u;
  uint8_t* wsm = smem;
  uint8_t* slots = smem + w_region;
  uint8_t* hid = slots + S * SLOT;
  uint64_t* full = reinterpret_cast<uint64_t*>(hid + kWsConsumers * Sh::TILE_H);
  uint64_t* empty = full + S;
  uint64_t* wbar = empty + S;
  uint64_t* done = wbar + 1;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + kWsConsumers);
  const int wg = threadIdx.x / kRows, t = threadIdx.x % kRows;
  const int alloc_warp = kWsEncoders * 4;  // first warp of the first consumer

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(&full[s], kRows);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(wbar, 1);
    for (int c = 0; c < kWsConsumers; ++c) tc::mbar_init(&done[c], 1);
    tc::fence_mbar_init();
  }
  if (int(threadIdx.x / 32) == alloc_warp) tc::tmem_alloc(tslot, TCOLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x == 0) {
    tc::mbar_arrive_expect_tx(wbar, a.w_bytes);
    for (uint32_t off = 0; off < a.w_bytes; off += 16384u) {
      const uint32_t nb = a.w_bytes - off < 16384u ? a.w_bytes - off : 16384u;
      tc::bulk_g2s(wsm + off, a.wimg + off, nb, wbar);
    }
  }
  const int n = fused_count(a.d_count, a.n_max);
  const long ntiles = (long(n) + kRows - 1) / kRows;
  bool ok = true;

  if (wg < kWsEncoders) {
    // ------------------------------------------------------------- encoders
    __syncwarp();
    tc::reg_dealloc<Cfg::RE>();
    for (int j = wg;; j += kWsEncoders) {
      const long tile = blockIdx.x + long(j) * gridDim.x;
      if (tile >= ntiles) break;
      const int s = j % S;
      const uint32_t r = uint32_t(j / S);
      if (!tc::mbar_wait(&empty[s], (r & 1u) ^ 1u)) {
        ok = false;
        break;
      }
      const long q = tile * kRows + t;
      float x[10];
#pragma unroll
      for (int d = 0; d < 10; ++d) x[d] = 0.f;
      if (q < n) {
        if (a.raw_mode)
          load_row(a.x, q, a.enc.n_input, x);
        else
          featurize<true>(a.enc, load3(a.pos, q), load3(a.wo, q), load3(a.nrm, q), a.rough[q], x);
      }
      // no loads ahead beside 8 slots, which leave the gathers 25 KB of L1: 500,000 queries of the
      // hash-grid network 249 us instead of 284 us
      encode_row<F, LEVELS, MODE, SHDEG, BINS, SMOOTH, false, true, S <= 6>(a, x, slots + s * SLOT, t);
      tc::fence_proxy_async();
      tc::mbar_arrive(&full[s]);
    }
    if (!ok) atomicExch(a.err, 5);
  } else {
    // ------------------------------------------------------------ consumers
    __syncwarp();
    tc::reg_alloc<Cfg::RC>();
    const int c = wg - kWsEncoders;
    const int bar = 1 + c;  // named barrier of this consumer warpgroup
    ok = bar_red_and(bar, kRows, tc::mbar_wait(wbar, 0));
    const uint32_t tmem = *tslot + uint32_t(c) * COLS;
    const uint32_t lane_addr = tmem + (uint32_t((t / 32) * 32) << 16);
    uint8_t* H = hid + c * Sh::TILE_H;
    const uint32_t w_addr = tc::smem_u32(wsm);
    const int nl = a.n_layers;
    uint32_t phase = 0;
    // Issues layer l's MMAs (one elected thread): A = `a_addr` tile of kin columns.
    auto issue = [&](int l, uint32_t a_addr) {
      issue_layer(a, l, tmem, a_addr, w_addr, l == 0 ? NENC : kWidth, l == nl - 1 ? a.n_out_pad : kWidth);
    };
    // Every exit below follows a bar.red over the group (or depends only on
    // j), so the 128 threads always leave together. (Issuing the next tile's
    // layer 0 before this tile's mixture epilogue measured 10% slower, both
    // with the issuing thread waiting for the next slot and when it issues
    // only if that slot is already full.)
    for (int j = c;; j += kWsConsumers) {
      const long tile = blockIdx.x + long(j) * gridDim.x;
      if (tile >= ntiles) break;
      const int s = j % S;
      const uint32_t r = uint32_t(j / S);
      const uint32_t h_addr = tc::smem_u32(H);
      bool got = true;
      if (t == 0) {
        got = tc::mbar_wait(&full[s], r & 1u);
        if (got) {
          tc::fence_after_sync();
          issue(0, tc::smem_u32(slots + s * SLOT));
          tc::mma_commit(&empty[s]);  // the slot is free once layer 0 has read it
          tc::mma_commit(&done[c]);
        }
      }
      ok = bar_red_and(bar, kRows, got && ok);
      if (!ok) break;
      float rr[NOUTMAX];
      bool last_ok = true;
      for (int l = 0; l < nl; ++l) {
        const bool last = l == nl - 1;
        const bool d = tc::mbar_wait(&done[c], phase);
        phase ^= 1u;
        tc::fence_after_sync();
        if (!last) {
          float v[kWidth];
          tc::tmem_load<kWidth / 16>(lane_addr, v);
#pragma unroll
          for (int cc = 0; cc < kWidth / 8; ++cc) store_chunk_relu(H, t, cc, kWidth / 8, v + 8 * cc, layer_fp16(a, l + 1));
          tc::fence_proxy_async();
          tc::fence_before_sync();
          ok = bar_red_and(bar, kRows, d);
          if (!ok) break;
          if (t == 0) {
            tc::fence_after_sync();
            issue(l + 1, h_addr);
            tc::mma_commit(&done[c]);
          }
        } else {
          if constexpr (!STREAM) {
            tc::tmem_load_n<NOUTMAX / 16>(lane_addr, rr, (a.n_out_pad + 15) / 16);
            tc::fence_before_sync();
          }
          last_ok = d;
        }
      }
      if (!ok) break;
      const long q = tile * kRows + t;
      if constexpr (STREAM) {
        // warp-collective TMEM reads: the group agrees on ok first, and the accumulator must
        // outlive every thread's reads, so the group meets again before the next layer 0
        ok = bar_red_and(bar, kRows, last_ok);
        if (!ok) break;
        query_epilogue_streamed<K>(a, q, q < n, lane_addr);
        tc::fence_before_sync();
        ok = bar_red_and(bar, kRows, ok);
        if (!ok) break;
      } else {
        ok = last_ok;  // reconciled across the group at the next tile's barrier
        if (q < n && ok) query_epilogue<K, NOUTMAX>(a, q, rr);
      }
    }
    if (!ok && t == 0) atomicExch(a.err, 6);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (int(threadIdx.x / 32) == alloc_warp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(*tslot, TCOLS);
  }
}

// ---------------------------------------------------------------------------
// The defaults give the mixture warpgroups of its own: a consumer that runs the
// MLP and then the mixture (WsCfg) took 11.4 us a tile, a third of it waiting
// for MMAs with the registers of 8 lobes per thread held idle, and held the
// encoders up. At 16 lobes G warpgroups share a tile: every query has G threads
// with 4 lobes each. The warps w, w + 4, ... of a tile's warpgroups read the
// same TMEM lane quadrant, hold the same rows and exchange through shared
// memory, each exchange behind a named barrier of those G warps: the lobe
// weights (every thread forms the total and scans the lobes itself, in the
// order of one thread per query, so that the selected lobe is the same bit for
// bit), the sampled direction, which the thread that holds the selected lobe
// computes, and the pdf's partial sums.

// Exchange of one tile: the rows' lobe weights (later the pdf's partial sums),
// then the sampled directions.
template <int K, int G> constexpr uint32_t ws_xch_bytes() { return G > 1 ? uint32_t(kRows) * (K + 4) * 4 : 0u; }

// One query's mixture split over G threads with KH lobes each, in the steps
// between which the kernels do other work. Part h of row t.
template <int K, int G>
struct SharedMixture {
  static constexpr int KH = K / G;
  static_assert(KH % 4 == 0, "16-column TMEM loads hold 4 lobes");
  Mix<KH> m;
  float inv;  // 1 / sum of the lobe weights
  int sel;
  f3 d;
  float* xl;   // [G][kRows][KH] weights, later pdf sums in the first of each KH
  float4* xd;  // [kRows] direction
  int t, h, xbar;

  NMG_D SharedMixture(uint8_t* xch, int row, int part, int barrier)
      : inv(0.f), sel(0), d{0.f, 0.f, 1.f}, xl(reinterpret_cast<float*>(xch)),
        xd(reinterpret_cast<float4*>(xl + kRows * K)), t(row), h(part), xbar(barrier) {}

  NMG_D void exchange() {
    if constexpr (G > 1) tc::bar_sync(xbar, 32 * G);
  }
  // Lobes [I0, I0 + 4) of the thread's from their raw outputs, with the cosine
  // lobe around mb (distribution.h:85-98, 184-195).
  template <int I0>
  NMG_D void activate(const FusedArgs& a, const float (&r)[16], f3 mb) {
    const float nb = prod_norm<true>(kCosineKappa);
#pragma unroll
    for (int i = I0; i < I0 + 4; ++i) {
      lobe_activate<true>(r[4 * (i - I0)], r[4 * (i - I0) + 1], r[4 * (i - I0) + 2], r[4 * (i - I0) + 3],
                          a.mix.kappa_softplus, m.lam[i], m.kap[i], m.mu[i]);
      if constexpr (K == 16) {
        // below M_EPSILON the lobe is uniform: kappa 0, and the branch-free normaliser
        const float kz = m.kap[i] < NMG_EPS ? 0.f : m.kap[i];
        m.nrm[i] = vmf_norm_sel(kz);
        if (!a.mix.cosine) m.kap[i] = kz;
      } else {
        m.nrm[i] = vmf_norm_flat(m.kap[i]);
      }
      if (a.mix.cosine) lobe_cosine_flat<K == 16>(mb, nb, m.lam[i], m.kap[i], m.mu[i], m.nrm[i]);
    }
  }
  NMG_D void share_weights() {
    if constexpr (G > 1) {
      static_assert(KH == 4, "a part's weights are one float4");
      reinterpret_cast<float4*>(xl)[h * kRows + t] = make_float4(m.lam[0], m.lam[1], m.lam[2], m.lam[3]);
      exchange();
    }
  }
  // The total, and the direction: wi, or sampled with u by the thread that
  // holds the selected lobe.
  NMG_D void direct(const FusedArgs& a, long q, bool valid, float4 u) {
    Mix<K> all;  // only the weights of every lobe
    if constexpr (G > 1) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 v = reinterpret_cast<const float4*>(xl)[g * kRows + t];
        all.w[4 * g] = v.x, all.w[4 * g + 1] = v.y, all.w[4 * g + 2] = v.z, all.w[4 * g + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < K; ++i) all.w[i] = m.lam[i];
    }
    all.total = 0.f;
    if constexpr (K == 16) {  // the two halves' sums
      float hi = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        all.total += all.w[i];
        hi += all.w[8 + i];
      }
      all.total += hi;
    } else {
#pragma unroll
      for (int i = 0; i < K; ++i) all.total += all.w[i];
    }
    if (a.mix.cosine) all.total = fmaxf(all.total, NMG_EPS);  // distribution.h:191
    inv = 1.f / all.total;
    if (a.wi) {
      if (valid) d = load3(a.wi, q);
    } else {
#pragma unroll
      for (int i = 0; i < K; ++i) all.w[i] *= inv;
      sel = mix_select<K>(all, u.y);
      if (G == 1 || sel / KH == h) {
        d = mix_sample_lobe<KH, true>(m, sel - KH * h, u.z, u.w);
        if (G > 1) xd[t] = make_float4(d.x, d.y, d.z, 0.f);
      }
    }
    exchange();  // the direction is there; every thread has read the weights
    if (G > 1 && !a.wi) {
      const float4 v = xd[t];
      d = f3{v.x, v.y, v.z};
    }
  }
  // The pdf at d (distribution.h:113-119), and the outputs.
  NMG_D void finish(const FusedArgs& a, long q, bool valid) {
    float pd = 0.f;
#pragma unroll
    for (int i = 0; i < KH; ++i) {
      const float k = m.kap[i];
      const float c = dot3(d, m.mu[i]);
      const float v = k < NMG_EPS ? NMG_INV_4PI : __expf(k * fminf(0.f, c - 1.f)) * m.nrm[i];
      pd += (m.lam[i] * inv) * v;
    }
    if constexpr (G > 1) {
      xl[(h * kRows + t) * KH] = pd;  // in its own weights' place: other rows' may not have been read yet
      exchange();
    }
    if (!valid) return;
    if (h == 0) {
#pragma unroll
      for (int g = 1; g < G; ++g) pd += xl[(g * kRows + t) * KH];
      a.pdf[q] = pd;
      if (!a.wi && a.lobe) a.lobe[q] = sel;
    }
    if (h == G - 1 && !a.wi) store3(a.dir, q, d);
  }
};

// The last part of a row takes the columns past the lobes (taddr), the
// selection logit and the padding, to their outputs. `ok`: the accumulator is
// there.
template <int K>
NMG_D void take_extra(const FusedArgs& a, uint32_t taddr, long q, bool ok) {
  float extra[16];
  tc::tmem_load<1>(taddr, extra);
  if (!ok) return;
  if (a.sel && a.selection && !a.raw_mode) a.sel[q] = logistic<true>(extra[0]);
  if (a.raw) {
    float4* dst = reinterpret_cast<float4*>(a.raw + q * a.n_out_pad + 4 * K);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      dst[c] = make_float4(extra[4 * c], extra[4 * c + 1], extra[4 * c + 2], extra[4 * c + 3]);
  }
}
// Columns [16 c16, 16 c16 + 16) of the raw row.
NMG_D void store_raw16(const FusedArgs& a, long q, int c16, const float (&r)[16]) {
  float4* dst = reinterpret_cast<float4*>(a.raw + q * a.n_out_pad) + 4 * c16;
#pragma unroll
  for (int c = 0; c < 4; ++c) dst[c] = make_float4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
}

// ---------------------------------------------------------------------------
// Three roles (the hash-grid networks): encoder warpgroups fill the ring; an
// MLP warpgroup takes tiles from it, two in flight, and leaves their raw
// outputs in a ring of TMEM accumulators; X mixture warpgroups take those, G
// per tile. The encoders gather all the time, which is what bounds the kernel
// (two roles, below: 600 us for the 2,073,600-query wavefront against 535 us;
// one warpgroup for MLP and mixture: 624 us).
// At 8 lobes two mixture warpgroups with a tile each keep up (88 registers hold
// a thread's 8 lobes); at 16 lobes the mixture takes as long as the gathers,
// and four warpgroups share a tile (two threads per query: 464 us for 900,000
// queries, now 318 us).
// SHARE, for launches of up to kShareTiles tiles per SM: every tile is encoded
// by all the encoder warpgroups, a part of the levels each, so that the first
// one is ready in a third of the time and the tiles follow one another. With
// one thread per row for a whole tile (the encoders' throughput is higher, as
// a thread's gathers run on from level to level) and shared, 8 / 16 lobes, us:
// 4,999 queries 17.0 / 17.2 and 14.1 / 14.6; 38,912 (2 tiles per SM) 23.7 / 27.8
// and 21.3 / 23.4; 77,824 (4 tiles) 36.9 / 43.8 and 36.2 / 39.9; 120,000 52.3 / 64.4
// and 55.3 / 66.8. The line is drawn on the launch's capacity: with both forms in one
// kernel, chosen by the device count, the encoders spill (2,073,600 queries 548
// instead of 538 us, 900,000 at 16 lobes 330 instead of 319). So 16 lobes with a
// count of one to two tiles per SM below a larger capacity take 27.5 us, as one
// tile's mixture follows the other's (shared 25.0, the kernel before the roles 25.1);
// every other count is faster than with that kernel.
constexpr int kShareTiles = 4;
template <int E_, int X_, int G_, int RE_, int RM_, int RX_>
struct WsRoles {
  static constexpr int E = E_, X = X_, G = G_, RE = RE_, RM = RM_, RX = RX_;
  static constexpr int P = X / G;  // tiles in the mixture role at a time
  static constexpr int S = 4;      // ring slots
  static constexpr int R = 4;      // raw-output accumulators
  static constexpr int FL = 2;     // tiles in flight in the MLP role
  static constexpr int THREADS = (E + 1 + X) * kRows, RL = 65536 / THREADS / 8 * 8;
  static_assert(E * RE + RM + X * RX <= (E + 1 + X) * RL, "register split within the launch allocation");
  static_assert(RE <= RL && RM <= RL && RX >= RL, "the encoders' and the MLP's registers go to the mixture");
  static_assert(2 + P + (G > 1 ? 4 * P : 0) <= 16, "named barriers: the MLP's, one per tile and one per lane quadrant");
};
using WsE4X2G1 = WsRoles<4, 2, 1, 64, 64, 88>;  // 8 lobes
using WsE3X4G4 = WsRoles<3, 4, 4, 56, 56, 72>;  // 16 lobes

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, class Cfg>
static size_t ws_roles_smem_bytes(uint32_t w_bytes) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  return size_t((w_bytes + 1023u) & ~1023u) + Cfg::S * size_t(Sh::TILE_IN) + Cfg::FL * size_t(Sh::TILE_H) +
         Cfg::P * size_t(ws_xch_bytes<K, Cfg::G>()) + (2 * Cfg::S + 2 * Cfg::R + Cfg::FL + 1) * 8 + 16;
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg, bool SHARE>
__global__ void __launch_bounds__(Cfg::THREADS, 1) k_fused_query_roles(const __grid_constant__ FusedArgs a) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  constexpr int NENC = Sh::NENC, S = Cfg::S, R = Cfg::R, E = Cfg::E, FL = Cfg::FL;
  constexpr int G = Cfg::G, P = Cfg::P, KH = K / G;
  constexpr uint32_t RCOLS = (NOUTMAX + 15) / 16 * 16;  // columns of a raw-output accumulator
  constexpr uint32_t CRAW = FL * kWidth;  // after the MLP's accumulators
  static_assert(CRAW + R * RCOLS <= 512, "TMEM columns");
  constexpr uint32_t TCOLS = CRAW + R * RCOLS <= 256 ? 256 : 512;
  extern __shared__ __align__(1024) uint8_t smem[];

  const uint32_t w_region = (a.w_bytes + 1023u) & ~1023u;
  uint8_t* wsm = smem;
  uint8_t* slots = smem + w_region;
  uint8_t* hid = slots + S * Sh::TILE_IN;  // the MLP's hidden tiles
  uint8_t* xch = hid + FL * Sh::TILE_H;
  uint64_t* full = reinterpret_cast<uint64_t*>(xch + P * ws_xch_bytes<K, G>());
  uint64_t* empty = full + S;
  uint64_t* rfull = empty + S;
  uint64_t* rempty = rfull + R;
  uint64_t* done = rempty + R;
  uint64_t* wbar = done + FL;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(wbar + 1);
  const int wg = threadIdx.x / kRows, t = threadIdx.x % kRows;
  const int alloc_warp = E * 4;  // the first MLP warp

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(&full[s], (SHARE ? E : 1) * kRows);
      tc::mbar_init(&empty[s], 1);
    }
    for (int r = 0; r < R; ++r) {
      tc::mbar_init(&rfull[r], 1);
      tc::mbar_init(&rempty[r], 1);
    }
    for (int i = 0; i < FL; ++i) tc::mbar_init(&done[i], 1);
    tc::mbar_init(wbar, 1);
    tc::fence_mbar_init();
  }
  if (int(threadIdx.x / 32) == alloc_warp) tc::tmem_alloc(tslot, TCOLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x == 0) {
    tc::mbar_arrive_expect_tx(wbar, a.w_bytes);
    for (uint32_t off = 0; off < a.w_bytes; off += 16384u) {
      const uint32_t nb = a.w_bytes - off < 16384u ? a.w_bytes - off : 16384u;
      tc::bulk_g2s(wsm + off, a.wimg + off, nb, wbar);
    }
  }
  const int n = fused_count(a.d_count, a.n_max);
  const long ntiles = (long(n) + kRows - 1) / kRows;
  // this CTA's tiles: blockIdx.x + j gridDim.x for j < nj
  const int nj = long(blockIdx.x) < ntiles ? int((ntiles - 1 - long(blockIdx.x)) / long(gridDim.x)) + 1 : 0;
  bool ok = true;

  if (wg < E) {
    // ------------------------------------------------------------- encoders
    __syncwarp();
    tc::reg_dealloc<Cfg::RE>();
    for (int j = SHARE ? 0 : wg; j < nj; j += SHARE ? 1 : E) {
      const int s = j % S;
      if (!tc::mbar_wait(&empty[s], (uint32_t(j / S) & 1u) ^ 1u)) {
        ok = false;
        break;
      }
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      float x[10];
#pragma unroll
      for (int d = 0; d < 10; ++d) x[d] = 0.f;
      if (q < n) {
        if (a.raw_mode)
          load_row(a.x, q, a.enc.n_input, x);
        else
          featurize<true>(a.enc, load3(a.pos, q), load3(a.wo, q), load3(a.nrm, q), a.rough[q], x);
      }
      if (SHARE)
        encode_row_part<F, LEVELS, MODE, SHDEG, BINS, SMOOTH, true>(a, x, slots + s * Sh::TILE_IN, t, wg, E);
      else
        encode_row<F, LEVELS, MODE, SHDEG, BINS, SMOOTH, false, true>(a, x, slots + s * Sh::TILE_IN, t);
      tc::fence_proxy_async();
      tc::mbar_arrive(&full[s]);
    }
    if (!ok) atomicExch(a.err, 5);
  } else if (wg == E) {
    // ------------------------------------------------------------------ MLP
    __syncwarp();
    tc::reg_dealloc<Cfg::RM>();
    const uint32_t tmem = *tslot, w_addr = tc::smem_u32(wsm);
    const uint32_t lane_off = uint32_t((t / 32) * 32) << 16;
    const int nl = a.n_layers, bar = 1;
    // Two tiles in flight take turns: while one waits for its MMAs the other's
    // epilogue runs. Per tile in flight: the layer whose MMAs run (-1: free), the
    // tile, the done barrier's phase; the turn's own in layer, tile and phase,
    // the other's in layer2, tile2 and phase2 (one copy of the code, no indexed
    // arrays). Every decision is the same in all 128 threads: it depends on
    // these, on a bar.red, or on *go, which the issuing thread writes before a
    // barrier of the group.
    volatile int* go = reinterpret_cast<volatile int*>(tslot + 1);
    int layer = -1, tile = 0, layer2 = -1, tile2 = 0;
    uint32_t phase = 0, phase2 = 0;
    int next = 0, busy = 0, i = 0;
    // Thread 32 i issues for tile i, so that neither tile's issue holds up the
    // other's epilogue. bad: one of its waits before an issue gave up (the group
    // learns of it at its next barrier).
    bool bad = false;
    ok = bar_red_and(bar, kRows, tc::mbar_wait(wbar, 0));
    auto issue = [&](int l, uint32_t a_addr, uint32_t d) {
      const int nout = l == nl - 1 ? a.n_out_pad : kWidth;
      if (l == 0)
        issue_layer_steps<NENC>(a, l, d, a_addr, w_addr, nout);
      else
        issue_layer_steps<kWidth>(a, l, d, a_addr, w_addr, nout);
    };
    while (ok && (next < nj || busy > 0)) {
      if (layer < 0) {
        if (next < nj) {
          // a new tile: waited for when nothing else is in flight, else only if it
          // is there (waiting for it regardless: 584 instead of 557 us)
          if (t == 32 * i) {
            const int s = next % S;
            const uint32_t par = uint32_t(next / S) & 1u;
            const bool there = busy == 0 ? tc::mbar_wait(&full[s], par) : tc::mbar_test(&full[s], par);
            if (there) {
              tc::fence_after_sync();
              issue(0, tc::smem_u32(slots + s * Sh::TILE_IN), tmem + i * kWidth);
              tc::mma_commit(&empty[s]);
              tc::mma_commit(&done[i]);
            }
            *go = bad ? -1 : (there ? 1 : (busy == 0 ? -1 : 0));
          }
          tc::bar_sync(bar, kRows);
          const int g = *go;
          tc::bar_sync(bar, kRows);  // *go is rewritten only when every thread has read it
          if (g < 0) ok = false;
          if (g > 0) {
            layer = 0;
            tile = next;
            ++next;
            ++busy;
          }
        }
      } else {
        const bool d = tc::mbar_wait(&done[i], phase);
        phase ^= 1u;
        tc::fence_after_sync();
        uint8_t* H = hid + i * Sh::TILE_H;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float v[kWidth / 2];
          tc::tmem_load<kWidth / 32>(tmem + lane_off + uint32_t(i * kWidth + c * (kWidth / 2)), v);
#pragma unroll
          for (int k = 0; k < kWidth / 16; ++k)
            store_chunk_relu(H, t, c * (kWidth / 16) + k, kWidth / 8, v + 8 * k, layer_fp16(a, layer + 1));
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = bar_red_and(bar, kRows, d && !bad);
        const bool last = layer + 1 == nl - 1;
        if (ok && t == 32 * i) {
          const int r = tile % R;
          if (last && !bad) bad = !tc::mbar_wait(&rempty[r], (uint32_t(tile / R) & 1u) ^ 1u);
          if (bad) {
            atomicExch(a.err, 6);
          } else {
            tc::fence_after_sync();
            issue(layer + 1, tc::smem_u32(H), last ? tmem + CRAW + r * RCOLS : tmem + i * kWidth);
            tc::mma_commit(last ? &rfull[r] : &done[i]);
          }
        }
        layer = last ? -1 : layer + 1;
        if (last) --busy;
      }
      const int lt = layer, tt = tile;
      const uint32_t pt = phase;
      layer = layer2, tile = tile2, phase = phase2;
      layer2 = lt, tile2 = tt, phase2 = pt;
      i ^= 1;
    }
    if (!ok && t == 0) atomicExch(a.err, 6);
    __syncwarp();
  } else {
    // -------------------------------------------------------------- mixture
    __syncwarp();
    tc::reg_alloc<Cfg::RX>();
    const int p = (wg - E - 1) / G, h = (wg - E - 1) % G;  // tile in flight, part of the row
    const int bar = 2 + p, xbar = 2 + P + 4 * p + t / 32;
    const bool leader = h == 0 && t == 0;
    const uint32_t lane_addr = *tslot + CRAW + (uint32_t((t / 32) * 32) << 16);
    // a tile's inputs are loaded before the last one's pdf
    f3 n3, wo3;
    float4 u;
    auto load_in = [&](int j) {
      n3 = wo3 = f3{0.f, 0.f, 1.f};
      u = make_float4(0.f, 0.f, 0.f, 0.f);
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      if (j >= nj || q >= n || a.raw_mode) return;
      if (a.mix.cosine) {
        n3 = load3(a.nrm, q);
        wo3 = load3(a.wo, q);
      }
      if (!a.wi) u = reinterpret_cast<const float4*>(a.u4)[q];
    };
    load_in(p);
    for (int j = p; j < nj; j += P) {
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      const bool valid = q < n;
      const int r = j % R;
      const bool d = tc::mbar_wait(&rfull[r], uint32_t(j / R) & 1u);
      tc::fence_after_sync();
      SharedMixture<K, G> sm(xch + p * ws_xch_bytes<K, G>(), t, h, xbar);
      const f3 mb = a.mix.cosine ? unit3<true>(face_fwd(n3, wo3)) : n3;
      const uint32_t raw_addr = lane_addr + uint32_t(r * RCOLS);
      // four lobes at a time, so that no more raw outputs are live
      auto take = [&](auto first) {
        constexpr int I0 = decltype(first)::value;
        float r16[16];
        tc::tmem_load<1>(raw_addr + uint32_t(4 * (KH * h + I0)), r16);
        if (a.raw && valid && d) store_raw16(a, q, (KH * h + I0) / 4, r16);
        if (!a.raw_mode) sm.template activate<I0>(a, r16, mb);
      };
      take(std::integral_constant<int, 0>());
      if constexpr (KH == 8) take(std::integral_constant<int, 4>());
      if (h == G - 1 && a.n_out_pad > 4 * K) take_extra<K>(a, raw_addr + uint32_t(4 * K), q, valid && d);
      tc::fence_before_sync();
      // every exit follows this barrier (or depends only on j), so a tile's warpgroups leave together
      ok = bar_red_and(bar, G * kRows, d);
      if (!ok) break;
      if (leader) tc::mbar_arrive(&rempty[r]);
      if (a.raw_mode) continue;
      sm.share_weights();
      sm.direct(a, q, valid, u);
      load_in(j + P);
      sm.finish(a, q, valid);
    }
    if (!ok && t == 0) atomicExch(a.err, 6);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (int(threadIdx.x / 32) == alloc_warp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(*tslot, TCOLS);
  }
}

// ---------------------------------------------------------------------------
// Two roles (the reference network): N network warpgroups, each of which
// encodes a tile and runs its MLP (the hidden activations overwrite the input
// tile), and X mixture warpgroups, which take the raw outputs from the network
// warpgroup's TMEM accumulator. A network warpgroup goes on to encode its next
// tile while the last layer runs and the mixture works. With 8 levels to gather
// instead of 16, an MLP warpgroup of its own would be busy all the time and
// bound the kernel (three roles: 122 us for the pdf of 550,001 queries; two:
// 110 us; one warpgroup for MLP and mixture: 150 us).
template <int N_, int X_, int G_, int RN_, int RX_>
struct WsDuo {
  static constexpr int N = N_, X = X_, G = G_, RN = RN_, RX = RX_;
  static constexpr int P = X / G;  // tiles in the mixture role at a time
  static constexpr int THREADS = (N + X) * kRows, RL = 65536 / THREADS / 8 * 8;
  static_assert(N * RN + X * RX <= (N + X) * RL, "register split within the launch allocation");
  static_assert(RN <= RL && RX >= RL, "the network warpgroups' registers go to the mixture");
  static_assert(1 + N + P + (G > 1 ? 4 * P : 0) <= 16, "named barriers: one per tile and one per lane quadrant");
};

using WsN4X2G1 = WsDuo<4, 2, 1, 64, 112>;

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, class Cfg>
static size_t ws_duo_smem_bytes(uint32_t w_bytes) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  return size_t((w_bytes + 1023u) & ~1023u) + Cfg::N * size_t(Sh::TILE_ANY) +
         Cfg::P * size_t(ws_xch_bytes<K, Cfg::G>()) + (3 * Cfg::N + 1) * 8 + 16;
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1) k_fused_query_duo(const __grid_constant__ FusedArgs a) {
  using Sh = WsShape<F, LEVELS, MODE, SHDEG, BINS>;
  constexpr int NENC = Sh::NENC, N = Cfg::N, G = Cfg::G, P = Cfg::P, KH = K / G;
  constexpr uint32_t SLOT = Sh::TILE_ANY;
  constexpr uint32_t COLS = NOUTMAX <= kWidth ? kWidth : (NOUTMAX + 15) / 16 * 16;  // a warpgroup's accumulator
  static_assert(COLS * N <= 512, "TMEM columns");
  constexpr uint32_t TCOLS = COLS * N <= 256 ? 256 : 512;
  extern __shared__ __align__(1024) uint8_t smem[];

  const uint32_t w_region = (a.w_bytes + 1023u) & ~1023u;
  uint8_t* wsm = smem;
  uint8_t* slots = smem + w_region;
  uint8_t* xch = slots + N * SLOT;
  uint64_t* done = reinterpret_cast<uint64_t*>(xch + P * ws_xch_bytes<K, G>());  // a layer's MMAs
  uint64_t* rfull = done + N;    // the raw outputs are in the accumulator
  uint64_t* rempty = rfull + N;  // ... and have been read
  uint64_t* wbar = rempty + N;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(wbar + 1);
  const int wg = threadIdx.x / kRows, t = threadIdx.x % kRows;

  // A CTA without tiles (a device count below n_max) leaves before it starts
  // anything: the weights are waited for before a warpgroup's first tile, so
  // nobody would wait for its copy, and a CTA must not exit with a copy into its
  // shared memory in flight.
  if (long(blockIdx.x) * kRows >= fused_count(a.d_count, a.n_max)) return;
  if (threadIdx.x == 0) {
    for (int i = 0; i < N; ++i) {
      tc::mbar_init(&done[i], 1);
      tc::mbar_init(&rfull[i], 1);
      tc::mbar_init(&rempty[i], 1);
    }
    tc::mbar_init(wbar, 1);
    tc::fence_mbar_init();
  }
  if (threadIdx.x < 32) tc::tmem_alloc(tslot, TCOLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x == 0) {
    tc::mbar_arrive_expect_tx(wbar, a.w_bytes);
    for (uint32_t off = 0; off < a.w_bytes; off += 16384u) {
      const uint32_t nb = a.w_bytes - off < 16384u ? a.w_bytes - off : 16384u;
      tc::bulk_g2s(wsm + off, a.wimg + off, nb, wbar);
    }
  }
  const int n = fused_count(a.d_count, a.n_max);
  const long ntiles = (long(n) + kRows - 1) / kRows;
  // this CTA's tiles: blockIdx.x + j gridDim.x for j < nj; tile j is warpgroup j % N's
  const int nj = long(blockIdx.x) < ntiles ? int((ntiles - 1 - long(blockIdx.x)) / long(gridDim.x)) + 1 : 0;
  bool ok = true;

  if (wg < N) {
    // -------------------------------------------------------------- network
    __syncwarp();
    tc::reg_dealloc<Cfg::RN>();
    const int bar = 1 + wg, nl = a.n_layers;
    const uint32_t tmem = *tslot + uint32_t(wg) * COLS, lane_addr = tmem + (uint32_t((t / 32) * 32) << 16);
    uint8_t* A = slots + wg * SLOT;
    const uint32_t a_addr = tc::smem_u32(A), w_addr = tc::smem_u32(wsm);
    uint32_t phase = 0, round = 0;
    auto issue = [&](int l) {
      tc::fence_after_sync();
      const int nout = l == nl - 1 ? a.n_out_pad : kWidth;
      if (l == 0)
        issue_layer_steps<NENC>(a, l, tmem, a_addr, w_addr, nout);
      else
        issue_layer_steps<kWidth>(a, l, tmem, a_addr, w_addr, nout);
      if (l == nl - 1) tc::mma_commit(&rfull[wg]);
      tc::mma_commit(&done[wg]);
    };
    // Every exit follows a bar.red over the warpgroup (or depends only on j), so
    // its threads leave together.
    for (int j = wg; j < nj; j += N, ++round) {
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      float x[10];
#pragma unroll
      for (int d = 0; d < 10; ++d) x[d] = 0.f;
      if (q < n) {
        if (a.raw_mode)
          load_row(a.x, q, a.enc.n_input, x);
        else
          featurize<true>(a.enc, load3(a.pos, q), load3(a.wo, q), load3(a.nrm, q), a.rough[q], x);
      }
      bool d = true;
      if (round > 0) {  // the last tile's last layer has read the slot
        d = tc::mbar_wait(&done[wg], phase);
        phase ^= 1u;
      }
      encode_row<F, LEVELS, MODE, SHDEG, BINS, SMOOTH, false, true>(a, x, A, t);
      if (round == 0) d = tc::mbar_wait(wbar, 0);
      tc::fence_proxy_async();
      ok = bar_red_and(bar, kRows, d);
      if (!ok) break;
      bool free_acc = true;
      if (t == 0) {  // the mixture has read the accumulator
        free_acc = tc::mbar_wait(&rempty[wg], (round & 1u) ^ 1u);
        if (free_acc) issue(0);
      }
      for (int l = 0; l < nl - 1; ++l) {
        d = tc::mbar_wait(&done[wg], phase);
        phase ^= 1u;
        tc::fence_after_sync();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float v[kWidth / 2];
          tc::tmem_load<kWidth / 32>(lane_addr + uint32_t(c * (kWidth / 2)), v);
#pragma unroll
          for (int k = 0; k < kWidth / 16; ++k)
            store_chunk_relu(A, t, c * (kWidth / 16) + k, kWidth / 8, v + 8 * k, layer_fp16(a, l + 1));
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = bar_red_and(bar, kRows, d && free_acc);
        if (!ok) break;
        if (t == 0) issue(l + 1);
      }
      if (!ok) break;
    }
    // the last tile's last layer, before the block's TMEM and shared memory go
    if (ok && round > 0) ok = bar_red_and(bar, kRows, tc::mbar_wait(&done[wg], phase));
    if (!ok && t == 0) atomicExch(a.err, 5);
  } else {
    // -------------------------------------------------------------- mixture
    __syncwarp();
    tc::reg_alloc<Cfg::RX>();
    const int p = (wg - N) / G, h = (wg - N) % G;  // tile in flight, part of the row
    const int bar = 1 + N + p, xbar = 1 + N + P + 4 * p + t / 32;
    const bool leader = h == 0 && t == 0;
    const uint32_t lane_addr = *tslot + (uint32_t((t / 32) * 32) << 16);
    // a tile's inputs are loaded before the last one's pdf
    f3 n3, wo3;
    float4 u;
    auto load_in = [&](int j) {
      n3 = wo3 = f3{0.f, 0.f, 1.f};
      u = make_float4(0.f, 0.f, 0.f, 0.f);
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      if (j >= nj || q >= n || a.raw_mode) return;
      if (a.mix.cosine) {
        n3 = load3(a.nrm, q);
        wo3 = load3(a.wo, q);
      }
      if (!a.wi) u = reinterpret_cast<const float4*>(a.u4)[q];
    };
    load_in(p);
    for (int j = p; j < nj; j += P) {
      const long q = (blockIdx.x + long(j) * gridDim.x) * kRows + t;
      const bool valid = q < n;
      const int r = j % N;
      const bool d = tc::mbar_wait(&rfull[r], uint32_t(j / N) & 1u);
      tc::fence_after_sync();
      SharedMixture<K, G> sm(xch + p * ws_xch_bytes<K, G>(), t, h, xbar);
      const f3 mb = a.mix.cosine ? unit3<true>(face_fwd(n3, wo3)) : n3;
      const uint32_t raw_addr = lane_addr + uint32_t(r) * COLS;
      // four lobes at a time, so that no more raw outputs are live
      auto take = [&](auto first) {
        constexpr int I0 = decltype(first)::value;
        float r16[16];
        tc::tmem_load<1>(raw_addr + uint32_t(4 * (KH * h + I0)), r16);
        if (a.raw && valid && d) store_raw16(a, q, (KH * h + I0) / 4, r16);
        if (!a.raw_mode) sm.template activate<I0>(a, r16, mb);
      };
      take(std::integral_constant<int, 0>());
      if constexpr (KH == 8) take(std::integral_constant<int, 4>());
      if (h == G - 1 && a.n_out_pad > 4 * K) take_extra<K>(a, raw_addr + uint32_t(4 * K), q, valid && d);
      tc::fence_before_sync();
      // every exit follows this barrier (or depends only on j), so a tile's warpgroups leave together
      ok = bar_red_and(bar, G * kRows, d);
      if (!ok) break;
      if (leader) tc::mbar_arrive(&rempty[r]);
      if (a.raw_mode) continue;
      sm.share_weights();
      sm.direct(a, q, valid, u);
      load_in(j + P);
      sm.finish(a, q, valid);
    }
    if (!ok && t == 0) atomicExch(a.err, 6);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc::fence_after_sync();
    tc::tmem_dealloc(*tslot, TCOLS);
  }
}

// Launch-time check of the register split: the kernel must have been
// compiled to exactly the launch registers per thread the split assumes.
template <class Kern>
static nmg_status ws_check_regs(Kern kern, int want) {
  cudaFuncAttributes attr;
  if (cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(kern)) != cudaSuccess) return NMG_ERR_CUDA;
  return attr.numRegs == want ? NMG_OK : NMG_ERR_UNSUPPORTED;
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg,
          bool STREAM = false>
static nmg_status launch_ws(const FusedArgs& a, cudaStream_t st) {
  auto kern = k_fused_query_ws<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, Cfg, STREAM>;
  static int regs_ok = 0;  // 1: checked and usable, -1: unusable
  if (regs_ok == 0) regs_ok = ws_check_regs(kern, Cfg::RL) == NMG_OK ? 1 : -1;
  if (regs_ok < 0)
    return set_error(NMG_ERR_UNSUPPORTED, "warp-specialised query kernel not compiled to %d registers", Cfg::RL);
  const size_t smem = ws_smem_bytes<F, LEVELS, MODE, SHDEG, BINS, Cfg>(a.w_bytes);
  nmg_status s = ensure_smem(reinterpret_cast<const void*>(kern), smem);
  if (s != NMG_OK) return s;
  const long tiles = (long(a.n_max) + kRows - 1) / kRows;
  int grid = sm_count();
  if (tiles < grid) grid = int(tiles > 0 ? tiles : 1);
  kern<<<grid, Cfg::THREADS, smem, st>>>(a);
  return check_launch("k_fused_query_ws");
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg>
static nmg_status launch_duo(const FusedArgs& a, cudaStream_t st) {
  auto kern = k_fused_query_duo<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, Cfg>;
  static int regs_ok = 0;  // 1: checked and usable, -1: unusable
  if (regs_ok == 0) regs_ok = ws_check_regs(kern, Cfg::RL) == NMG_OK ? 1 : -1;
  if (regs_ok < 0)
    return set_error(NMG_ERR_UNSUPPORTED, "warp-specialised query kernel not compiled to %d registers", Cfg::RL);
  const size_t smem = ws_duo_smem_bytes<F, LEVELS, MODE, SHDEG, BINS, K, Cfg>(a.w_bytes);
  nmg_status s = ensure_smem(reinterpret_cast<const void*>(kern), smem);
  if (s != NMG_OK) return s;
  const long tiles = (long(a.n_max) + kRows - 1) / kRows;
  int grid = sm_count();
  if (tiles < grid) grid = int(tiles > 0 ? tiles : 1);
  kern<<<grid, Cfg::THREADS, smem, st>>>(a);
  return check_launch("k_fused_query_duo");
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg, bool SHARE>
static nmg_status launch_roles_kernel(const FusedArgs& a, int grid, cudaStream_t st) {
  auto kern = k_fused_query_roles<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, Cfg, SHARE>;
  static int regs_ok = 0;  // 1: checked and usable, -1: unusable
  if (regs_ok == 0) regs_ok = ws_check_regs(kern, Cfg::RL) == NMG_OK ? 1 : -1;
  if (regs_ok < 0)
    return set_error(NMG_ERR_UNSUPPORTED, "warp-specialised query kernel not compiled to %d registers", Cfg::RL);
  const size_t smem = ws_roles_smem_bytes<F, LEVELS, MODE, SHDEG, BINS, K, Cfg>(a.w_bytes);
  nmg_status s = ensure_smem(reinterpret_cast<const void*>(kern), smem);
  if (s != NMG_OK) return s;
  kern<<<grid, Cfg::THREADS, smem, st>>>(a);
  return check_launch("k_fused_query_roles");
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH, class Cfg>
static nmg_status launch_roles(const FusedArgs& a, cudaStream_t st) {
  const long tiles = (long(a.n_max) + kRows - 1) / kRows;
  int grid = sm_count();
  if (tiles < grid) grid = int(tiles > 0 ? tiles : 1);
  if (tiles <= long(kShareTiles) * grid)
    return launch_roles_kernel<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, Cfg, true>(a, grid, st);
  return launch_roles_kernel<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, Cfg, false>(a, grid, st);
}

// Whether the one MLP warpgroup of the three roles would bound a launch: deep
// networks beyond the launches whose tiles the encoders share. The two roles run
// the MLP in four warpgroups. us, three roles / two, the hash-grid network (with
// half the levels to gather, the two roles hold at six layers on any size):
//   hidden layers      4            5            6            7
//   query 2,000,000    590 / 599    642 / 620    704 / 654    761 / 675
//   pdf   2,000,000    581 / 585    627 / 606    693 / 640    748 / 660
//   pdf   100,001       48 / 44      50 / 46      57 / 48      60 / 50
//   raw   2,000,000    612 / 659    618 / 681    698 / 717    764 / 740
//   raw   500,000      165 / 173    169 / 179    190 / 188    207 / 195
static bool roles_mlp_bound(const FusedArgs& a) {
  const long tiles = (long(a.n_max) + kRows - 1) / kRows, per_sm = (tiles + sm_count() - 1) / sm_count();
  const int hidden = a.n_layers - 1;
  if (per_sm <= kShareTiles) return false;
  // A query takes the same kernel whether it returns its raw outputs or not, so that it gives the same
  // bits (returned, three roles / two: 699 / 718 at five layers, 743 / 757 at six, 797 / 781 at seven).
  if (!a.raw_mode) return hidden >= 5;
  return hidden >= 7 || (hidden == 6 && (a.enc.levels <= 8 || per_sm <= 32));
}

template <int F, int LEVELS, int MODE, int SHDEG, int BINS, int K, int NOUTMAX, bool SMOOTH>
static nmg_status launch_ws_tiling(int tiling, const FusedArgs& a, cudaStream_t st) {
  switch (tiling) {
    case 8: return launch_duo<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsN4X2G1>(a, st);
    case 9: return launch_ws<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsE5C1>(a, st);
    case 10: return launch_ws<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsE6C2>(a, st);
    case 11: return launch_ws<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsE4C2S8>(a, st);
    case 12:
      if (roles_mlp_bound(a)) return launch_duo<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsN4X2G1>(a, st);
      return launch_roles<F, LEVELS, MODE, SHDEG, BINS, K, NOUTMAX, SMOOTH, WsE4X2G1>(a, st);
  }
  return set_error(NMG_ERR_INVALID_ARG, "tiling %d is not a warp-specialised one", tiling);
}

nmg_status launch_query_ws(int preset, int tiling, const FusedArgs& a, cudaStream_t st) {
  switch (preset) {
    case 1: return launch_ws_tiling<2, 16, 1, 4, 4, 8, 48, false>(tiling, a, st);
    case 2:
      if (tiling == kTilingPair) return launch_roles<2, 16, 1, 4, 4, 16, 80, false, WsE3X4G4>(a, st);
      if (!a.raw && !a.raw_mode) return launch_ws<2, 16, 1, 4, 4, 16, 80, false, WsE4C2, true>(a, st);
      return launch_ws<2, 16, 1, 4, 4, 16, 80, false, WsE4C2>(a, st);
    case 3: return launch_ws_tiling<4, 8, 0, 2, 4, 8, 48, true>(tiling, a, st);
  }
  return set_error(NMG_ERR_UNSUPPORTED, "configuration has no fused kernel");
}

}  // namespace nmg
