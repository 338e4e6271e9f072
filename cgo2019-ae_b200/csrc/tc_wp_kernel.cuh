// The output-resident fp64 kernel for outputs of several column tiles and contractions of at most three K steps: the
// row operand's tile is RESIDENT too.
//
// tc_wc_dmma_kernel (tc_wc_kernel.cuh) fetches both operands of every tile.  Where K is short, that is as much data as the
// tile of C itself (K = 40: 61 KB of operands for 64 KB of C each way), the gather of an awkward operand is repeated for
// every tile, and the ring both operands need leaves shared memory for one consumer group only, whose epilogue the tensor
// pipe then waits for.  Here a CTA takes a PANEL -- 128 rows of X over the whole contraction, at most three K steps -- into
// shared memory and walks over columns of Y:
//
//   * operand traffic falls to the 64 columns of Y per tile, and X is gathered once per panel;
//   * the ring holds Y alone, so two consumer groups (four warps of 64 x 32 each) fit, each with a ring and an output-tile
//     buffer of its own: one group's epilogue and hand-overs run beside the other's products;
//   * a panel's K steps are handed over one by one: the last tile of a panel releases a step as soon as it has read it,
//     and the next panel's step is fetched while that tile is still at work.
//
// Warps: 0-7 consumers (two groups), 8-11 fetch Y (two per group), 12 and 13 the groups' C threads (tiles of C in and out,
// as in tc_wc_dmma_kernel, one buffer per group: it is stored, read out and refilled while the group multiplies the next
// tile, which takes twice as long), 14 and 15 fetch the panels.  No two warps of a role meet at a barrier: each keeps the
// offsets it needs in a table of its own.
//
// Measured (one B200, both kernels in turn): triples term 24/16, K = 24, X gathered by element: 156 -> 129 us (91 at the
// copy bandwidth); one GPU's eighth of the 40^6 output, K = 40: 1 799 -> 1 733 us under the board's
// power cap, 1 736 -> 1 633 in bursts that stay below it (floor 1 255).
//
// Every mbarrier wait is bounded (args.spin_limit) and reports through args.status; a role that gives up leaves when what it
// has under way has landed.
#pragma once
#include "tc_wc_kernel.cuh"

namespace tck {

template <int MODEX_, int MODEY_>
struct WpCfg {
  using T = double;
  static constexpr int BM = 128, BN = 64, BK = 16;
  static constexpr int MODEX = MODEX_, MODEY = MODEY_;
  static constexpr int GROUPS = 2, WGM = 2, WGN = 2, CW = WGM * WGN;  // consumer warps of a group
  static constexpr int WM = BM / WGM, WN = BN / WGN;
  static constexpr int CONSUMER_WARPS = GROUPS * CW, Y_WARPS = 2, X_WARPS = 2;  // Y_WARPS per group
  static constexpr int CTA_THREADS = 512;
  // Registers follow the roles: what the consumers gain is what the other half of the CTA gives up.
  static constexpr int CONSUMER_REGS = 200, OTHER_REGS = 56;
  static_assert(CONSUMER_REGS + OTHER_REGS == 2 * (65536 / CTA_THREADS), "register split");
  static constexpr int LDK = BK + 2;
  static constexpr int LDX = MODEX == LM_K_VEC ? LDK : MODEX == LM_TMA_K ? BK : BM + 4;
  static constexpr int LDY = MODEY == LM_K_VEC ? LDK : MODEY == LM_TMA_K ? BK : BN + 4;
  static constexpr int round128(int x) { return (x + 127) / 128 * 128; }  // images start on 1024 bytes
  static constexpr int XIMG = round128(MODEX == LM_K_VEC ? BM * LDK : MODEX == LM_TMA_K ? BM * BK : BK * (BM + 4));
  static constexpr int YIMG = round128(MODEY == LM_K_VEC ? BN * LDK : MODEY == LM_TMA_K ? BN * BK : BK * (BN + 4));
  static constexpr int CTILE_ELEMS = BM * BN;
  static constexpr int MAX_STEPS = 3, MAX_STAGES = 4;  // K steps of a panel, stages of a group's ring
  static constexpr int TABLE_ELEMS = X_WARPS * BM + GROUPS * Y_WARPS * BN;  // one table per fetching warp
  static constexpr int NBARS = 2 * MAX_STEPS + GROUPS * (2 * MAX_STAGES + 2);
  static constexpr int SMEM_BYTES = 232448;
  // stages of a group's ring beside a panel of nk steps
  static constexpr int stages_for(int nk) {
    const int left = SMEM_BYTES / 8 - nk * XIMG - GROUPS * CTILE_ELEMS - TABLE_ELEMS - NBARS;
    const int n = left / (GROUPS * YIMG);
    return n > MAX_STAGES ? MAX_STAGES : n;
  }
  static_assert(stages_for(MAX_STEPS) >= 2, "shared memory");
};
// A consumer thread's products into the tile buffer `tb`: buffer (+)= alpha * acc.  `dense`: the tile is BM consecutive
// rows by all of its columns; else its rows lie where `mo` says (see the kernel).
template <int BM, int MB2, int NB2>
__device__ __forceinline__ void resident_add(double* tb, const double (&acc)[2 * NB2][2 * MB2][2], double alpha, bool accumulate, bool dense, int wm0,
                                             int wn0, int g, int t, int b0, int tile_n, const int (&mo)[MB2][2]) {
  const int h0 = g & 1;  // which 16-byte half of its 32 bytes a thread visits first (see the header)
  // (tiles that are plain ranges keep addresses the compiler knows: the general form cost 2.5 % on the 40^6 slab)
  if (dense) {
#pragma unroll
    for (int nb = 0; nb < 2 * NB2; ++nb) {
      double* row = tb + (wn0 + 16 * (nb >> 1) + 2 * g + (nb & 1)) * BM + wm0 + 4 * t;
#pragma unroll
      for (int i = 0; i < MB2; ++i) {
        double2* q = reinterpret_cast<double2*>(row + 16 * i);
        // the thread's four consecutive outputs: lo = (m, m+1), hi = (m+2, m+3)
        const double2 lo = make_double2(alpha * acc[nb][2 * i][0], alpha * acc[nb][2 * i + 1][0]);
        const double2 hi = make_double2(alpha * acc[nb][2 * i][1], alpha * acc[nb][2 * i + 1][1]);
        double2 first_v = h0 ? hi : lo, second_v = h0 ? lo : hi;
        if (accumulate) {
          const double2 c0 = q[h0], c1 = q[h0 ^ 1];
          first_v.x += c0.x; first_v.y += c0.y;
          second_v.x += c1.x; second_v.y += c1.y;
        }
        q[h0] = first_v;
        q[h0 ^ 1] = second_v;
      }
    }
  } else {
#pragma unroll
    for (int nb = 0; nb < 2 * NB2; ++nb) {
      const int n = wn0 + 16 * (nb >> 1) + 2 * g + (nb & 1);
      if (n >= tile_n) continue;
      double* row = tb + n * b0;
#pragma unroll
      for (int i = 0; i < MB2; ++i) {
        // the thread's four outputs: lo = (m, m+1), hi = (m+2, m+3), each pair in one run
        const double2 lo = make_double2(alpha * acc[nb][2 * i][0], alpha * acc[nb][2 * i + 1][0]);
        const double2 hi = make_double2(alpha * acc[nb][2 * i][1], alpha * acc[nb][2 * i + 1][1]);
        const int q0 = h0 ? mo[i][1] : mo[i][0], q1 = h0 ? mo[i][0] : mo[i][1];
        double2 first_v = h0 ? hi : lo, second_v = h0 ? lo : hi;
        double2* f = reinterpret_cast<double2*>(row + q0);
        double2* l = reinterpret_cast<double2*>(row + q1);
        if (accumulate) {
          const double2 c0 = q0 >= 0 ? *f : make_double2(0.0, 0.0), c1 = q1 >= 0 ? *l : make_double2(0.0, 0.0);
          first_v.x += c0.x; first_v.y += c0.y;
          second_v.x += c1.x; second_v.y += c1.y;
        }
        if (q0 >= 0) *f = first_v;
        if (q1 >= 0) *l = second_v;
      }
    }
  }
}

// The threads of one fetching role, as the shared loaders see them.
template <int THREADS_>
struct WpLoad {
  static constexpr int THREADS = THREADS_, BK = 16, LDK = BK + 2;
};

// The panels of a CTA, in order, as segments (panel, first and last column tile).  While there is a panel for every CTA, each
// takes a whole one -- at any time all CTAs are at about the same columns, and neighbours write neighbouring rows; the tiles
// of the panels left over are dealt in equal runs.
struct PanelWalk {
  uint32_t panel, n0, n1;
  uint32_t cta, ctas, tiles_n, rounds, l, l_end, round;
  __device__ __forceinline__ PanelWalk(const TcKernelArgs& p) {
    cta = blockIdx.x;
    ctas = gridDim.x;
    tiles_n = p.tiles_n;
    rounds = p.tiles_m / ctas;
    const uint64_t left = (uint64_t)(p.tiles_m - rounds * ctas) * tiles_n;
    l = (uint32_t)(left * cta / ctas);
    l_end = (uint32_t)(left * (cta + 1) / ctas);
    round = 0;
  }
  __device__ __forceinline__ bool next() {
    if (round < rounds) {
      panel = round * ctas + cta;
      n0 = 0;
      n1 = tiles_n;
      ++round;
      return true;
    }
    if (l >= l_end) return false;
    const uint32_t q = l / tiles_n;
    panel = rounds * ctas + q;
    n0 = l - q * tiles_n;
    n1 = min(tiles_n, n0 + (l_end - l));
    l += n1 - n0;
    return true;
  }
};
// ... and the tiles of one group: every other one of the CTA's.
struct GroupWalk {
  PanelWalk w;
  uint32_t tm, tn, pos, group;
  bool any;
  __device__ __forceinline__ GroupWalk(const TcKernelArgs& p, uint32_t gi) : w(p), pos(0), group(gi), any(false) {}
  __device__ __forceinline__ bool next() {
    if (any) tn += 2;
    while (!any || tn >= w.n1) {
      if (!w.next()) return false;
      any = true;
      tm = w.panel;
      tn = w.n0 + ((group ^ pos) & 1u);
      pos += w.n1 - w.n0;
    }
    return true;
  }
};

template <class CF>
__global__ void __launch_bounds__(CF::CTA_THREADS, 1) tc_wp_dmma_kernel(const __grid_constant__ TcKernelArgs p,
                                                                         double* __restrict__ C,
                                                                         const double* __restrict__ X,
                                                                         const double* __restrict__ Y) {
  constexpr int BM = CF::BM, BN = CF::BN, BK = CF::BK, LDX = CF::LDX, LDY = CF::LDY, CW = CF::CW;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const int nk = (int)((p.Kflat + BK - 1) / BK);  // <= MAX_STEPS
  const uint32_t S = (uint32_t)p.ring_stages;
  const uint32_t kend = p.Kflat;
  const bool accumulate = p.beta != 0;
  double* panel = reinterpret_cast<double*>(smem_raw);  // [nk][XIMG]; images lead: TMA boxes need 1024-byte alignment
  double* rings = panel + nk * CF::XIMG;                // [groups][S][YIMG]
  double* cbufs = rings + CF::GROUPS * S * CF::YIMG;    // [groups][CTILE_ELEMS]
  int64_t* tables = reinterpret_cast<int64_t*>(cbufs + CF::GROUPS * CF::CTILE_ELEMS);
  uint64_t* pfull = reinterpret_cast<uint64_t*>(tables + CF::TABLE_ELEMS);  // [steps] a panel's K step has landed
  uint64_t* pempty = pfull + CF::MAX_STEPS;                                 // [steps] ... and nobody reads it any more

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto group_bars = [&](int g) { return pempty + CF::MAX_STEPS + g * (2 * CF::MAX_STAGES + 2); };
  constexpr int X_ARRIVALS = CF::MODEX == LM_TMA_K ? 1 : 32 * CF::X_WARPS, Y_ARRIVALS = CF::MODEY == LM_TMA_K ? 1 : 32 * CF::Y_WARPS;
  if (tid == 32) {  // descriptors into the copy engine's cache before the first copy needs them
    if constexpr (CF::MODEX == LM_TMA_K) asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_x)) : "memory");
    if constexpr (CF::MODEY == LM_TMA_K) asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_y)) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_ct)) : "memory");
  }
  if (tid == 0) {
    for (int ks = 0; ks < CF::MAX_STEPS; ++ks) { mbar_init(pfull + ks, X_ARRIVALS); mbar_init(pempty + ks, CF::CONSUMER_WARPS); }
    for (int g = 0; g < CF::GROUPS; ++g) {
      uint64_t* b = group_bars(g);
      for (int s = 0; s < CF::MAX_STAGES; ++s) { mbar_init(b + s, Y_ARRIVALS); mbar_init(b + CF::MAX_STAGES + s, CW); }
      mbar_init(b + 2 * CF::MAX_STAGES, 1);
      mbar_init(b + 2 * CF::MAX_STAGES + 1, CW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();

  if (warp >= CF::CONSUMER_WARPS) {
    reg_dec<CF::OTHER_REGS>();
    const int role = warp - CF::CONSUMER_WARPS;
    if (role < CF::GROUPS * CF::Y_WARPS) {
      // ------------------------------------------------------------ fetch Y ----
      const int gi = role / CF::Y_WARPS, ptid = tid - 32 * (CF::CONSUMER_WARPS + gi * CF::Y_WARPS);
      uint64_t *full = group_bars(gi), *empty = full + CF::MAX_STAGES;
      int64_t* offy_n = tables + CF::X_WARPS * BM + role * BN;
      double* ring = rings + gi * S * CF::YIMG;
      // element copies: 0 = lanes walk the external index, else the step between the positions of the 4 lanes that walk k
      const int lgy = p.lanes_k_y == 1 ? 0 : p.kstep_y;
      uint32_t it = 0, s = 0, use = 0;
      for (GroupWalk w(p, gi); w.next();) {
        const CutTile nt = cut_tile(p.ncut, w.tn);
        if constexpr (CF::MODEY != LM_TMA_K) {
          __syncwarp();
          for (int i = lane; i < BN; i += 32) {
            int64_t unused;
            decode(p.N, cut_flat(p.ncut, nt, i), p.Nflat, &offy_n[i], &unused);
          }
          __syncwarp();
        }
        int64_t ky = ws_koff(p.koff_y, 0, kend, lane);
        for (int ks = 0; ks < nk; ++ks, ++it) {
          const int64_t ny = ws_koff(p.koff_y, (uint32_t)(ks + 1) * BK, kend, lane);
          // (one decision per warp: the loaders below shuffle)
          if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], (use & 1u) ^ 1u, p.status, 2, p.spin_limit))) {
            copies_landed();
            if (CF::MODEY == LM_TMA_K && ptid == 0) fills_landed(full, it, S, p.status, p.spin_limit);
            return;
          }
          double* ys = ring + s * CF::YIMG;
          // tests only: one thread of CTA 0 never announces its copies of one stage
          const bool skip = p.test_fault == 1 && blockIdx.x == 0 && gi == 0 && it == 1;
          if constexpr (CF::MODEY == LM_TMA_K) {
            if (ptid == 0 && !skip) {
              mbar_arrive_expect_tx(&full[s], BN * BK * 8);
              tma_load_2d(ys, &p.tmap_y, ks * BK, (int)cut_flat(p.ncut, nt, 0), &full[s]);
            }
          } else {
            ws_load<WpLoad<32 * CF::Y_WARPS>, BN, CF::MODEY>(ys, Y, offy_n, ky, ptid, lgy, p.rows_across_y, (int)p.ncut.b0);
            if (!(skip && ptid == 7)) mbar_arrive_on_copies(&full[s]);
          }
          ky = ny;
          if (++s == S) { s = 0; ++use; }
        }
      }
      return;
    }
    if (role < CF::GROUPS * CF::Y_WARPS + CF::GROUPS) {
      // ----------------------------------------------------------- C thread ----
      if (lane != 0) return;
      const int gi = role - CF::GROUPS * CF::Y_WARPS;
      uint64_t *c_ready = group_bars(gi) + 2 * CF::MAX_STAGES, *c_staged = c_ready + 1;
      const uint32_t buf = smem_u32(cbufs + gi * CF::CTILE_ELEMS);
      const uint64_t tmap = reinterpret_cast<uint64_t>(&p.tmap_ct);
      auto fetch = [&](const int (&c)[5]) {  // a tile into the buffer (or just: the buffer is free)
        if (!accumulate) { mbar_arrive(c_ready); return; }
        mbar_arrive_expect_tx(c_ready, p.mcut.b0 * p.mcut.b1 * p.ncut.b0 * p.ncut.b1 * 8u);
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n" ::"r"(buf),
            "l"(tmap), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(smem_u32(c_ready))
            : "memory");
      };
      GroupWalk w(p, gi);
      int c[5];
      bool more = w.next();
      if (more) {
        tile_box_coords(p, w.tm, w.tn, c);
        fetch(c);
      }
      for (uint32_t j = 0; more; ++j) {
        int next[5] = {0, 0, 0, 0, 0};  // (its divisions are done while the consumers work)
        more = w.next();
        if (more) tile_box_coords(p, w.tm, w.tn, next);
        if (!mbar_wait(c_staged, j & 1u, p.status, 6, p.spin_limit)) {  // the tile on its way into the buffer lands first
          mbar_wait(c_ready, j & 1u, p.status, 6, p.spin_limit);
          break;
        }
        asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4, %5}], [%6];\n" ::"l"(tmap), "r"(c[0]),
                     "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(buf)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        if (more) {
          asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // the store has read the buffer: it may be refilled
          fetch(next);
        }
#pragma unroll
        for (int d = 0; d < 5; ++d) c[d] = next[d];
      }
      asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
      return;
    }
    // --------------------------------------------------------- fetch panels ----
    const int ptid = tid - 32 * (CF::CONSUMER_WARPS + CF::GROUPS * CF::Y_WARPS + CF::GROUPS);
    int64_t* offx_m = tables + (ptid >> 5) * BM;
    const int lgx = p.lanes_k_x == 1 ? 0 : p.kstep_x;
    PanelWalk w(p);
    for (uint32_t seg = 0; w.next(); ++seg) {
      const CutTile mt = cut_tile(p.mcut, w.panel);
      if constexpr (CF::MODEX != LM_TMA_K) {
        __syncwarp();
        for (int i = lane; i < BM; i += 32) {
          int64_t unused;
          decode(p.M, cut_flat(p.mcut, mt, i), p.Mflat, &offx_m[i], &unused);
        }
        __syncwarp();
      }
      int64_t kx = ws_koff(p.koff_x, 0, kend, lane);
      for (int ks = 0; ks < nk; ++ks) {
        const int64_t nx = ws_koff(p.koff_x, (uint32_t)(ks + 1) * BK, kend, lane);
        if (!__all_sync(0xffffffffu, mbar_wait(&pempty[ks], (seg & 1u) ^ 1u, p.status, 1, p.spin_limit))) {
          copies_landed();
          if (CF::MODEX == LM_TMA_K && ptid == 0) fills_landed(pfull, seg * nk + ks, nk, p.status, p.spin_limit);
          return;
        }
        double* xs = panel + ks * CF::XIMG;
        if constexpr (CF::MODEX == LM_TMA_K) {
          if (ptid == 0) {
            mbar_arrive_expect_tx(&pfull[ks], BM * BK * 8);
            tma_load_2d(xs, &p.tmap_x, ks * BK, (int)cut_flat(p.mcut, mt, 0), &pfull[ks]);
          }
        } else {
          ws_load<WpLoad<32 * CF::X_WARPS>, BM, CF::MODEX>(xs, X, offx_m, kx, ptid, lgx, p.rows_across_x, (int)p.mcut.b0);
          mbar_arrive_on_copies(&pfull[ks]);
        }
        kx = nx;
      }
    }
    return;
  }

  // -------------------------------------------------------------- consumer ----
  reg_inc<CF::CONSUMER_REGS>();
  constexpr int WM = CF::WM, WN = CF::WN, MB2 = WM / 16, NB2 = WN / 16;
  const int gi = warp / CW, cw = warp % CW;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (cw % CF::WGM) * WM, wn0 = (cw / CF::WGM) * WN;
  const double alpha = p.alpha;
  uint64_t *full = group_bars(gi), *empty = full + CF::MAX_STAGES, *c_ready = empty + CF::MAX_STAGES, *c_staged = c_ready + 1;
  const double* ring = rings + gi * S * CF::YIMG;
  double* tb = cbufs + gi * CF::CTILE_ELEMS;
  // where this thread's pairs of rows lie in a tile buffer (see tc_wc_dmma_kernel)
  const int b0 = (int)p.mcut.b0, tile_n = (int)(p.ncut.b0 * p.ncut.b1), tile_m = (int)(p.mcut.b0 * p.mcut.b1);
  const bool dense = b0 == BM && tile_n == BN;
  int mo[MB2][2];
#pragma unroll
  for (int i = 0; i < MB2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = wm0 + 16 * i + 4 * t + 2 * h;
      mo[i][h] = m < tile_m ? m % b0 + m / b0 * (b0 * tile_n) : -1;
    }
  uint32_t s = 0, use = 0, j = 0, seg = 0, pos = 0;
  for (PanelWalk w(p); w.next(); ++seg) {
    uint32_t tn = w.n0 + (((uint32_t)gi ^ pos) & 1u);
    pos += w.n1 - w.n0;
    if (tn >= w.n1) {  // no tile of this panel is the group's: it only passes the panel on
      for (int ks = 0; ks < nk; ++ks) {
        if (!mbar_wait(&pfull[ks], seg & 1u, p.status, 5, p.spin_limit)) return;
        __syncwarp();
        if (lane == 0) mbar_arrive(&pempty[ks]);
      }
      continue;
    }
    for (bool first = true; tn < w.n1; tn += 2, ++j, first = false) {
      const bool last = tn + 2 >= w.n1;
      double acc[2 * NB2][2 * MB2][2];
#pragma unroll
      for (int jj = 0; jj < 2 * NB2; ++jj)
#pragma unroll
        for (int i = 0; i < 2 * MB2; ++i) { acc[jj][i][0] = 0.0; acc[jj][i][1] = 0.0; }
      for (int ks = 0; ks < nk; ++ks) {
        if (first && !mbar_wait(&pfull[ks], seg & 1u, p.status, 5, p.spin_limit)) return;
        if (!mbar_wait(&full[s], use & 1u, p.status, 3, p.spin_limit)) return;
        const double* xs = panel + ks * CF::XIMG;
        const double* ys = ring + s * CF::YIMG;
        const int kleft = (int)kend - ks * BK;
        const int nks = kleft >= BK ? BK / 4 : (kleft + 3) / 4;
#pragma unroll
        for (int kq = 0; kq < BK / 4; ++kq) {
          if (kq < nks) {
            const int k = kq * 4 + t;
            double2 xf[MB2], yf[NB2];
#pragma unroll
            for (int i = 0; i < MB2; ++i) xf[i] = ws_frag<CF::MODEX, LDX>(xs, wm0 + 2 * g + i * 16, k);
#pragma unroll
            for (int jj = 0; jj < NB2; ++jj) yf[jj] = ws_frag<CF::MODEY, LDY>(ys, wn0 + 2 * g + jj * 16, k);
#pragma unroll
            for (int jj = 0; jj < NB2; ++jj)
#pragma unroll
              for (int i = 0; i < MB2; ++i) {
                dmma884(acc[2 * jj][2 * i][0], acc[2 * jj][2 * i][1], yf[jj].x, xf[i].x);
                dmma884(acc[2 * jj][2 * i + 1][0], acc[2 * jj][2 * i + 1][1], yf[jj].x, xf[i].y);
                dmma884(acc[2 * jj + 1][2 * i][0], acc[2 * jj + 1][2 * i][1], yf[jj].y, xf[i].x);
                dmma884(acc[2 * jj + 1][2 * i + 1][0], acc[2 * jj + 1][2 * i + 1][1], yf[jj].y, xf[i].y);
              }
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&empty[s]);  // this warp no longer reads the stage
          if (last) mbar_arrive(&pempty[ks]);  // ... nor this step of the panel
        }
        if (++s == S) { s = 0; ++use; }
      }
      // ---- epilogue: buffer (+)= alpha * acc in shared memory; the C thread stores the buffer ----
      if (!mbar_wait(c_ready, j & 1u, p.status, 4, p.spin_limit)) return;
      resident_add<BM, MB2, NB2>(tb, acc, alpha, accumulate, dense, wm0, wn0, g, t, b0, tile_n, mo);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(c_staged);  // release: this warp's part of the tile is in the buffer
    }
  }
}

}  // namespace tck
