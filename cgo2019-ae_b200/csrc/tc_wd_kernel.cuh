// Persistent fp32 contraction kernel for sm_100a on PAIRS of CTAs: 256 x 256 tiles, three TF32 products per fp32 product on
// tcgen05.mma.cta_group::2.
//
// Same arithmetic, split (v = hi + lo), image layouts and accumulation chains as tc_wt_tf32_kernel (tc_wt_kernel.cuh), for
// long contractions whose operands both arrive in tiled TMA boxes.  There a K step of a 128 x 128 tile takes about 1 200
// cycles of which the six MMAs are 440: what bounds it is the chain conversion -> hand-over -> MMA, whose length does not
// depend on how much the MMAs do.  Here the two CTAs of a cluster (two SMs) work on one tile: each fetches and converts 128
// rows of X and 128 rows of Y per K step, exactly as before, and the MMA -- issued by the first CTA's one thread for both --
// multiplies all 256 by all 256 of them: twice the products per SM for the same conversion and hand-over, and half the
// operand bytes per product from L2.
//
//   warps 0-7   EPILOGUE  a thread holds one row (n) and half of the columns (128 m) of its CTA's 128 x 256 half of the tile
//                         IN REGISTERS: segments of at most 512 products leave the accumulator by tcgen05.ld and are added
//                         up there in round-to-nearest fp32, so one accumulator serves (it is free again as soon as it has
//                         been read) and no tile buffer is needed; at the end the row goes to C through a small staging
//                         area, 16 columns at a time, as bulk reduce-adds (`+=`, `-=`) or stores (`=`).
//   warps 8-15  SPLIT     stage -> registers -> hi / lo: X into images in shared memory, Y into tensor memory.
//   warp 16     LOADER    one thread, one box per operand and stage.
//   warp 17     MMA       (first CTA of the pair) waits until both CTAs' images are written, issues, commits to both.
//   warps 18-19 no work.
//
// Measured (one B200, against the kernels these problems ran on before): 4096 x 4096 x 2048 554 -> 314 us in short runs (219
// TFLOP/s; the MMAs alone take 207 in four rounds of 74 tiles, 181 with the last one halved) and 555 -> 352 in long ones, under
// the board's power cap; 720 x 2064 x 3664 365 -> 133, 1496 x 1120 x 400 42 -> 25; 80 matrices of 200 to 4096 rows and
// columns, K = 256 to 4096, 0.99 to 6.6 times as fast, 2.4 in the mean.  With the copies, the conversion or two of the three
// MMAs taken out in turn 4096 x 4096 x 2048 took 279, 320 and 357 of the 361 us it stood at: what is left is all three meeting
// in 227 KB.  Bulk reduce-adds keep subnormal sums; adding to C in registers was 1 to 19 % slower.
//
// Barriers that both CTAs arrive on live in the first CTA (arrivals of the second go there through the cluster's shared
// memory); commits arrive on both CTAs' barriers.  Neither CTA leaves before the other has finished (cluster barrier), and
// tensor memory is freed after that.  Every mbarrier wait is bounded and reports through args.status.
#pragma once
#include "tc_wt_kernel.cuh"

namespace tck {

template <int MODEX_, int MODEY_>
struct WdCfg {
  using T = float;
  // 3: box of rows of 32 k (128-byte swizzle), 4: the external index is the fastest (32 rows of k, dense)
  static constexpr int MODEX = MODEX_, MODEY = MODEY_;
  static constexpr int BM = 256, BN = 256, HALF = 128;  // the pair's tile; rows of each operand per CTA
  // Stages and image slots are units of 32 k: what a unit costs beside its conversion and its MMAs -- waits, fences,
  // arrivals, and the copy engine's work per row of a box -- does not depend on its length (units of 16 k in both: 502 us
  // on 4096 x 4096 x 2048, in the slots alone 420, in neither 361; a third slot, for which the output staging shrank, 336).
  static constexpr int UK = 32;
  static constexpr int IMG = HALF * UK;                          // elements of one operand's box, and of one image
  static constexpr uint32_t TMA_BYTES = 2 * IMG * 4;
  static constexpr int UMMA_ELEMS = 2 * IMG;                     // hi and lo images of X for one unit
  static constexpr int CTA_THREADS = 640;
  static constexpr int SPLIT_WARPS = 8, EPI_WARPS = 8;
  static constexpr int SEG_UNITS = 16;                           // units per accumulation chain: 512 products
  static constexpr int STAGES = 3, SLOTS = 3;
  static constexpr int TMEM_COLS = 512, A_COLS = 256, A_SLOT_COLS = 64;
  static constexpr int OUT_COLS = 16, OUT_PITCH = OUT_COLS + 4;  // staging: 16 columns of a row, conflict-free 16-byte accesses
  static constexpr int OUT_ELEMS = 32 * OUT_PITCH;               // per epilogue warp
  static constexpr int NBARS = 2 * STAGES + 2 * SLOTS + 4;
  static constexpr int HEAD_BYTES = NBARS * 8 + 16;
  static constexpr int SMEM_BYTES = (STAGES * 2 * IMG + SLOTS * UMMA_ELEMS + EPI_WARPS * OUT_ELEMS) * 4 + HEAD_BYTES;
  static_assert(SMEM_BYTES <= 232448 && NBARS % 2 == 0, "shared memory");
  // 640 threads start with 96 registers; what the epilogue gains the other three warpgroups give up.
  static constexpr int LAUNCH_REGS = 96, EPILOGUE_REGS = 168, SPLIT_REGS = 48, OTHER_REGS = 40;
  static_assert(256 * EPILOGUE_REGS + 256 * SPLIT_REGS + 128 * OTHER_REGS <= CTA_THREADS * LAUNCH_REGS, "register split");
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
// Arrival on the barrier at the same place in the pair's first CTA.
__device__ __forceinline__ void mbar_arrive_first(uint64_t* bar) {
  asm volatile(
      "{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %0, 0;\n mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n}\n" ::"r"(smem_u32(bar))
      : "memory");
}
// Bounded wait that also orders what the other CTA's threads did before they arrived.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status, int code, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  atomicCAS(status, 0, code);
  return false;
}
// D (+)= A * B^T over the pair: 256 rows (128 per CTA, A in each CTA's tensor memory) by N columns (half of B's rows in each
// CTA's shared memory, at the same address).
__device__ __forceinline__ void tc05_pair_mma_tf32(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0)
      : "memory");
}
// One arrival on `bar` of each CTA of the pair once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void tc05_pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

template <class CF>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CF::CTA_THREADS, 1)
    tc_wd_tf32_kernel(const __grid_constant__ TcKernelArgs p, float* __restrict__ C, const float* __restrict__ X, const float* __restrict__ Y) {
  constexpr int UK = CF::UK, HALF = CF::HALF, STAGES = CF::STAGES, SLOTS = CF::SLOTS;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float* stages = reinterpret_cast<float*>(smem_raw);             // [STAGES][X box | Y box]
  float* images = stages + STAGES * 2 * CF::IMG;                  // [SLOTS][X hi | X lo]
  float* outs = images + SLOTS * CF::UMMA_ELEMS;                  // [EPI_WARPS][32][OUT_PITCH]
  uint64_t* full = reinterpret_cast<uint64_t*>(outs + CF::EPI_WARPS * CF::OUT_ELEMS);  // [STAGES] boxes have landed
  uint64_t* empty = full + STAGES;      // [STAGES] the split warps have read them
  uint64_t* img_full = empty + STAGES;  // [SLOTS] (first CTA) both CTAs' images of a K step are written
  uint64_t* img_free = img_full + SLOTS;  // [SLOTS] ... and the MMAs that read them have completed
  uint64_t* acc_full = img_free + SLOTS;  // the accumulator holds a finished segment
  uint64_t* acc_free = acc_full + 1;      // (first CTA) both CTAs have read it out
  uint64_t* drained = acc_full + 2;       // the MMAs of a role that gave up have completed
  uint32_t* slot = reinterpret_cast<uint32_t*>(full + CF::NBARS);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, CF::SPLIT_WARPS); }
    for (int h = 0; h < SLOTS; ++h) { mbar_init(img_full + h, 2 * CF::SPLIT_WARPS); mbar_init(img_free + h, 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, 2 * CF::EPI_WARPS);
    mbar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_x)) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_y)) : "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)), "r"(CF::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
  tc05_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA's barriers are set up too
  tc05_fence_after();
  const uint32_t tmem = *slot;

  // Items: tiles, and -- where the last round would leave half of the pairs without one -- the last round's tiles as halves
  // of 128 columns.
  const uint32_t first = blockIdx.x >> 1, step = gridDim.x >> 1, tiles = p.tiles_m * p.tiles_n;
  const uint32_t left = tiles % step, halved = 2 * left <= step ? left : 0u, whole = tiles - halved, total = whole + 2 * halved;
  struct Place { uint32_t m0, n0; bool half; };
  auto place = [&](uint32_t item) {
    const uint32_t h = item < whole ? 0u : item - whole;
    uint32_t tm, tn;
    tile_coords(p, item < whole ? item : whole + (h >> 1), &tm, &tn);
    return Place{tm * CF::BM + (h & 1u) * HALF, tn * CF::BN + rank * HALF, item >= whole};
  };
  const uint32_t kend = p.Kflat;
  const int nu = (int)((kend + UK - 1) / UK);
  const int nseg = (nu + CF::SEG_UNITS - 1) / CF::SEG_UNITS;
  auto seg_begin = [&](int seg) { return (int)((int64_t)seg * nu / nseg); };  // segments of (almost) equal length, none empty
  const uint32_t limit = p.spin_limit;

  if (warp < 8) {
    // ------------------------------------------------------------ epilogue ----
    reg_inc<CF::EPILOGUE_REGS>();
    constexpr int COLS = 128;  // columns of a thread: half (warp / 4) of the tile's m
    const float alpha = (float)p.alpha;
    const bool accumulate = p.beta != 0;
    float* row = outs + warp * CF::OUT_ELEMS + lane * CF::OUT_PITCH;  // this thread's: nobody else touches it
    auto out_off = [&](const TcDims& d, uint32_t flat) -> int64_t {
      if (d.n == 1) return (int64_t)flat * d.s_out[0];
      int64_t unused, o;
      decode(d, flat, 0xffffffffu, &unused, &o);
      return o;
    };
    uint32_t unit = 0;
    bool alive = true;
    for (uint32_t item = first; alive && item < total; item += step) {
      const Place at = place(item);
      const int cols = at.half ? COLS / 2 : COLS;
      const uint32_t cbase = (uint32_t)((warp >> 2) * cols), taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + cbase;
      float sum[COLS];
      for (int seg = 0; seg < nseg; ++seg, ++unit) {
        if (!mbar_wait(acc_full, unit & 1u, p.status, 10, limit)) { alive = false; break; }
        tc05_fence_after();
        if (seg == 0) {
#pragma unroll
          for (int c = 0; c < COLS; c += 16)
            if (c < cols) tc05_ld16(taddr + c, sum + c);
          tc05_wait_ld();
        } else {
#pragma unroll
          for (int c = 0; c < COLS; c += 16) {
            if (c >= cols) break;
            float v[16];
            tc05_ld16(taddr + c, v);
            tc05_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[c + i] += v[i];
          }
        }
        // the accumulator is in registers: the next segment may overwrite it
        tc05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_first(acc_free);
      }
      if (!alive) break;
      const uint32_t n = at.n0 + 32 * (warp & 3) + lane, m0 = at.m0 + cbase;
      const int64_t noff = n < p.Nflat ? out_off(p.N, n) : -1;
#pragma unroll
      for (int c = 0; c < COLS; c += CF::OUT_COLS) {
        if (c >= cols) break;
        asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // the copy before has read the row
#pragma unroll
        for (int i = 0; i < CF::OUT_COLS; i += 4)
          *reinterpret_cast<float4*>(row + i) = make_float4(alpha * sum[c + i], alpha * sum[c + i + 1], alpha * sum[c + i + 2], alpha * sum[c + i + 3]);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // these writes -> the copy that reads them
        const uint32_t m = m0 + c;
        if (noff >= 0 && m < p.Mflat) {
          float* dst = C + noff + out_off(p.M, m);  // 16 values from a multiple of 16 on are neighbours in C
          const uint32_t bytes = min((uint32_t)CF::OUT_COLS, p.Mflat - m) * 4u;
          if (accumulate) bulk_reduce_add(dst, smem_u32(row), bytes);
          else bulk_store(dst, smem_u32(row), bytes);
        }
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      }
    }
    asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
  } else if (warp < 16) {
    // --------------------------------------------------------------- split ----
    reg_dec<CF::SPLIT_REGS>();
    // Thread -> one 16-byte chunk of each operand per group of eight k: row r and the four k = 4 kc .. + 3, kc = 2 h + q.
    const int stid = tid - 256, r = stid % HALF, q = stid / HALF;
    auto chunk = [&](const float* img, int kc, int mode) {
      // rows of 32 k in 16-byte chunks, chunk c at position c ^ (r % 8) (128-byte swizzle)
      if (mode == 3) return *reinterpret_cast<const float4*>(img + r * UK + 4 * (kc ^ (r & 7)));
      const float* src = img + (4 * kc) * HALF + r;
      return make_float4(src[0], src[HALF], src[2 * HALF], src[3 * HALF]);
    };
    const uint32_t ylane = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + CF::A_COLS + 4u * (uint32_t)q;
    uint32_t s = 0, sl = 0, sphase = 0, lphase = 0, done = 0;
    bool alive = true;
    for (uint32_t item = first; alive && item < total; item += step) {
      const bool has_x = item < whole || r < HALF / 2;
      for (int u = 0; u < nu; ++u) {
        const int nh = (int)min(4u, (kend - (uint32_t)u * UK + 7u) / 8u);  // groups of eight k
        if (!mbar_wait(full + s, sphase, p.status, 12, limit)) { alive = false; break; }
        const float* xs = stages + s * 2 * CF::IMG;
        const float* ys = xs + CF::IMG;
        float4 vy[2], vx[2];
        auto load = [&](int h0) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            vy[h] = chunk(ys, 2 * (h0 + h) + q, CF::MODEY);
            if (has_x) vx[h] = chunk(xs, 2 * (h0 + h) + q, CF::MODEX);
          }
        };
        float4* hi_img = reinterpret_cast<float4*>(images + sl * CF::UMMA_ELEMS);
        float4* lo_img = hi_img + CF::IMG / 4;
        auto store = [&](int h0) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h0 + h >= nh) break;
            float4 hi, lo;
            split_tf32_bits(vy[h].x, hi.x, lo.x); split_tf32_bits(vy[h].y, hi.y, lo.y);
            split_tf32_bits(vy[h].z, hi.z, lo.z); split_tf32_bits(vy[h].w, hi.w, lo.w);
            const uint32_t col = ylane + sl * CF::A_SLOT_COLS + (h0 + h) * 16u;
            tc05_st4(col, hi);
            tc05_st4(col + 8u, lo);
            if (!has_x) continue;
            split_tf32_bits(vx[h].x, hi.x, lo.x); split_tf32_bits(vx[h].y, hi.y, lo.y);
            split_tf32_bits(vx[h].z, hi.z, lo.z); split_tf32_bits(vx[h].w, hi.w, lo.w);
            const int d = ((r >> 3) * (UK / 4) + 2 * (h0 + h) + q) * 8 + (r & 7);
            hi_img[d] = hi;
            lo_img[d] = lo;
          }
        };
        load(0);
        if (done >= (uint32_t)SLOTS && !mbar_wait(img_free + sl, lphase ^ 1u, p.status, 13, limit)) { alive = false; break; }
        tc05_fence_after();
        store(0);
        if (nh > 2) {
          load(2);
          store(2);
        }
        __syncwarp();
        tc05_wait_st();
        tc05_fence_before();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // generic writes -> the MMA's reads; reads -> the refill
        __syncwarp();
        if (lane == 0) { mbar_arrive(empty + s); mbar_arrive_first(img_full + sl); }
        ++done;
        if (++s == STAGES) { s = 0; sphase ^= 1u; }
        if (++sl == SLOTS) { sl = 0; lphase ^= 1u; }
      }
    }
  } else {
    reg_dec<CF::OTHER_REGS>();
    if (warp == 16 && lane == 0) {
      // ------------------------------------------------------------ loader ----
      uint32_t g = 0;
      bool alive = true;
      for (uint32_t item = first; alive && item < total; item += step) {
        const Place at = place(item);
        const int m0 = (int)(at.m0 + rank * (at.half ? HALF / 2 : HALF)), n0 = (int)at.n0;
        for (int k0 = 0; k0 < (int)kend; k0 += UK, ++g) {
          const uint32_t s = g % STAGES;
          if (g >= (uint32_t)STAGES && !mbar_wait(empty + s, ((g / STAGES) - 1) & 1u, p.status, 14, limit)) { alive = false; break; }
          // tests only: one stage is left unannounced, so that the waits on it run out
          if (p.test_fault == 1 && blockIdx.x == 0 && g == 1) continue;
          float* xs = stages + s * 2 * CF::IMG;
          float* ys = xs + CF::IMG;
          mbar_arrive_expect_tx(full + s, CF::TMA_BYTES);
          if constexpr (CF::MODEX == 3) tma_load_2d(xs, &p.tmap_x, k0, m0, full + s);
          else tma_load_2d(xs, &p.tmap_x, m0, k0, full + s);
          if constexpr (CF::MODEY == 3) tma_load_2d(ys, &p.tmap_y, k0, n0, full + s);
          else tma_load_2d(ys, &p.tmap_y, n0, k0, full + s);
        }
      }
      // A loader that gave up waits (with a limit) for the boxes it has under way.
      if (!alive)
        for (uint32_t q = g > (uint32_t)STAGES ? g - STAGES : 0u; q < g; ++q)
          if (!(p.test_fault == 1 && blockIdx.x == 0 && q == 1)) mbar_wait(full + q % STAGES, (q / STAGES) & 1u, p.status, 14, limit);
    } else if (warp == 17 && lane == 0 && rank == 0) {
      // --------------------------------------------------------------- MMA ----
      const uint64_t bh0 = umma_desc_k(smem_u32(images), 128, (UK / 4) * 128);
      const uint32_t a0 = tmem + CF::A_COLS;
      uint32_t sl = 0, phase = 0, unit = 0;
      bool alive = true;
      for (uint32_t item = first; alive && item < total; item += step)
        for (int seg = 0; alive && seg < nseg; ++seg, ++unit) {
          const uint32_t idesc = item < whole ? umma_idesc_tf32(CF::BN, CF::BM) : umma_idesc_tf32(CF::BN, HALF);
          if (unit >= 1 && !mbar_wait_cluster(acc_free, (unit - 1) & 1u, p.status, 15, limit)) { alive = false; break; }
          tc05_fence_after();
          const int u_begin = seg_begin(seg), u_end = seg_begin(seg + 1);
          for (int u = u_begin; u < u_end; ++u) {
            const int nh = (int)min(4u, (kend - (uint32_t)u * UK + 7u) / 8u);
            if (!mbar_wait_cluster(img_full + sl, phase, p.status, 16, limit)) { alive = false; break; }
            tc05_fence_after();
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              if (h >= nh) break;
              const uint32_t ah = a0 + sl * CF::A_SLOT_COLS + h * 16u, al = ah + 8u;
              const uint64_t bh = bh0 + (uint64_t)(sl * (uint32_t)(CF::UMMA_ELEMS * 4 / 16) + h * 16u);
              const uint64_t bl = bh + (uint64_t)(CF::IMG * 4 / 16);
              tc05_pair_mma_tf32(tmem, al, bh, idesc, (u > u_begin || h > 0) ? 1u : 0u);
              tc05_pair_mma_tf32(tmem, ah, bl, idesc, 1u);
              tc05_pair_mma_tf32(tmem, ah, bh, idesc, 1u);
            }
            tc05_pair_commit(img_free + sl);
            if (++sl == SLOTS) { sl = 0; phase ^= 1u; }
          }
          if (alive) tc05_pair_commit(acc_full);
        }
      if (!alive) {  // what is under way must not outlive the memory it works on
        tc05_pair_commit(drained);
        mbar_wait(drained, 0u, p.status, 16, limit);
      }
    }
  }
  __syncwarp();
  tc05_fence_before();
  cluster_sync();  // both CTAs are done with each other's shared and tensor memory
  tc05_fence_after();
  if (warp == 17)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(CF::TMEM_COLS) : "memory");
}

}  // namespace tck
