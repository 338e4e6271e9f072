// Several fp64 contractions into one output, operands in tiled TMA boxes: the kernel of tc_fused.cu for plans whose
// inputs all start with the (single, even) contraction index and carry at most four output indices.
//
// A box of the output -- b_i consecutive values of every index, b_i a power of two or the whole extent, 4096 elements
// at most -- lives in shared memory while every term adds its (rows x cols) product to it, as in tc_fused_kernel.
// What bounded that kernel was not the pipe (23 % busy) but issue and latency: operands gathered by every thread,
// tables read again for each box, one barrier per 16 k.  Here
//   * CTAs are persistent, two per SM, and walk the boxes; tables are read once;
//   * one PRODUCER thread issues two tiled copies per stage (16 k x 64 rows of each input, rank 5, 128-byte swizzle,
//     zeros outside the tensor), up to kBoxStages stages ahead and across terms and boxes;
//   * eight CONSUMER warps (32 x 16 products each) wait per stage on mbarriers and once per term, before they
//     add the term's products to the box, for the other warps' additions of the term before;
//   * the first term's products are stored, the others' added; C's old values are read and the box added to them
//     once, at the end, as in tc_fused_kernel: one rounding against C's magnitude however many terms there are (a box
//     that starts from C has every term rounded against it; no faster either, 3.94 ms).
//
// Shared-memory layouts.  Operand images are [row][16 k], the 16-byte chunk c of row r at chunk position c ^ (r & 7).
// A thread reads two consecutive k at once; MMA number 2 h + e of a stage takes k = 8 h + 2 t + e in slot t, for both
// operands, so the sums are over the same k.  Block row g of an MMA stands for row perm(g) = (g & 1) * 4 + g / 2:
// the two rows a quarter warp reads then differ in bit 2 and their chunks fall into different halves of the banks.
// Box element e sits at position box_hash(e): its low four bits are XORed with a 4-bit code per higher bit.  Half a warp's
// accumulators vary over both bits of one input's first index and over one bit each of the other input's first two; the
// codes (found by search) make these four independent, so without bank conflicts, for every term of the CCSD(T) doubles
// and for four in five of all assignments of six indices (two-way at most in the rest).
//
// Measured (nine doubles terms of CCSD(T), all extents 24, one B200): 9.78 ms on tc_fused_kernel, 3.94 ms here (20.9
// TFLOP/s, 57 % of the DMMA rate; floor 2.23 ms of products).  On the way: one block barrier per term 4.76 ms; a barrier
// that warps only arrive at when their additions are done, 104 registers a thread, eight old values read together 4.49;
// positions as byte offsets, no tests in whole terms 4.14; conflict-free codes and both halves' reads first 3.95; the
// first term stored, C added at the end 3.94.  Without any loads 4.43 of the 4.49 remained, the loads alone take 2.07,
// without the additions 3.68: what is left is the chain of a term (wait, fragments, products, additions) with two CTAs
// of eight warps to cover it.
#pragma once
#include "tc_ws_kernel.cuh"

namespace tcbox {

constexpr int kMaxTerms = 16;
constexpr int kMaxRank = 8;
constexpr int kBox = 64;           // rows / columns of a term inside a box, at most
constexpr int kBoxElems = 4096;
constexpr int kBoxStages = 4;
constexpr int kConsumers = 256;    // eight warps
constexpr int kBoxThreads = kConsumers + 128;  // + a warpgroup whose first lane is the producer
// registers: launched with 80 a thread (two CTAs of 384); what the consumers take is less than the producer's warpgroup gives
constexpr int kProducerRegs = 24, kConsumerRegs = 104;
static_assert(128 * kProducerRegs + 256 * kConsumerRegs <= 384 * 80, "register shares");
constexpr int kImgBytes = kBox * 128;
constexpr int kMapDims = 4;        // output indices an input may carry

struct BoxTerm {
  uint32_t kflat, bytes;             // contraction length; bytes of one stage's two boxes
  int8_t px[kMapDims], py[kMapDims];  // output index of dimension 1 + d of the left / right input's map (-1: padding)
  int32_t full;                       // 64 rows and 64 columns
  double alpha;
};

struct BoxArgs {
  TcTensorMap x[kMaxTerms], y[kMaxTerms];
  BoxTerm term[kMaxTerms];
  int32_t n_terms, rank;
  uint32_t b[kMaxRank], ext[kMaxRank], tiles[kMaxRank];
  uint32_t lg[kMaxRank];     // bits of index i in a box position
  int64_t sc[kMaxRank];
  uint32_t total_boxes;
  uint32_t spin_limit;
  int32_t test_fault;        // tests only: 1 = the first CTA's producer leaves its second stage out
  const int32_t* pos;        // [terms][2][64] hashed box position, in bytes, of row r / column c, -1 beyond the term's rows
  int* status;               // host-visible word: code of a wait that gave up
};

// 4-bit code XORed into the low bits of a box position for each of its bits 4..11.
__host__ __device__ constexpr uint32_t box_code(int bit) {
  constexpr uint32_t code[12] = {0, 0, 0, 0, 15, 12, 5, 2, 11, 8, 14, 12};
  return code[bit];
}
__host__ __device__ constexpr uint32_t box_hash(uint32_t e) {
  uint32_t r = e;
  for (int bit = 4; bit < 12; ++bit)
    if ((e >> bit) & 1u) r ^= box_code(bit);
  return r;
}

__device__ __forceinline__ bool box_wait(uint64_t* bar, uint32_t parity, int* status, int code, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i)
    if (tck::mbar_try_wait(bar, parity)) return true;
  *reinterpret_cast<volatile int*>(status) = code;
  __threadfence_system();
  return false;
}

__device__ __forceinline__ void box_load(uint32_t dst, const TcTensorMap* map, int k0, const int (&c)[4], uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(k0), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(tck::smem_u32(bar))
      : "memory");
}

__global__ void __launch_bounds__(kBoxThreads, 2) tc_fused_box_kernel(const __grid_constant__ BoxArgs p, double* __restrict__ C) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  double* box = reinterpret_cast<double*>(smem_raw + kBoxStages * 2 * kImgBytes);
  int32_t* s_pos = reinterpret_cast<int32_t*>(box + kBoxElems);               // [terms][2][64]
  uint64_t* full = reinterpret_cast<uint64_t*>(s_pos + kMaxTerms * 2 * kBox);  // [stages]
  uint64_t* empty = full + kBoxStages;
  uint64_t* added = empty + kBoxStages;  // every warp has added its products of a term to the box
  uint64_t* left = added + 1;            // every warp has read its part of the finished box
  unsigned char* box_b = reinterpret_cast<unsigned char*>(box);
  const uint32_t stage0 = tck::smem_u32(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kBoxStages; ++s) { tck::mbar_init(full + s, 1); tck::mbar_init(empty + s, kConsumers / 32); }
    tck::mbar_init(added, kConsumers / 32);
    tck::mbar_init(left, kConsumers / 32);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  for (int i = tid; i < p.n_terms * 2 * kBox; i += kBoxThreads) s_pos[i] = p.pos[i];
  __syncthreads();

  if (warp >= kConsumers / 32) {
    // ------------------------------------------------------------ producer ----
    tck::reg_dec<kProducerRegs>();
    if (tid != kConsumers) return;
    uint32_t it = 0;
    auto drain = [&]() {  // copies land while this CTA has its shared memory, also where the consumers have given up
      for (uint32_t j = it > kBoxStages ? it - kBoxStages : 0u; j < it; ++j)
        box_wait(&full[j % kBoxStages], (j / kBoxStages) & 1, p.status, 7, p.spin_limit);
    };
    for (uint32_t bx = blockIdx.x; bx < p.total_boxes; bx += gridDim.x) {
      for (int k = 0; k < p.n_terms; ++k) {
        int cx[4] = {0, 0, 0, 0}, cy[4] = {0, 0, 0, 0};
        uint32_t r = bx;
        for (int i = 0; i < p.rank; ++i) {
          const uint32_t q = r / p.tiles[i];
          const int at = (int)((r - q * p.tiles[i]) * p.b[i]);
          r = q;
#pragma unroll
          for (int d = 0; d < kMapDims; ++d) {
            if (p.term[k].px[d] == i) cx[d] = at;
            if (p.term[k].py[d] == i) cy[d] = at;
          }
        }
        const uint32_t kfl = p.term[k].kflat, bytes = p.term[k].bytes;
        for (uint32_t k0 = 0; k0 < kfl; k0 += 16, ++it) {
          const uint32_t s = it % kBoxStages;
          if (!box_wait(&empty[s], ((it / kBoxStages) & 1) ^ 1, p.status, 2, p.spin_limit)) { drain(); return; }
          if (p.test_fault == 1 && blockIdx.x == 0 && it == 1) continue;
          tck::mbar_arrive_expect_tx(&full[s], bytes);
          box_load(stage0 + s * 2 * kImgBytes, &p.x[k], (int)k0, cx, &full[s]);
          box_load(stage0 + s * 2 * kImgBytes + kImgBytes, &p.y[k], (int)k0, cy, &full[s]);
        }
      }
    }
    drain();
    return;
  }

  // -------------------------------------------------------------- consumer ----
  tck::reg_inc<kConsumerRegs>();
  const int g = lane >> 2, t = lane & 3;
  const int pg = ((g & 1) << 2) | (g >> 1);
  const int wm0 = (warp & 1) * 32, wn0 = (warp >> 1) * 16;
  const uint32_t chunk = (uint32_t)((t ^ pg) << 4);
  const uint32_t fx = (uint32_t)(wm0 + pg) * 128u + chunk, fy = (uint32_t)(kImgBytes + (wn0 + pg) * 128) + chunk;
  // A wait gave up: the warp goes on to the end of its box without waiting or announcing anything and leaves there.  The
  // other warps' waits on it run out too, so none of this box reaches C.  (Leaving at the next term takes a vote
  // between every wait and its additions: 3.94 -> 3.96 ms on the nine terms.)
  bool dead = false;

  // this thread's box elements e = tid + 256 i: offset in C and coordinates are those of tid plus those of 256 i
  int64_t off_lo = 0;
  uint64_t crd_lo = 0;
  auto split = [&](uint32_t e, int64_t* off, uint64_t* crd) {
    int64_t o = 0;
    uint64_t c = 0;
    int sh = 0;
    for (int i = 0; i < p.rank; ++i) {
      const uint32_t v = (e >> sh) & ((1u << p.lg[i]) - 1u);
      sh += (int)p.lg[i];
      o += (int64_t)v * p.sc[i];
      c |= (uint64_t)v << (8 * i);
    }
    if (e >> sh) c = 0x4040404040404040ull;  // beyond the box (coordinates end at 63)
    *off = o;
    *crd = c;
  };
  split((uint32_t)tid, &off_lo, &crd_lo);
  int64_t* s_off_hi = reinterpret_cast<int64_t*>(left + 1);              // [16]
  uint64_t* s_crd_hi = reinterpret_cast<uint64_t*>(s_off_hi + 16);      // [16]
  if (tid < 16) split((uint32_t)tid << 8, &s_off_hi[tid], &s_crd_hi[tid]);
  const uint32_t pos_lo = box_hash((uint32_t)tid);
  asm volatile("bar.sync 1, %0;\n" ::"n"(kConsumers) : "memory");

  // corner of box bx in C, and per index the last valid coordinate inside it (one byte each, top bit set)
  auto corner_of = [&](uint32_t bx, int64_t* base, uint64_t* last) {
    int64_t o = 0;
    uint64_t l = 0x8080808080808080ull;
    uint32_t r = bx;
    for (int i = 0; i < p.rank; ++i) {
      const uint32_t q = r / p.tiles[i];
      const uint32_t at = (r - q * p.tiles[i]) * p.b[i];
      r = q;
      o += (int64_t)at * p.sc[i];
      l |= (uint64_t)(min(p.ext[i] - at, p.b[i]) - 1u) << (8 * i);
    }
    *base = o;
    *last = l;
  };
  auto valid = [&](uint64_t crd, uint64_t last) { return ((last - crd) & 0x8080808080808080ull) == 0x8080808080808080ull; };

  int64_t base = 0;
  uint64_t last = 0;
  uint32_t it = 0, terms = 0, boxes = 0;  // stages, terms and boxes so far
  for (uint32_t bx = blockIdx.x; bx < p.total_boxes; bx += gridDim.x, ++boxes) {
    corner_of(bx, &base, &last);
    for (int k = 0; k < p.n_terms; ++k) {
      double acc[2][4][2];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc[j][i][0] = 0.0; acc[j][i][1] = 0.0; }
      const int kfl = (int)p.term[k].kflat;
      for (int k0 = 0; k0 < kfl; k0 += 16, ++it) {
        const uint32_t s = it % kBoxStages;
        if (!dead && !box_wait(&full[s], (it / kBoxStages) & 1, p.status, 3, p.spin_limit)) dead = true;
        const unsigned char* img = smem_raw + s * 2 * kImgBytes;
        // (both halves of a whole stage are read before the first product: behind a branch the second half's reads would
        // wait for the first half's products)
        auto halves = [&](auto count) {
          constexpr int H = decltype(count)::value;
          double2 xf[H][4], yf[H][2];
#pragma unroll
          for (int h = 0; h < H; ++h) {
#pragma unroll
            for (int i = 0; i < 4; ++i) xf[h][i] = *reinterpret_cast<const double2*>(img + (fx ^ (h * 64u)) + i * 1024);
#pragma unroll
            for (int j = 0; j < 2; ++j) yf[h][j] = *reinterpret_cast<const double2*>(img + (fy ^ (h * 64u)) + j * 1024);
          }
#pragma unroll
          for (int h = 0; h < H; ++h) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int i = 0; i < 4; ++i) tck::dmma884(acc[j][i][0], acc[j][i][1], yf[h][j].x, xf[h][i].x);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int i = 0; i < 4; ++i) tck::dmma884(acc[j][i][0], acc[j][i][1], yf[h][j].y, xf[h][i].y);
          }
        };
        if (kfl - k0 > 8) halves(std::integral_constant<int, 2>{});
        else halves(std::integral_constant<int, 1>{});
        __syncwarp();
        if (lane == 0 && !dead) tck::mbar_arrive(&empty[s]);
      }
      // The products of this term go into the box: every (row, column) is one distinct element, and a term's rows and
      // columns are the whole box.  Another warp may hold the same element in the term before (or, for the first term,
      // still read it out): a warp waits for all warps' additions of that term (for the box before to have left), and
      // has its own term's products meanwhile.  Eight elements are read before any is written: one by one, which is
      // what the compiler must do where they could meet, costs sixteen round trips.
      const int32_t* pm = s_pos + k * 2 * kBox + wm0 + t;
      const int32_t* pn = s_pos + k * 2 * kBox + kBox + wn0 + pg;
      const double alpha = p.term[k].alpha;
      int qm[8], qn[2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) qm[2 * i + h] = pm[8 * i + 4 * h];
#pragma unroll
      for (int j = 0; j < 2; ++j) qn[j] = pn[8 * j];
      if (!dead && !(k == 0 ? boxes == 0 || box_wait(left, (boxes - 1) & 1, p.status, 4, p.spin_limit) : box_wait(added, (terms - 1) & 1, p.status, 5, p.spin_limit)))
        dead = true;
      if (k == 0) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if ((qm[i] | qn[j]) >= 0) *reinterpret_cast<double*>(box_b + (qm[i] ^ qn[j])) = alpha * acc[j][i >> 1][i & 1];
      } else if (p.term[k].full) {  // 64 rows and columns: nothing to test
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double old[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) old[i] = *reinterpret_cast<const double*>(box_b + (qm[i] ^ qn[j]));
#pragma unroll
          for (int i = 0; i < 8; ++i) *reinterpret_cast<double*>(box_b + (qm[i] ^ qn[j])) = fma(alpha, acc[j][i >> 1][i & 1], old[i]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double old[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if ((qm[i] | qn[j]) >= 0) old[i] = *reinterpret_cast<const double*>(box_b + (qm[i] ^ qn[j]));
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if ((qm[i] | qn[j]) >= 0) *reinterpret_cast<double*>(box_b + (qm[i] ^ qn[j])) = fma(alpha, acc[j][i >> 1][i & 1], old[i]);
        }
      }
      __syncwarp();
      if (lane == 0 && !dead) tck::mbar_arrive(added);
      ++terms;
    }
    // ---- the box is added to C: the old values are on their way before the last term's additions are waited for ----
    double old[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) old[i] = valid(crd_lo + s_crd_hi[i], last) ? C[base + off_lo + s_off_hi[i]] : 0.0;
    if (!__all_sync(0xffffffffu, !dead && box_wait(added, (terms - 1) & 1, p.status, 6, p.spin_limit))) return;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (valid(crd_lo + s_crd_hi[i], last)) C[base + off_lo + s_off_hi[i]] = old[i] + box[pos_lo ^ box_hash((uint32_t)i << 8)];
    __syncwarp();
    if (lane == 0) tck::mbar_arrive(left);
  }
}

constexpr int box_smem_bytes() { return kBoxStages * 2 * kImgBytes + kBoxElems * 8 + kMaxTerms * 2 * kBox * 4 + (2 * kBoxStages + 2) * 8 + 32 * 8; }

}  // namespace tcbox
