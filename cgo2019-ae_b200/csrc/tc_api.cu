// C ABI: plan / execute / free, the seeded input generator and small utilities.
// Declarations and the reference interfaces they replace are in include/tc_b200.h.
#include <cuda_runtime.h>
#include <stdlib.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>

#include "tc_inst.cuh"
#include "tc_internal.h"
#include "tc_tensor_map.h"

// ---------------------------------------------------------------- errors ----
static thread_local char g_cuda_error[256] = "";

void tc_note_cuda_error(int code, const char* what) {
  std::snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s (%d)", what, cudaGetErrorString((cudaError_t)code), code);
}

extern "C" const char* tc_last_cuda_error(void) { return g_cuda_error; }

extern "C" const char* tc_status_string(int s) {
  switch (s) {
    case TC_OK: return "ok";
    case TC_ERR_PARSE: return "expression rejected by the grammar";
    case TC_ERR_INVALID_ARG: return "invalid argument";
    case TC_ERR_UNSUPPORTED: return "unsupported contraction";
    case TC_ERR_EXTENT: return "bad extent or stride";
    case TC_ERR_CUDA: return "CUDA error";
    case TC_ERR_ALIGNMENT: return "misaligned tensor pointer";
    case TC_ERR_STATE: return "call order violated";
    case TC_ERR_WORKSPACE: return "workspace missing or too small";
    case TC_ERR_DEVICE_WAIT: return "a bounded wait inside a kernel gave up";
    default: return "unknown status";
  }
}

extern "C" const char* tc_version(void) { return "tc_b200 0.2 (sm_100a)"; }

static void copy_out(const std::string& s, char* buf, size_t cap) {
  if (!buf || cap == 0) return;
  const size_t n = std::min(cap - 1, s.size());
  std::memcpy(buf, s.data(), n);
  buf[n] = '\0';
}

// ------------------------------------------------------------ expression ----
extern "C" int tc_expr_describe(const char* expr, char* buf, size_t cap) {
  TcExpr e;
  std::string why;
  const int st = tc_parse_expr(expr, &e, &why);
  copy_out(st == TC_OK ? tc_expr_to_json(e) : "{\"error\":\"" + why + "\"}", buf, cap);
  return st;
}

// -------------------------------------------------------- kernel dispatch ----
#include "tc_kernel_list.h"

#define TC_DECLARE(NAME, T, MATH, BM, BN, WMN, WNN, STAGES, MINB, VARIANT) \
  extern "C" int tc_inst_##NAME(int, int, const TcKernelArgs*, void*, const void*, const void*, cudaStream_t, int, int*, int*);
TC_KERNEL_LIST(TC_DECLARE)
#undef TC_DECLARE
#define TC_DECLARE_WS(NAME, BM, BN, STAGES, VARIANT) \
  extern "C" int tc_inst_##NAME(int, int, const TcKernelArgs*, void*, const void*, const void*, cudaStream_t, int, int*, int*);
TC_WS_KERNEL_LIST(TC_DECLARE_WS)
#undef TC_DECLARE_WS
#define TC_DECLARE_WC(NAME, BM, BN, WGM, WGN, STAGES, VARIANT) \
  extern "C" int tc_inst_##NAME(int, int, const TcKernelArgs*, void*, const void*, const void*, cudaStream_t, int, int*, int*);
TC_WC_KERNEL_LIST(TC_DECLARE_WC)
#undef TC_DECLARE_WC
#define TC_DECLARE_WT(NAME, BM, VARIANT) \
  extern "C" int tc_inst_##NAME(int, int, const TcKernelArgs*, void*, const void*, const void*, cudaStream_t, int, int*, int*);
TC_WT_KERNEL_LIST(TC_DECLARE_WT)
#undef TC_DECLARE_WT

namespace {
struct KernelEntry {
  const char* name;
  int dtype, math, bm, bn, variant;
  tc_inst_fn fn;
};
template <typename T> constexpr int dtype_of() { return sizeof(T) == 8 ? TC_F64 : TC_F32; }
#define TC_ENTRY(NAME, T, MATH, BM, BN, WMN, WNN, STAGES, MINB, VARIANT) {#NAME, dtype_of<T>(), MATH, BM, BN, VARIANT, tc_inst_##NAME},
#define TC_WS_ENTRY(NAME, BM, BN, STAGES, VARIANT) {#NAME, TC_F64, TC_MATH_DMMA, BM, BN, VARIANT, tc_inst_##NAME},
#define TC_WC_ENTRY(NAME, BM, BN, WGM, WGN, STAGES, VARIANT) {#NAME, TC_F64, TC_MATH_DMMA, BM, BN, VARIANT, tc_inst_##NAME},
#define TC_WT_ENTRY(NAME, BM, VARIANT) {#NAME, TC_F32, TC_MATH_TF32TC, BM, 128, VARIANT, tc_inst_##NAME},
const KernelEntry kKernels[] = {TC_KERNEL_LIST(TC_ENTRY) TC_WS_KERNEL_LIST(TC_WS_ENTRY) TC_WC_KERNEL_LIST(TC_WC_ENTRY)
                                TC_WT_KERNEL_LIST(TC_WT_ENTRY)};
#undef TC_WT_ENTRY
#undef TC_ENTRY
#undef TC_WS_ENTRY
#undef TC_WC_ENTRY

const KernelEntry* find_kernel(int dtype, int math, int bm, int bn, int variant) {
  for (const KernelEntry& k : kKernels)
    if (k.dtype == dtype && k.math == math && k.bm == bm && k.bn == bn && k.variant == variant) return &k;
  return nullptr;
}
}  // namespace

bool tc_kernel_exists(int dtype, int math, int bm, int bn, int variant) {
  return find_kernel(dtype, math, bm, bn, variant) != nullptr;
}

const char* tc_kernel_name(const TcKernelChoice& c) {
  const KernelEntry* k = find_kernel(c.dtype, c.math, c.bm, c.bn, c.variant);
  return k ? k->name : "?";
}

static tc_inst_fn pick_inst(const TcKernelChoice& c) {
  const KernelEntry* k = find_kernel(c.dtype, c.math, c.bm, c.bn, c.variant);
  return k ? k->fn : nullptr;
}

static int mode_of(bool ext_vec, bool k_vec) { return ext_vec ? 1 : k_vec ? 2 : 0; }

// The transposed operand matrix (fp32): dimension 0 = flattened external index (stride 1), dimension 1 = contraction
// index at `pitch` elements; box = rows x kbox, no swizzle, zero fill outside the tensor.
static bool encode_operand_map_ext(TcTensorMap* out, const void* base, uint64_t ext_extent, uint64_t k_extent,
                                   uint64_t pitch, uint32_t rows, uint32_t kbox = TC_BK) {
  const tc_encode_fn fn = tc_tensor_map_encoder();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) || (pitch * 4) % 16 != 0 || rows > 256 || rows % 4 != 0) return false;
  const cuuint64_t dims[2] = {ext_extent, k_extent};
  const cuuint64_t strides[1] = {pitch * 4};
  const cuuint32_t box[2] = {rows, kbox};
  const cuuint32_t estr[2] = {1, 1};
  return fn(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tiled TMA descriptor of an operand seen as a 2-D matrix of `es`-byte elements: dimension 0 = contraction index
// (stride 1), dimension 1 = flattened external index at `pitch` elements; box = kbox x rows, swizzled over the box
// row (128 bytes for fp64 and pairs of fp32 K steps, 64 for one fp32 K step), zero fill outside the tensor.
static bool encode_operand_map(TcTensorMap* out, const void* base, uint64_t k_extent, uint64_t ext_extent,
                               uint64_t pitch, uint32_t rows, int es = 8, uint32_t kbox = TC_BK) {
  const tc_encode_fn fn = tc_tensor_map_encoder();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) || (pitch * es) % 16 != 0 || rows > 256) return false;
  const cuuint64_t dims[2] = {k_extent, ext_extent};
  const cuuint64_t strides[1] = {pitch * (uint64_t)es};
  const cuuint32_t box[2] = {kbox, rows};
  const cuuint32_t estr[2] = {1, 1};
  static_assert(sizeof(CUtensorMap) == sizeof(TcTensorMap), "tensor map storage");
  return fn(reinterpret_cast<CUtensorMap*>(out), es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
            const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            kbox * es == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Rank-5 tiled TMA descriptor of the fp64 output for the persistent kernel's epilogue.  Dimensions, fastest
// first: the contiguous run of the fastest M dimensions; the parity of n; n / 2 inside N's fastest dimensions;
// then the remaining N and M dimensions (at most two together, padded with extent 1).
// Box = (bw, bh, bq, 1, 1): (warp rows, 1, 8) for the 8 rows one consumer warp stages at a time, or
// (bm, 2, bn / 2) for a whole tile.  No swizzle, no fill.
static bool encode_output_map(TcTensorMap* out, const void* base, const TcOutMap& o, uint32_t bw, uint32_t bh,
                              uint32_t bq) {
  const tc_encode_fn fn = tc_tensor_map_encoder();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) || bw > 256 || bq > 256 || o.e0 == 0 || o.f0 < 2 || o.ne + o.me > 2) return false;
  cuuint64_t dims[5] = {o.e0, 2, o.f0 / 2, 1, 1};
  cuuint64_t strides[4] = {(cuuint64_t)o.stride_n * 8, (cuuint64_t)o.stride_n * 16, 0, 0};
  int r = 3;
  for (int d = 0; d < o.ne + o.me; ++d, ++r) { dims[r] = o.ext[d]; strides[r - 1] = (cuuint64_t)o.stride[d] * 8; }
  for (; r < 5; ++r) strides[r - 1] = strides[r - 2] * dims[r - 1];  // extent-1 padding: any aligned stride
  for (int i = 0; i < 4; ++i)
    if (strides[i] % 16 != 0 || strides[i] >= (cuuint64_t(1) << 40)) return false;
  const cuuint32_t box[5] = {bw, bh, bq, 1, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return fn(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, const_cast<void*>(base), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same output as the boxes of the output-resident kernel's cut tiles (TcBoxMap).
static bool encode_box_output_map(TcTensorMap* out, const void* base, const TcBoxMap& o) {
  const tc_encode_fn fn = tc_tensor_map_encoder();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) || o.rank < 1 || o.rank > 5) return false;
  cuuint64_t dims[5] = {1, 1, 1, 1, 1}, strides[4];
  cuuint32_t box[5] = {1, 1, 1, 1, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  for (int d = 0; d < o.rank; ++d) {
    dims[d] = o.ext[d];
    box[d] = o.box[d];
    if (d > 0) strides[d - 1] = (cuuint64_t)o.stride[d] * 8;
    if (box[d] > 256) return false;
  }
  for (int d = std::max(o.rank, 1); d < 5; ++d) strides[d - 1] = d > 1 ? strides[d - 2] * dims[d - 1] : (dims[0] + 1) / 2 * 16;  // extent-1 padding
  for (int i = 0; i < 4; ++i)
    if (strides[i] % 16 != 0 || strides[i] >= (cuuint64_t(1) << 40)) return false;
  return fn(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, const_cast<void*>(base), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int tc_kernel_shape(const TcKernelChoice& c, int* threads, int* smem_bytes, int* bk) {
  if (bk) *bk = TC_BK;
  tc_inst_fn fn = pick_inst(c);
  if (!fn) return TC_ERR_UNSUPPORTED;
  return fn(mode_of(c.vec_x, c.kvec_x), mode_of(c.vec_y, c.kvec_y), nullptr, nullptr, nullptr, nullptr, nullptr, TC_INST_QUERY, threads, smem_bytes);
}

static int kernels_prepare_one(const TcKernelChoice& c);
int tc_kernels_prepare(const TcKernelChoice& c) {
  int st = kernels_prepare_one(c);
  if (st == TC_OK && tc_kernel_is_c_resident(c)) {  // its stand-in for outputs the copy engine cannot address as boxes
    TcKernelChoice alt = c;
    alt.variant = 2;
    st = kernels_prepare_one(alt);
  }
  if (st == TC_OK && c.pair) {  // compiled with the persistent kernel of single CTAs
    TcKernelChoice alt = c;
    alt.variant = 1;
    st = kernels_prepare_one(alt);
  }
  if (st == TC_OK && tc_kernel_is_tmem_persistent(c)) {  // its stand-in for outputs without 16-byte alignment
    TcKernelChoice alt = c;
    alt.variant = 0;
    st = kernels_prepare_one(alt);
  }
  return st;
}
static int kernels_prepare_one(const TcKernelChoice& c) {
  // Both loader variants of each operand: a misaligned base pointer at execute
  // time demotes 16-byte loads to element loads.
  tc_inst_fn fn = pick_inst(c);
  if (!fn) return TC_ERR_UNSUPPORTED;
  const int mx = mode_of(c.vec_x, c.kvec_x), my = mode_of(c.vec_y, c.kvec_y);
  const bool ws = tc_kernel_is_persistent(c) && (c.math == TC_MATH_DMMA || tc_kernel_is_tmem_persistent(c));
  const bool wt = tc_kernel_is_tmem_persistent(c);
  const int xs[4] = {0, mx, (ws && c.tma_x) ? 3 : 0, (wt && c.tma_xe) ? 4 : 0};
  const int ys[4] = {0, my, (ws && c.tma_y) ? 3 : 0, (wt && c.tma_ye) ? 4 : 0};
  for (int vx : xs)
    for (int vy : ys) {
      const int st = fn(vx, vy, nullptr, nullptr, nullptr, nullptr, nullptr, TC_INST_PREPARE, nullptr, nullptr);
      if (st != TC_OK) return st;
    }
  return TC_OK;
}

// Resident CTAs of the chosen kernel on the whole device (0 on failure).
static int resident_ctas(const TcKernelChoice& c) {
  tc_inst_fn fn = pick_inst(c);
  int per_sm = 0, dev = 0, sms = 0;
  if (!fn || fn(mode_of(c.vec_x, c.kvec_x), mode_of(c.vec_y, c.kvec_y), nullptr, nullptr, nullptr, nullptr, nullptr, TC_INST_OCCUPANCY, &per_sm, nullptr) != TC_OK) return 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return per_sm * sms;
}

int tc_launch_contraction(const tc_plan& p, const TcKernelArgs& args, void* C, const void* X, const void* Y,
                          cudaStream_t stream) {
  const TcKernelChoice& c = p.choice;
  TcKernelArgs a = args;
  // Alignment-driven demotions (base pointers are the only run-time unknowns).
  const bool x16 = (reinterpret_cast<uintptr_t>(X) & 15) == 0, y16 = (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
  const uintptr_t cu = reinterpret_cast<uintptr_t>(C);
  if ((cu & 15) != 0) a.vec_c = 1;
  int vx = x16 ? mode_of(c.vec_x, c.kvec_x) : 0, vy = y16 ? mode_of(c.vec_y, c.kvec_y) : 0;
  // The C-resident kernel moves whole output tiles as boxes of a view of C: the view must exist and the base must be
  // 16-byte aligned.  Otherwise the same tiles run on the persistent kernel that reaches C through reduce-adds or plain
  // read-modify-writes.
  const bool resident = tc_kernel_is_c_resident(c) && c.box_c && encode_box_output_map(&a.tmap_ct, C, a.cbox);
  // Persistent kernels fetch operands that are plain 2-D matrices with one tiled TMA copy per stage.
  if (tc_kernel_is_persistent(c) && c.math == TC_MATH_DMMA && p.opt.tma != 1) {
    const bool operands = p.opt.tma == 0 || p.opt.tma == 2 || p.opt.tma == 4, output = !resident && (p.opt.tma == 0 || p.opt.tma == 3 || p.opt.tma == 4);
    if (operands && c.tma_x && encode_operand_map(&a.tmap_x, X, a.Kflat, a.Mflat, (uint64_t)a.M.s_in[0], (uint32_t)a.bm)) vx = 3;
    if (operands && c.tma_y && encode_operand_map(&a.tmap_y, Y, a.Kflat, a.Nflat, (uint64_t)a.N.s_in[0], (uint32_t)a.bn)) vy = 3;
    a.c_tensor = (output && c.tma_c && a.c_mode == 2 &&
                  encode_output_map(&a.tmap_c, C, a.cmap, (uint32_t)a.bm / 2 /* rows of a consumer warp's block */, 1, 8)) ? 1 : 0;
    if (a.c_tensor == 1 && c.tma_ct && p.opt.tma != 4 &&
        encode_output_map(&a.tmap_ct, C, a.cmap, (uint32_t)a.bm, 2, (uint32_t)a.bn / 2))
      a.c_tensor = 2;
  }
  tc_inst_fn fn = pick_inst(c);
  int passes = p.passes;
  auto operand_boxes = [&](uint32_t kbox) {  // fp32 operands that are plain matrices, in either orientation
    if (c.tma_x && encode_operand_map(&a.tmap_x, X, a.Kflat, a.Mflat, (uint64_t)a.M.s_in[0], (uint32_t)a.bm, 4, kbox)) vx = 3;
    if (c.tma_y && encode_operand_map(&a.tmap_y, Y, a.Kflat, a.Nflat, (uint64_t)a.N.s_in[0], (uint32_t)a.bn, 4, kbox)) vy = 3;
    if (c.tma_xe && encode_operand_map_ext(&a.tmap_x, X, a.Mflat, a.Kflat, (uint64_t)p.kdims.s_in[0], (uint32_t)a.bm, kbox)) vx = 4;
    if (c.tma_ye && encode_operand_map_ext(&a.tmap_y, Y, a.Nflat, a.Kflat, (uint64_t)p.kdims.s_out[0], (uint32_t)a.bn, kbox)) vy = 4;
  };
  if (c.pair && (cu & 15) == 0 && x16 && y16) {
    const int mx = vx, my = vy;
    operand_boxes(32);
    a.pair = vx >= 3 && vy >= 3;
    if (!a.pair) { vx = mx; vy = my; }
  }
  if (a.pair) {
    TcKernelChoice alt = c;
    alt.variant = 1;  // (the pairs' kernel is compiled with the single CTAs' one)
    fn = pick_inst(alt);
    passes = 1;
    a.tiles_m = (a.Mflat + 255) / 256;
    a.tiles_n = (a.Nflat + 255) / 256;
    a.mblock_w = a.tiles_m > 32 && a.tiles_n > 1 ? 16 : 0;
    if (!fn) return TC_ERR_UNSUPPORTED;
    __atomic_store_n(&p.ran, (int)TC_ROUTE_PAIRS, __ATOMIC_RELAXED);
    return fn(vx, vy, &a, C, X, Y, stream, TC_INST_LAUNCH, nullptr, nullptr);
  }
  // (a plan for the pairs that runs without them: on the single CTAs' kernel of its variant)
  TcRoute route = c.pair ? TC_ROUTE_KERNEL : tc_plan_route(p);
  if (tc_kernel_is_c_resident(c) && !resident) {
    route = TC_ROUTE_STANDIN;
    a.vec_c = std::min(a.vec_c, a.standin_vec_c);
    TcKernelChoice alt = c;
    alt.variant = 2;
    fn = pick_inst(alt);
  }
  if (tc_kernel_is_tmem_persistent(c) && ((cu & 15) != 0 || p.opt.c_path == 2)) {
    // The persistent tcgen05 kernel moves its output tiles as bulk copies of 16-byte aligned chunks; an output
    // without that alignment (or accumulators that are to start from the output) runs the same tiles one CTA per tile.
    route = TC_ROUTE_STANDIN;
    TcKernelChoice alt = c;
    alt.variant = 0;
    fn = pick_inst(alt);
    // ... as sequential passes where the persistent kernel would have cut the accumulation chain itself
    const int64_t steps = (a.Kflat + TC_BK - 1) / TC_BK, want = (steps + 31) / 32;
    if (want > 1) {
      passes = (int)want;
      a.k_chunk = (uint32_t)(((steps + want - 1) / want) * TC_BK);
    }
  } else if (tc_kernel_is_tmem_persistent(c)) {
    // Operands that are plain 2-D matrices -- contraction index fastest, or the flattened external index fastest and
    // the contraction index at a constant pitch -- arrive as one tiled TMA box per stage.  A box always holds sixteen
    // k: contraction lengths that would leave more than a fifth of the boxes' k outside the tensor keep the
    // per-thread copies (K = 24: boxes of either kind measured 2-3 % slower; long contractions a fifth faster).
    const bool boxes_pay = (uint64_t)a.Kflat * 5 >= (uint64_t)((a.Kflat + TC_BK - 1) / TC_BK * TC_BK) * 4;
    if (p.opt.tma != 1 && p.opt.tma != 3 && boxes_pay) operand_boxes(TC_BK);
    // How the kernel's shared memory is carved.  Short contractions are bound by the output stream: tile buffers,
    // so that enough of C is in flight.  Long ones are bound by the MMAs: one tile buffer, a second image set and
    // every operand stage that fits.  (Swept on B200 over both kernels and contractions of 24 to 2048: no other
    // split of the 227 KB measured more than a per cent better; one buffer on short contractions a sixth worse.)
    const int64_t steps = (a.Kflat + TC_BK - 1) / TC_BK;
    a.out_bufs = steps >= 16 ? 1 : (a.bm <= 96 ? 3 : 2);
    a.img_sets = steps >= 16 ? 2 : 1;
    int stages = 0;
    const int st = fn(vx, vy, &a, nullptr, nullptr, nullptr, nullptr, TC_INST_CARVE, &stages, nullptr);
    if (st != TC_OK) return st;
    a.ring_stages = stages;
  }
  if (!fn) return TC_ERR_UNSUPPORTED;
  __atomic_store_n(&p.ran, (int)route, __ATOMIC_RELAXED);
  // Plans whose contraction runs as sequential passes (fp32 tensor-core chains kept short on outputs too large
  // for slice scratch): one launch per range of k, the first with the expression's operator, the rest adding.
  for (int pass = 0; pass < passes; ++pass) {
    TcKernelArgs b = a;
    if (passes > 1) {
      b.k_first = (uint32_t)pass * a.k_chunk;
      b.Kflat = std::min<uint32_t>(a.Kflat, b.k_first + a.k_chunk);
      if (pass > 0) b.beta = 1;
    }
    const int st = fn(vx, vy, &b, C, X, Y, stream, TC_INST_LAUNCH, nullptr, nullptr);
    if (st != TC_OK) return st;
  }
  if (a.ksplit > 1) {
    const unsigned tiles = a.tiles_m * a.tiles_n, most = (unsigned)(a.bm * a.bn + 255) / 256;
    const unsigned want = (8u * (unsigned)p.sm_count + tiles - 1) / tiles;  // eight CTAs of 256 threads fill an SM
    const dim3 grid(tiles, std::max(1u, std::min(want, most)));
    const size_t smem = (size_t)(a.bm + a.bn) * sizeof(int64_t);
    if (p.dtype == TC_F64) TC_CUDA_OK(tck::launch_chained(true, tck::tc_combine_kernel<double>, grid, 256, smem, stream, a, static_cast<double*>(C)));
    else TC_CUDA_OK(tck::launch_chained(true, tck::tc_combine_kernel<float>, grid, 256, smem, stream, a, static_cast<float*>(C)));
  }
  return TC_OK;
}

// ------------------------------------------------------------------ plan ----
extern "C" int tc_plan_create(const char* expr, int dtype, const tc_options* options, tc_plan** out) {
  if (!expr || !out) return TC_ERR_INVALID_ARG;
  *out = nullptr;
  if (dtype != TC_F64 && dtype != TC_F32) return TC_ERR_INVALID_ARG;
  TcExpr e;
  std::string why;
  const int st = tc_parse_expr(expr, &e, &why);
  if (st != TC_OK) return st;
  tc_plan* p = new (std::nothrow) tc_plan();
  if (!p) return TC_ERR_INVALID_ARG;
  p->expr = e;
  p->dtype = dtype;
  if (options) p->opt = *options;
  if (p->opt.path < TC_PATH_AUTO || p->opt.path > TC_PATH_TCGEN05 || p->opt.split_k < 0 || p->opt.test_fault < 0 ||
      p->opt.test_fault > 1) {
    delete p;
    return TC_ERR_INVALID_ARG;
  }
  p->host_mu = new (std::nothrow) std::mutex();
  if (!p->host_mu) { delete p; return TC_ERR_INVALID_ARG; }
  for (size_t i = 0; i < e.out_idx.size(); ++i) { p->idx_names.push_back(e.out_idx[i]); p->idx_extent.push_back(e.out_ext[i]); }
  for (size_t i = 0; i < e.sum_idx.size(); ++i) { p->idx_names.push_back(e.sum_idx[i]); p->idx_extent.push_back(e.sum_ext[i]); }
  *out = p;
  return TC_OK;
}

extern "C" int tc_plan_set_extents(tc_plan* p, int n, const char* const* names, const int64_t* extents) {
  if (!p || n < 0 || (n > 0 && (!names || !extents))) return TC_ERR_INVALID_ARG;
  if (p->committed) return TC_ERR_STATE;
  std::vector<int64_t> next = p->idx_extent;
  for (int i = 0; i < n; ++i) {
    if (!names[i]) return TC_ERR_INVALID_ARG;
    if (extents[i] <= 0) return TC_ERR_EXTENT;
    size_t j = 0;
    for (; j < p->idx_names.size(); ++j)
      if (p->idx_names[j] == names[i]) break;
    if (j == p->idx_names.size()) return TC_ERR_INVALID_ARG;
    next[j] = extents[i];
  }
  p->idx_extent = next;
  return TC_OK;
}

extern "C" int tc_plan_set_extents_ordered(tc_plan* p, int n, const int64_t* extents) {
  if (!p || n < 0 || (n > 0 && !extents)) return TC_ERR_INVALID_ARG;
  if (p->committed) return TC_ERR_STATE;
  if ((size_t)n != p->idx_names.size()) return TC_ERR_INVALID_ARG;
  for (int i = 0; i < n; ++i)
    if (extents[i] <= 0) return TC_ERR_EXTENT;
  p->idx_extent.assign(extents, extents + n);
  return TC_OK;
}

extern "C" int tc_plan_set_strides(tc_plan* p, int tensor, int n, const int64_t* strides) {
  if (!p || tensor < 0 || tensor > 2 || n < 0 || (n > 0 && !strides)) return TC_ERR_INVALID_ARG;
  if (p->committed) return TC_ERR_STATE;
  const size_t rank = tensor == 0 ? p->expr.out_idx.size() : tensor == 1 ? p->expr.left_idx.size() : p->expr.right_idx.size();
  if ((size_t)n != rank) return TC_ERR_INVALID_ARG;
  for (int i = 0; i < n; ++i)
    if (strides[i] <= 0) return TC_ERR_EXTENT;
  p->strides[tensor].assign(strides, strides + n);
  p->custom_strides[tensor] = true;
  return TC_OK;
}

// K-slice scratch that lives in the library image instead of in allocated memory (tc_execute_noalloc).
// Every GPU that loads the library carries these 8 MiB until the process exits.
static __device__ __align__(256) unsigned char g_tc_static_ws[TC_NOALLOC_MAX_WORKSPACE_BYTES];

namespace {
constexpr int kMaxDevices = 64;
// Device address of g_tc_static_ws per device.  In host code the array's name is only a handle for
// the runtime, not an address a kernel can use; the real address comes from cudaGetSymbolAddress,
// asked once per device with that device current.
void* g_static_ws_addr[kMaxDevices] = {};
int g_sm_count[kMaxDevices] = {};

// Resolves the static scratch array on the current device (once) and makes sure the combine kernels'
// module is resident, so that an allocation-free execute later neither looks anything up nor triggers
// the lazy load of that module (which allocates device memory).
int prepare_static_scratch(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return TC_ERR_STATE;
  if (__atomic_load_n(&g_static_ws_addr[dev], __ATOMIC_ACQUIRE)) return TC_OK;
  void* addr = nullptr;
  TC_CUDA_OK(cudaGetSymbolAddress(&addr, g_tc_static_ws));
  if (!addr) return TC_ERR_CUDA;
  cudaFuncAttributes fa;
  TC_CUDA_OK(cudaFuncGetAttributes(&fa, tck::tc_combine_kernel<double>));
  TC_CUDA_OK(cudaFuncGetAttributes(&fa, tck::tc_combine_kernel<float>));
  __atomic_store_n(&g_static_ws_addr[dev], addr, __ATOMIC_RELEASE);  // same value from every thread
  return TC_OK;
}

int device_sm_count(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return TC_DEFAULT_SMS;
  int n = __atomic_load_n(&g_sm_count[dev], __ATOMIC_RELAXED);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return TC_DEFAULT_SMS;
  __atomic_store_n(&g_sm_count[dev], n, __ATOMIC_RELAXED);
  return n;
}
}  // namespace

extern "C" int tc_plan_commit(tc_plan* p) {
  if (!p) return TC_ERR_INVALID_ARG;
  if (p->committed) return TC_OK;
  int dev = 0;
  TC_CUDA_OK(cudaGetDevice(&dev));
  p->sm_count = device_sm_count(dev);  // the tile rules fill THIS device's multiprocessors
  int st = tc_plan_build(p, &p->why);
  if (st != TC_OK) return st;
  st = tc_kernels_prepare(p->choice);
  if (st != TC_OK) return st;
  // How the result reaches C (tc_options.c_path) and whether output tiles are prefetched into L2.
  // Defaults follow the B200 measurements: persistent kernels hand their tiles to the memory system as
  // bulk reduce-adds and need no prefetch; the one-CTA-per-tile kernels read-modify-write behind a prefetch.
  const bool persistent = tc_kernel_is_persistent(p->choice);
  const int c_path = p->opt.c_path;
  p->args.c_mode = c_path > 0 ? c_path - 1 : ((persistent || p->choice.math != TC_MATH_DMMA) ? 2 : 0);
  // The persistent tcgen05 kernel stages the output tile in shared memory either way: by default the tile holds the
  // products only and leaves as bulk reduce-adds (measured faster on every shape tried: 0.292 against 0.311 ms on the
  // fp32 benchmark configuration); with c_path 1 the tile's old values are fetched and the sums stored.
  if (tc_kernel_is_tmem_persistent(p->choice)) p->args.c_mode = c_path == 1 ? 0 : 2;
  p->args.c_stream = 0;
  const bool bulk_out = p->args.c_mode == 2 && (persistent || p->args.epi_run > 0);
  // ... unless the whole problem is a fraction of one wave: then the tile is in flight anyway and the prefetch
  // only lengthens a latency-bound kernel (measured on the 64 x 48 x 32 configuration: 10.7 -> 9.4 us).
  const bool tiny = (int64_t)p->args.tiles_m * p->args.tiles_n * p->args.ksplit < p->sm_count;
  const bool prefetch = p->opt.l2_prefetch == 2 || (p->opt.l2_prefetch == 0 && !bulk_out && !tiny);
  p->args.prefetch_dist = prefetch ? (uint32_t)resident_ctas(p->choice) : 0u;
  p->args.spin_limit = p->opt.test_fault ? (1u << 14) : TC_SPIN_LIMIT;
  p->args.test_fault = p->opt.test_fault;
  const size_t kb = p->h_koff_x.size() * sizeof(int64_t);
  TC_CUDA_OK(cudaMalloc(&p->d_koff, 2 * kb));
  TC_CUDA_OK(cudaMemcpy(p->d_koff, p->h_koff_x.data(), kb, cudaMemcpyHostToDevice));
  TC_CUDA_OK(cudaMemcpy(static_cast<char*>(p->d_koff) + kb, p->h_koff_y.data(), kb, cudaMemcpyHostToDevice));
  p->args.koff_x = static_cast<const int64_t*>(p->d_koff);
  p->args.koff_y = p->args.koff_x + p->h_koff_x.size();
  if (p->ws_bytes) {
    TC_CUDA_OK(cudaMalloc(&p->d_ws, p->ws_bytes));
    if (p->ws_bytes <= (size_t)TC_NOALLOC_MAX_WORKSPACE_BYTES) {  // the plan may later run through tc_execute_noalloc
      st = prepare_static_scratch(dev);
      if (st != TC_OK) return st;
    }
  }
  TC_CUDA_OK(cudaMalloc(&p->d_status, sizeof(int)));
  TC_CUDA_OK(cudaMemset(p->d_status, 0, sizeof(int)));
  p->args.status = p->d_status;
  p->device = dev;
  p->committed = true;
  return TC_OK;
}

struct TcHostPipe;
static void host_pipe_destroy(TcHostPipe* h);

extern "C" void tc_plan_destroy(tc_plan* p) {
  if (!p) return;
  if (p->d_koff) cudaFree(p->d_koff);
  if (p->d_ws) cudaFree(p->d_ws);
  if (p->d_status) cudaFree(p->d_status);
  host_pipe_destroy(p->host);
  delete p->host_mu;
  delete p;
}

extern "C" int tc_plan_describe(const tc_plan* p, char* buf, size_t cap) {
  if (!p) return TC_ERR_INVALID_ARG;
  if (p->committed) { copy_out(tc_plan_to_json(*p), buf, cap); return TC_OK; }
  // Not committed yet: run the host-side planner on a copy (needs no GPU).
  tc_plan tmp = *p;
  std::string why;
  const int st = tc_plan_build(&tmp, &why);
  if (st != TC_OK) { copy_out("{\"error\":\"" + why + "\"}", buf, cap); return st; }
  tmp.committed = true;
  std::string js = tc_plan_to_json(tmp);
  tmp.committed = false;
  copy_out(js, buf, cap);
  return TC_OK;
}

extern "C" int tc_plan_cost(const tc_plan* p, double* flops, double* bytes) {
  if (!p) return TC_ERR_INVALID_ARG;
  tc_plan tmp = *p;
  if (!p->committed) {
    std::string why;
    const int st = tc_plan_build(&tmp, &why);
    if (st != TC_OK) return st;
  }
  if (flops) *flops = tmp.flops;
  if (bytes) *bytes = tmp.bytes;
  return TC_OK;
}

extern "C" int tc_plan_status(tc_plan* p, int* device_status) {
  if (!p || !device_status) return TC_ERR_INVALID_ARG;
  if (!p->committed) return TC_ERR_STATE;
  // a plain cudaMemcpy is ordered after the legacy stream only: work on non-blocking streams needs this
  TC_CUDA_OK(cudaDeviceSynchronize());
  TC_CUDA_OK(cudaMemcpy(device_status, p->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  return TC_OK;
}

extern "C" int tc_plan_status_reset(tc_plan* p) {
  if (!p) return TC_ERR_INVALID_ARG;
  if (!p->committed) return TC_ERR_STATE;
  TC_CUDA_OK(cudaDeviceSynchronize());
  TC_CUDA_OK(cudaMemset(p->d_status, 0, sizeof(int)));
  return TC_OK;
}

extern "C" int tc_plan_launches(const tc_plan* p) { return p && p->committed ? p->launches : -1; }

extern "C" int tc_plan_workspace_bytes(const tc_plan* p, size_t* bytes) {
  if (!p || !bytes) return TC_ERR_INVALID_ARG;
  if (!p->committed) return TC_ERR_STATE;
  *bytes = p->ws_bytes;
  return TC_OK;
}

// --------------------------------------------------------------- execute ----
static int execute_impl(tc_plan* p, void* C, const void* A, const void* B, void* ws, size_t ws_bytes, void* stream) {
  if (!p || !C || !A || !B) return TC_ERR_INVALID_ARG;
  if (!p->committed) {
    const int st = tc_plan_commit(p);
    if (st != TC_OK) return st;
  }
  int dev = 0;
  TC_CUDA_OK(cudaGetDevice(&dev));
  if (dev != p->device) return TC_ERR_STATE;
  const uintptr_t es = p->dtype == TC_F64 ? 8 : 4;
  if ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & (es - 1))
    return TC_ERR_ALIGNMENT;
  TcKernelArgs a = p->args;
  if (a.ksplit > 1) {
    if (!ws || ws_bytes < p->ws_bytes || (reinterpret_cast<uintptr_t>(ws) & 15)) return TC_ERR_WORKSPACE;
    a.ws = ws;
  }
  const void* X = p->swapped ? B : A;
  const void* Y = p->swapped ? A : B;
  return tc_launch_contraction(*p, a, C, X, Y, static_cast<cudaStream_t>(stream));
}

extern "C" int tc_execute(tc_plan* p, void* C, const void* A, const void* B, void* stream) {
  if (p && !p->committed) {
    const int st = tc_plan_commit(p);
    if (st != TC_OK) return st;
  }
  return execute_impl(p, C, A, B, p ? p->d_ws : nullptr, p ? p->ws_bytes : 0, stream);
}

extern "C" int tc_execute_ws(tc_plan* p, void* C, const void* A, const void* B, void* ws, size_t ws_bytes, void* stream) {
  return execute_impl(p, C, A, B, ws, ws_bytes, stream);
}

// ---------------------------------------------------- execute without allocating ----
// For callers that must not allocate device memory at call time and have none to lend: an application
// whose own pool already owns the whole device (the reference's competitors pre-claim memory this way,
// nwchem-tccg/memory.cu:74-163), or a latency-critical loop where cudaMalloc's implicit device-wide
// synchronisation is not acceptable.  Same work as tc_execute on a committed plan; a plan that slices
// the contraction takes its slice scratch from the static array g_tc_static_ws.
//   * The plan must already be committed (committing uploads tables, which allocates): TC_ERR_STATE otherwise.
//   * Plans that need more than TC_NOALLOC_MAX_WORKSPACE_BYTES of scratch are refused with TC_ERR_WORKSPACE.
//   * tc_plan_commit of a K-sliced plan has already looked up the array's device address and loaded the
//     combine kernels, so this call finds everything resident.  Only if that address is missing (no
//     K-sliced plan was committed on this device through this library image) is it looked up here;
//     such a first call belongs before any stream capture.
//   * All calls on a device share the one array and it keeps whatever the last call left in it.  Nothing
//     in it has to start at zero: every slice overwrites its whole partial tile before the combine step
//     reads it.  Two calls whose kernels overlap on the GPU (different streams) race on it: serialise them.
extern "C" int tc_execute_noalloc(tc_plan* p, void* C, const void* A, const void* B, void* stream) {
  if (!p || !C || !A || !B) return TC_ERR_INVALID_ARG;
  if (!p->committed) return TC_ERR_STATE;
  if (p->ws_bytes > (size_t)TC_NOALLOC_MAX_WORKSPACE_BYTES) return TC_ERR_WORKSPACE;
  int dev = 0;
  TC_CUDA_OK(cudaGetDevice(&dev));
  if (dev != p->device || dev < 0 || dev >= kMaxDevices) return TC_ERR_STATE;
  void* ws = nullptr;
  if (p->ws_bytes) {
    ws = __atomic_load_n(&g_static_ws_addr[dev], __ATOMIC_ACQUIRE);
    if (!ws) {
      const int st = prepare_static_scratch(dev);
      if (st != TC_OK) return st;
      ws = __atomic_load_n(&g_static_ws_addr[dev], __ATOMIC_ACQUIRE);
    }
  }
  return execute_impl(p, C, A, B, ws, (size_t)TC_NOALLOC_MAX_WORKSPACE_BYTES, stream);
}

// Host-pointer path.  The reference's wrapper copies everything in, runs, copies the output back
// (cogent/src/codes/others/tc_pre_CUDA_Malloc.py:6-47, tc_interface.py:1368-1388).  Here the output's
// slowest index is cut into slabs and the slabs are pipelined over two streams: while slab i computes, slab
// i+1 is on its way in and slab i-1 on its way out, so a pass costs about max(bytes in, bytes out) over
// PCIe instead of their sum.  Inputs that carry the cut index as THEIR slowest index travel slab by slab
// too; the others go first, whole.  Device buffers, streams and the slab plans are created on the first
// call and kept with the plan.
//
// Pageable host memory (plain malloc -- what the reference drivers pass, code_main_tccg_02.c:53-62) cannot
// be copied asynchronously, so it travels through pinned bounce buffers owned by the plan: on the way in the
// calling thread fills a bounce buffer (several helper threads share the memcpy) and enqueues its copy; on
// the way out a drain thread enqueues the device-to-host copies behind each slab's kernel and empties the
// bounce buffers into the caller's memory while the next slab is still being staged.
#include <condition_variable>
#include <deque>
#include <map>
#include <memory>
#include <thread>
#include <sched.h>

namespace {

// memcpy shared by helper threads.  One set of them per process, made when a plan first sees pageable memory and joined when the
// last such plan is destroyed: every plan's copies, in and out, from any thread, take their helpers from it, so that neither
// several plans nor a driver that makes plan after plan has more threads than the cores call for.
class CopyPool {
 public:
  static std::shared_ptr<CopyPool> get() {
    static std::mutex mu;
    static std::weak_ptr<CopyPool> kept;
    std::lock_guard<std::mutex> l(mu);
    std::shared_ptr<CopyPool> p = kept.lock();
    if (!p) kept = p = std::make_shared<CopyPool>();
    return p;
  }
  CopyPool() {
    cpu_set_t set;
    const int cores = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : (int)std::thread::hardware_concurrency();
    const int n = std::min(12, std::max(1, cores - 2));  // (beside the caller and the thread that empties the buffers)
    try {
      for (int i = 0; i < n; ++i) workers_.emplace_back([this] { loop(); });
    } catch (const std::exception&) {  // no more threads to be had: with those there are, or the callers alone
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (std::thread& t : workers_) t.join();
  }
  void copy(void* dst, const void* src, size_t bytes) {
    const size_t n = workers_.size();
    if (bytes < (1u << 20) || n == 0) { std::memcpy(dst, src, bytes); return; }
    Job j = {static_cast<char*>(dst), static_cast<const char*>(src), bytes, ((bytes + n) / (n + 1) + 4095) / 4096 * 4096, 0, bytes, nullptr, nullptr};
    std::unique_lock<std::mutex> l(mu_);
    j.prev = last_;
    (last_ ? last_->next : first_) = &j;
    last_ = &j;
    l.unlock();
    cv_.notify_all();
    l.lock();
    while (j.at < j.bytes) take(&j, l);  // the caller copies too
    done_.wait(l, [&] { return j.left == 0; });
  }

 private:
  struct Job {  // lives on its caller's stack until nothing of it is left
    char* dst;
    const char* src;
    size_t bytes, piece, at, left;  // at: first byte that nobody has taken; left: bytes not copied yet
    Job *prev, *next;
  };
  void take(Job* j, std::unique_lock<std::mutex>& l) {
    const size_t lo = j->at, hi = std::min(j->bytes, lo + j->piece);
    j->at = hi;
    if (hi == j->bytes) {  // all of it is taken: out of the queue
      (j->prev ? j->prev->next : first_) = j->next;
      (j->next ? j->next->prev : last_) = j->prev;
    }
    l.unlock();
    std::memcpy(j->dst + lo, j->src + lo, hi - lo);
    l.lock();
    j->left -= hi - lo;
    if (j->left == 0) done_.notify_all();
  }
  void loop() {
    std::unique_lock<std::mutex> l(mu_);
    for (;;) {
      cv_.wait(l, [&] { return stop_ || first_; });
      if (stop_) return;
      take(first_, l);
    }
  }
  std::vector<std::thread> workers_;
  std::mutex mu_;
  std::condition_variable cv_, done_;
  bool stop_ = false;
  Job *first_ = nullptr, *last_ = nullptr;  // jobs with bytes that nobody has taken
};

// Small buffers and many helpers: a copy over the link starts when its buffer is filled, so the first and the last buffer are
// not overlapped with anything.  48^4 outputs and inputs (85 MB in, 42 MB out) on 16 cores, each direction with helpers of its
// own: 9.0 ms with three buffers of 8 MB and four helpers, 6.6 with twelve, 4.9 with 2 MB and six, 4.0 with 2 MB and twelve.
// Twelve for both directions together (in turn, medians): 48^4 3.7 -> 3.6 ms, 56^4 7.1 -> 6.5, 64^4 7.7 -> 6.9, 80^4 17.2 -> 15.1.
// Calls that move more are bound by the host's memory and by the hand-over per piece, and take whole buffers (64^4, 268 MB
// in: 10.5 ms in pieces of 2 MB, 9.5 in 4, 9.8 in 8; 96^4, 1.36 GB in: 51, 39, 47; with six or four helpers 42 to 52).
constexpr size_t kBounceBytes = size_t(4) << 20, kShortPiece = size_t(2) << 20, kShortCall = size_t(192) << 20;
constexpr int kBounceCount = 6;

bool is_pageable(const void* ptr) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) { cudaGetLastError(); return true; }
  return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

struct TcHostPipe {
  void *dC = nullptr, *dA = nullptr, *dB = nullptr;
  cudaStream_t stream[2] = {nullptr, nullptr};
  cudaStream_t out_stream = nullptr;  // device-to-host copies of pageable outputs
  cudaEvent_t inputs_ready = nullptr;
  int cut = -1;                 // position of the cut index in idx_names (-1: no slabs)
  int64_t extent = 1, slab = 1; // extent of the cut index, values per slab
  int64_t step[3] = {0, 0, 0};  // element stride of the cut index where the tensor travels slab by slab (0: whole, first)
  int64_t rest[3] = {0, 0, 0};  // elements one value of the cut index spans in such a tensor
  int64_t view[3] = {0, 0, 0};  // element stride of the cut index in C, A, B (0: the tensor does not carry it)
  tc_plan* plan_slab = nullptr; // slab-sized sub-plan (strides of the full tensors)
  tc_plan* plan_tail = nullptr; // last, shorter slab
  int* h_status = nullptr;      // pinned: status words of the three plans after a call
  // pageable staging
  void* bounce_in[kBounceCount] = {};
  void* bounce_out[kBounceCount] = {};
  size_t piece = kBounceBytes;  // bytes of a buffer that the present call fills
  cudaEvent_t in_done[kBounceCount] = {};
  cudaEvent_t out_done[kBounceCount] = {};
  int in_next = 0;
  std::shared_ptr<CopyPool> pool;
  std::vector<cudaEvent_t> slab_done;  // kernel of slab i finished (recorded on its stream)
  std::vector<cudaEvent_t> slab_in;    // inputs of slab i have arrived (page-locked callers: copies on their own stream)
};

static void host_pipe_destroy(TcHostPipe* h) {
  if (!h) return;
  if (h->dC) cudaFree(h->dC);
  if (h->dA) cudaFree(h->dA);
  if (h->dB) cudaFree(h->dB);
  for (cudaStream_t s : h->stream)
    if (s) cudaStreamDestroy(s);
  if (h->out_stream) cudaStreamDestroy(h->out_stream);
  if (h->inputs_ready) cudaEventDestroy(h->inputs_ready);
  if (h->plan_slab) tc_plan_destroy(h->plan_slab);
  if (h->plan_tail) tc_plan_destroy(h->plan_tail);
  if (h->h_status) cudaFreeHost(h->h_status);
  for (int i = 0; i < kBounceCount; ++i) {
    if (h->bounce_in[i]) cudaFreeHost(h->bounce_in[i]);
    if (h->bounce_out[i]) cudaFreeHost(h->bounce_out[i]);
    if (h->in_done[i]) cudaEventDestroy(h->in_done[i]);
    if (h->out_done[i]) cudaEventDestroy(h->out_done[i]);
  }
  for (cudaEvent_t e : h->slab_done) cudaEventDestroy(e);
  for (cudaEvent_t e : h->slab_in) cudaEventDestroy(e);
  delete h;
}

// Element strides of tensor t (0 output, 1 left, 2 right) in written order: the caller's, or compact.
static std::vector<int64_t> effective_strides(const tc_plan* p, int t) {
  if (p->custom_strides[t]) return p->strides[t];
  const std::vector<std::string>& idx = t == 0 ? p->expr.out_idx : t == 1 ? p->expr.left_idx : p->expr.right_idx;
  std::vector<int64_t> s;
  int64_t acc = 1;
  for (const std::string& n : idx) {
    s.push_back(acc);
    for (size_t j = 0; j < p->idx_names.size(); ++j)
      if (p->idx_names[j] == n) acc *= p->idx_extent[j];
  }
  return s;
}

static int make_slab_plan(const tc_plan* p, int cut, int64_t count, tc_plan** out) {
  tc_plan* q = nullptr;
  // same expression, options and strides; only the cut index is shorter
  q = new (std::nothrow) tc_plan();
  if (!q) return TC_ERR_INVALID_ARG;
  q->expr = p->expr;
  q->dtype = p->dtype;
  q->opt = p->opt;
  q->idx_names = p->idx_names;
  q->idx_extent = p->idx_extent;
  q->idx_extent[cut] = count;
  q->host_mu = new (std::nothrow) std::mutex();
  for (int t = 0; t < 3; ++t) {
    q->strides[t] = effective_strides(p, t);
    q->custom_strides[t] = true;
  }
  const int st = q->host_mu ? tc_plan_commit(q) : TC_ERR_INVALID_ARG;
  if (st != TC_OK) { tc_plan_destroy(q); return st; }
  *out = q;
  return TC_OK;
}

static int host_pipe_create(tc_plan* p) {
  TcHostPipe* h = new (std::nothrow) TcHostPipe();
  if (!h) return TC_ERR_INVALID_ARG;
  p->host = h;
  const size_t es = p->dtype == TC_F64 ? 8 : 4;
  TC_CUDA_OK(cudaMalloc(&h->dC, p->size_c * es));
  TC_CUDA_OK(cudaMalloc(&h->dA, p->size_a * es));
  TC_CUDA_OK(cudaMalloc(&h->dB, p->size_b * es));
  for (cudaStream_t& s : h->stream) TC_CUDA_OK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  TC_CUDA_OK(cudaEventCreateWithFlags(&h->inputs_ready, cudaEventDisableTiming));
  TC_CUDA_OK(cudaMallocHost(reinterpret_cast<void**>(&h->h_status), 4 * sizeof(int)));
  // Slabs for outputs worth pipelining (>= 32 MB) and plans that do not slice K: the cut index is the output
  // index with the largest stride, provided everything else of the output fits below that stride (then a range
  // of its values is one contiguous range of addresses -- compact tensors and per-rank views alike).
  const TcExpr& e = p->expr;
  if (e.out_idx.empty() || p->count_c * (int64_t)es < (32 << 20) || p->args.ksplit > 1) return TC_OK;
  const std::vector<std::string>* tidx[3] = {&e.out_idx, &e.left_idx, &e.right_idx};
  std::vector<int64_t> str[3], ext[3];
  for (int t = 0; t < 3; ++t) {
    str[t] = effective_strides(p, t);
    for (const std::string& n : *tidx[t])
      for (size_t j = 0; j < p->idx_names.size(); ++j)
        if (p->idx_names[j] == n) ext[t].push_back(p->idx_extent[j]);
  }
  int pos = -1;
  for (size_t i = 0; i < e.out_idx.size(); ++i)
    if (ext[0][i] > 1 && (pos < 0 || str[0][i] > str[0][pos])) pos = (int)i;
  if (pos < 0) return TC_OK;
  const std::string& name = e.out_idx[pos];
  int cut = -1;
  for (size_t j = 0; j < p->idx_names.size(); ++j)
    if (p->idx_names[j] == name) cut = (int)j;
  const int64_t extent = p->idx_extent[cut];
  if (extent < 4) return TC_OK;
  // per tensor: does it carry the cut index, and as its outermost one?
  for (int t = 0; t < 3; ++t) {
    int64_t rest = 1, sc = 0;
    for (size_t i = 0; i < tidx[t]->size(); ++i) {
      if ((*tidx[t])[i] == name) sc = str[t][i];
      else rest += (ext[t][i] - 1) * str[t][i];
    }
    h->view[t] = sc;
    if (sc > 0 && rest <= sc) { h->step[t] = sc; h->rest[t] = rest; }
  }
  if (!h->step[0]) { h->view[0] = h->view[1] = h->view[2] = 0; return TC_OK; }  // the output's slabs are not contiguous ranges
  const int64_t nslabs = std::min<int64_t>(extent, 12);
  h->slab = (extent + nslabs - 1) / nslabs;
  h->extent = extent;
  int st = make_slab_plan(p, cut, h->slab, &h->plan_slab);
  if (st != TC_OK) return st;
  if (extent % h->slab) {
    st = make_slab_plan(p, cut, extent % h->slab, &h->plan_tail);
    if (st != TC_OK) return st;
  }
  if (h->plan_slab->args.ksplit > 1 || (h->plan_tail && h->plan_tail->args.ksplit > 1)) return TC_OK;  // keep one stream
  h->cut = cut;
  return TC_OK;
}

// Bounce buffers, helper threads and the drain stream: only plans that ever see pageable memory pay for them.
static int host_pipe_enable_staging(TcHostPipe* h) {
  if (h->pool) return TC_OK;
  for (int i = 0; i < kBounceCount; ++i) {
    TC_CUDA_OK(cudaMallocHost(&h->bounce_in[i], kBounceBytes));
    TC_CUDA_OK(cudaMallocHost(&h->bounce_out[i], kBounceBytes));
    TC_CUDA_OK(cudaEventCreateWithFlags(&h->in_done[i], cudaEventDisableTiming));
    TC_CUDA_OK(cudaEventCreateWithFlags(&h->out_done[i], cudaEventDisableTiming));
  }
  TC_CUDA_OK(cudaStreamCreateWithFlags(&h->out_stream, cudaStreamNonBlocking));
  try {
    h->pool = CopyPool::get();
  } catch (const std::exception&) {
    return TC_ERR_INVALID_ARG;
  }
  return TC_OK;
}

// Host -> device on `s`: directly from pinned memory, through the bounce buffers otherwise.
static int copy_in(TcHostPipe* h, char* dst, const char* src, size_t bytes, bool pageable, cudaStream_t s) {
  if (!pageable) {
    TC_CUDA_OK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    return TC_OK;
  }
  for (size_t off = 0; off < bytes; off += h->piece) {
    const size_t n = std::min(h->piece, bytes - off);
    const int b = h->in_next;
    h->in_next = (b + 1) % kBounceCount;
    TC_CUDA_OK(cudaEventSynchronize(h->in_done[b]));  // the copy that last used this buffer has read it
    h->pool->copy(h->bounce_in[b], src + off, n);
    TC_CUDA_OK(cudaMemcpyAsync(dst + off, h->bounce_in[b], n, cudaMemcpyHostToDevice, s));
    TC_CUDA_OK(cudaEventRecord(h->in_done[b], s));
  }
  return TC_OK;
}

namespace {
// Device -> pageable host, run by the drain thread: ranges become ready in order (each behind an event).
struct DrainJob { const char* src; char* dst; size_t bytes; cudaEvent_t after; };
struct Drain {
  TcHostPipe* h;
  int device;
  std::mutex mu;
  std::condition_variable cv;
  std::deque<DrainJob> jobs;
  bool closed = false;
  int status = TC_OK;
  void push(const DrainJob& j) { { std::lock_guard<std::mutex> l(mu); jobs.push_back(j); } cv.notify_one(); }
  void close() { { std::lock_guard<std::mutex> l(mu); closed = true; } cv.notify_one(); }
  int run_job(const DrainJob& j) {
    TC_CUDA_OK(cudaStreamWaitEvent(h->out_stream, j.after, 0));
    // the copies of the next chunks are in flight while chunk c is emptied into the caller's memory
    size_t issued = 0, drained = 0;
    int bi = 0, bd = 0;
    size_t len[kBounceCount] = {};
    while (drained < j.bytes) {
      while (issued < j.bytes && bi - bd < kBounceCount - 1) {
        const size_t n = std::min(h->piece, j.bytes - issued);
        const int b = bi % kBounceCount;
        TC_CUDA_OK(cudaMemcpyAsync(h->bounce_out[b], j.src + issued, n, cudaMemcpyDeviceToHost, h->out_stream));
        TC_CUDA_OK(cudaEventRecord(h->out_done[b], h->out_stream));
        len[b] = n;
        issued += n;
        ++bi;
      }
      const int b = bd % kBounceCount;
      TC_CUDA_OK(cudaEventSynchronize(h->out_done[b]));
      h->pool->copy(j.dst + drained, h->bounce_out[b], len[b]);
      drained += len[b];
      ++bd;
    }
    return TC_OK;
  }
  void loop() {
    if (cudaSetDevice(device) != cudaSuccess) { status = TC_ERR_CUDA; }
    for (;;) {
      std::unique_lock<std::mutex> l(mu);
      cv.wait(l, [this] { return closed || !jobs.empty(); });
      if (jobs.empty()) return;
      DrainJob j = jobs.front();
      jobs.pop_front();
      l.unlock();
      if (status == TC_OK) status = run_job(j);
    }
  }
};
}  // namespace

static int execute_host_locked(tc_plan* p, void* C, const void* A, const void* B) {
  if (!p->host) {
    const int st = host_pipe_create(p);
    if (st != TC_OK) { host_pipe_destroy(p->host); p->host = nullptr; return st; }
  }
  TcHostPipe* h = p->host;
  const size_t es = p->dtype == TC_F64 ? 8 : 4;
  char* hC = static_cast<char*>(C);
  const char* hA = static_cast<const char*>(A);
  const char* hB = static_cast<const char*>(B);
  char *dC = static_cast<char*>(h->dC), *dA = static_cast<char*>(h->dA), *dB = static_cast<char*>(h->dB);
  const bool page_c = is_pageable(C), page_a = is_pageable(A), page_b = is_pageable(B);
  if (page_c || page_a || page_b) {
    const int st = host_pipe_enable_staging(h);
    if (st != TC_OK) return st;
    h->piece = (p->size_a + p->size_b + p->size_c) * es <= kShortCall ? kShortPiece : kBounceBytes;
  }
  const bool read_c = p->args.beta || p->size_c != p->count_c;
  cudaStream_t s0 = h->stream[0];
  tc_plan* used[3] = {p, nullptr, nullptr};
  int st = TC_OK;

  if (h->cut < 0) {  // one piece
    st = copy_in(h, dA, hA, p->size_a * es, page_a, s0);
    if (st == TC_OK) st = copy_in(h, dB, hB, p->size_b * es, page_b, s0);
    if (st == TC_OK && read_c) st = copy_in(h, dC, hC, p->size_c * es, page_c, s0);
    if (st == TC_OK) st = execute_impl(p, dC, dA, dB, p->d_ws, p->ws_bytes, s0);
    if (st != TC_OK) return st;
    TC_CUDA_OK(cudaMemcpyAsync(hC, dC, p->size_c * es, cudaMemcpyDeviceToHost, s0));  // pageable: the driver stages it
  } else {
    used[0] = nullptr;
    used[1] = h->plan_slab;
    used[2] = h->plan_tail;
    // inputs that are not sliced go first, whole
    if (!h->step[1]) st = copy_in(h, dA, hA, p->size_a * es, page_a, s0);
    if (st == TC_OK && !h->step[2]) st = copy_in(h, dB, hB, p->size_b * es, page_b, s0);
    if (st != TC_OK) return st;
    TC_CUDA_OK(cudaEventRecord(h->inputs_ready, s0));
    Drain drain;
    std::thread drainer;
    if (page_c) {
      drain.h = h;
      drain.device = p->device;
      drainer = std::thread([&drain] { drain.loop(); });
    }
    auto finish = [&](int code) {
      if (page_c) { drain.close(); drainer.join(); if (code == TC_OK) code = drain.status; }
      return code;
    };
    // Page-locked callers: copies in, kernels and copies out each on a stream of their own, chained slab by slab
    // through events.  The whole tensors are resident on the device, so the copies in never wait for a copy out and
    // both directions of the link stay busy for the whole call.  (Measured on the sharded benchmark configuration,
    // 65.6 GB per call: 0.81 s, the same as with two streams that each did copy in, kernel, copy out for every other
    // slab -- 81 GB/s over both directions together is what the link of these hosts gives.)
    if (!page_c && !page_a && !page_b) {
      if (!h->out_stream) TC_CUDA_OK(cudaStreamCreateWithFlags(&h->out_stream, cudaStreamNonBlocking));
      cudaStream_t s_in = h->stream[0], s_k = h->stream[1], s_out = h->out_stream;
      auto event_of = [&](std::vector<cudaEvent_t>& pool, int k, cudaEvent_t* ev) {
        while ((int)pool.size() <= k) {
          cudaEvent_t e;
          if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return TC_ERR_CUDA;
          pool.push_back(e);
        }
        *ev = pool[k];
        return TC_OK;
      };
      int k = 0;
      for (int64_t v = 0; v < h->extent; v += h->slab, ++k) {
        const int64_t n = std::min(h->slab, h->extent - v);
        tc_plan* q = n == h->slab ? h->plan_slab : h->plan_tail;
        auto range = [&](int t, size_t* off, size_t* bytes) {
          *off = (size_t)(v * h->step[t]) * es;
          *bytes = (size_t)((n - 1) * h->step[t] + h->rest[t]) * es;
        };
        size_t oc, bc, oa, ba, ob, bb;
        range(0, &oc, &bc);
        range(1, &oa, &ba);
        range(2, &ob, &bb);
        if (read_c) TC_CUDA_OK(cudaMemcpyAsync(dC + oc, hC + oc, bc, cudaMemcpyHostToDevice, s_in));
        if (h->step[1]) TC_CUDA_OK(cudaMemcpyAsync(dA + oa, hA + oa, ba, cudaMemcpyHostToDevice, s_in));
        if (h->step[2]) TC_CUDA_OK(cudaMemcpyAsync(dB + ob, hB + ob, bb, cudaMemcpyHostToDevice, s_in));
        cudaEvent_t in_ev, k_ev;
        st = event_of(h->slab_in, k, &in_ev);
        if (st == TC_OK) st = event_of(h->slab_done, k, &k_ev);
        if (st != TC_OK) return st;
        TC_CUDA_OK(cudaEventRecord(in_ev, s_in));      // (the whole inputs went first on this stream)
        TC_CUDA_OK(cudaStreamWaitEvent(s_k, in_ev, 0));
        st = execute_impl(q, dC + oc, dA + (size_t)(v * h->view[1]) * es, dB + (size_t)(v * h->view[2]) * es, q->d_ws,
                          q->ws_bytes, s_k);
        if (st != TC_OK) return st;
        TC_CUDA_OK(cudaEventRecord(k_ev, s_k));
        TC_CUDA_OK(cudaStreamWaitEvent(s_out, k_ev, 0));
        TC_CUDA_OK(cudaMemcpyAsync(hC + oc, dC + oc, bc, cudaMemcpyDeviceToHost, s_out));
      }
    }
    int i = 0;
    for (int64_t v = 0; (page_c || page_a || page_b) && v < h->extent; v += h->slab, ++i) {
      const int64_t n = std::min(h->slab, h->extent - v);
      tc_plan* q = n == h->slab ? h->plan_slab : h->plan_tail;
      cudaStream_t s = h->stream[i & 1];
      auto range = [&](int t, size_t* off, size_t* bytes) {
        *off = (size_t)(v * h->step[t]) * es;
        *bytes = (size_t)((n - 1) * h->step[t] + h->rest[t]) * es;
      };
      size_t oc, bc, oa, ba, ob, bb;
      range(0, &oc, &bc);
      range(1, &oa, &ba);
      range(2, &ob, &bb);
      if (read_c) st = copy_in(h, dC + oc, hC + oc, bc, page_c, s);
      if (st == TC_OK && h->step[1]) st = copy_in(h, dA + oa, hA + oa, ba, page_a, s);
      if (st == TC_OK && h->step[2]) st = copy_in(h, dB + ob, hB + ob, bb, page_b, s);
      if (st != TC_OK) return finish(st);
      if (s != s0) TC_CUDA_OK(cudaStreamWaitEvent(s, h->inputs_ready, 0));
      st = execute_impl(q, dC + oc, dA + (size_t)(v * h->view[1]) * es, dB + (size_t)(v * h->view[2]) * es, q->d_ws,
                        q->ws_bytes, s);
      if (st != TC_OK) return finish(st);
      if (!page_c) {
        TC_CUDA_OK(cudaMemcpyAsync(hC + oc, dC + oc, bc, cudaMemcpyDeviceToHost, s));
      } else {
        if ((int)h->slab_done.size() <= i) {
          cudaEvent_t ev;
          TC_CUDA_OK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
          h->slab_done.push_back(ev);
        }
        TC_CUDA_OK(cudaEventRecord(h->slab_done[i], s));
        drain.push(DrainJob{dC + oc, hC + oc, bc, h->slab_done[i]});
      }
    }
    st = finish(TC_OK);
    if (st != TC_OK) return st;
  }
  TC_CUDA_OK(cudaStreamSynchronize(h->stream[1]));
  if (h->out_stream) TC_CUDA_OK(cudaStreamSynchronize(h->out_stream));
  TC_CUDA_OK(cudaStreamSynchronize(s0));
  // Status words of the plans that ran (read once every kernel of the call has finished): a wait that gave up leaves
  // the output invalid.
  int k = 0;
  for (tc_plan* q : used)
    if (q) { TC_CUDA_OK(cudaMemcpyAsync(h->h_status + k, q->d_status, sizeof(int), cudaMemcpyDeviceToHost, s0)); ++k; }
  TC_CUDA_OK(cudaStreamSynchronize(s0));
  for (int q = 0; q < k; ++q)
    if (h->h_status[q] != 0) {
      int code = h->h_status[q];
      cudaMemcpy(p->d_status, &code, sizeof(int), cudaMemcpyHostToDevice);  // visible through tc_plan_status of the caller's plan
      return TC_ERR_DEVICE_WAIT;
    }
  return TC_OK;
}

extern "C" int tc_execute_host(tc_plan* p, void* C, const void* A, const void* B) {
  if (!p || !C || !A || !B) return TC_ERR_INVALID_ARG;
  if (!p->committed) {
    const int st = tc_plan_commit(p);
    if (st != TC_OK) return st;
  }
  int dev = 0;
  TC_CUDA_OK(cudaGetDevice(&dev));
  if (dev != p->device) return TC_ERR_STATE;
  std::lock_guard<std::mutex> lock(*p->host_mu);  // the plan's device buffers, streams and bounce buffers are shared
  return execute_host_locked(p, C, A, B);
}

// Frees what the host-pointer path keeps on the device for this plan (it is rebuilt on the next call).
static void host_pipe_release(tc_plan* p) {
  std::lock_guard<std::mutex> lock(*p->host_mu);
  host_pipe_destroy(p->host);
  p->host = nullptr;
}

// ------------------------------------------- drop-in for sd_t_d2_fusion_ ----
extern "C" int tc_sd_t_d2_fusion(const char* expr, int dtype, int n_sizes, const int* sizes, void* t3, const void* t2,
                                 const void* v2) {
  if (!expr || !sizes || !t3 || !t2 || !v2 || n_sizes < 0) return TC_ERR_INVALID_ARG;
  // Plans are kept per (expression, dtype, sizes), like the generated code's statics; the device buffers of
  // the host-pointer path are kept only for the most recently used plan, so a driver that sweeps many sizes
  // holds one problem's tensors on the device at a time (the reference frees after every call,
  // cogent/src/codes/others/tc_pre_CUDA_Malloc.py).
  static std::mutex mu;
  static std::map<std::string, tc_plan*> cache;
  static tc_plan* last = nullptr;
  constexpr size_t kMaxCached = 256;
  std::string key = std::string(expr) + "|" + std::to_string(dtype);
  for (int i = 0; i < n_sizes; ++i) key += "," + std::to_string(sizes[i]);
  tc_plan* plan = nullptr;
  bool cached = true;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) plan = it->second;
  }
  if (!plan) {
    int st = tc_plan_create(expr, dtype, nullptr, &plan);
    if (st != TC_OK) return st;
    std::vector<int64_t> ext(sizes, sizes + n_sizes);
    st = tc_plan_set_extents_ordered(plan, n_sizes, ext.data());
    if (st == TC_OK) st = tc_plan_commit(plan);
    if (st != TC_OK) { tc_plan_destroy(plan); return st; }
    std::lock_guard<std::mutex> lock(mu);
    if (cache.size() >= kMaxCached) cached = false;  // beyond that: plan, run, free, like the reference
    else {
      auto ins = cache.emplace(key, plan);
      if (!ins.second) { tc_plan_destroy(plan); plan = ins.first->second; }
    }
  }
  if (cached) {
    tc_plan* prev = nullptr;
    {
      std::lock_guard<std::mutex> lock(mu);
      if (last != plan) { prev = last; last = plan; }
    }
    if (prev) host_pipe_release(prev);
  }
  const int st = tc_execute_host(plan, t3, t2, v2);
  if (!cached) tc_plan_destroy(plan);
  return st;
}

// -------------------------------------------------------- seeded inputs ----
namespace {

__host__ __device__ inline uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

template <typename T>
__global__ void fill_kernel(T* dst, int64_t count, uint64_t key, int64_t first) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < count; i += stride) {
    const uint64_t x = splitmix64(key ^ (uint64_t)(first + i));
    if constexpr (sizeof(T) == 8) dst[i] = (double)(x >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    else dst[i] = (float)(x >> 40) * (1.0f / 16777216.0f) * 2.0f - 1.0f;
  }
}

template <typename T>
__global__ void axpy_kernel(T* y, const T* x, int64_t count, T alpha) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < count; i += stride) y[i] += alpha * x[i];
}

int grid_for(int64_t count) {
  int dev = 0;
  cudaGetDevice(&dev);
  int64_t g = (count + 255) / 256;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)device_sm_count(dev) * 16));
}

}  // namespace

extern "C" int tc_fill_uniform(void* dst, int64_t count, int dtype, uint64_t seed, int tensor_id, int64_t first_index,
                               void* stream) {
  if (!dst || count < 0 || tensor_id < 0 || tensor_id > 15 || (dtype != TC_F64 && dtype != TC_F32)) return TC_ERR_INVALID_ARG;
  if (count == 0) return TC_OK;
  const uint64_t key = (seed * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)tensor_id << 60);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == TC_F64) fill_kernel<double><<<grid_for(count), 256, 0, s>>>(static_cast<double*>(dst), count, key, first_index);
  else fill_kernel<float><<<grid_for(count), 256, 0, s>>>(static_cast<float*>(dst), count, key, first_index);
  TC_CUDA_OK(cudaGetLastError());
  return TC_OK;
}

extern "C" int tc_axpy(void* y, const void* x, int64_t count, int dtype, double alpha, void* stream) {
  if (!y || !x || count < 0 || (dtype != TC_F64 && dtype != TC_F32)) return TC_ERR_INVALID_ARG;
  if (count == 0) return TC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == TC_F64) axpy_kernel<double><<<grid_for(count), 256, 0, s>>>(static_cast<double*>(y), static_cast<const double*>(x), count, alpha);
  else axpy_kernel<float><<<grid_for(count), 256, 0, s>>>(static_cast<float*>(y), static_cast<const float*>(x), count, (float)alpha);
  TC_CUDA_OK(cudaGetLastError());
  return TC_OK;
}
