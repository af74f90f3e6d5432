// C ABI of the B200 back end: argument checks, launch configuration, error reporting.
// The kernels live in the .cuh files included below; this is the only translation unit.
#include <cuda_runtime.h>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include <stdlib.h>
#include <string.h>

#include "../../include/arcq_b200.h"
#include "ptx.cuh"
#include "act_quant.cuh"
#include "group_quant.cuh"
#include "act_quant_tile.cuh"
#include "codes.cuh"
#include "packed_gemm.cuh"
#include "gemm_ws.cuh"
#include "gemm_pair.cuh"
#include "gemm_pair_dense.cuh"
#include "add_layernorm.cuh"
#include "ln_act_quant.cuh"
#include "attention.cuh"
#include "small_linear.cuh"
#include "patch_embed.cuh"
#include <cudaTypedefs.h>

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(ARCQ_E_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

__device__ int g_status_word = 0;
// which GEMM kernel the last GEMM entry point of this host thread launched (arcq_debug_last_gemm_kernel)
thread_local int g_last_gemm_kernel = 0;
long long* g_trace_buf = nullptr;   // set by arcq_debug_trace; 64 timestamps per CTA

int* status_ptr() {
  // one address per device; looked up once per device and cached
  static thread_local int cached_dev = -1;
  static thread_local int* cached = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != cached_dev) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess) return nullptr;
    cached = static_cast<int*>(p);
    cached_dev = dev;
  }
  return cached;
}

int sm_count() {
  static thread_local int cached_dev = -1;
  static thread_local int sms = 148;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != cached_dev) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cached_dev = dev;
  }
  return sms;
}

// Tuning options.  Each has a built-in default; an environment variable of the same name, read once when the
// library is first used, or arcq_debug_set_option() at any time, overrides it.  Normal use sets none of them.
enum Opt {
  O_WS_BN, O_WS_SA, O_WS_WS, O_WS_STATIONARY, O_WS_NBB, O_WS_GRID, O_WS_TMA_STORE, O_WS_ROTATE,
  O_ACT_QUANT_V1, O_LN_PLAIN,
  O_PAIR, O_PAIR_MIN_M, O_PAIR_BN, O_PAIR_SA, O_PAIR_KS, O_PAIR_NBB, O_PAIR_LUT, O_PAIR_PAIRS, O_PAIR_STATIONARY,
  O_PAIR_WS, O_LNQ_SMALL, O_AQ2_MIN_GROUPS, O_PDL, O_GELU_GEMM, O_GEMM_UNPACK, O_POLL_LIMIT, O_SPIN_LIMIT, O_LAUNCH_REGS,
  O_SMALL_LINEAR, O_SMALL_R, O_SMALL_BN, O_PAIR_SPLIT, O_PAIR_STAGGER,
  O_COUNT
};
struct OptDef { const char* name; int dflt; };
const OptDef kOptDefs[O_COUNT] = {
    {"ARCQ_WS_BN", 0},        {"ARCQ_WS_SA", 0},          {"ARCQ_WS_WS", 0},       {"ARCQ_WS_STATIONARY", -1},
    {"ARCQ_WS_NBB", 0},       {"ARCQ_WS_GRID", 0},        {"ARCQ_WS_TMA_STORE", 1}, {"ARCQ_WS_ROTATE", 1},
    {"ARCQ_ACT_QUANT_V1", 0}, {"ARCQ_LN_PLAIN", 0},
    {"ARCQ_PAIR", 1},         {"ARCQ_PAIR_MIN_M", 1024},  {"ARCQ_PAIR_BN", 0},     {"ARCQ_PAIR_SA", 0},
    {"ARCQ_PAIR_KS", 0},      {"ARCQ_PAIR_NBB", 0},       {"ARCQ_PAIR_LUT", 0},    {"ARCQ_PAIR_PAIRS", 0},
    {"ARCQ_PAIR_STATIONARY", -1}, {"ARCQ_PAIR_WS", 0}, {"ARCQ_LNQ_SMALL", 1}, {"ARCQ_AQ2_MIN_GROUPS", 0}, {"ARCQ_PDL", 1},
    {"ARCQ_GELU_GEMM", -1}, {"ARCQ_GEMM_UNPACK", 1},
    {"ARCQ_POLL_LIMIT", 1 << 21}, {"ARCQ_SPIN_LIMIT", 1 << 25}, {"ARCQ_LAUNCH_REGS", 0},
    {"ARCQ_SMALL_LINEAR", -1}, {"ARCQ_SMALL_R", 0}, {"ARCQ_SMALL_BN", 0}, {"ARCQ_PAIR_SPLIT", 1}, {"ARCQ_PAIR_STAGGER", -1},
};
int g_opt[O_COUNT];
void load_options() {
  static const bool once = [] {
    for (int i = 0; i < O_COUNT; ++i) {
      const char* v = getenv(kOptDefs[i].name);
      g_opt[i] = (v != nullptr && *v != 0) ? atoi(v) : kOptDefs[i].dflt;
    }
    return true;
  }();
  (void)once;
}
int opt(Opt o) {
  load_options();
  return g_opt[o];
}

// Launch as a programmatic dependent of the kernel before it in the stream (unless ARCQ_PDL is 0): the grid may
// become resident while that kernel drains; every kernel launched this way calls pdl_wait() before it reads
// anything a predecessor writes.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = opt(O_PDL) != 0 ? 1 : 0;
  return cudaLaunchKernelEx(&lc, kernel, static_cast<KArgs>(args)...);
}

// Set-up of a kernel whose warp groups hand registers over: its shared-memory limit, and whether a launch brings the registers a
// thread that the hand-over counts on.  An increase beyond them waits for good, and a changed flag or compiler is enough for that, so
// such a build is refused here.  ARCQ_LAUNCH_REGS stands for what the compiled kernel says, in tests.
template <typename Kernel> int prepare_register_kernel(Kernel kernel, size_t smem, int regs, const char* what) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  cudaFuncAttributes a = {};
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return cuda_fail(e, what);
  const int got = opt(O_LAUNCH_REGS) > 0 ? opt(O_LAUNCH_REGS) : a.numRegs;
  if (got < regs) return fail(ARCQ_E_CUDA, "%s: compiled for %d registers a thread, its warp groups share out %d", what, got, regs);
  return ARCQ_OK;
}

bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

int grid_for(long long work_items, int per_block, int blocks_per_sm) {
  long long need = (work_items + per_block - 1) / per_block;
  long long cap = static_cast<long long>(sm_count()) * blocks_per_sm;
  if (need < 1) need = 1;
  return static_cast<int>(need < cap ? need : cap);
}

template <typename T, int BITS, int PRE = 0>
cudaError_t launch_act_quant(const void* x, long long groups, const float* th, const float* cb, uint8_t* packed,
                             float* mu, float* sg, float* cs, void* xhat, int xhat_dtype, cudaStream_t st,
                             int one_fma, const arcq::UnpackJobs& jobs) {
  const int grid = grid_for((groups + 3) / 4, 8, 8) + jobs.blocks;
  const T* xt = static_cast<const T*>(x);
  if (xhat == nullptr) {
    launch_pdl(arcq::act_quant_kernel<T, BITS, float, false, PRE>, grid, 256, 0, st, xt, groups, th, cb, packed, mu, sg, cs, static_cast<float*>(nullptr), one_fma, jobs);
  } else if (xhat_dtype == ARCQ_DT_F32) {
    launch_pdl(arcq::act_quant_kernel<T, BITS, float, true, PRE>, grid, 256, 0, st, xt, groups, th, cb, packed, mu, sg, cs, static_cast<float*>(xhat), one_fma, jobs);
  } else if (xhat_dtype == ARCQ_DT_F16) {
    launch_pdl(arcq::act_quant_kernel<T, BITS, __half, true, PRE>, grid, 256, 0, st, xt, groups, th, cb, packed, mu, sg, cs, static_cast<__half*>(xhat), one_fma, jobs);
  } else {
    launch_pdl(arcq::act_quant_kernel<T, BITS, __nv_bfloat16, true, PRE>, grid, 256, 0, st, xt, groups, th, cb, packed, mu, sg, cs, static_cast<__nv_bfloat16*>(xhat), one_fma, jobs);
  }
  return cudaGetLastError();
}

// ---- tensor maps (driver entry point fetched through the runtime, so libcuda is not linked) ----
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {   // resolved once; the initialisation is thread-safe
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
  }();
  return fn;
}

// Row-major tensor [rows, cols] of `elem_bytes`-byte elements, or `planes` of them one after the other (0: a matrix), box
// [box_cols x box_rows].  A descriptor depends only on these values (not on what the memory holds), so the last few are kept
// per host thread: a model's layers present the same (pointer, shape) again on every forward.
struct TensorMapKey {
  const void* base;
  uint64_t planes, rows, cols;
  uint32_t box_cols, box_rows;
  int dt, swz;
  bool operator==(const TensorMapKey& o) const {
    return base == o.base && planes == o.planes && rows == o.rows && cols == o.cols && box_cols == o.box_cols &&
           box_rows == o.box_rows && dt == o.dt && swz == o.swz;
  }
};
bool make_tensor_map(CUtensorMap* tm, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t planes, uint64_t rows,
                     uint64_t cols, uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swz) {
  constexpr int kSlots = 256;
  struct Slot { TensorMapKey key; CUtensorMap map; bool used; };
  static thread_local Slot cache[kSlots] = {};
  const TensorMapKey key{base, planes, rows, cols, box_cols, box_rows, static_cast<int>(dt), static_cast<int>(swz)};
  uint64_t h = (reinterpret_cast<uintptr_t>(base) >> 4) ^ (planes << 50);
  h = (h ^ (rows * 0x9E3779B97F4A7C15ull) ^ (cols << 7) ^ (static_cast<uint64_t>(box_rows) << 29) ^ (static_cast<uint64_t>(box_cols) << 41)) * 0xD6E8FEB86659FD93ull;
  Slot& slot = cache[(h >> 40) % kSlots];
  if (slot.used && slot.key == key) {
    *tm = slot.map;
    return true;
  }
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc == nullptr) return false;
  const cuuint64_t row_bytes = cols * static_cast<uint64_t>(elem_bytes);
  cuuint64_t dims[3] = {cols, rows, planes};
  cuuint64_t strides[2] = {row_bytes, rows * row_bytes};
  cuuint32_t box[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  if (enc(tm, dt, planes > 0 ? 3 : 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  slot.key = key;
  slot.map = *tm;
  slot.used = true;
  return true;
}
bool make_tensor_map_2d(CUtensorMap* tm, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t rows,
                        uint64_t cols, uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swz) {
  return make_tensor_map(tm, base, dt, elem_bytes, 0, rows, cols, box_cols, box_rows, swz);
}

// Tile form of the quantizer (a thread per group, tiles by TMA): taken when the buffers are aligned for 16-byte accesses and
// the reconstruction, if asked for, is fp16 or has the input's element type.
template <typename T, int BITS, int PRE, typename XH, bool WX, bool WP>
cudaError_t launch_act_quant_tile(const void* x, long long groups, const float* th, const float* cb, uint8_t* packed,
                                  float* mu, float* sg, float* cs, void* xhat, cudaStream_t st, int one_fma,
                                  const arcq::UnpackJobs& jobs) {
  auto k = arcq::act_quant_tile_kernel<T, BITS, XH, WX, PRE, WP>;
  using Shape = arcq::AqtShape<T, WP>;
  constexpr int smem = Shape::kSmem;
  static thread_local int done_dev = -1;      // shared-memory ceiling raised once per (host thread, device)
  int dev = 0;
  cudaGetDevice(&dev);
  if (done_dev != dev) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    done_dev = dev;
  }
  // a group is one row of 64 16-bit values, or two rows of 32 fp32 values
  auto map = [&](CUtensorMap* tm, const void* p, int bytes, CUtensorMapDataType dt) {
    const int rows_per = bytes == 4 ? 2 : 1;
    return make_tensor_map_2d(tm, p, dt, bytes, static_cast<uint64_t>(groups) * rows_per, 64 / rows_per, 64 / rows_per,
                              Shape::kGroups * rows_per,
                              CU_TENSOR_MAP_SWIZZLE_128B);
  };
  auto type_of = [](auto v) {
    using V = decltype(v);
    return sizeof(V) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                          : std::is_same<V, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  };
  CUtensorMap tm_x, tm_out;
  if (!map(&tm_x, x, static_cast<int>(sizeof(T)), type_of(T{}))) return cudaErrorInvalidValue;
  if (WX) {
    if (!map(&tm_out, xhat, static_cast<int>(sizeof(XH)), type_of(XH{}))) return cudaErrorInvalidValue;
  } else {
    tm_out = tm_x;
  }
  constexpr int per_block = Shape::kWarps * Shape::kGroups;
  const long long blocks = (groups + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(sm_count()) * Shape::kBlocksPerSm;
  launch_pdl(k, static_cast<unsigned>((blocks < cap ? blocks : cap) + jobs.blocks), Shape::kThreads, smem, st, tm_x, tm_out, groups, th, cb,
             packed, mu, sg, cs, one_fma, status_ptr(), jobs);
  return cudaGetLastError();
}

template <typename T, int BITS, int PRE, typename XH>
cudaError_t launch_act_quant_tile_outputs(const void* x, long long groups, const float* th, const float* cb, uint8_t* packed,
                                          float* mu, float* sg, float* cs, void* xhat, cudaStream_t st, int one_fma,
                                  const arcq::UnpackJobs& jobs) {
  if (xhat == nullptr) return launch_act_quant_tile<T, BITS, PRE, XH, false, true>(x, groups, th, cb, packed, mu, sg, cs, xhat, st, one_fma, jobs);
  if (packed == nullptr) return launch_act_quant_tile<T, BITS, PRE, XH, true, false>(x, groups, th, cb, packed, mu, sg, cs, xhat, st, one_fma, jobs);
  return launch_act_quant_tile<T, BITS, PRE, XH, true, true>(x, groups, th, cb, packed, mu, sg, cs, xhat, st, one_fma, jobs);
}

template <typename T, int BITS, int PRE>
cudaError_t dispatch_act_quant_tile(const void* x, long long groups, const float* th, const float* cb, uint8_t* packed, float* mu,
                                    float* sg, float* cs, void* xhat, bool xhat_f16, cudaStream_t st, int one_fma,
                                  const arcq::UnpackJobs& jobs) {
  if constexpr (!std::is_same<T, __half>::value) {
    if (xhat != nullptr && xhat_f16)
      return launch_act_quant_tile_outputs<T, BITS, PRE, __half>(x, groups, th, cb, packed, mu, sg, cs, xhat, st, one_fma, jobs);
  }
  return launch_act_quant_tile_outputs<T, BITS, PRE, T>(x, groups, th, cb, packed, mu, sg, cs, xhat, st, one_fma, jobs);
}

template <typename T, int PRE>
cudaError_t dispatch_act_quant_bits(int bits, const void* x, int x_dtype, long long groups, const float* th,
                                    const float* cb, uint8_t* packed, float* mu, float* sg, float* cs, void* xhat,
                                    int xhat_dtype, cudaStream_t st, int one_fma,
                                  const arcq::UnpackJobs& jobs) {
  // The one-thread-per-group kernel needs enough groups to half fill the machine (256 per SM of 4 blocks x 128
  // threads); below that the 8-lanes-per-group kernel has 8 times the parallelism and lower latency.
  const long long min_groups = opt(O_AQ2_MIN_GROUPS) > 0 ? opt(O_AQ2_MIN_GROUPS) : static_cast<long long>(sm_count()) * 256;
  const bool xhat_f16 = xhat != nullptr && xhat_dtype == ARCQ_DT_F16;
  const bool tile = groups >= min_groups && groups < (1ll << 30) && opt(O_ACT_QUANT_V1) == 0 && aligned(x, 16) &&
                    (packed == nullptr || aligned(packed, 16)) &&
                    (xhat == nullptr || ((xhat_dtype == x_dtype || xhat_f16) && aligned(xhat, 16)));
  if (tile) {
    switch (bits) {
      case 4: return dispatch_act_quant_tile<T, 4, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_f16, st, one_fma, jobs);
      case 3: return dispatch_act_quant_tile<T, 3, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_f16, st, one_fma, jobs);
      default: return dispatch_act_quant_tile<T, 2, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_f16, st, one_fma, jobs);
    }
  }
  switch (bits) {
    case 4: return launch_act_quant<T, 4, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_dtype, st, one_fma, jobs);
    case 3: return launch_act_quant<T, 3, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_dtype, st, one_fma, jobs);
    default: return launch_act_quant<T, 2, PRE>(x, groups, th, cb, packed, mu, sg, cs, xhat, xhat_dtype, st, one_fma, jobs);
  }
}

// Tile width for the packed GEMM: the widest multiple of 16 (<= 256) that divides N, narrowed while
// the grid would leave most of the SMs idle.
int choose_bn(long long M, long long N) {
  static const int cand[] = {256, 192, 128, 96, 64, 48, 32, 16};
  const long long tiles_m = (M + arcq::kTileM - 1) / arcq::kTileM;
  int widest = 0, narrowest = 0;
  for (int c : cand) {
    if (N % c != 0) continue;
    if (widest == 0) widest = c;
    if (tiles_m * (N / c) >= sm_count()) return c;  // widest tile that still fills the machine
    if (c >= 32 || narrowest == 0) narrowest = c;
  }
  if (widest != 0) return narrowest;
  const long long r = (N + 15) / 16 * 16;  // N not a multiple of 16: pad the last tile column
  return static_cast<int>(r < 256 ? r : 256);
}


struct WsConfig {
  int bn, ws, sa, nbb, stationary, grid;
  size_t smem;
};

// Shared memory one CTA may ask for on B200 (227 KB) minus the 1 KB alignment slack.
constexpr size_t kSmemBudget = 232448 - 1024;

// Pick slab width, ring depths and grid for the warp-specialised GEMM; false if the shape is not
// one it handles (the caller then reports ARCQ_E_UNSUPPORTED).
bool choose_ws_config(long long M, long long N, long long K, int bits, bool dense, WsConfig* c) {
  const int G = static_cast<int>(K / 64);
  const long long tiles_m = (M + arcq::kTileM - 1) / arcq::kTileM;
  const int sms = sm_count();
  static const int cand[] = {192, 256, 128, 96, 64, 48, 32, 16};
  int best_bn = 0;
  long long best_ctas = -1;
  for (int bn : cand) {
    if (N % bn != 0) continue;
    const long long slabs = N / bn;
    if (slabs > sms) continue;
    const long long per = sms / slabs;
    const long long ctas = slabs * (tiles_m < per ? tiles_m : per);
    if (ctas * 4 >= 3LL * sms) { best_bn = bn; best_ctas = ctas; break; }  // first (widest) that fills 3/4 of the SMs
    if (ctas > best_ctas) { best_ctas = ctas; best_bn = bn; }
  }
  const int force_bn = opt(O_WS_BN);
  if (force_bn > 0 && force_bn % 16 == 0 && force_bn <= 256 && N % force_bn == 0) best_bn = force_bn;
  if (best_bn == 0) return false;
  c->bn = best_bn;
  const long long slabs = N / best_bn;
  const long long per = sms / slabs;
  c->grid = static_cast<int>(slabs * (tiles_m < per ? tiles_m : per));
  const int force_grid = opt(O_WS_GRID);
  if (force_grid > 0 && force_grid <= sms) c->grid = force_grid;
  const int force_stat = opt(O_WS_STATIONARY), force_sa = opt(O_WS_SA);
  const int force_ws = opt(O_WS_WS), force_nbb = opt(O_WS_NBB);
  // stationary if all G sub-tiles plus two A stages fit
  for (int stationary = 1; stationary >= 0; --stationary) {
    if (force_stat >= 0 && stationary != force_stat) continue;
    const int stream_slots = dense ? 4 : 3;
    int ws = stationary ? G : (G < stream_slots ? G : stream_slots);
    if (!stationary && force_ws > 0 && force_ws <= 16) ws = force_ws;
    if (ws > (stationary ? 32 : 16)) continue;   // barrier slots: 16 full/empty pairs for a ring, 32 full for a stationary slab
    for (int sa = 8; sa >= 2; --sa) {
      if (force_sa > 0 && sa != force_sa) continue;
      const size_t need = arcq::ws_smem_layout(best_bn, ws, sa, bits, G, stationary != 0, dense).total;
      if (need <= kSmemBudget) {
        c->ws = ws; c->sa = sa; c->stationary = stationary;
        c->nbb = stationary ? 1 : 2;
        if (force_nbb == 1 || force_nbb == 2) c->nbb = force_nbb;
        c->smem = need + 1024;
        return true;
      }
    }
  }
  return false;
}


// A one-CTA kernel whose only job is to let a bounded wait run out: it initialises an mbarrier that nothing
// ever arrives on, waits for it with the given poll limit, and leaves kStatusDebugTimeout in the status word.
// Exercises the error path of the kernels' waits (status set, kernel returns) without hanging anything.
constexpr int kStatusDebugTimeout = 0x7E57;
__global__ void debug_wait_timeout_kernel(uint32_t poll_limit, int* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    arcq::mbar_init(&bar, 1);
    arcq::mbar_fence_init();
  }
  __syncthreads();
  const bool ok = arcq::mbar_wait_sleep_a(arcq::smem_u32(&bar), 0u, poll_limit, 32);
  if (!ok && threadIdx.x == 0) atomicExch(status, kStatusDebugTimeout);
}

// ---- CTA-pair kernel: configuration ----
struct PairConfig {
  int bn, ws, sa, ks, nbb, stationary, lut_shift, pairs;
  size_t smem;
};

// How many two-CTA clusters of the pair kernel can be resident at once (each takes two whole SMs).
int max_resident_pairs(int bits, size_t smem) {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev == cached_dev && cached > 0) return cached;
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count() / 2 * 2));
  cfg.blockDim = dim3(arcq::kPairThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaErrorUnknown;
  if (bits == 4) e = cudaOccupancyMaxActiveClusters(&n, arcq::packed_weight_gemm_pair_kernel<4, true>, &cfg);
  else if (bits == 3) e = cudaOccupancyMaxActiveClusters(&n, arcq::packed_weight_gemm_pair_kernel<3, true>, &cfg);
  else e = cudaOccupancyMaxActiveClusters(&n, arcq::packed_weight_gemm_pair_kernel<2, true>, &cfg);
  if (e != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = sm_count() / 2;
  }
  if (n > sm_count() / 2) n = sm_count() / 2;
  cached = n;
  cached_dev = dev;
  return n;
}

template <int B>
cudaError_t pair_set_smem(size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(arcq::packed_weight_gemm_pair_kernel<B, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(arcq::packed_weight_gemm_pair_kernel<B, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(smem));
}

// Slab width, stages and grid for the CTA-pair kernel; false when the shape is left to the one-CTA kernel
// (small M, N without a slab width that is a multiple of 32, ...).  The cost model counts tensor-pipe
// cycles per SM: a 256 x bn x 64 stage is four instructions of bn/2 cycles each; rebuilding one
// [bn/2 x 64] sub-tile costs about 300 + 6.5 * bn/2 cycles on the eight producer warps.
bool choose_pair_config(long long M, long long N, long long K, int bits, bool y_f32, PairConfig* c) {
  if (opt(O_PAIR) == 0 || M < opt(O_PAIR_MIN_M)) return false;
  const int G = static_cast<int>(K / 64);
  if (G < 1 || G > 64) return false;
  const long long tiles_m = (M + arcq::kPairTileM - 1) / arcq::kPairTileM;
  const size_t full_smem = kSmemBudget + 1024;
  {
    // raise the kernel's dynamic shared-memory ceiling once per (host thread, device, code width)
    static thread_local int done_dev[5] = {-1, -1, -1, -1, -1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (done_dev[bits] != dev) {
      if (bits == 4 ? pair_set_smem<4>(full_smem) != cudaSuccess
                    : bits == 3 ? pair_set_smem<3>(full_smem) != cudaSuccess : pair_set_smem<2>(full_smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      done_dev[bits] = dev;
    }
  }
  int max_pairs = max_resident_pairs(bits, full_smem);
  if (opt(O_PAIR_PAIRS) > 0 && opt(O_PAIR_PAIRS) < max_pairs) max_pairs = opt(O_PAIR_PAIRS);
  static const int cand[] = {192, 160, 128, 96, 64, 32};     // at most arcq::kPairMaxBn
  double best_cost = 0;
  bool found = false;
  PairConfig best = {};
  for (int bn : cand) {
    if (N % bn != 0) continue;
    if (opt(O_PAIR_BN) > 0 && bn != opt(O_PAIR_BN)) continue;
    const long long slabs = N / bn;
    if (slabs > max_pairs) continue;
    const int hb = bn / 2;
    long long per = max_pairs / slabs;
    if (per > tiles_m) per = tiles_m;
    const long long tiles_pp = (tiles_m + per - 1) / per;
    // Cost model in microseconds, constants from time stamps taken inside the kernel on the DeiT shapes: a tile is
    // bound by its output stores (about 22 GB/s per SM) or by the issuing thread (about 110 cycles per
    // instruction plus 0.15 us per stage); a sub-tile rebuild takes 0.12 + 0.0026 * rows us when both warp
    // groups build (stationary slab) and about twice that when only the weight warps do (streaming ring).
    const int esize = y_f32 ? 4 : 2;
    const double t_write = 128.0 * bn * esize / 22.0e3;
    const double t_l2 = static_cast<double>(slabs) * M * K * 2.0 / 5.0e6;    // every slab streams the whole activation
    for (int stationary = 1; stationary >= 0; --stationary) {
      if (opt(O_PAIR_STATIONARY) >= 0 && stationary != opt(O_PAIR_STATIONARY)) continue;
      PairConfig k = {};
      k.bn = bn; k.stationary = stationary; k.pairs = static_cast<int>(slabs * per);
      k.nbb = stationary ? 1 : 2;
      if (opt(O_PAIR_NBB) == 1 || opt(O_PAIR_NBB) == 2) k.nbb = opt(O_PAIR_NBB);
      // two 64-wide sub-tiles per stage: one wait and one pair of commits per eight instructions keeps the
      // issuing thread ahead of the tensor pipe
      k.ks = (G % 2 == 0) ? 2 : (G % 3 == 0) ? 3 : 1;
      if (opt(O_PAIR_KS) > 0 && G % opt(O_PAIR_KS) == 0) k.ks = opt(O_PAIR_KS);
      k.ws = stationary ? G : (opt(O_PAIR_WS) > 0 ? opt(O_PAIR_WS) : (k.ks == 2 || k.ks == 3 ? 6 : 4));
      if (!stationary && k.ws > G) k.ws = G;
      if (k.ws > (stationary ? 32 : 16) || k.ws < k.ks || (!stationary && k.ws % k.ks != 0)) continue;
      // eight copies of the pair table (more did not measure faster); as many A stages as fit, eight sub-stages at most
      bool fits = false;
      for (int lut = (opt(O_PAIR_LUT) > 0 ? opt(O_PAIR_LUT) : 3); lut >= 3 && !fits; --lut) {
        for (int sa = 8; sa >= 2 && !fits; --sa) {
          if (opt(O_PAIR_SA) > 0 && sa != opt(O_PAIR_SA)) continue;
          if (sa * k.ks > 8 && opt(O_PAIR_SA) == 0) continue;            // eight 16 KB sub-stages are plenty
          const size_t need = arcq::pair_smem_layout(bn, k.ws, sa, k.ks, G, stationary != 0, lut).total;
          if (need <= kSmemBudget) {
            k.sa = sa; k.lut_shift = lut; k.smem = need + 1024; fits = true;
          }
        }
        if (opt(O_PAIR_LUT) > 0) break;
      }
      if (!fits) continue;
      const double t_issue = (G / k.ks) * (k.ks * 4 * 0.056 + 0.15);
      double cost;
      if (stationary) {
        const double t_tile = (t_write > t_issue ? t_write : t_issue) + 0.15;
        const double path = G * (0.12 + 0.0026 * hb) + tiles_pp * t_tile;
        cost = 2.2 + (path > t_l2 ? path : t_l2);
      } else {
        double path = 0;
        for (long long t = 0; t < tiles_pp; t += k.nbb) {
          const long long nb = (tiles_pp - t) < k.nbb ? (tiles_pp - t) : k.nbb;
          const double build = G * (0.25 + 0.0055 * hb), issue = nb * t_issue;
          path += (build > issue ? build : issue) * 1.2 + nb * (t_write + 0.15);
        }
        cost = 2.2 + (path > t_l2 ? path : t_l2);
      }
      if (!found || cost < best_cost) { best = k; best_cost = cost; found = true; }
    }
  }
  if (!found) return false;
  *c = best;
  return true;
}


// ---- dense-weight CTA-pair kernel: configuration ----
struct PairDenseConfig {
  int bn, sa, ks, pairs, stationary, split_last, stagger;
  size_t smem;
  double cost;     // of the model that chose it
};

// CTA pairs of a form of the kernel that are resident at once with all of the shared memory, kept per host thread and device.
// The limit is raised before the question, whichever entry point asks first; a question that fails is not remembered.
struct ResidentPairs {
  int dev = -1, n = 0;
};
template <typename Kernel> int max_resident_dense_pairs(Kernel kernel, int threads, ResidentPairs* known) {
  const size_t smem = kSmemBudget + 1024;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev == known->dev) return known->n;
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count() / 2 * 2));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return sm_count() / 2;
  }
  if (n > sm_count() / 2) n = sm_count() / 2;
  *known = {dev, n};
  return n;
}

// Pairs of a launch: as many for each slab that stays, else up to one for each (row tile, slab).
long long dense_pairs(long long slabs, long long tiles_m, long long max_pairs, bool stationary) {
  if (!stationary) return slabs * tiles_m < max_pairs ? slabs * tiles_m : max_pairs;
  const long long per = max_pairs / slabs;
  return slabs * (per < tiles_m ? per : tiles_m);
}

// Slab width, stages and grid for the dense-weight pair kernel; false leaves the shape to the one-CTA kernel.
// Cost model in microseconds: a tile is bound by its output stores (about 24 GB/s per SM) or by the issuing thread, and every slab
// streams the whole activation from L2.
bool choose_pair_dense_config(long long M, long long N, long long K, bool y_f32, PairDenseConfig* c) {
  // No row threshold (ARCQ_PAIR_MIN_M gates the packed-weight pair kernel only): with nothing to rebuild, the pair
  // form measured faster than the one-CTA form from one row tile on (DeiT-S batch 1: 0.55 against 0.68 ms).
  if (opt(O_PAIR) == 0) return false;
  const int G = static_cast<int>(K / 64);
  if (G < 1) return false;
  const long long tiles_m = (M + arcq::kPairTileM - 1) / arcq::kPairTileM;
  const size_t full_smem = kSmemBudget + 1024;
  {
    static thread_local int done_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (done_dev != dev) {
      if (cudaFuncSetAttribute(arcq::dense_weight_gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(full_smem)) != cudaSuccess ||
          cudaFuncSetAttribute(arcq::dense_weight_gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(full_smem)) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      done_dev = dev;
    }
  }
  static thread_local ResidentPairs known;
  int max_pairs = max_resident_dense_pairs(arcq::dense_weight_gemm_pair_kernel<true>, arcq::kPairDenseThreads, &known);
  if (opt(O_PAIR_PAIRS) > 0 && opt(O_PAIR_PAIRS) < max_pairs) max_pairs = opt(O_PAIR_PAIRS);
  static const int cand[] = {256, 192, 160, 128, 96, 64, 32};
  bool found = false;
  PairDenseConfig best = {};
  // Up to four row tiles (batch 1-5 of a ViT): the launch is a latency chain, not a throughput problem, and the narrowest slab that gives
  // every (tile, slab) its own pair is the shortest chain, as long as that is no more than 40 pairs: every pair beyond them costs the launch
  // more than a narrower slab saves (K = 384, N = 1536: 197 rows 64 columns 4.4 us, 32 4.9; 394 rows 96 columns 4.6, 64 5.1; K = 768, N = 2304,
  // 197 rows 64 columns 5.6, 32 6.7).  Where 40 pairs leave only slabs of more than 128 columns the model below has it: a tile is then
  // longer than a few pairs more cost (K = 768, N = 2304, 788 rows: 256 columns on 36 pairs 7.7 us, 128 on 72 6.6; N = 3072, 394 rows 192 columns 6.7,
  // 128 6.1).  Over the same layers with 197 to 788 rows the slab chosen is 0.03 % slower than the fastest, 2.7 % at worst; without the
  // limit on its width 1.4 and 22 %, with up to two row tiles and all pairs 4.6 and 26 %.
  constexpr int kLatencyTiles = 4, kLatencyPairs = 40, kLatencyColumns = 128;
  int narrow_bn = 0;
  if (tiles_m <= kLatencyTiles && opt(O_PAIR_BN) == 0)
    for (int bn : cand)
      if (bn <= kLatencyColumns && N % bn == 0 && (N / bn) * tiles_m <= (max_pairs < kLatencyPairs ? max_pairs : kLatencyPairs))
        narrow_bn = bn;                                        // candidates descend: keeps the narrowest
  for (int bn : cand) {
    if (N % bn != 0) continue;
    if (opt(O_PAIR_BN) > 0 && bn != opt(O_PAIR_BN)) continue;
    if (narrow_bn != 0 && bn != narrow_bn) continue;
    const long long slabs = N / bn;
    if (slabs > max_pairs) continue;
    long long per = max_pairs / slabs;
    if (per > tiles_m) per = tiles_m;
    const int esize = y_f32 ? 4 : 2;
    const double t_write = 128.0 * bn * esize / 24.4e3;
    for (int stationary = 1; stationary >= 0; --stationary) {
      if (opt(O_PAIR_STATIONARY) >= 0 && stationary != opt(O_PAIR_STATIONARY)) continue;
      if (stationary && G > 32) continue;
      PairDenseConfig k = {};
      k.bn = bn; k.stationary = stationary;
      k.pairs = static_cast<int>(dense_pairs(slabs, tiles_m, max_pairs, stationary));
      const long long tiles_pp = stationary ? (tiles_m + per - 1) / per : (slabs * tiles_m + k.pairs - 1) / k.pairs;
      k.ks = (G % 2 == 0) ? 2 : (G % 3 == 0) ? 3 : 1;
      if (opt(O_PAIR_KS) > 0 && G % opt(O_PAIR_KS) == 0) k.ks = opt(O_PAIR_KS);
      bool fits = false;
      for (int sa = 16; sa >= 2 && !fits; --sa) {
        if (opt(O_PAIR_SA) > 0 && sa != opt(O_PAIR_SA)) continue;
        if (sa * k.ks > 8 && opt(O_PAIR_SA) == 0) continue;             // eight sub-stages in flight are plenty
        const size_t need = arcq::pair_dense_smem_layout(bn, sa, k.ks, G, stationary != 0).total;
        if (need <= kSmemBudget) { k.sa = sa; k.smem = need + 1024; fits = true; }
      }
      if (!fits) continue;
      if (stationary && opt(O_PAIR_STATIONARY) < 0 && (k.sa * k.ks < 4 || tiles_pp < 3))
        continue;   // too little room left for A, or too few tiles to pay for loading the whole slab first
      const double t_issue = (G / k.ks) * (k.ks * 4 * (bn > 128 ? 0.056 * bn / 192.0 : 0.04) + 0.1);
      // what goes through L2 into shared memory: every tile streams its A rows, and its W16 rows too unless the slab is stationary
      const double fill_mb = (static_cast<double>(slabs) * M * K * 2.0 +
                              (stationary ? static_cast<double>(k.pairs) : static_cast<double>(slabs * tiles_m)) * bn * K * 2.0) / 1.0e6;
      // A tile's stores or its issue, whichever is longer, 0.6 us a tile that neither accounts for, and a twentieth of a microsecond
      // for every megabyte of fill: it is hidden in part only, behind wide slabs as behind narrow ones.  Fitted to every slab width, with
      // and without a slab that stays and half tiles, on 600 shapes (twelve layers of the three widths, 197 to 50 432 rows, both output
      // types): the slab chosen is 1.1 % slower than the fastest on average, 24 % at worst (3001 rows of 192 x 192 to fp32, 32 columns 4.7 us, 64
      // 3.8), eight shapes by more than 10 %.  The constants fitted to the former order of the tiles (22 GB/s, 0.8 us, a half tile as half
      // a tile) had 1.6 %, and took 16 % more time than that order for K = 1536, N = 384, 9850 rows (17.1 us, 14.9 with this slab) and 7 %
      // for K = 384, N = 1536, 18 912 rows (23.5, 22.0).
      const double tile = t_write > t_issue ? t_write : t_issue;
      double cost = tiles_pp * (tile + 0.6) + fill_mb / 20.0;
      // Tiles that would fill half of another round at most come as halves (a half has to be a width of the instruction's), from K =
      // 1024 on: 12 608 rows of K = 1536, N = 384 are 100 tiles on 74 pairs, 19.8 us whole and 18.4 with the last 26 halved; a slab of 256
      // columns is 10 % faster so on average, of 192 6, of 128 2.  In the choice of a width a half counts as nine tenths of a tile: its
      // stores are half, its latency is not.  From K = 768 down it does not pay: K = 384, N = 384 7.5 / 7.8 us, K = 768, N = 768 25.1 / 25.4, N = 2304 38.7 / 37.9.
      const long long left = slabs * tiles_m % k.pairs;
      k.split_last = !stationary && opt(O_PAIR_SPLIT) != 0 && G >= 16 && slabs * tiles_m > k.pairs && left > 0 && 2 * left <= k.pairs && bn % 64 == 0;
      if (k.split_last) cost -= tile / 10;
      // fp32 outputs at least twice as wide as the rows of A: pairs that keep their slabs and start at different row tiles, where that
      // takes no more rounds and A, read for each slab anew, is well inside L2; beyond 16 MB of A only if the last round is 0.3 full at least (a
      // shorter one is over sooner with the tiles dealt out).  K = 768, N = 2304, 5517 rows 25.9 -> 24.6 us, 8471 rows, a last round of 10 pairs,
      // 39.4 -> 37.9, 9850 rows 42.7 -> 40.5; N = 3072, 7289 rows 42.0 -> 39.9; 15 760 rows, a last round of 4 pairs, 79.8 against 83.4 dealt out;
      // N = 768 the same either way, fp16 outputs 1 to 2 % slower.
      if (!stationary && !k.split_last && slabs * tiles_m > k.pairs && opt(O_PAIR_STAGGER) != 0) {
        const bool rule = y_f32 && N >= 2 * K && (tiles_m + per - 1) / per == tiles_pp && (left == 0 || 10 * left >= 3 * k.pairs || M * K <= (8ll << 20)) &&
                          M * K <= (24ll << 20);
        if (rule || opt(O_PAIR_STAGGER) > 0) { k.pairs = static_cast<int>(slabs * per); k.stagger = 1; }
      }
      k.cost = cost;
      if (!found || cost < best.cost) { best = k; found = true; }
    }
  }
  if (!found) return false;
  *c = best;
  return true;
}

// Slab width, stages and grid of the form with GELU and quantizer in its epilogue; false: none fits.
bool choose_pair_quant_config(long long M, long long N, long long K, PairDenseConfig* c) {
  if (opt(O_PAIR) == 0) return false;
  const int G = static_cast<int>(K / 64);
  const long long tiles_m = (M + arcq::kPairTileM - 1) / arcq::kPairTileM;
  static thread_local ResidentPairs known;
  int max_pairs = max_resident_dense_pairs(arcq::dense_weight_gemm_pair_kernel<true, false, 4>, arcq::kPairQuantThreads, &known);
  if (opt(O_PAIR_PAIRS) > 0 && opt(O_PAIR_PAIRS) < max_pairs) max_pairs = opt(O_PAIR_PAIRS);
  static const int cand[] = {192, 128, 64};                  // whole groups, at most one per epilogue warp of a lane quarter
  bool found = false;
  for (int bn : cand) {
    if (N % bn != 0 || (opt(O_PAIR_BN) > 0 && bn != opt(O_PAIR_BN))) continue;
    const long long slabs = N / bn;
    if (slabs > max_pairs) continue;
    long long per = max_pairs / slabs;
    if (per > tiles_m) per = tiles_m;
    // The epilogue bounds every tile: one, two or three warps per scheduler share its issue slots (a single tile of
    // 64 / 128 / 192 columns, K = 384: 8.7 / 9.8 / 11.4 us).
    for (int stationary = 1; stationary >= 0; --stationary) {
      PairDenseConfig k = {};
      k.bn = bn; k.stationary = stationary;
      k.pairs = static_cast<int>(dense_pairs(slabs, tiles_m, max_pairs, stationary));
      const long long tiles_pp = stationary ? (tiles_m + per - 1) / per : (slabs * tiles_m + k.pairs - 1) / k.pairs;
      if (stationary && (G > 32 || tiles_pp < 3)) continue;    // too few tiles to pay for loading the whole slab first
      k.ks = (G % 2 == 0) ? 2 : (G % 3 == 0) ? 3 : 1;
      bool fits = false;
      for (int sa = 8 / k.ks; sa >= 2 && !fits; --sa) {
        const size_t need = arcq::pair_dense_smem_layout(bn, sa, k.ks, G, stationary != 0, true).total;
        if (need <= kSmemBudget) { k.sa = sa; k.smem = need + 1024; fits = true; }
      }
      if (!fits || (stationary && k.sa * k.ks < 4)) continue;
      k.cost = tiles_pp * (2.5 + 0.9 * (bn / 64));
      if (!found || k.cost < c->cost) *c = k;
      found = true;
      break;                                                   // a slab that can stay does
    }
  }
  return found;
}

// Small inputs, where most SMs would get no 128-group tile, take the twelve-warp form of LayerNorm + quantizer (48 groups per
// block, lower latency).  Both forms give the same bits.  The line is where they measured equal: 4 137 groups 3.4 against 5.9 us,
// 8 274 groups 6.5 against 5.6 us, 18 912 groups 9.8 against 6.0 us.
bool small_layernorm_quant(long long M, long long K) {
  return M * (K / 64) < static_cast<long long>(sm_count()) * 48 && opt(O_LNQ_SMALL) != 0;
}

// fc1 with GELU and quantizer in its epilogue, or GEMM and quantizer kernel?  Whole forwards through a graph, microseconds, two
// kernels / one.  The epilogue's 12 warps hide latency worse than the quantizer kernel's 16, so it is rounds that decide: of the
// fused form's tiles on the pairs against the quantizer's blocks (512 groups an SM).  The line below is fitted to 62 batch sizes of
// DeiT-T, DeiT-S and DeiT-B (DeiT-T batch 32: 679 / 685, 37, where the quantizer has started a second round: 760 / 713; DeiT-S batch 16: 729 /
// 737, 18: 799 / 749, 64: 1413 / 1379): the worst it does there is two kernels for DeiT-T batch 48, 789 / 781.  The line fitted when every
// slab had the same number of pairs chose two kernels at thirteen of them, up to 5 % slower (DeiT-T batch 80: 1009 / 956).  Always where
// the products under the epilogue are long (DeiT-B batch 8: 880 / 871) or the matrix between the two no longer stays in L2 (DeiT-S
// batch 128: 2483 / 2377, DeiT-B: 6860 / 6188).  Where the quantizer takes its form for small inputs: one round of tiles (DeiT-S
// batch 6 / 8: 564 / 533, 661 / 608; DeiT-T batch 12: 525 / 496, but 8: 473 / 483), but not below five row tiles (DeiT-T batch 2: 449 / 463,
// although DeiT-S batch 4: 510 / 503).
bool choose_gelu_quant(long long M, long long N, long long K, PairDenseConfig* pc) {
  const int force = opt(O_GELU_GEMM);
  if (force == 0 || N % 64 != 0 || !choose_pair_quant_config(M, N, K, pc)) return false;
  if (force > 0 || K >= 768 || M >= 20000) return true;
  const long long groups = M * (N / 64), sms = sm_count();
  PairDenseConfig plain;
  if (groups < sms * 256 || !choose_pair_dense_config(M, N, K, false, &plain))
    return M > 1024 && 1ll * pc->pairs * pc->bn >= (M + arcq::kPairTileM - 1) / arcq::kPairTileM * N;
  const double rounds = static_cast<double>((groups + sms * 512 - 1) / (sms * 512));
  return 1.2 * pc->cost < 5.7 * rounds + plain.cost - 0.3;
}

// ---- packed linear in one launch: configuration ----
struct SmallLinearConfig {
  int R, bn;
  unsigned blocks;
  size_t smem;
  bool captured;     // the faster way in GPU time too
};
// Rows and columns of a block, and whether the one launch is taken: microseconds of GPU time, fitted to every (R, bn) and to the two
// launches on 312 combinations of 20 layers and 1 to 1000 rows, in graphs.  A block's time is passes of 96 groups, rounds of unpacking
// and the products' chain over k; the pair chosen is 1 % slower than the fastest on average, 12 % at worst.  For the comparison the blocks
// count too (3 % rms, the two launches 6 %).
//
// In a captured graph a call costs what the GPU needs, so there the one launch has to be below 0.96 of the two: 88 of the 312, 9 % faster on
// average, 2.5 % slower at worst (64 x 256, 1000 rows).  Elsewhere the host needs 8.8 to 10.2 us for a call of two launches and 5.3 for the one.
// While the two are no longer than that on the GPU, 0.8 us more of it by these costs are taken: K = 192, N = 192, 197 rows 6.0 us against 5.6 in a
// graph, 6.0 against 8.8 a call; 192 x 768, 197 rows 7.0 / 5.6 (the worst of the 312), 7.1 / 8.7 a call; 384 x 1536, 48 rows 7.6 / 7.0 and 7.6 / 8.7; only
// 768 x 3072 with 16 to 24 rows is slower both ways, 10.5 / 9.3 and 10.5 / 10.2.
bool search_small_linear(long long M, long long N, long long K, SmallLinearConfig* c) {
  const int force = opt(O_SMALL_LINEAR);
  const int G = static_cast<int>(K / 64), n = static_cast<int>(N), sms = sm_count();
  constexpr int kPass = arcq::kSmallLinearThreads / 8, kRound = arcq::kSmallLinearThreads * 4;
  // More than one round of blocks can take with four times 96 groups and 384 columns of a group a block: calls on many rows end here.
  if (force < 0 && M * N * G * G > 4ll * sms * kPass * 384) return false;
  const auto part = [](int of, int whole) { return of < whole ? static_cast<double>(of) / whole : 1.0; };
  const auto more = [](int of, int whole) { return (of + whole - 1) / whole - 1; };
  double best = 1.0e9;
  for (int R : {8, 16, 32, 64, 128}) {
    if (opt(O_SMALL_R) > 0 && R != opt(O_SMALL_R)) continue;
    if (R > 8 && R / 2 >= M) break;
    const int row_blocks = (static_cast<int>(M) + R - 1) / R, groups = static_cast<int>(M < R ? M : R) * G;
    const double rows_cost = 4.40 + 2.10 * more(groups, kPass) + 1.23 * part(groups, kPass) + 0.072 * G;
    if (rows_cost > best) break;                               // more rows a block only cost more
    for (int bn : {16, 32, 48, 64, 96, 128, 192, 256}) {
      if (row_blocks * (n / bn) > sms || n % bn != 0 || (opt(O_SMALL_BN) > 0 && bn != opt(O_SMALL_BN))) continue;
      const int chunks = bn * G * 8;
      const double cost = rows_cost + 1.77 * more(chunks, kRound) + 1.77 * part(chunks, kRound);
      if (cost > best) break;
      const size_t smem = arcq::small_linear_smem_layout(R, bn, G).total;
      if (smem > kSmemBudget) break;
      *c = {R, bn, static_cast<unsigned>(row_blocks * (n / bn)), smem, false};
      best = cost;
    }
  }
  if (best == 1.0e9) return false;
  const int groups = static_cast<int>(M < c->R ? M : c->R) * G, chunks = c->bn * G * 8;
  const double one = 4.0 + 2.04 * more(groups, kPass) + 1.2 * part(groups, kPass) + 0.115 * G + 1.78 * more(chunks, kRound) +
                     1.39 * part(chunks, kRound) + 0.63 * c->blocks / sms;
  const double two = 4.38 + 0.0021 * static_cast<double>(K) + 1.365e-6 * static_cast<double>(N * K) + 0.112 * std::log2(static_cast<double>(M));
  c->captured = force > 0 || one <= 0.96 * two;
  return c->captured || one <= (two < 10.0 ? two + 0.8 : two);
}
// The last answer is kept, for the call that follows the question.
bool choose_small_linear(long long M, long long N, long long K, SmallLinearConfig* c) {
  if (opt(O_SMALL_LINEAR) == 0 || M <= 0 || M > 4096 || K % 64 != 0 || N % 16 != 0 || K > (1 << 16) || N > (1 << 20)) return false;
  struct Answer {
    long long M, N, K;
    int force, R, bn, sms;
    bool found;
    SmallLinearConfig c;
  };
  static thread_local Answer last = {};
  const int force = opt(O_SMALL_LINEAR), R = opt(O_SMALL_R), bn = opt(O_SMALL_BN), sms = sm_count();
  if (last.M != M || last.N != N || last.K != K || last.force != force || last.R != R || last.bn != bn || last.sms != sms) {
    last = {M, N, K, force, R, bn, sms, false, {}};
    last.found = search_small_linear(M, N, K, &last.c);
  }
  *c = last.c;
  return last.found;
}

}  // namespace

extern "C" {

int arcq_version(void) { return ARCQ_B200_VERSION; }

const char* arcq_last_error_string(void) { return g_err; }

int arcq_debug_trace(void* device_buffer) {
  g_trace_buf = static_cast<long long*>(device_buffer);
  return ARCQ_OK;
}

int arcq_debug_set_option(const char* name, int value) {
  if (name == nullptr) return fail(ARCQ_E_BAD_ARG, "null option name");
  load_options();
  for (int i = 0; i < O_COUNT; ++i) {
    if (strcmp(name, kOptDefs[i].name) == 0) {
      g_opt[i] = value;
      return ARCQ_OK;
    }
  }
  return fail(ARCQ_E_BAD_ARG, "unknown option %s", name);
}

int arcq_debug_last_gemm_kernel(void) { return g_last_gemm_kernel; }

int arcq_debug_get_option(const char* name, int* value_out) {
  if (name == nullptr || value_out == nullptr) return fail(ARCQ_E_BAD_ARG, "null argument");
  load_options();
  for (int i = 0; i < O_COUNT; ++i) {
    if (strcmp(name, kOptDefs[i].name) == 0) {
      *value_out = g_opt[i];
      return ARCQ_OK;
    }
  }
  return fail(ARCQ_E_BAD_ARG, "unknown option %s", name);
}

int arcq_debug_wait_timeout(unsigned poll_limit, void* stream) {
  if (poll_limit > (1u << 16)) return fail(ARCQ_E_BAD_ARG, "poll_limit above 65536: this entry point is for short waits");
  int* st = status_ptr();
  if (st == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  debug_wait_timeout_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(poll_limit, st);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "debug_wait_timeout launch");
  return ARCQ_OK;
}

int arcq_device_status(void) {
  int v = 0, zero = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return fail(ARCQ_E_CUDA, "device synchronize failed: %s",
                                                          cudaGetErrorString(cudaGetLastError()));
  if (cudaMemcpyFromSymbol(&v, g_status_word, sizeof(int)) != cudaSuccess) return fail(ARCQ_E_CUDA, "status read failed");
  if (v != 0) cudaMemcpyToSymbol(g_status_word, &zero, sizeof(int));
  return v;
}

// The unpack jobs of a call as kernel argument.  Blocks of 128 threads or more, each thread taking four 16-byte chunks a
// round: enough blocks for one round, two per SM at most (they share the SMs with the kernel's own blocks).
static int make_unpack_jobs(const arcq_unpack_job* jobs, int n, arcq::UnpackJobs* out, int max_blocks = 0) {
  *out = arcq::UnpackJobs{};
  if (n == 0) return ARCQ_OK;
  if (jobs == nullptr || n < 0 || n > 2) return fail(ARCQ_E_BAD_ARG, "between 0 and 2 unpack jobs");
  long long chunks = 0;
  for (int i = 0; i < n; ++i) {
    const arcq_unpack_job& j = jobs[i];
    if (!j.packed || !j.mu || !j.sigma || !j.codesum || !j.codebook || !j.out) return fail(ARCQ_E_BAD_ARG, "null pointer in an unpack job");
    if (j.bits < 2 || j.bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", j.bits);
    if (j.rows <= 0 || j.K <= 0 || j.K % 64 != 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape of a weight: rows=%lld K=%lld", (long long)j.rows, (long long)j.K);
    if (!aligned(j.packed, 4) || !aligned(j.out, 16)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte, out 16-byte aligned");
    out->job[i] = arcq::UnpackWeightJob{j.packed, j.mu, j.sigma, j.codesum, j.codebook, static_cast<__half*>(j.out),
                                        static_cast<long long>(j.rows), static_cast<int>(j.K), j.bits};
    chunks += j.rows * (j.K / 8);
  }
  const long long want = (chunks + 511) / 512, cap = max_blocks > 0 ? max_blocks : 2ll * sm_count();
  out->blocks = static_cast<int>(want < cap ? want : cap);
  return ARCQ_OK;
}

// The jobs alone, where there is no kernel for them to go beside.
static int run_unpack_jobs(const arcq_unpack_job* unpack, int n, void* stream) {
  arcq::UnpackJobs jobs;
  if (const int rc = make_unpack_jobs(unpack, n, &jobs)) return rc;
  if (n == 0) return ARCQ_OK;
  launch_pdl(arcq::unpack_jobs_kernel, jobs.blocks, 256, 0, static_cast<cudaStream_t>(stream), jobs);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "unpack launch");
  return ARCQ_OK;
}

static int act_quant_impl(int pre, const void* x, int x_dtype, int64_t M, int64_t K, const float* thresholds,
                          const float* codebook, int bits, int group_size, uint8_t* packed_out, float* mu_out,
                          float* sigma_out, float* codesum_out, void* xhat_out, int xhat_dtype, int one_fma,
                          const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  if (x == nullptr || thresholds == nullptr || codebook == nullptr) return fail(ARCQ_E_BAD_ARG, "null input pointer");
  if (packed_out == nullptr && xhat_out == nullptr) return fail(ARCQ_E_BAD_ARG, "no output requested");
  if ((mu_out != nullptr) != (sigma_out != nullptr)) return fail(ARCQ_E_BAD_ARG, "mu_out and sigma_out go together");
  if (packed_out != nullptr && mu_out == nullptr) return fail(ARCQ_E_BAD_ARG, "packed_out needs mu_out and sigma_out");
  if (codesum_out != nullptr && mu_out == nullptr) return fail(ARCQ_E_BAD_ARG, "codesum_out needs mu_out");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (x_dtype < ARCQ_DT_F32 || x_dtype > ARCQ_DT_BF16) return fail(ARCQ_E_BAD_ARG, "bad x_dtype %d", x_dtype);
  if (xhat_out != nullptr && (xhat_dtype < ARCQ_DT_F32 || xhat_dtype > ARCQ_DT_BF16))
    return fail(ARCQ_E_BAD_ARG, "bad xhat_dtype %d", xhat_dtype);
  if (M < 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
  if (group_size <= 0 || K % group_size != 0)
    return fail(ARCQ_E_BAD_SHAPE, "K=%lld is not a multiple of group_size=%d", (long long)K, group_size);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (packed_out != nullptr && !aligned(packed_out, 4)) return fail(ARCQ_E_ALIGN, "packed_out must be 4-byte aligned");
  if (M == 0) return run_unpack_jobs(unpack, n_unpack, stream);
  arcq::UnpackJobs jobs;
  if (const int rc = make_unpack_jobs(unpack, n_unpack, &jobs)) return rc;
  const long long groups = static_cast<long long>(M) * (K / 64);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (pre == 1) {
    if (x_dtype != ARCQ_DT_F16) return fail(ARCQ_E_UNSUPPORTED, "the fused GELU is built for fp16 input only");
    e = dispatch_act_quant_bits<__half, 1>(bits, x, x_dtype, groups, thresholds, codebook, packed_out, mu_out,
                                           sigma_out, codesum_out, xhat_out, xhat_dtype, st, one_fma, jobs);
  } else if (x_dtype == ARCQ_DT_F32)
    e = dispatch_act_quant_bits<float, 0>(bits, x, x_dtype, groups, thresholds, codebook, packed_out, mu_out, sigma_out,
                                          codesum_out, xhat_out, xhat_dtype, st, one_fma, jobs);
  else if (x_dtype == ARCQ_DT_F16)
    e = dispatch_act_quant_bits<__half, 0>(bits, x, x_dtype, groups, thresholds, codebook, packed_out, mu_out, sigma_out,
                                           codesum_out, xhat_out, xhat_dtype, st, one_fma, jobs);
  else
    e = dispatch_act_quant_bits<__nv_bfloat16, 0>(bits, x, x_dtype, groups, thresholds, codebook, packed_out, mu_out,
                                                  sigma_out, codesum_out, xhat_out, xhat_dtype, st, one_fma, jobs);
  if (e != cudaSuccess) return cuda_fail(e, "act_quant launch");
  return ARCQ_OK;
}

int arcq_act_quant(const void* x, int x_dtype, int64_t M, int64_t K, const float* thresholds, const float* codebook,
                   int bits, int group_size, uint8_t* packed_out, float* mu_out, float* sigma_out, float* codesum_out,
                   void* xhat_out, int xhat_dtype, void* stream) {
  return act_quant_impl(0, x, x_dtype, M, K, thresholds, codebook, bits, group_size, packed_out, mu_out, sigma_out,
                        codesum_out, xhat_out, xhat_dtype, 0, nullptr, 0, stream);
}

int arcq_gelu_act_quant(const void* x, int x_dtype, int64_t M, int64_t K, const float* thresholds,
                        const float* codebook, int bits, int group_size, uint8_t* packed_out, float* mu_out,
                        float* sigma_out, float* codesum_out, void* xhat_out, int xhat_dtype, void* stream) {
  return act_quant_impl(1, x, x_dtype, M, K, thresholds, codebook, bits, group_size, packed_out, mu_out, sigma_out,
                        codesum_out, xhat_out, xhat_dtype, 0, nullptr, 0, stream);
}

int arcq_act_quant_unpack(int pre_gelu, const void* x, int x_dtype, int64_t M, int64_t K, const float* thresholds,
                          const float* codebook, int bits, int group_size, void* xhat_out, int xhat_dtype, int one_fma,
                          const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  return act_quant_impl(pre_gelu != 0, x, x_dtype, M, K, thresholds, codebook, bits, group_size, nullptr, nullptr, nullptr, nullptr,
                        xhat_out, xhat_dtype, one_fma != 0, unpack, n_unpack, stream);
}

int arcq_packed_gemm(const uint8_t* packed_x, const float* mu_a, const float* sigma_a, const float* codesum_a,
                     const uint8_t* packed_w, const float* mu_w, const float* sigma_w, const float* codesum_w,
                     const float* act_codebook, const float* w_codebook, const float* bias, int bits, int group_size,
                     int64_t M, int64_t N, int64_t K, void* y, int y_dtype, void* stream) {
  if (!packed_x || !mu_a || !sigma_a || !codesum_a || !packed_w || !mu_w || !sigma_w || !codesum_w ||
      !act_codebook || !w_codebook || !y)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (group_size <= 0 || K % group_size != 0)
    return fail(ARCQ_E_BAD_SHAPE, "K=%lld is not a multiple of group_size=%d", (long long)K, group_size);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (N % 8 != 0) return fail(ARCQ_E_BAD_SHAPE, "N=%lld must be a multiple of 8", (long long)N);
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(packed_x, 4) || !aligned(packed_w, 4)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte aligned");
  if (!aligned(y, 16)) return fail(ARCQ_E_ALIGN, "y must be 16-byte aligned");
  if (M == 0) return ARCQ_OK;

  arcq::GemmParams p;
  p.pa = packed_x; p.mu_a = mu_a; p.sg_a = sigma_a; p.cs_a = codesum_a;
  p.pw = packed_w; p.mu_w = mu_w; p.sg_w = sigma_w; p.cs_w = codesum_w;
  p.cb_a = act_codebook; p.cb_w = w_codebook; p.bias = bias; p.y = y;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K); p.G = static_cast<int>(K / 64);
  p.pc = static_cast<int>(K * bits / 8);
  p.bn = choose_bn(M, N);
  p.y_f32 = (y_dtype == ARCQ_DT_F32) ? 1 : 0;
  p.status = status_ptr();
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");

  const size_t smem = arcq::packed_gemm_smem_bytes(p.bn);
  dim3 grid(static_cast<unsigned>((M + arcq::kTileM - 1) / arcq::kTileM), static_cast<unsigned>((N + p.bn - 1) / p.bn));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
#define ARCQ_LAUNCH_GEMM(B)                                                                                  \
  do {                                                                                                       \
    e = cudaFuncSetAttribute(arcq::packed_gemm_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                             static_cast<int>(smem));                                                        \
    if (e == cudaSuccess) {                                                                                  \
      launch_pdl(arcq::packed_gemm_kernel<B>, grid, arcq::kGemmThreads, smem, st, p);                         \
      e = cudaGetLastError();                                                                                \
    }                                                                                                        \
  } while (0)
  if (bits == 4) ARCQ_LAUNCH_GEMM(4);
  else if (bits == 3) ARCQ_LAUNCH_GEMM(3);
  else ARCQ_LAUNCH_GEMM(2);
#undef ARCQ_LAUNCH_GEMM
  if (e != cudaSuccess) return cuda_fail(e, "packed_gemm launch");
  return ARCQ_OK;
}


// Launch of the persistent GEMM for either weight form: packed codes + statistics (rebuilt in shared
// memory) or an fp16 matrix (`dense`; mu_w .. w_codebook unused).  Arguments are already validated.
static int launch_ws_gemm(bool dense, const void* xhat, const void* w, const float* mu_w, const float* sigma_w,
                          const float* codesum_w, const float* w_codebook, const float* bias, int bits, int64_t M,
                          int64_t N, int64_t K, void* y, int y_dtype, void* stream) {
  g_last_gemm_kernel = dense ? ARCQ_GEMM_ONE_CTA_DENSE : ARCQ_GEMM_ONE_CTA_PACKED;
  WsConfig cfg;
  if (!choose_ws_config(M, N, K, bits, dense, &cfg)) return fail(ARCQ_E_UNSUPPORTED, "no tile configuration for this shape");

  CUtensorMap tm_a, tm_w;
  if (!make_tensor_map_2d(&tm_a, xhat, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(M),
                          static_cast<uint64_t>(K), 64, arcq::kTileM, CU_TENSOR_MAP_SWIZZLE_128B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the activation matrix");
  if (dense) {
    if (!make_tensor_map_2d(&tm_w, w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(N),
                            static_cast<uint64_t>(K), 64, cfg.bn, CU_TENSOR_MAP_SWIZZLE_128B))
      return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the weight matrix");
  } else if (!make_tensor_map_2d(&tm_w, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, static_cast<uint64_t>(N),
                                 static_cast<uint64_t>(K * bits / 8), arcq::raw_row_bytes(bits), cfg.bn,
                                 CU_TENSOR_MAP_SWIZZLE_NONE)) {
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the packed weight");
  }

  // output tensor map for the TMA-store epilogue: 32-row blocks of 64 bytes (32 fp16 / 16 fp32 columns)
  const int out_cw = (y_dtype == ARCQ_DT_F32) ? 16 : 32;
  const bool use_tma_store = (cfg.bn % out_cw == 0) && opt(O_WS_TMA_STORE) != 0;
  CUtensorMap tm_y;
  if (!make_tensor_map_2d(&tm_y, y, (y_dtype == ARCQ_DT_F32) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                          (y_dtype == ARCQ_DT_F32) ? 4 : 2, static_cast<uint64_t>(M), static_cast<uint64_t>(N),
                          out_cw, 32, CU_TENSOR_MAP_SWIZZLE_64B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the output matrix");

  arcq::WsParams p;
  p.tma_store = use_tma_store ? 1 : 0;
  p.rotate = opt(O_WS_ROTATE);
  p.mu_w = mu_w; p.sg_w = sigma_w; p.cs_w = codesum_w; p.cb_w = w_codebook; p.bias = bias; p.y = y;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K); p.G = static_cast<int>(K / 64);
  p.bn = cfg.bn; p.ws = cfg.ws; p.sa = cfg.sa; p.nbb = cfg.nbb; p.stationary = cfg.stationary;
  p.dense = dense ? 1 : 0;
  p.y_f32 = (y_dtype == ARCQ_DT_F32) ? 1 : 0;
  p.status = status_ptr();
  p.trace = g_trace_buf;
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
#define ARCQ_LAUNCH_WS_T(B, T)                                                                                     \
  do {                                                                                                             \
    e = cudaFuncSetAttribute(arcq::packed_weight_gemm_ws_kernel<B, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                             static_cast<int>(cfg.smem));                                                          \
    if (e == cudaSuccess) {                                                                                        \
      launch_pdl(arcq::packed_weight_gemm_ws_kernel<B, T>, cfg.grid, arcq::kWsThreads, cfg.smem, st, tm_a, tm_w, tm_y, p); \
      e = cudaGetLastError();                                                                                      \
    }                                                                                                              \
  } while (0)
  // the instantiation with time stamps runs only while arcq_debug_trace() has a buffer registered
#define ARCQ_LAUNCH_WS(B)                                                                                          \
  do {                                                                                                             \
    if (p.trace != nullptr) ARCQ_LAUNCH_WS_T(B, true);                                                             \
    else ARCQ_LAUNCH_WS_T(B, false);                                                                               \
  } while (0)
  if (bits == 4) ARCQ_LAUNCH_WS(4);
  else if (bits == 3) ARCQ_LAUNCH_WS(3);
  else ARCQ_LAUNCH_WS(2);
#undef ARCQ_LAUNCH_WS_T
#undef ARCQ_LAUNCH_WS
  if (e != cudaSuccess) return cuda_fail(e, "packed_weight_gemm launch");
  return ARCQ_OK;
}

// Launch of the CTA-pair kernel (packed weight form only).  Arguments are already validated.
static int launch_pair_gemm(const PairConfig& cfg, const void* xhat, const void* w, const float* mu_w,
                            const float* sigma_w, const float* codesum_w, const float* w_codebook, const float* bias,
                            int bits, int64_t M, int64_t N, int64_t K, void* y, int y_dtype, void* stream) {
  CUtensorMap tm_a, tm_y;
  if (!make_tensor_map_2d(&tm_a, xhat, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(M),
                          static_cast<uint64_t>(K), 64, arcq::kTileM, CU_TENSOR_MAP_SWIZZLE_128B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the activation matrix");
  const int out_cw = (y_dtype == ARCQ_DT_F32) ? 16 : 32;
  if (!make_tensor_map_2d(&tm_y, y, (y_dtype == ARCQ_DT_F32) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                          (y_dtype == ARCQ_DT_F32) ? 4 : 2, static_cast<uint64_t>(M), static_cast<uint64_t>(N),
                          out_cw, 32, CU_TENSOR_MAP_SWIZZLE_64B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the output matrix");
  arcq::PairParams p;
  p.pw = static_cast<const uint8_t*>(w); p.pc = static_cast<int>(K * bits / 8);
  p.mu_w = mu_w; p.sg_w = sigma_w; p.cs_w = codesum_w; p.cb_w = w_codebook; p.bias = bias; p.y = y;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K); p.G = static_cast<int>(K / 64);
  p.bn = cfg.bn; p.ws = cfg.ws; p.sa = cfg.sa; p.ks = cfg.ks; p.nbb = cfg.nbb; p.stationary = cfg.stationary;
  p.lut_shift = cfg.lut_shift;
  p.y_f32 = (y_dtype == ARCQ_DT_F32) ? 1 : 0;
  p.poll_limit = static_cast<uint32_t>(opt(O_POLL_LIMIT));
  p.spin_limit = static_cast<uint32_t>(opt(O_SPIN_LIMIT));
  p.status = status_ptr();
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = static_cast<unsigned>(2 * cfg.pairs);
  // the dynamic shared-memory ceiling of the kernel was raised when the configuration was chosen
#define ARCQ_LAUNCH_PAIR(B)                                                                                              \
  do {                                                                                                                  \
    if (cfg.stationary)                                                                                                 \
      launch_pdl(arcq::packed_weight_gemm_pair_kernel<B, true>, grid, arcq::kPairThreads, cfg.smem, st, tm_a, tm_y, p);  \
    else                                                                                                                \
      launch_pdl(arcq::packed_weight_gemm_pair_kernel<B, false>, grid, arcq::kPairThreads, cfg.smem, st, tm_a, tm_y, p); \
  } while (0)
  if (bits == 4) ARCQ_LAUNCH_PAIR(4);
  else if (bits == 3) ARCQ_LAUNCH_PAIR(3);
  else ARCQ_LAUNCH_PAIR(2);
#undef ARCQ_LAUNCH_PAIR
  g_last_gemm_kernel = ARCQ_GEMM_PAIR_PACKED;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "packed_weight_gemm (pair) launch");
  return ARCQ_OK;
}

static int launch_pair_dense_gemm(const PairDenseConfig& cfg, const void* xhat, const void* w16, const float* bias,
                                  int64_t M, int64_t N, int64_t K, void* y, int y_dtype, void* stream,
                                  const arcq::UnpackWeightJob* next = nullptr, const arcq::UnpackJobs& jobs = {},
                                  const float* q_thresholds = nullptr, const float* q_codebook = nullptr, int q_bits = 0) {
  CUtensorMap tm_a, tm_w, tm_y;
  if (!make_tensor_map_2d(&tm_a, xhat, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(M),
                          static_cast<uint64_t>(K), 64, arcq::kTileM, CU_TENSOR_MAP_SWIZZLE_128B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the activation matrix");
  if (!make_tensor_map_2d(&tm_w, w16, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(N),
                          static_cast<uint64_t>(K), 64, cfg.bn / 2, CU_TENSOR_MAP_SWIZZLE_128B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the weight matrix");
  // 64 bytes of a row per store; a whole group of 64 values in the quantizer form
  const int out_cw = q_bits != 0 ? 64 : (y_dtype == ARCQ_DT_F32) ? 16 : 32;
  if (!make_tensor_map_2d(&tm_y, y, (y_dtype == ARCQ_DT_F32) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                          (y_dtype == ARCQ_DT_F32) ? 4 : 2, static_cast<uint64_t>(M), static_cast<uint64_t>(N),
                          out_cw, 32, q_bits != 0 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the output matrix");
  arcq::PairDenseParams p;
  p.pairs = cfg.pairs;
  p.thresholds = q_thresholds;
  p.codebook = q_codebook;
  p.bias = bias;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K); p.G = static_cast<int>(K / 64);
  p.bn = cfg.bn; p.sa = cfg.sa; p.ks = cfg.ks; p.split_last = cfg.split_last; p.stagger = cfg.stagger;
  p.y_f32 = (y_dtype == ARCQ_DT_F32) ? 1 : 0;
  p.poll_limit = static_cast<uint32_t>(opt(O_POLL_LIMIT));
  p.spin_limit = static_cast<uint32_t>(opt(O_SPIN_LIMIT));
  p.status = status_ptr();
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  p.next = arcq::UnpackWeightJob{};
  if (next != nullptr) p.next = *next;
  const unsigned grid = static_cast<unsigned>(2 * cfg.pairs + jobs.blocks);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (q_bits != 0) {
    auto launch = [&](auto kernel, int* done_dev) {
      int dev = 0;
      cudaGetDevice(&dev);
      if (*done_dev != dev) {                   // once per (thread, device)
        const int rc = prepare_register_kernel(kernel, kSmemBudget + 1024, arcq::kPairQuantLaunchRegs, "dense_weight_gemm_gelu_quant");
        if (rc != ARCQ_OK) return rc;
        *done_dev = dev;
      }
      launch_pdl(kernel, grid, arcq::kPairQuantThreads, cfg.smem, st, tm_a, tm_w, tm_y, p, jobs);
      const cudaError_t e = cudaGetLastError();
      return e != cudaSuccess ? cuda_fail(e, "dense_weight_gemm_gelu_quant launch") : ARCQ_OK;
    };
    static thread_local int done[6] = {-1, -1, -1, -1, -1, -1};
    int rc;
    if (cfg.stationary)
      rc = q_bits == 4 ? launch(arcq::dense_weight_gemm_pair_kernel<true, false, 4>, done)
          : q_bits == 3 ? launch(arcq::dense_weight_gemm_pair_kernel<true, false, 3>, done + 1)
                        : launch(arcq::dense_weight_gemm_pair_kernel<true, false, 2>, done + 2);
    else
      rc = q_bits == 4 ? launch(arcq::dense_weight_gemm_pair_kernel<false, false, 4>, done + 3)
          : q_bits == 3 ? launch(arcq::dense_weight_gemm_pair_kernel<false, false, 3>, done + 4)
                        : launch(arcq::dense_weight_gemm_pair_kernel<false, false, 2>, done + 5);
    g_last_gemm_kernel = ARCQ_GEMM_PAIR_DENSE_GELU_QUANT;
    return rc;
  }
  if (next != nullptr) {
    static thread_local int done_dev = -1;      // the prefetch form's shared-memory ceiling, once per (thread, device)
    int dev = 0;
    cudaGetDevice(&dev);
    if (done_dev != dev) {
      cudaFuncSetAttribute(arcq::dense_weight_gemm_pair_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemBudget + 1024));
      cudaFuncSetAttribute(arcq::dense_weight_gemm_pair_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemBudget + 1024));
      done_dev = dev;
    }
    if (cfg.stationary)
      launch_pdl(arcq::dense_weight_gemm_pair_kernel<true, true>, grid, arcq::kPairDenseThreads, cfg.smem, st, tm_a, tm_w, tm_y, p, jobs);
    else
      launch_pdl(arcq::dense_weight_gemm_pair_kernel<false, true>, grid, arcq::kPairDenseThreads, cfg.smem, st, tm_a, tm_w, tm_y, p, jobs);
  } else if (cfg.stationary) {
    launch_pdl(arcq::dense_weight_gemm_pair_kernel<true>, grid, arcq::kPairDenseThreads, cfg.smem, st, tm_a, tm_w, tm_y, p, jobs);
  } else {
    launch_pdl(arcq::dense_weight_gemm_pair_kernel<false>, grid, arcq::kPairDenseThreads, cfg.smem, st, tm_a, tm_w, tm_y, p, jobs);
  }
  g_last_gemm_kernel = next != nullptr ? ARCQ_GEMM_PAIR_DENSE_PREFETCH : ARCQ_GEMM_PAIR_DENSE;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "dense_weight_gemm (pair) launch");
  return ARCQ_OK;
}

int arcq_packed_weight_gemm(const void* xhat, const uint8_t* packed_w, const float* mu_w, const float* sigma_w,
                            const float* codesum_w, const float* w_codebook, const float* bias, int bits,
                            int group_size, int64_t M, int64_t N, int64_t K, void* y, int y_dtype, void* stream) {
  if (!xhat || !packed_w || !mu_w || !sigma_w || !codesum_w || !w_codebook || !y)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (group_size <= 0 || K % group_size != 0)
    return fail(ARCQ_E_BAD_SHAPE, "K=%lld is not a multiple of group_size=%d", (long long)K, group_size);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (N % 16 != 0) return fail(ARCQ_E_UNSUPPORTED, "N=%lld: this entry point needs N %% 16 == 0", (long long)N);
  if ((K * bits / 8) % 16 != 0)
    return fail(ARCQ_E_UNSUPPORTED, "packed row of %lld bytes is not a multiple of 16 (TMA stride rule)",
                (long long)(K * bits / 8));
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(xhat, 16) || !aligned(packed_w, 16) || !aligned(y, 16))
    return fail(ARCQ_E_ALIGN, "xhat, packed_w and y must be 16-byte aligned");
  if (M == 0) return ARCQ_OK;
  PairConfig pc;
  if (choose_pair_config(M, N, K, bits, y_dtype == ARCQ_DT_F32, &pc))
    return launch_pair_gemm(pc, xhat, packed_w, mu_w, sigma_w, codesum_w, w_codebook, bias, bits, M, N, K, y, y_dtype,
                            stream);
  return launch_ws_gemm(false, xhat, packed_w, mu_w, sigma_w, codesum_w, w_codebook, bias, bits, M, N, K, y, y_dtype,
                        stream);
}

// Unpack jobs for the SMs that `pairs` CTA pairs leave idle, in whole pairs of blocks.
static int make_idle_jobs(const arcq_unpack_job* unpack, int n_unpack, int pairs, arcq::UnpackJobs* jobs) {
  const int idle = sm_count() - 2 * pairs;
  const int rc = make_unpack_jobs(unpack, n_unpack, jobs, idle > 2 ? idle : 2);
  jobs->blocks = (jobs->blocks + 1) / 2 * 2;
  return rc;
}

static int dense_weight_gemm_impl(const void* xhat, const void* w16, const float* bias, int64_t M, int64_t N, int64_t K,
                                  void* y, int y_dtype, const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  if (!xhat || !w16 || !y) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (K % 64 != 0) return fail(ARCQ_E_UNSUPPORTED, "K=%lld: this entry point needs K %% 64 == 0", (long long)K);
  if (N % 16 != 0) return fail(ARCQ_E_UNSUPPORTED, "N=%lld: this entry point needs N %% 16 == 0", (long long)N);
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(xhat, 16) || !aligned(w16, 16) || !aligned(y, 16))
    return fail(ARCQ_E_ALIGN, "xhat, w16 and y must be 16-byte aligned");
  if (M == 0 && n_unpack == 0) return ARCQ_OK;
  PairDenseConfig pc;
  if (M > 0 && choose_pair_dense_config(M, N, K, y_dtype == ARCQ_DT_F32, &pc)) {
    arcq::UnpackJobs jobs;
    if (const int rc = make_idle_jobs(unpack, n_unpack, pc.pairs, &jobs)) return rc;
    return launch_pair_dense_gemm(pc, xhat, w16, bias, M, N, K, y, y_dtype, stream, nullptr, jobs);
  }
  // no pair configuration (or nothing to multiply): the unpack by its own kernel
  if (const int rc = run_unpack_jobs(unpack, n_unpack, stream)) return rc;
  if (M == 0) return ARCQ_OK;
  return launch_ws_gemm(true, xhat, w16, nullptr, nullptr, nullptr, nullptr, bias, 4, M, N, K, y, y_dtype, stream);
}

int arcq_dense_weight_gemm(const void* xhat, const void* w16, const float* bias, int64_t M, int64_t N, int64_t K,
                           void* y, int y_dtype, void* stream) {
  return dense_weight_gemm_impl(xhat, w16, bias, M, N, K, y, y_dtype, nullptr, 0, stream);
}

int arcq_dense_weight_gemm_unpack(const void* xhat, const void* w16, const float* bias, int64_t M, int64_t N, int64_t K,
                                  void* y, int y_dtype, const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  if (n_unpack < 0 || n_unpack > 2 || (n_unpack > 0 && unpack == nullptr)) return fail(ARCQ_E_BAD_ARG, "between 0 and 2 unpack jobs");
  return dense_weight_gemm_impl(xhat, w16, bias, M, N, K, y, y_dtype, unpack, n_unpack, stream);
}

// Unpack jobs beside GEMMs or beside the LayerNorm + quantizer: where that takes its latency form, blocks added to it lengthen
// it, and where it takes the tile form they do not.  Whole forwards through a graph (LayerNorm / GEMM): DeiT-S batch 1 554 / 506,
// batch 6 714 / 628, batch 8 724 / 772 us; DeiT-T batch 12 613 / 570, batch 16 656 / 689 us; DeiT-B batch 3 898 / 793, batch 4
// 867 / 923 us: the line between the two forms runs through each of these.
int arcq_unpack_beside_gemm(int64_t M, int64_t width) { return small_layernorm_quant(M, width) && opt(O_GEMM_UNPACK) != 0 ? 1 : 0; }

int64_t arcq_dense_weight_gemm_unpack_room(int64_t M, int64_t N, int64_t K, int gelu_quant) {
  PairDenseConfig pc;
  if (M <= 0 || N <= 0 || K <= 0 || K % 64 != 0 || N % 16 != 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return 0;
  if (!(gelu_quant ? choose_gelu_quant(M, N, K, &pc) : choose_pair_dense_config(M, N, K, false, &pc))) return 0;
  // five rounds of four chunks of eight values per thread: about what a GEMM of a few hundred rows takes itself
  const long long idle = sm_count() - 2 * pc.pairs;
  return idle > 0 ? idle * arcq::kPairDenseThreads * 160 : 0;
}

int arcq_dense_weight_gemm_gelu_quant_applies(int64_t M, int64_t N, int64_t K) {
  PairDenseConfig pc;
  if (M <= 0 || N <= 0 || K <= 0 || K % 64 != 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return 0;
  return choose_gelu_quant(M, N, K, &pc) ? 1 : 0;
}

int arcq_dense_weight_gemm_gelu_quant(const void* xhat, const void* w16, const float* bias, int64_t M, int64_t N, int64_t K,
                                      const float* thresholds, const float* codebook, int bits, int group_size, void* out,
                                      const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  if (!xhat || !w16 || !out || !thresholds || !codebook) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (K % 64 != 0 || N % 64 != 0) return fail(ARCQ_E_UNSUPPORTED, "K=%lld, N=%lld: this entry point needs multiples of 64", (long long)K, (long long)N);
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(xhat, 16) || !aligned(w16, 16) || !aligned(out, 16))
    return fail(ARCQ_E_ALIGN, "xhat, w16 and out must be 16-byte aligned");
  if (M == 0 && n_unpack != 0) return fail(ARCQ_E_BAD_SHAPE, "no rows to unpack weights beside");
  if (M == 0) return ARCQ_OK;
  PairDenseConfig pc;
  if (!choose_gelu_quant(M, N, K, &pc))
    return fail(ARCQ_E_UNSUPPORTED, "M=%lld, N=%lld, K=%lld: left to arcq_dense_weight_gemm and arcq_gelu_act_quant", (long long)M, (long long)N, (long long)K);
  arcq::UnpackJobs jobs;
  if (const int rc = make_idle_jobs(unpack, n_unpack, pc.pairs, &jobs)) return rc;
  return launch_pair_dense_gemm(pc, xhat, w16, bias, M, N, K, out, ARCQ_DT_F16, stream, nullptr, jobs, thresholds, codebook, bits);
}

int arcq_packed_linear_small_applies(int64_t M, int64_t N, int64_t K) {
  SmallLinearConfig c;
  return choose_small_linear(M, N, K, &c) ? 1 : 0;
}

int arcq_packed_linear_small_applies_captured(int64_t M, int64_t N, int64_t K) {
  SmallLinearConfig c;
  return choose_small_linear(M, N, K, &c) && c.captured ? 1 : 0;
}

int arcq_packed_linear_small(int pre_gelu, const void* x, int x_dtype, int64_t M, const float* thresholds, const float* codebook,
                             int one_fma, const arcq_unpack_job* weight, const float* bias, void* y, int y_dtype, void* stream) {
  if (!x || !thresholds || !codebook || !weight || !weight->packed || !weight->mu || !weight->sigma || !weight->codesum || !weight->codebook || !y)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  const int bits = weight->bits;
  const int64_t N = weight->rows, K = weight->K;
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (x_dtype < ARCQ_DT_F32 || x_dtype > ARCQ_DT_BF16) return fail(ARCQ_E_BAD_ARG, "bad x_dtype %d", x_dtype);
  if (pre_gelu && x_dtype != ARCQ_DT_F16) return fail(ARCQ_E_UNSUPPORTED, "the fused GELU is built for fp16 input only");
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
  if (K % 64 != 0 || N % 16 != 0) return fail(ARCQ_E_UNSUPPORTED, "K=%lld, N=%lld: this entry point needs multiples of 64 and 16", (long long)K, (long long)N);
  if (!aligned(weight->packed, 4) || !aligned(y, 16)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte, y 16-byte aligned");
  if (M == 0) return ARCQ_OK;
  SmallLinearConfig c;
  if (!choose_small_linear(M, N, K, &c))
    return fail(ARCQ_E_UNSUPPORTED, "M=%lld, N=%lld, K=%lld: left to arcq_act_quant_unpack and arcq_dense_weight_gemm", (long long)M, (long long)N, (long long)K);
  arcq::SmallLinearParams p;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K); p.G = static_cast<int>(K / 64);
  p.R = c.R; p.bn = c.bn;
  p.thresholds = thresholds; p.codebook = codebook; p.one_fma = one_fma != 0;
  p.weight = arcq::UnpackWeightJob{weight->packed, weight->mu, weight->sigma, weight->codesum, weight->codebook, nullptr, N, p.K, bits};
  p.bias = bias; p.y = y; p.y_f32 = y_dtype == ARCQ_DT_F32;
  p.tmem_cols = 32;
  while (p.tmem_cols < static_cast<uint32_t>(c.bn)) p.tmem_cols *= 2;
  p.poll_limit = static_cast<uint32_t>(opt(O_POLL_LIMIT));
  p.status = status_ptr();
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  auto launch = [&](auto kernel, auto type, int* done_dev) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (*done_dev != dev) {                   // once per (thread, device)
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemBudget));
      if (e != cudaSuccess) return cuda_fail(e, "packed_linear_small");
      *done_dev = dev;
    }
    launch_pdl(kernel, c.blocks, arcq::kSmallLinearThreads, c.smem, static_cast<cudaStream_t>(stream), static_cast<const decltype(type)*>(x), p);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? cuda_fail(e, "packed_linear_small launch") : ARCQ_OK;
  };
  static thread_local int done[12] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
  auto by_bits = [&](auto type, auto pre, int* d) {
    using T = decltype(type);
    constexpr int PRE = decltype(pre)::value;
    return bits == 4 ? launch(arcq::small_linear_kernel<T, 4, PRE>, type, d)
           : bits == 3 ? launch(arcq::small_linear_kernel<T, 3, PRE>, type, d + 1) : launch(arcq::small_linear_kernel<T, 2, PRE>, type, d + 2);
  };
  g_last_gemm_kernel = ARCQ_GEMM_SMALL_LINEAR;
  if (pre_gelu) return by_bits(__half(), std::integral_constant<int, 1>(), done);
  if (x_dtype == ARCQ_DT_F16) return by_bits(__half(), std::integral_constant<int, 0>(), done + 3);
  if (x_dtype == ARCQ_DT_F32) return by_bits(float(), std::integral_constant<int, 0>(), done + 6);
  return by_bits(__nv_bfloat16(), std::integral_constant<int, 0>(), done + 9);
}

int arcq_dense_weight_gemm_prefetch(const void* xhat, const void* w16, const float* bias, int64_t M, int64_t N,
                                    int64_t K, void* y, int y_dtype, const uint8_t* next_packed, const float* next_mu,
                                    const float* next_sigma, const float* next_codesum, const float* next_codebook,
                                    int next_bits, int next_group_size, int64_t next_rows, int64_t next_K,
                                    void* next_out, void* stream) {
  if (!next_packed || !next_mu || !next_sigma || !next_codesum || !next_codebook || !next_out)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (next_bits < 2 || next_bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", next_bits);
  if (next_group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", next_group_size);
  if (next_rows <= 0 || next_K <= 0 || next_K % 64 != 0)
    return fail(ARCQ_E_BAD_SHAPE, "bad shape of the next weight: rows=%lld K=%lld", (long long)next_rows, (long long)next_K);
  if (!aligned(next_packed, 4) || !aligned(next_out, 16))
    return fail(ARCQ_E_ALIGN, "next packed codes must be 4-byte, next_out 16-byte aligned");
  if (!xhat || !w16 || !y) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (K % 64 != 0) return fail(ARCQ_E_UNSUPPORTED, "K=%lld: this entry point needs K %% 64 == 0", (long long)K);
  if (N % 16 != 0) return fail(ARCQ_E_UNSUPPORTED, "N=%lld: this entry point needs N %% 16 == 0", (long long)N);
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(xhat, 16) || !aligned(w16, 16) || !aligned(y, 16))
    return fail(ARCQ_E_ALIGN, "xhat, w16 and y must be 16-byte aligned");
  const arcq::UnpackWeightJob job = {next_packed, next_mu, next_sigma, next_codesum, next_codebook,
                                     static_cast<__half*>(next_out), static_cast<long long>(next_rows),
                                     static_cast<int>(next_K), next_bits};
  PairDenseConfig pc;
  if (M > 0 && choose_pair_dense_config(M, N, K, y_dtype == ARCQ_DT_F32, &pc))
    return launch_pair_dense_gemm(pc, xhat, w16, bias, M, N, K, y, y_dtype, stream, &job);
  // no pair configuration (or nothing to multiply): the GEMM by the one-CTA kernel, the unpack by its own kernel
  if (M > 0) {
    const int rc = launch_ws_gemm(true, xhat, w16, nullptr, nullptr, nullptr, nullptr, bias, 4, M, N, K, y, y_dtype, stream);
    if (rc != ARCQ_OK) return rc;
  }
  return arcq_unpack_weight_f16(next_packed, next_mu, next_sigma, next_codesum, next_codebook, next_bits, next_group_size,
                                next_rows, next_K, next_out, stream);
}

int arcq_add_layernorm(const void* x, const void* y, const float* gamma, const float* beta, float eps, int64_t M,
                       int64_t K, void* sum_out, void* h_out, void* stream) {
  return arcq_add_layernorm_strided(x, y, gamma, beta, ARCQ_DT_F32, eps, M, K, K, sum_out, h_out, stream);
}

int arcq_add_layernorm_strided(const void* x, const void* y, const void* gamma, const void* beta, int param_dtype, float eps,
                               int64_t M, int64_t K, int64_t ld, void* sum_out, void* h_out, void* stream) {
  if (x == nullptr || gamma == nullptr || beta == nullptr || h_out == nullptr)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (param_dtype < ARCQ_DT_F32 || param_dtype > ARCQ_DT_BF16) return fail(ARCQ_E_BAD_ARG, "bad param_dtype %d", param_dtype);
  if (M < 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
  if (K % 8 != 0) return fail(ARCQ_E_BAD_SHAPE, "K=%lld must be a multiple of 8", (long long)K);
  if (ld < K || ld % 8 != 0) return fail(ARCQ_E_BAD_SHAPE, "row stride %lld must be a multiple of 8, at least K", (long long)ld);
  if (K > 32 * 8 * arcq::kLnMaxChunks) return fail(ARCQ_E_TOO_LARGE, "rows longer than %d values are not built", 32 * 8 * arcq::kLnMaxChunks);
  if (!aligned(x, 16) || !aligned(h_out, 16) || (y != nullptr && !aligned(y, 16)) ||
      (sum_out != nullptr && !aligned(sum_out, 16)) || !aligned(gamma, 16) || !aligned(beta, 16))
    return fail(ARCQ_E_ALIGN, "all buffers must be 16-byte aligned");
  if (M == 0) return ARCQ_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half *xh = static_cast<const __half*>(x), *yh = static_cast<const __half*>(y);
  __half *so = static_cast<__half*>(sum_out), *ho = static_cast<__half*>(h_out);
  const arcq::NormParams np = {gamma, beta, param_dtype};
  const bool plain = opt(O_LN_PLAIN) != 0;
  if (K == 384 && !plain) {          // 16 lanes per row, 2 rows per warp
    launch_pdl(arcq::add_layernorm_rows_kernel<16>, grid_for(M, 16, 6), 256, 0, st, xh, yh, np, eps, M, ld, so, ho);
  } else if (K == 192 && !plain) {
    launch_pdl(arcq::add_layernorm_rows_kernel<8>, grid_for(M, 32, 6), 256, 0, st, xh, yh, np, eps, M, ld, so, ho);
  } else if (K == 768 && !plain) {
    launch_pdl(arcq::add_layernorm_rows_kernel<32>, grid_for(M, 8, 6), 256, 0, st, xh, yh, np, eps, M, ld, so, ho);
  } else {
    launch_pdl(arcq::add_layernorm_kernel, grid_for(M, 8, 8), 256, 0, st, xh, yh, np, eps, M, static_cast<int>(K), ld, so, ho);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "add_layernorm launch");
  return ARCQ_OK;
}

int arcq_add_layernorm_act_quant(const void* x, const void* y, const float* gamma, const float* beta, float eps,
                                 int64_t M, int64_t K, const float* thresholds, const float* codebook, int bits,
                                 int group_size, void* sum_out, void* h_out, void* xhat, void* stream) {
  return arcq_add_layernorm_act_quant_unpack(x, y, gamma, beta, ARCQ_DT_F32, eps, M, K, thresholds, codebook, bits, group_size,
                                             sum_out, h_out, xhat, 0, nullptr, 0, stream);
}

int arcq_add_layernorm_act_quant_unpack(const void* x, const void* y, const void* gamma, const void* beta, int param_dtype,
                                        float eps, int64_t M, int64_t K, const float* thresholds, const float* codebook,
                                        int bits, int group_size, void* sum_out, void* h_out, void* xhat, int one_fma,
                                        const arcq_unpack_job* unpack, int n_unpack, void* stream) {
  if (x == nullptr || gamma == nullptr || beta == nullptr || thresholds == nullptr || codebook == nullptr || xhat == nullptr)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (param_dtype < ARCQ_DT_F32 || param_dtype > ARCQ_DT_BF16) return fail(ARCQ_E_BAD_ARG, "bad param_dtype %d", param_dtype);
  if (M < 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
  if (K % 64 != 0) return fail(ARCQ_E_BAD_SHAPE, "K=%lld is not a multiple of the group size 64", (long long)K);
  if (K != 192 && K != 384 && K != 768)
    return fail(ARCQ_E_UNSUPPORTED, "K=%lld: the merged kernel is built for rows of 192, 384 and 768 values", (long long)K);
  if (y == nullptr && sum_out != nullptr) return fail(ARCQ_E_BAD_ARG, "sum_out without y");
  if (!aligned(x, 16) || !aligned(xhat, 16) || (y != nullptr && !aligned(y, 16)) ||
      (sum_out != nullptr && !aligned(sum_out, 16)) || (h_out != nullptr && !aligned(h_out, 16)) || !aligned(gamma, 16) || !aligned(beta, 16))
    return fail(ARCQ_E_ALIGN, "all matrices and the parameters must be 16-byte aligned");
  if (M == 0) return run_unpack_jobs(unpack, n_unpack, stream);
  arcq::UnpackJobs jobs;
  if (const int rc = make_unpack_jobs(unpack, n_unpack, &jobs)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const arcq::NormParams np = {gamma, beta, param_dtype};
  const int G = static_cast<int>(K / 64);
  {
    const bool small = small_layernorm_quant(M, K);
    if (small) {
      const __half *xs = static_cast<const __half*>(x), *ys = static_cast<const __half*>(y);
      __half *so2 = static_cast<__half*>(sum_out), *ho2 = static_cast<__half*>(h_out), *xo2 = static_cast<__half*>(xhat);
      const int lanes = static_cast<int>(K / 24), rows_tile = 4 * (32 / lanes);
      const long long tiles2 = (M + rows_tile - 1) / rows_tile;
      const long long cap2 = static_cast<long long>(sm_count()) * 8;
      const unsigned grid2 = static_cast<unsigned>((tiles2 < cap2 ? tiles2 : cap2) + jobs.blocks);
#define ARCQ_LAUNCH_LNQ_ROWS(LN, B, HASY)                                                                            \
  launch_pdl(arcq::add_layernorm_act_quant_rows_kernel<LN, B, HASY>, grid2, arcq::kLnqRowsThreads, 0, st, xs, ys, np, eps,     \
             static_cast<long long>(M), thresholds, codebook, so2, ho2, xo2, one_fma, jobs)
#define ARCQ_LNQ_ROWS_BITS(LN, HASY)                                                                                  \
  do {                                                                                                                \
    if (bits == 4) ARCQ_LAUNCH_LNQ_ROWS(LN, 4, HASY);                                                                  \
    else if (bits == 3) ARCQ_LAUNCH_LNQ_ROWS(LN, 3, HASY);                                                             \
    else ARCQ_LAUNCH_LNQ_ROWS(LN, 2, HASY);                                                                            \
  } while (0)
      if (y != nullptr) {
        if (lanes == 8) ARCQ_LNQ_ROWS_BITS(8, true); else if (lanes == 16) ARCQ_LNQ_ROWS_BITS(16, true); else ARCQ_LNQ_ROWS_BITS(32, true);
      } else {
        if (lanes == 8) ARCQ_LNQ_ROWS_BITS(8, false); else if (lanes == 16) ARCQ_LNQ_ROWS_BITS(16, false); else ARCQ_LNQ_ROWS_BITS(32, false);
      }
#undef ARCQ_LNQ_ROWS_BITS
#undef ARCQ_LAUNCH_LNQ_ROWS
      cudaError_t e2 = cudaGetLastError();
      if (e2 != cudaSuccess) return cuda_fail(e2, "add_layernorm_act_quant (rows) launch");
      return ARCQ_OK;
    }
  }
  const long long tiles = (M * G + arcq::kLnqThreads - 1) / arcq::kLnqThreads;
  const long long cap = static_cast<long long>(sm_count()) * 4;
  const unsigned grid = static_cast<unsigned>((tiles < cap ? tiles : cap) + jobs.blocks);
  const __half *xh = static_cast<const __half*>(x), *yh = static_cast<const __half*>(y);
  __half *so = static_cast<__half*>(sum_out), *ho = static_cast<__half*>(h_out);
  if (M * G >= (1ll << 30)) return fail(ARCQ_E_TOO_LARGE, "too many groups");
  CUtensorMap tm_out;
  if (!make_tensor_map_2d(&tm_out, xhat, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(M * G), 64, 64, 32,
                          CU_TENSOR_MAP_SWIZZLE_128B))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed for the reconstruction");
  int* const status = status_ptr();
  if (status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
#define ARCQ_LAUNCH_LNQ(LN, B, HASY)                                                                                   \
  do {                                                                                                                 \
    auto k = arcq::add_layernorm_act_quant_kernel<LN, B, HASY>;                                                        \
    constexpr int smem = arcq::lnq_smem_layout(LN, HASY).total;                                                        \
    static thread_local int done_dev = -1;      /* shared-memory ceiling raised once per (host thread, device) */      \
    int dev = 0;                                                                                                       \
    cudaGetDevice(&dev);                                                                                               \
    if (done_dev != dev) {                                                                                             \
      const cudaError_t e1 = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);               \
      if (e1 != cudaSuccess) return cuda_fail(e1, "add_layernorm_act_quant");                                          \
      done_dev = dev;                                                                                                  \
    }                                                                                                                  \
    launch_pdl(k, grid, arcq::kLnqThreads, smem, st, tm_out, xh, yh, np, eps, static_cast<long long>(M), thresholds,   \
               codebook, so, ho, one_fma, static_cast<uint32_t>(opt(O_POLL_LIMIT)), status, jobs);                     \
  } while (0)
#define ARCQ_LNQ_BITS(LN, HASY)                                                                                         \
  do {                                                                                                                  \
    if (bits == 4) ARCQ_LAUNCH_LNQ(LN, 4, HASY);                                                                         \
    else if (bits == 3) ARCQ_LAUNCH_LNQ(LN, 3, HASY);                                                                    \
    else ARCQ_LAUNCH_LNQ(LN, 2, HASY);                                                                                   \
  } while (0)
  {
    const int lanes = static_cast<int>(K / 24);
    if (y != nullptr) {
      if (lanes == 8) ARCQ_LNQ_BITS(8, true); else if (lanes == 16) ARCQ_LNQ_BITS(16, true); else ARCQ_LNQ_BITS(32, true);
    } else {
      if (lanes == 8) ARCQ_LNQ_BITS(8, false); else if (lanes == 16) ARCQ_LNQ_BITS(16, false); else ARCQ_LNQ_BITS(32, false);
    }
  }
#undef ARCQ_LNQ_BITS
#undef ARCQ_LAUNCH_LNQ
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "add_layernorm_act_quant launch");
  return ARCQ_OK;
}

static int launch_attention(const void* qkv, int64_t B, int64_t T, int64_t H, int head_dim, const float* thresholds,
                            const float* codebook, int bits, int one_fma, void* out, void* stream) {
  // (tensors of an empty batch have null pointers)
  if (B != 0 && (qkv == nullptr || out == nullptr)) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (head_dim != 64) return fail(ARCQ_E_UNSUPPORTED, "head_dim %d: only 64 is built", head_dim);
  if (B < 0 || T <= 0 || H <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape B=%lld T=%lld H=%lld", (long long)B, (long long)T, (long long)H);
  if (T > arcq::kAttnMaxT) return fail(ARCQ_E_TOO_LARGE, "sequences longer than %d tokens are not built", arcq::kAttnMaxT);
  // (a matrix of 2^30 heads would be 400 GB)
  if (B > 0x3fffffffLL || H > 0x7fffffLL || B * H > 0x3fffffffLL) return fail(ARCQ_E_TOO_LARGE, "too many (image, head) pairs");
  if (!aligned(qkv, 16) || !aligned(out, 16)) return fail(ARCQ_E_ALIGN, "qkv and out must be 16-byte aligned");
  if (B == 0) return ARCQ_OK;
  arcq::AttnParams p;
  p.T = static_cast<int>(T); p.H = static_cast<int>(H);
  p.tk = static_cast<int>((T + 15) / 16 * 16);
  p.qtiles = static_cast<int>((T + arcq::kAttnQueries - 1) / arcq::kAttnQueries);
  p.items = static_cast<int>(B * H * p.qtiles);
  p.thresholds = thresholds;
  p.codebook = codebook;
  p.one_fma = one_fma;
  p.poll_limit = static_cast<uint32_t>(opt(O_POLL_LIMIT));
  p.status = status_ptr();
  if (p.status == nullptr) return fail(ARCQ_E_CUDA, "device status word not reachable");
  CUtensorMap tm_q, tm_kv, tm_out;
  auto map = [&](CUtensorMap* tm, const void* base, int64_t cols, int box_rows) {
    return make_tensor_map(tm, base, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, static_cast<uint64_t>(B), static_cast<uint64_t>(T),
                           static_cast<uint64_t>(cols), 64, static_cast<uint32_t>(box_rows), CU_TENSOR_MAP_SWIZZLE_128B);
  };
  if (!map(&tm_q, qkv, 3 * H * 64, arcq::kAttnQueries) || !map(&tm_kv, qkv, 3 * H * 64, p.tk) || !map(&tm_out, out, H * 64, 32))
    return fail(ARCQ_E_CUDA, "cuTensorMapEncodeTiled failed");
  const size_t smem = arcq::attn_smem_layout(p.tk).total;
  const int cap = sm_count();
  const unsigned grid = static_cast<unsigned>(p.items < cap ? p.items : cap);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define ARCQ_LAUNCH_ATTN(Q, BT)                                                                                      \
  do {                                                                                                                \
    static thread_local int done_dev = -1;                                                                            \
    int dev = 0;                                                                                                      \
    cudaGetDevice(&dev);                                                                                              \
    if (done_dev != dev) {                                                                                            \
      const int rc = prepare_register_kernel(arcq::attention_kernel<Q, BT>, arcq::attn_smem_layout(arcq::kAttnMaxT).total, \
                                             arcq::kAttnLaunchRegs, "attention");                                    \
      if (rc != ARCQ_OK) return rc;                                                                                   \
      done_dev = dev;                                                                                                 \
    }                                                                                                                 \
    launch_pdl(arcq::attention_kernel<Q, BT>, grid, arcq::kAttnThreads, smem, st, tm_q, tm_kv, tm_out, p);            \
  } while (0)
  if (thresholds == nullptr) ARCQ_LAUNCH_ATTN(false, 4);
  else if (bits == 4) ARCQ_LAUNCH_ATTN(true, 4);
  else if (bits == 3) ARCQ_LAUNCH_ATTN(true, 3);
  else ARCQ_LAUNCH_ATTN(true, 2);
#undef ARCQ_LAUNCH_ATTN
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "attention launch");
  return ARCQ_OK;
}

int arcq_attention(const void* qkv, int64_t B, int64_t T, int64_t H, int head_dim, void* out, void* stream) {
  return launch_attention(qkv, B, T, H, head_dim, nullptr, nullptr, 4, 0, out, stream);
}

int arcq_attention_act_quant_form(const void* qkv, int64_t B, int64_t T, int64_t H, int head_dim, const float* thresholds,
                                  const float* codebook, int bits, int group_size, void* xhat, int one_fma, void* stream) {
  if (thresholds == nullptr || codebook == nullptr) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  return launch_attention(qkv, B, T, H, head_dim, thresholds, codebook, bits, one_fma, xhat, stream);
}

int arcq_attention_act_quant(const void* qkv, int64_t B, int64_t T, int64_t H, int head_dim, const float* thresholds,
                             const float* codebook, int bits, int group_size, void* xhat, void* stream) {
  return arcq_attention_act_quant_form(qkv, B, T, H, head_dim, thresholds, codebook, bits, group_size, xhat, 0, stream);
}

int arcq_patchify(const void* images, int64_t B, int64_t C, int64_t H, int64_t W, int patch, void* rows, void* stream) {
  if (images == nullptr || rows == nullptr) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (B < 0 || C <= 0 || H <= 0 || W <= 0 || patch <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape");
  if (patch % 8 != 0 || H % patch != 0 || W % patch != 0)
    return fail(ARCQ_E_UNSUPPORTED, "patch %d: must be a multiple of 8 that divides H=%lld and W=%lld", patch, (long long)H, (long long)W);
  if (B * C * H * W > 0x7fffffffffLL) return fail(ARCQ_E_TOO_LARGE, "image batch too large");
  if (!aligned(images, 16) || !aligned(rows, 16)) return fail(ARCQ_E_ALIGN, "images and rows must be 16-byte aligned");
  if (B == 0) return ARCQ_OK;
  const long long chunks = B * C * H * W / 8;
  launch_pdl(arcq::patchify_kernel, grid_for(chunks, 256, 8), 256, 0, static_cast<cudaStream_t>(stream),
             static_cast<const __half*>(images), static_cast<int>(B), static_cast<int>(C), static_cast<int>(H),
             static_cast<int>(W), patch, static_cast<__half*>(rows));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "patchify launch");
  return ARCQ_OK;
}

int arcq_assemble_tokens(const void* patches, const void* cls_token, const void* pos_embed, int64_t B, int64_t T, int64_t D,
                         void* tokens, void* stream) {
  if (patches == nullptr || cls_token == nullptr || pos_embed == nullptr || tokens == nullptr)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (B < 0 || T <= 0 || D <= 0 || D % 8 != 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape B=%lld T=%lld D=%lld", (long long)B, (long long)T, (long long)D);
  if (!aligned(patches, 16) || !aligned(cls_token, 16) || !aligned(pos_embed, 16) || !aligned(tokens, 16))
    return fail(ARCQ_E_ALIGN, "all buffers must be 16-byte aligned");
  if (B == 0) return ARCQ_OK;
  const long long chunks = B * (T + 1) * (D / 8);
  launch_pdl(arcq::assemble_tokens_kernel, grid_for(chunks, 256, 8), 256, 0, static_cast<cudaStream_t>(stream),
             static_cast<const __half*>(patches), static_cast<const __half*>(cls_token),
             static_cast<const __half*>(pos_embed), static_cast<int>(B), static_cast<int>(T), static_cast<int>(D),
             static_cast<__half*>(tokens));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "assemble_tokens launch");
  return ARCQ_OK;
}

int arcq_unpack_codes(const uint8_t* packed, int64_t rows, int64_t length, int bits, uint8_t* codes_out, void* stream) {
  if (!packed || !codes_out) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (rows < 0 || length < 0) return fail(ARCQ_E_BAD_SHAPE, "negative shape");
  if (rows == 0 || length == 0) return ARCQ_OK;
  const long long pc = (length * bits + 7) / 8;
  arcq::unpack_codes_kernel<<<grid_for(rows * length, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      packed, rows, length, pc, bits, codes_out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "unpack launch");
  return ARCQ_OK;
}

int arcq_pack_codes(const uint8_t* codes, int64_t rows, int64_t length, int bits, uint8_t* packed_out, void* stream) {
  if (!codes || !packed_out) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (rows < 0 || length < 0) return fail(ARCQ_E_BAD_SHAPE, "negative shape");
  if (rows == 0 || length == 0) return ARCQ_OK;
  const long long pc = (length * bits + 7) / 8;
  arcq::pack_codes_kernel<<<grid_for(rows * pc, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      codes, rows, length, pc, bits, packed_out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "pack launch");
  return ARCQ_OK;
}

int arcq_unpack_weight_f16(const uint8_t* packed, const float* mu, const float* sigma, const float* codesum,
                           const float* codebook, int bits, int group_size, int64_t rows, int64_t K, void* out,
                           void* stream) {
  if (!packed || !mu || !sigma || !codesum || !codebook || !out) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (rows < 0 || K <= 0 || K % 64 != 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape rows=%lld K=%lld", (long long)rows, (long long)K);
  if (!aligned(packed, 4) || !aligned(out, 16)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte, out 16-byte aligned");
  if (rows == 0) return ARCQ_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(rows * (K / 8), 256, 8);
  const int k = static_cast<int>(K);
  __half* o = static_cast<__half*>(out);
  if (bits == 4) arcq::unpack_weight_f16_kernel<4><<<grid, 256, 0, st>>>(packed, mu, sigma, codesum, codebook, rows, k, o);
  else if (bits == 3) arcq::unpack_weight_f16_kernel<3><<<grid, 256, 0, st>>>(packed, mu, sigma, codesum, codebook, rows, k, o);
  else arcq::unpack_weight_f16_kernel<2><<<grid, 256, 0, st>>>(packed, mu, sigma, codesum, codebook, rows, k, o);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "unpack_weight_f16 launch");
  return ARCQ_OK;
}

int arcq_dequant(const uint8_t* packed, const float* mu, const float* sigma, const float* codesum, const float* codebook,
                 int bits, int group_size, int64_t rows, int64_t K, void* out, int out_dtype, void* stream) {
  if (!packed || !mu || !sigma || !codesum || !codebook || !out) return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (out_dtype != ARCQ_DT_F16 && out_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "out_dtype must be f16 or f32");
  if (rows < 0 || K <= 0 || group_size <= 0 || K % group_size != 0 || group_size % 8 != 0)
    return fail(ARCQ_E_BAD_SHAPE, "bad shape rows=%lld K=%lld group_size=%d", (long long)rows, (long long)K, group_size);
  if (!aligned(packed, 4)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte aligned");
  if (rows == 0) return ARCQ_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(rows * (K / 8), 256, 8);
  const int k = static_cast<int>(K);
  const bool wide = group_size == 64 && aligned(out, 16);
  const long long chunks = rows * (K / 8);
  const int grid64 = grid_for(chunks, 512, 8);
#define ARCQ_LAUNCH_DQ(B)                                                                                          \
  do {                                                                                                             \
    if (wide && out_dtype == ARCQ_DT_F32)                                                                          \
      launch_pdl(arcq::dequant64_kernel<B, float>, grid64, 256, 0, st, packed, mu, sigma, codesum, codebook, chunks, \
                 static_cast<float*>(out));                                                                        \
    else if (wide)                                                                                                 \
      launch_pdl(arcq::dequant64_kernel<B, __half>, grid64, 256, 0, st, packed, mu, sigma, codesum, codebook, chunks, \
                 static_cast<__half*>(out));                                                                       \
    else if (out_dtype == ARCQ_DT_F32)                                                                                  \
      arcq::dequant_kernel<B, float><<<grid, 256, 0, st>>>(packed, mu, sigma, codesum, codebook, rows, k,          \
                                                           group_size, static_cast<float*>(out));                 \
    else                                                                                                           \
      arcq::dequant_kernel<B, __half><<<grid, 256, 0, st>>>(packed, mu, sigma, codesum, codebook, rows, k,         \
                                                            group_size, static_cast<__half*>(out));               \
  } while (0)
  if (bits == 4) ARCQ_LAUNCH_DQ(4);
  else if (bits == 3) ARCQ_LAUNCH_DQ(3);
  else ARCQ_LAUNCH_DQ(2);
#undef ARCQ_LAUNCH_DQ
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "dequant launch");
  return ARCQ_OK;
}

// ---------------------------------------------------------------------------------------------------------
// Linear with the library's own weight scratch.
//
// The dense route above needs room for the unpacked fp16 weight, and so far the caller brings it.  Some
// callers have no way to: a C host that binds this ABI from a runtime whose device memory was handed out in
// full at start-up, or a serving loop in which a device allocation (and the device-wide wait it may imply) is
// not acceptable once requests are flowing.  For them the scratch lives in the library image itself: a
// file-scope device array, sized for the largest DeiT-B linear (768 x 3072 fp16 values, 4.5 MB per device).
// Nothing here allocates or frees memory.
//  * Set-up: the array's device address is looked up once per device, on the first call made with that
//    device current.  That look-up is host-side work of the CUDA runtime; make the first call outside any
//    stream capture, later calls only launch kernels.
//  * Nothing has to start at zero: every element the contraction reads was written by the unpack kernel of
//    the same call, which is ordered before it on `stream`.
//  * One array per device: two calls in flight at once on the same device (different streams or host
//    threads) would overwrite each other's weight.  Calls must be ordered one after the other.
constexpr long long kStaticWeightElems = ARCQ_STATIC_WEIGHT_ELEMS;
static __device__ __align__(256) __half g_static_w16[kStaticWeightElems];

static __half* static_weight_scratch() {
  constexpr int kMaxDevices = 64;
  static __half* cached[kMaxDevices] = {};
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    fail(ARCQ_E_CUDA, "no current CUDA device (or device index above %d)", kMaxDevices - 1);
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_w16);
    if (e != cudaSuccess || p == nullptr) {
      cuda_fail(e, "address of the static weight scratch");
      return nullptr;
    }
    cached[dev] = static_cast<__half*>(p);
  }
  return cached[dev];
}

int arcq_packed_linear_static_scratch(const void* xhat, const uint8_t* packed_w, const float* mu_w,
                                      const float* sigma_w, const float* codesum_w, const float* w_codebook,
                                      const float* bias, int bits, int group_size, int64_t M, int64_t N, int64_t K,
                                      void* y, int y_dtype, void* stream) {
  if (!xhat || !packed_w || !mu_w || !sigma_w || !codesum_w || !w_codebook || !y)
    return fail(ARCQ_E_BAD_ARG, "null pointer argument");
  if (M < 0 || N <= 0 || K <= 0) return fail(ARCQ_E_BAD_SHAPE, "bad shape M=%lld N=%lld K=%lld", (long long)M,
                                              (long long)N, (long long)K);
  if (group_size != 64) return fail(ARCQ_E_UNSUPPORTED, "group_size %d: only 64 is built", group_size);
  if (N > kStaticWeightElems || K > kStaticWeightElems || N * K > kStaticWeightElems)
    return fail(ARCQ_E_TOO_LARGE, "weight of %lld x %lld values exceeds the static scratch of %lld values; "
                                  "use arcq_dequant + arcq_dense_weight_gemm with a buffer of your own",
                (long long)N, (long long)K, (long long)kStaticWeightElems);
  // everything the two launches below would reject is rejected here, before the first of them runs and
  // overwrites the shared scratch
  if (bits < 2 || bits > 4) return fail(ARCQ_E_BAD_ARG, "bits must be 2, 3 or 4, got %d", bits);
  if (y_dtype != ARCQ_DT_F16 && y_dtype != ARCQ_DT_F32) return fail(ARCQ_E_BAD_ARG, "y_dtype must be f16 or f32");
  if (K % 64 != 0) return fail(ARCQ_E_UNSUPPORTED, "K=%lld: this entry point needs K %% 64 == 0", (long long)K);
  if (N % 16 != 0) return fail(ARCQ_E_UNSUPPORTED, "N=%lld: this entry point needs N %% 16 == 0", (long long)N);
  if (M > 0x7fffffffLL || N > 0x7fffffffLL || K > (1 << 20)) return fail(ARCQ_E_TOO_LARGE, "shape too large");
  if (!aligned(xhat, 16) || !aligned(y, 16)) return fail(ARCQ_E_ALIGN, "xhat and y must be 16-byte aligned");
  if (!aligned(packed_w, 4)) return fail(ARCQ_E_ALIGN, "packed codes must be 4-byte aligned");
  if (M > 0) {
    WsConfig probe;
    if (!choose_ws_config(M, N, K, 4, true, &probe)) return fail(ARCQ_E_UNSUPPORTED, "no tile configuration for this shape");
  }
  __half* const w16 = static_weight_scratch();
  if (w16 == nullptr) return ARCQ_E_CUDA;
  if (M == 0) return ARCQ_OK;
  const int rc = arcq_dequant(packed_w, mu_w, sigma_w, codesum_w, w_codebook, bits, group_size, N, K, w16,
                              ARCQ_DT_F16, stream);
  if (rc != ARCQ_OK) return rc;
  return arcq_dense_weight_gemm(xhat, w16, bias, M, N, K, y, y_dtype, stream);
}

}  // extern "C"
