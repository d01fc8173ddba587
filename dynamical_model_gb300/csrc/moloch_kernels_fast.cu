// FP64 and FP32-storage kernels with multiply-add contraction allowed.
#define MOLOCH_KNS kfast
#define MOLOCH_LEAN_FP64 1  // FP64 expressions written for few FP64 operations
#include "../../include/moloch_gb300.h"
#include "moloch_kernels.cuh"

namespace moloch {
namespace kfast {
template int launch_prediag<double>(const View<double>&, cudaStream_t, const PhaseFlags&);
template int launch_sound<double>(View<double>&, cudaStream_t, const PhaseFlags&);
template int launch_advection<double>(View<double>&, cudaStream_t);
template int launch_postdiag<double>(View<double>&, cudaStream_t, const PhaseFlags&, const double*, const double*);
template int launch_diag<double>(const View<double>&, cudaStream_t);
template int launch_prediag<float>(const View<float>&, cudaStream_t, const PhaseFlags&);
template int launch_sound<float>(View<float>&, cudaStream_t, const PhaseFlags&);
template int launch_advection<float>(View<float>&, cudaStream_t);
template int launch_postdiag<float>(View<float>&, cudaStream_t, const PhaseFlags&, const float*, const float*);
template int launch_diag<float>(const View<float>&, cudaStream_t);
template int blaunch_step<double>(const Batch<double>&, cudaStream_t, const PhaseFlags&, int&, int&);
template int blaunch_step<float>(const Batch<float>&, cudaStream_t, const PhaseFlags&, int&, int&);
template int blaunch_advection<double>(const Batch<double>&, cudaStream_t, int&, int&);
template int blaunch_advection<float>(const Batch<float>&, cudaStream_t, int&, int&);
}  // namespace kfast
}  // namespace moloch

// ---- tensor maps of the staged column kernel --------------------------------
#include <mutex>

namespace moloch {
namespace kfast {
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}
// dense FP32 field (nj, ni, nk), j fastest, as boxes of cols x rows x levels
bool map3(EncodeTiledFn fn, CUtensorMap* m, const float* base, int nj, int ni, int nk, int cols, int rows, int levels) {
  const cuuint64_t dims[3] = {(cuuint64_t)nj, (cuuint64_t)ni, (cuuint64_t)nk};
  const cuuint64_t strides[2] = {(cuuint64_t)nj * 4, (cuuint64_t)nj * ni * 4};
  const cuuint32_t box[3] = {(cuuint32_t)cols, (cuuint32_t)rows, (cuuint32_t)levels};
  const cuuint32_t es[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

int column_maps_bytes() { return (int)(2 * sizeof(ColumnMaps)); }
int column_map_set_bytes() { return (int)sizeof(ColumnMaps); }

// Warps of a column tile side by side along j (8, 4, 2 or 1): the shape that
// covers the domain with the fewest tiles, the widest of equals (longer runs
// of DRAM: moloch_column_tm.cuh)
int column_wide(int nj, int ni) {
  int best = 1;
  long tiles = 0;
  for (int w = kTwWarps; w >= 1; w /= 2) {
    const long n = (long)((nj + 32 * w - 1) / (32 * w)) * ((ni * w + kTwWarps - 1) / kTwWarps);
    if (!tiles || n < tiles) { tiles = n; best = w; }
  }
  return best;
}

bool build_column_maps(const View<float>& v, void* out) {
  if (v.kz > kTwMaxKz || v.kz < 2 || v.nj % 4 != 0 || ((uintptr_t)out & 63)) return false;
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  // for the handle's device: the attribute is a device's own
  cudaFuncSetAttribute(k_sound_column_tw<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, TwCfg<0>::smem);
  cudaFuncSetAttribute(k_sound_column_tw<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, TwCfg<1>::smem);
  cudaFuncSetAttribute(kb_sound_column_tw<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, TwCfg<0>::smem);
  cudaFuncSetAttribute(kb_sound_column_tw<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, TwCfg<1>::smem);
  ColumnMaps* cm = static_cast<ColumnMaps*>(out);
  const int nj = v.nj, ni = v.ni, kz = v.kz;
  const int cols = 32 * v.twide, rows = kTwWarps / v.twide, lev = TwCfg<0>::kct;
  auto map = [&](CUtensorMap* m, const float* base, int nk) { return map3(fn, m, base, nj, ni, nk, cols, rows, lev); };
  for (int set = 0; set < 2; ++set) {
    CUtensorMap* m = cm[set].m;
    const bool ok = map(&m[CM_W], v.w, kz + 1) && map(&m[CM_FMZF], v.fmzf, kz + 1) &&
                    map(&m[CM_QV], v.fset[set][5], kz) && map(&m[CM_TET], v.fset[set][0], kz) &&
                    map(&m[CM_PAI], v.fset[set][1], kz) && map(&m[CM_QSAT], v.qsat, kz) &&
                    map(&m[CM_ZD], v.zdiv2b, kz) && map(&m[CM_FMZ], v.fmz, kz) && map(&m[CM_T], v.t, kz) &&
                    map(&m[CM_QC], v.fset[set][6], kz) && map(&m[CM_QWL], v.qwltot, kz) &&
                    map(&m[CM_QWI], v.qwitot, kz) && map(&m[CM_S], v.s, kz + 1);
    if (!ok) return false;
  }
  return cudaGetLastError() == cudaSuccess;
}
}  // namespace kfast
}  // namespace moloch

// ---- arithmetic check of the FP32 quotient with one correction --------------
namespace moloch {
namespace kfast {
__global__ void k_check_division(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ qc,
                                 float* __restrict__ qi, int n) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    qc[q] = div_corr(a[q], b[q]);
    qi[q] = a[q] / b[q];
  }
}
__global__ void k_check_division_f64(const double* __restrict__ a, const double* __restrict__ b,
                                     double* __restrict__ qn, double* __restrict__ qi, int n) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    qn[q] = qdiv(a[q], b[q]);  // quot_rn in this build
    qi[q] = a[q] / b[q];
  }
}
__global__ void k_check_math_f64(int op, const double* __restrict__ a, const double* __restrict__ b,
                                 double* __restrict__ out, double* __restrict__ ref, int n) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const double x = a[q], y = b[q];
    switch (op) {
      case 0: out[q] = quot_rn(x, rcp_rn_of(y)); ref[q] = x / y; break;
      case 1: out[q] = inv_rn(y); ref[q] = 1.0 / y; break;
      case 2: out[q] = pivot_rcp(y); ref[q] = 1.0 / y; break;
      default: out[q] = pow_cpovr(x); ref[q] = pow(x, kCpovr); break;
    }
  }
}
}  // namespace kfast
}  // namespace moloch

// div_corr (the quotient of the FP32 Exner/theta update) and CUDA's IEEE
// FP32 quotient of the same device arrays, for tests of its error bound
extern "C" int moloch_gpu_check_division(const float* a, const float* b, float* q_corr, float* q_ieee, int n,
                                         void* stream) {
  if (!a || !b || !q_corr || !q_ieee || n < 0) return MOLOCH_ERR_ARG;
  if (n == 0) return MOLOCH_OK;
  const int blocks = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
  moloch::kfast::k_check_division<<<blocks, 256, 0, (cudaStream_t)stream>>>(a, b, q_corr, q_ieee, n);
  return cudaPeekAtLastError() == cudaSuccess ? MOLOCH_OK : MOLOCH_ERR_CUDA;
}
extern "C" int moloch_gpu_check_division_f64(const double* a, const double* b, double* q_nr, double* q_ieee, int n,
                                             void* stream) {
  if (!a || !b || !q_nr || !q_ieee || n < 0) return MOLOCH_ERR_ARG;
  if (n == 0) return MOLOCH_OK;
  const int blocks = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
  moloch::kfast::k_check_division_f64<<<blocks, 256, 0, (cudaStream_t)stream>>>(a, b, q_nr, q_ieee, n);
  return cudaPeekAtLastError() == cudaSuccess ? MOLOCH_OK : MOLOCH_ERR_CUDA;
}
extern "C" int moloch_gpu_check_math_f64(int op, const double* a, const double* b, double* out, double* ref, int n,
                                         void* stream) {
  if (op < 0 || op > 3 || !a || !b || !out || !ref || n < 0) return MOLOCH_ERR_ARG;
  if (n == 0) return MOLOCH_OK;
  const int blocks = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
  moloch::kfast::k_check_math_f64<<<blocks, 256, 0, (cudaStream_t)stream>>>(op, a, b, out, ref, n);
  return cudaPeekAtLastError() == cudaSuccess ? MOLOCH_OK : MOLOCH_ERR_CUDA;
}
