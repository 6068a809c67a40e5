// sphg_hostio.cu -- upload and download that read and write the caller's host
// arrays from the device.
//
// On a Grace-Blackwell node the GPU reaches pageable host memory directly
// (cudaDevAttrPageableMemoryAccess, address translation through the host's
// page tables), so the FP64 <-> device-representation conversion of
// sphg_upload / sphg_download runs as one kernel over the caller's arrays:
// no pinned staging copy and no host conversion loop.  Used when the device
// reports the capability (sphg_set_host_access can turn it off); the results
// are those of the staging path.
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/sphg.h"
#include "sphg_internal.cuh"
#include "sphg_neighbor.cuh"

namespace sphg {
namespace {

// floor(t / cs) exactly as the FP64 division rounds it, from t * (1 / cs):
// the product is within 3 ulp of the quotient, so away from an integer (and
// for |q| < 1e6) its floor is the quotient's; near one the division decides.
__device__ __forceinline__ double floor_div(double t, double cs, double inv_cs) {
  const double q = __dmul_rn(t, inv_cs);
  const double f = floor(q);
  const double r = __dsub_rn(q, f);
  if (r > 1.0e-9 && r < 1.0 - 1.0e-9 && fabs(q) < 1.0e6) return f;
  return floor(__ddiv_rn(t, cs));
}

// Whether the state is valid by its error words, which go into the handle's pinned
// block (the host reads them after the synchronisation that ends the call).
__device__ __forceinline__ bool state_valid(const HostErrors& e, bool report) {
  bool valid = true;
#pragma unroll
  for (int k = 0; k < kErrorWords; ++k) {
    const uint32_t w = *e.word[k];
    valid = valid && w == 0u;
    if (report) e.out[k] = w;
  }
  return valid;
}

// An FP64 position as its cell (clamped to [0, cmax]) and FP32 offset in it.
// FUSED: c cs taken off x - lo with one rounding, as the host code that stages a
// served request rounds it where its compiler contracts (Arm does); an upload has
// always rounded the product first.
template <bool FUSED>
__device__ __forceinline__ float2 split_position(const InstDesc& d, double x, double y, int cmx, int cmy, int& cx,
                                                 int& cy) {
  const double qx = floor_div(__dsub_rn(x, d.lo_xd), d.cs_xd, d.inv_cs_xd);
  const double qy = floor_div(__dsub_rn(y, d.lo_yd), d.cs_yd, d.inv_cs_yd);
  cx = !(qx < (double)cmx) ? cmx : (qx < 0.0 ? 0 : (int)qx);
  cy = !(qy < (double)cmy) ? cmy : (qy < 0.0 ? 0 : (int)qy);
  const double tx = __dsub_rn(x, d.lo_xd), ty = __dsub_rn(y, d.lo_yd);
  float fx = __double2float_rn(FUSED ? __fma_rn(-(double)cx, d.cs_xd, tx) : __dsub_rn(tx, __dmul_rn((double)cx, d.cs_xd)));
  float fy = __double2float_rn(FUSED ? __fma_rn(-(double)cy, d.cs_yd, ty) : __dsub_rn(ty, __dmul_rn((double)cy, d.cs_yd)));
  if ((double)fx >= d.cs_xd) fx = nextafterf(fx, 0.0f);
  if ((double)fy >= d.cs_yd) fy = nextafterf(fy, 0.0f);
  return make_float2(fx, fy);
}

// One particle of the caller's FP64 state into the device representation
// (false: not finite, nothing written).
__device__ __forceinline__ bool upload_one(const StepArgs& a, int precision, int64_t i, double xi, double yi,
                                           double vxi, double vyi, float2& pos, float2& vel, uint32_t& key) {
  if (!isfinite(xi) || !isfinite(yi) || !isfinite(vxi) || !isfinite(vyi)) return false;
  vel = make_float2((float)vxi, (float)vyi);
  if (precision == SPHG_PRECISION_SPLIT) {
    const InstDesc& d = inst_ref<true>(a, i);
    const int cmx = d.periodic ? d.nxr - 1 : d.nx - 1;
    const int cmy = d.periodic ? d.nyr - 1 : d.ny - 1;
    int cx, cy;
    pos = split_position<false>(d, xi, yi, cmx, cmy, cx, cy);
    key = d.cell_base + local_code(d, cx, cy);
  } else {
    pos = make_float2((float)xi, (float)yi);
  }
  return true;
}

__global__ void upload_direct_kernel(StepArgs a, int precision, const double* __restrict__ x,
                                     const double* __restrict__ y, const double* __restrict__ vx,
                                     const double* __restrict__ vy, uint32_t* first_bad, volatile uint32_t* any_bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  float2 pos, vel;
  uint32_t key = 0;
  if (!upload_one(a, precision, i, x[i], y[i], vx[i], vy[i], pos, vel, key)) {
    atomicMin(first_bad, (uint32_t)i);
    *any_bad = 1u;
    return;
  }
  a.velB[i] = vel;
  a.posB[i] = pos;
  if (precision == SPHG_PRECISION_SPLIT) a.keyA[i] = key;
  if (a.track_ids) a.idsB[i] = (int32_t)i;
}

// Two consecutive particles a thread, 16-byte reads of the caller's arrays
// (all four 16-byte aligned; n odd: the last particle alone).
__global__ void upload_direct_kernel2(StepArgs a, int precision, const double2* __restrict__ x,
                                      const double2* __restrict__ y, const double2* __restrict__ vx,
                                      const double2* __restrict__ vy, uint32_t* first_bad, volatile uint32_t* any_bad) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i0 = 2 * t;
  if (i0 >= a.n) return;
  if (i0 + 1 == a.n) {  // the odd last particle
    const double* xs = reinterpret_cast<const double*>(x);
    const double* ys = reinterpret_cast<const double*>(y);
    const double* vxs = reinterpret_cast<const double*>(vx);
    const double* vys = reinterpret_cast<const double*>(vy);
    float2 pos, vel;
    uint32_t key = 0;
    if (!upload_one(a, precision, i0, xs[i0], ys[i0], vxs[i0], vys[i0], pos, vel, key)) {
      atomicMin(first_bad, (uint32_t)i0);
      *any_bad = 1u;
      return;
    }
    a.velB[i0] = vel;
    a.posB[i0] = pos;
    if (precision == SPHG_PRECISION_SPLIT) a.keyA[i0] = key;
    if (a.track_ids) a.idsB[i0] = (int32_t)i0;
    return;
  }
  const double2 xv = x[t], yv = y[t], vxv = vx[t], vyv = vy[t];
  float2 p0, p1, v0, v1;
  uint32_t k0 = 0, k1 = 0;
  const bool ok0 = upload_one(a, precision, i0, xv.x, yv.x, vxv.x, vyv.x, p0, v0, k0);
  const bool ok1 = upload_one(a, precision, i0 + 1, xv.y, yv.y, vxv.y, vyv.y, p1, v1, k1);
  if (!ok0 || !ok1) {
    atomicMin(first_bad, (uint32_t)(ok0 ? i0 + 1 : i0));
    *any_bad = 1u;
    if (!ok0 && !ok1) return;
  }
  if (ok0 && ok1) {
    reinterpret_cast<float4*>(a.velB)[t] = make_float4(v0.x, v0.y, v1.x, v1.y);
    reinterpret_cast<float4*>(a.posB)[t] = make_float4(p0.x, p0.y, p1.x, p1.y);
    if (precision == SPHG_PRECISION_SPLIT) reinterpret_cast<uint2*>(a.keyA)[t] = make_uint2(k0, k1);
    if (a.track_ids) reinterpret_cast<int2*>(a.idsB)[t] = make_int2((int32_t)i0, (int32_t)(i0 + 1));
    return;
  }
  const int64_t i = ok0 ? i0 : i0 + 1;  // the finite one of the pair
  a.velB[i] = ok0 ? v0 : v1;
  a.posB[i] = ok0 ? p0 : p1;
  if (precision == SPHG_PRECISION_SPLIT) a.keyA[i] = ok0 ? k0 : k1;
  if (a.track_ids) a.idsB[i] = (int32_t)i;
}

// One position coordinate (axis 0 or 1) of slot i in the caller's FP64 representation
// (lo + c cs in one rounding, as the contracted host code of the staged download).
__device__ __forceinline__ double download_position(const StepArgs& a, int precision, int64_t i, int axis) {
  const float2 p = a.posA[i];
  const double o = axis ? p.y : p.x;
  if (precision != SPHG_PRECISION_SPLIT) return o;
  const InstDesc& d = inst_ref<true>(a, i);
  int cx, cy;
  decode_code(d, a.keyA[i] - d.cell_base, cx, cy);
  return axis ? __dadd_rn(__fma_rn((double)cy, d.cs_yd, d.lo_yd), o)
              : __dadd_rn(__fma_rn((double)cx, d.cs_xd, d.lo_xd), o);
}

// Entry of `out` that thread t writes: t less the entries between the 128-byte
// line the array starts in and its first one, so that a warp's stores cover
// whole lines wherever the caller's array lies (malloc's large blocks start 16
// bytes into a page: 170 GB/s of the host link with lines split between warps,
// 192 with whole ones -- what the link takes of writes).
template <class T>
__device__ __forceinline__ int64_t line_entry(const T* out, int64_t t) {
  return t - (int64_t)((reinterpret_cast<uintptr_t>(out) & 127u) / sizeof(T));
}
constexpr int kLineEntries = 32;  // at most this many threads more than entries

__global__ void download_direct_kernel(StepArgs a, int precision, double* __restrict__ x, double* __restrict__ y,
                                       double* __restrict__ vx, double* __restrict__ vy,
                                       double* __restrict__ rho, double* __restrict__ fx,
                                       double* __restrict__ fy, int32_t* __restrict__ ids, HostErrors errors) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = state_valid(errors, t == 0);  // else the call fails: the arrays stay as they are
  auto write = [&](auto* out, auto&& value) {
    if (!out) return;
    const int64_t i = line_entry(out, t);
    if (i < 0 || i >= a.n) return;
    const auto v = value(i);  // loaded beside the words
    if (valid) out[i] = v;
  };
  write(x, [&](int64_t i) { return download_position(a, precision, i, 0); });
  write(y, [&](int64_t i) { return download_position(a, precision, i, 1); });
  write(vx, [&](int64_t i) { return (double)a.velpA[i].x; });
  write(vy, [&](int64_t i) { return (double)a.velpA[i].y; });
  write(rho, [&](int64_t i) { return (double)a.rho[i]; });
  write(fx, [&](int64_t i) { return (double)a.acc[i].x; });
  write(fy, [&](int64_t i) { return (double)a.acc[i].y; });
  write(ids, [&](int64_t i) { return a.track_ids ? a.idsA[i] : -1; });
}

// A served request's host arrays into the admission staging: device
// representation, instance-local cell code of the held position, creation index.
__global__ void stage_direct_kernel(InstDesc d, int precision, int64_t n, const double* __restrict__ x,
                                    const double* __restrict__ y, const double* __restrict__ vx,
                                    const double* __restrict__ vy, float2* __restrict__ pos, float2* __restrict__ vel,
                                    uint32_t* __restrict__ key, int32_t* __restrict__ ids) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int cmx = d.periodic ? d.nxr - 1 : d.nx - 1;
  const int cmy = d.periodic ? d.nyr - 1 : d.ny - 1;
  int cx, cy;
  float2 p;
  if (precision == SPHG_PRECISION_SPLIT) {
    p = split_position<true>(d, x[i], y[i], cmx, cmy, cx, cy);
  } else {
    p = make_float2((float)x[i], (float)y[i]);
    cx = cell_coord(p.x, d.lo_x, d.inv_cs_x, d.lo_xd, d.cs_xd, cmx);
    cy = cell_coord(p.y, d.lo_y, d.inv_cs_y, d.lo_yd, d.cs_yd, cmy);
  }
  pos[i] = p;
  vel[i] = make_float2((float)vx[i], (float)vy[i]);
  key[i] = local_code(d, cx, cy);
  if (ids) ids[i] = (int32_t)i;
}

// Slots [first, first + n) as a result: x, y, vx, vy, rho (FP64) and the creation
// indices, n entries each, one after the other.
__global__ void result_kernel(StepArgs a, int precision, int64_t first, int64_t n, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t q = first + i;
  const float4 v = a.velpA[q];
  out[i] = download_position(a, precision, q, 0);
  out[n + i] = download_position(a, precision, q, 1);
  out[2 * n + i] = v.x;
  out[3 * n + i] = v.y;
  out[4 * n + i] = a.rho[q];
  reinterpret_cast<int32_t*>(out + 5 * n)[i] = a.track_ids ? a.idsA[q] : -1;
}

__global__ void host_copy_kernel(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, int64_t words) {
  const int64_t i = line_entry(dst, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= 0 && i < words) dst[i] = src[i];
}

bool aligned(const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; }

}  // namespace

cudaError_t launch_upload_direct(const StepArgs& a, int precision, const double* x, const double* y,
                                 const double* vx, const double* vy, uint32_t* first_bad, uint32_t* any_bad,
                                 cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  if (aligned(x, 16) && aligned(y, 16) && aligned(vx, 16) && aligned(vy, 16)) {
    const int64_t pairs = (a.n + 1) / 2;
    upload_direct_kernel2<<<(unsigned)((pairs + 255) / 256), 256, 0, st>>>(
        a, precision, reinterpret_cast<const double2*>(x), reinterpret_cast<const double2*>(y),
        reinterpret_cast<const double2*>(vx), reinterpret_cast<const double2*>(vy), first_bad, any_bad);
  } else {
    upload_direct_kernel<<<(unsigned)((a.n + 255) / 256), 256, 0, st>>>(a, precision, x, y, vx, vy, first_bad,
                                                                          any_bad);
  }
  return cudaGetLastError();
}

cudaError_t launch_stage_direct(const InstDesc& d, int precision, int64_t n, const double* x, const double* y,
                                const double* vx, const double* vy, float2* pos, float2* vel, uint32_t* key,
                                int32_t* ids, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  stage_direct_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, precision, n, x, y, vx, vy, pos, vel, key, ids);
  return cudaGetLastError();
}

cudaError_t launch_result(const StepArgs& a, int precision, int64_t first, int64_t n, double* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  result_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, precision, first, n, out);
  return cudaGetLastError();
}

cudaError_t launch_host_copy(uint32_t* dst, const uint32_t* src, int64_t words, cudaStream_t st) {
  if (words <= 0) return cudaSuccess;
  host_copy_kernel<<<(unsigned)((words + kLineEntries + 255) / 256), 256, 0, st>>>(dst, src, words);
  return cudaGetLastError();
}

cudaError_t launch_download_direct(const StepArgs& a, int precision, double* x, double* y, double* vx, double* vy,
                                   double* rho, double* fx, double* fy, int32_t* ids, const HostErrors& errors,
                                   cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const unsigned g = (unsigned)((a.n + kLineEntries + 255) / 256);
  download_direct_kernel<<<g, 256, 0, st>>>(a, precision, x, y, vx, vy, rho, fx, fy, ids, errors);
  return cudaGetLastError();
}

}  // namespace sphg
