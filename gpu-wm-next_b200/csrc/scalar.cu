// scalar.cu — advance_scalar_ssprk3 (src/dycore/dry_transport.cu:285-325): SSPRK3 of a
// scalar field under a constant advection velocity with first-order upwind differences
// (upwind_stage_kernel, :13-37), on the global owned array (nz, ny, nx) in device memory.
//
// One kernel per step: a warp marches down the rows of 32 columns in the direction of the
// wind and computes the three stages
//   q1 = L(q),  q2 = 0.75 q + 0.25 L(q1),  q' = 1/3 q + 2/3 L(q2)
// of a row together: the upwind row's values stay in registers, the upwind column's come from
// the neighbouring lane, and each stage is valid one column and one row further downwind, so
// 29 columns and all but the first three rows of a segment are written.  A step reads q and
// writes q' once, 8 B per cell, where a kernel per stage moved 32.  The steps alternate
// between q and one scratch array.
// with L(x) = x - dt (u dx/dx + v dx/dy).  The roundings are the reference build's: the
// divisions, fma(-dt, fma(u, dqx, v*dqy), q) for the stage and fma(wa, a, wb*b) for the
// blend (the contractions its compiler makes of the written expressions, identified on
// its golden vectors), written out so that no compiler choice can change them.  The
// stencil's halo is the periodic image, or zero beyond an open side: what the
// reference's halo exchange gives its virtual ranks (an absent neighbour sends zeros).
#include "../../include/gwm_b200.h"
#include "common.cuh"
#include "device_memory.cuh"
#include "physics.cuh"
#include "stencil.cuh"

namespace gwmb {
namespace {

struct ScalarStep {
  int nx, ny, px, py;
  float u, v, dt, dx, dy;
  const float* in;
  float* out;
};

constexpr int kSLanes = 29;  // columns a warp writes: 32 less one per stage
constexpr int kSRows = 32;   // rows it writes
constexpr int kSWarps = 4;

// NEAR: dx and dy lie in [2^-20, 2^20], so a quotient by them may take the residual steps of
// fp::div_by, which give the division's value for the differences tested here (the others
// divide); six IEEE divisions per cell and step were most of the kernel.
template <bool NEAR>
__global__ void __launch_bounds__(32 * kSWarps) k_scalar_step(const ScalarStep a) {
  const int lane = threadIdx.x & 31, seg = blockIdx.y * kSWarps + (threadIdx.x >> 5);
  const int j0 = seg * kSRows, j1 = min(j0 + kSRows, a.ny);
  if (j0 >= a.ny) return;  // the whole warp
  const size_t level = (size_t)blockIdx.z * ((size_t)a.nx * a.ny);
  const bool west = a.u >= 0.0f, south = a.v >= 0.0f;  // where the wind comes from
  const int i = blockIdx.x * kSLanes + lane - (west ? 3 : 0);
  const bool own = (west ? lane >= 3 : lane < kSLanes) && i < a.nx;
  const bool in_x = a.px || (i >= 0 && i < a.nx);
  auto wrap = [](int q, int n) {
    if (q >= 0 && q < n) return q;
    q %= n;
    return q < 0 ? q + n : q;
  };
  const float* col = a.in + level + wrap(i, a.nx);
  // row n of the march: three rows upwind of the segment first
  const int rows = j1 - j0 + 3;
  auto row = [&](int n) { return south ? j0 - 3 + n : j1 + 2 - n; };
  auto inside = [&](int j) { return in_x && (a.py || (j >= 0 && j < a.ny)); };
  auto load = [&](int n) {
    const int j = row(n);
    return n < rows && inside(j) ? __ldg(col + (size_t)wrap(j, a.ny) * a.nx) : 0.0f;
  };
  const float ydx = fp::recip(a.dx), ydy = fp::recip(a.dy);
  // +0 (div_by loses the sign of -0), or a magnitude in [2^-79, 2^100]; on the value rotated by
  // its sign, which costs nothing (testing it beside the magnitude: 5 % of the kernel)
  auto residual_safe = [](float e) {
    const unsigned x = __float_as_uint(e), r = (x << 1) | (x >> 31);
    return r == 0u || r - 0x30000000u <= 0xe3000001u - 0x30000000u;
  };
  // the reference build's contractions of q - dt*(u*dqx + v*dqy) and wa*a + wb*b
  auto stage = [&](float q, float qy) {
    const float qx = west ? __shfl_up_sync(0xffffffffu, q, 1) : __shfl_down_sync(0xffffffffu, q, 1);
    const float ex = west ? q - qx : qx - q, ey = south ? q - qy : qy - q;
    float dqx, dqy;
    if (NEAR && residual_safe(ex) && residual_safe(ey)) {
      dqx = fp::div_by(ex, a.dx, ydx);
      dqy = fp::div_by(ey, a.dy, ydy);
    } else {
      dqx = ex / a.dx;
      dqy = ey / a.dy;
    }
    return __fmaf_rn(-a.dt, __fmaf_rn(a.u, dqx, __fmul_rn(a.v, dqy)), q);
  };
  float n0 = load(0), n1 = load(1);        // two rows ahead
  float p0 = 0.0f, p1 = 0.0f, p2 = 0.0f;   // the upwind row's q, q1, q2
  for (int n = 0; n < rows; ++n) {
    const float q = n0;
    n0 = n1;
    n1 = load(n + 2);
    const int j = row(n);
    const bool in = inside(j);  // beyond an open side every stage reads zeros
    float q1 = stage(q, p0);
    if (!in) q1 = 0.0f;
    float q2 = __fmaf_rn(0.75f, q, __fmul_rn(0.25f, stage(q1, p1)));
    if (!in) q2 = 0.0f;
    const float out = __fmaf_rn(1.0f / 3.0f, q, __fmul_rn(2.0f / 3.0f, stage(q2, p2)));
    if (own && n >= 3) a.out[level + (size_t)j * a.nx + i] = out;
    p0 = q;
    p1 = q1;
    p2 = q2;
  }
}

}  // namespace
}  // namespace gwmb

extern "C" int gwm_b200_scalar_ssprk3(const gwm_b200_scalar_desc* d, float* q, int nsteps, void* stream) {
  using namespace gwmb;
  if (!d || !q || d->nx <= 0 || d->ny <= 0 || d->nz <= 0 || nsteps < 0 || d->nz > 65535 || !(d->dx > 0.0f) ||
      !(d->dy > 0.0f))
    return GWM_B200_ERR_ARG;
  if (nsteps == 0) {
    trim_scratch();
    return GWM_B200_OK;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = (size_t)d->nx * d->ny * d->nz;
  float* tmp = nullptr;
  if (scratch_alloc((void**)&tmp, n * sizeof(float), s) != cudaSuccess) return GWM_B200_ERR_CUDA;
  ScalarStep a{d->nx, d->ny, d->periodic_x, d->periodic_y, d->u_adv, d->v_adv, d->dt, d->dx, d->dy, q, tmp};
  auto mid = [](float x) { return x >= 9.5367431640625e-7f && x <= 1048576.0f; };
  const bool near = mid(d->dx) && mid(d->dy);
  const int segs = (d->ny + kSRows - 1) / kSRows;
  const dim3 grid((d->nx + kSLanes - 1) / kSLanes, (segs + kSWarps - 1) / kSWarps, d->nz);
  for (int step = 0; step < nsteps; ++step) {
    if (near) k_scalar_step<true><<<grid, 32 * kSWarps, 0, s>>>(a);
    else k_scalar_step<false><<<grid, 32 * kSWarps, 0, s>>>(a);
    a.in = a.out;
    a.out = a.out == q ? tmp : q;
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && nsteps % 2)  // the result is in the scratch
    e = cudaMemcpyAsync(q, tmp, n * sizeof(float), cudaMemcpyDeviceToDevice, s);
  cudaFreeAsync(tmp, s);
  if (e != cudaSuccess) return GWM_B200_ERR_CUDA;
  return cudaStreamSynchronize(s) == cudaSuccess ? GWM_B200_OK : GWM_B200_ERR_CUDA;
}
