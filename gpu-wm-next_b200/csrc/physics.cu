// physics.cu — sm_100a kernels for the moist part of the step: the fused
// three-tracer SSPRK3 stage and the warm-rain column kernel.
#include "dycore.cuh"
#include "physics.cuh"
#include "stencil.cuh"
#include "zsplit.cuh"
#include "rain_cell.cuh"

namespace gwmb {
namespace {

constexpr int BX = 32;
constexpr int NTR = 3;

struct TrCol {
  float rho, uf, vf, wf;
  float rq[NTR], q[NTR];
};

__device__ __forceinline__ TrCol tr_load(const TracerArgs& a, bool valid, int base, int kk) {
  TrCol c{};
  if (!valid) return c;
  const int o = base + kk * a.g.plane;
  if (kk < a.g.nz) {
    c.rho = __ldg(a.rho + o);
    c.uf = __ldg(a.u + o);
    c.vf = __ldg(a.v + o);
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      if (t < a.ntracers) c.rq[t] = __ldg(a.q_in[t] + o);
  }
  if (kk <= a.g.nz) c.wf = __ldg(a.w + o);
  return c;
}

__device__ __forceinline__ void tr_mix(TrCol& c) {
  const float rr = fmaxf(c.rho, 1.0e-6f), y = fp::recip(rr);
#pragma unroll
  for (int t = 0; t < NTR; ++t) c.q[t] = fp::quotient(c.rq[t], rr, y);  // mixing ratio: dry_transport.cu:91-94
}

template <int TBY>
__global__ void __launch_bounds__(BX * TBY) k_tracer_stage(const TracerArgs a) {
  const Geom& g = a.g;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int gi = blockIdx.x * (BX - 2) - 1 + tx;
  const int gj = blockIdx.y * (TBY - 2) - 1 + ty;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const bool valid = gi >= -1 && gi <= nx + 1 && gj >= -1 && gj <= ny + 1;
  const bool inner = tx >= 1 && tx <= BX - 2 && ty >= 1 && ty <= TBY - 2;
  const bool own_c = inner && gi >= 0 && gi < nx && gj >= 0 && gj < ny;
  const int base = valid ? gidx(g, gi, gj, 0) : 0;
  const int ilo = blockIdx.x * (BX - 2), jlo = blockIdx.y * (TBY - 2);
  const bool edge = (g.per_x && (ilo <= 1 || ilo + BX - 3 >= nx - 1)) ||
                    (g.per_y && (jlo <= 1 || jlo + TBY - 3 >= ny - 1));
  const float idx = g.inv_dx, idy = g.inv_dy;
  const bool blend = a.q0[0] != nullptr;

  __shared__ float s_q[NTR][2][TBY][BX];
  __shared__ float s_u[2][TBY][BX], s_v[2][TBY][BX];

  TrCol cm{}, cc = tr_load(a, valid, base, 0), cn = tr_load(a, valid, base, 1);
  TrCol c2 = tr_load(a, valid, base, 2);
  tr_mix(cc);
  tr_mix(cn);
  for (int k = 0; k < nz; ++k) {
    const int pb = k & 1;
    const TrCol c3 = tr_load(a, valid, base, k + 3);
    float q0v[NTR] = {0.f, 0.f, 0.f};
    const int o = base + k * g.plane;
    if (own_c && blend) {
#pragma unroll
      for (int t = 0; t < NTR; ++t)
        if (t < a.ntracers) q0v[t] = __ldg(a.q0[t] + o);
    }
    const float idz = own_c ? (a.terrain ? __ldg(a.idz_c + o) : __ldg(a.idz_c + k)) : 0.f;
#pragma unroll
    for (int t = 0; t < NTR; ++t) s_q[t][pb][ty][tx] = cc.q[t];
    s_u[pb][ty][tx] = cc.uf;
    s_v[pb][ty][tx] = cc.vf;
    __syncthreads();
    if (own_c) {
      const float fw = cc.uf, fe = s_u[pb][ty][tx + 1], fs = cc.vf, fn = s_v[pb][ty + 1][tx];
      const float fb = cc.wf, ft = cn.wf;
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        if (t >= a.ntracers) break;
        const float qc = cc.q[t];
        const float qw = s_q[t][pb][ty][tx - 1], qe = s_q[t][pb][ty][tx + 1];
        const float qs = s_q[t][pb][ty - 1][tx], qn = s_q[t][pb][ty + 1][tx];
        const float qb = (k > 0) ? cm.q[t] : qc;
        const float qt = (k + 1 < nz) ? cn.q[t] : qc;
        const float gw = fp::upwind(fw, qw, qc), ge = fp::upwind(fe, qc, qe);
        const float gs = fp::upwind(fs, qs, qc), gn = fp::upwind(fn, qc, qn);
        const float gb = fp::upwind(fb, qb, qc), gt = fp::upwind(ft, qc, qt);
        const float div = fp::divergence(ge, gw, gn, gs, gt, gb, idx, idy, idz);
        float out = fp::update(cc.rq[t], -a.dt, div, 0.0f);
        if (blend) out = fp::blend(a.wa, q0v[t], a.wb, out);
        store_tile(a.q_out[t], g, kCell, gi, gj, k, out, edge);
      }
    }
    cm = cc;
    cc = cn;
    cn = c2;
    tr_mix(cn);
    c2 = c3;
  }
}


// Warm rain and fallout.  A warp takes 32 columns of one row; a CTA's kRW warps are WX along
// the row and kRW / WX up the levels.  What falls out of a cell depends on that cell alone, so
// only the top cell of a warp's levels waits for its inflow, from the warp above through
// shared memory.  Small grids take all warps up the levels: a column sweep is a serial chain
// of nz cells there (109 us at 128 x 128 x 64; 33 us in eight chunks).  Large grids take long
// rows, whose loads are contiguous (1024 x 1024 x 64: 948 us with 32 columns per CTA).
constexpr int kRW = 8;  // warps per CTA

// MICRO = false: fallout only, on a state whose microphysics was already applied
// (the surrogate's network kernel); the reference applies each cell's microphysics
// before the rain from above arrives, so the split is exact.
template <bool MICRO, int WX>
__global__ void __launch_bounds__(32 * kRW) k_warm_rain(const RainArgs a) {
  constexpr int WZ = kRW / WX;
  const Geom& g = a.g;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wx = wid % WX, wz = wid / WX;
  const int per = (g.nz + WZ - 1) / WZ;
  const int k0 = wz * per, k1 = min(k0 + per, g.nz);  // the warp's levels (none when k0 >= nz)
  __shared__ long long s_th[kMaxNz][WX];
  __shared__ float s_out[kRW][32];  // outflow of each warp's lowest cell
  // fallout of a layer: its floored inverse depth, its depth, the fraction that falls out
  struct Layer {
    float idz, dz, frac;
  };
  __shared__ Layer s_layer[kMaxNz];  // flat terrain: one per level
  auto layer = [&](float v) {
    const float idz = fmaxf(v, 1.0e-6f);
    return Layer{idz, 1.0f / idz, fminf(fmaxf(a.vt * a.dt * idz, 0.0f), 1.0f)};
  };
  if (a.fallout_mode == 1 && !a.terrain) {
    for (int k = threadIdx.x; k < g.nz; k += 32 * kRW) s_layer[k] = layer(__ldg(a.idz_c + k));
    __syncthreads();
  }
  const bool need_rt = MICRO || a.th_acc;
  {
    const int gj = blockIdx.y, ilo = (blockIdx.x * WX + wx) * 32, gi = ilo + lane;
    const bool active = gi < g.nx;
    const bool edge = (g.per_x && (ilo <= 1 || ilo + 31 >= g.nx - 1)) || (g.per_y && (gj <= 1 || gj >= g.ny - 1));
    float out = 0.0f;                     // falling out of the cell above
    float top_kept = 0.0f, top_f = 0.0f;  // top cell: water kept, and the factor to a density
    const bool waits = k1 < g.nz && k0 < k1 && a.fallout_mode != 0;  // its inflow comes from another warp
    // one-cell-ahead prefetch down the levels
    float n_rho = 0.f, n_rt = 0.f, n_qv = 0.f, n_qc = 0.f, n_qr = 0.f;
    auto fetch = [&](int k) {
      const int o = gidx(g, gi, gj, k);
      n_rho = __ldg(a.rho + o);
      n_qr = a.qr[o];
      if (need_rt) n_rt = a.rt[o];
      if (MICRO) { n_qv = a.qv[o]; n_qc = a.qc[o]; }
    };
    if (active && k0 < k1) fetch(k1 - 1);
    for (int k = k1 - 1; k >= k0; --k) {
      long long th_sum = 0;
      const float c_rho = n_rho, c_rt = n_rt, c_qv = n_qv, c_qc = n_qc, c_qr = n_qr;
      if (active && k > k0) fetch(k - 1);
      if (active) {
        const float rho_d = c_rho;
        float rho = 0.0f, th = 0.0f, qv = 0.0f, qc = 0.0f, rqr = c_qr;
        // a / max(rho, 1e-6) of several a by one reciprocal
        const float rr = fmaxf(rho_d, 1.0e-6f), y = fp::recip(rr);
        auto quotient = [&](float v) {
          return fp::quotient(v, rr, y);
        };
        if (MICRO) {  // warm_rain_kernel: warm_rain.cu:36-120
          MicroCell mc;
          if (a.thr >= 0.0f && surely_quiet(rho_d, c_rt, c_qv, c_qc, c_qr)) {
            // micro_step leaves the cell as micro_state derives it: only the mixing ratios
            // and theta are needed, not the temperature, pressure or saturation
            mc.rho = rr;
            mc.th = quotient(c_rt);
            mc.qv = fmaxf(quotient(c_qv), 0.0f);
            mc.qc = 0.0f;  // no cloud or rain water above zero: clipped at zero
            mc.qr = 0.0f;
          } else {
            mc = micro_state(rho_d, c_rt, c_qv, c_qc, c_qr);
            micro_step(mc, MicroParams{a.dt, a.relax, a.thr, a.rate, a.evap, a.latent});
          }
          rho = mc.rho; th = mc.th; qv = mc.qv; qc = mc.qc;
          rqr = rho * mc.qr;
        }
        // fallout of this cell, fed by the cell above
        const bool top = waits && k == k1 - 1;
        if (a.fallout_mode == 1) {  // rain_fallout_metric_kernel: warm_rain.cu:156-191
          const Layer l = a.terrain ? layer(__ldg(a.idz_c + gidx(g, gi, gj, k))) : s_layer[k];
          const float idz = l.idz, dz = l.dz, frac = l.frac;
          const float old_a = fmaxf(rqr, 0.0f) * dz;
          const float fall = frac * old_a;
          rqr = ((old_a - fall) + out) * idz;
          if (top) { top_kept = old_a - fall; top_f = idz; }
          out = fall;
        } else if (a.fallout_mode == 2) {  // rain_fallout_nominal_kernel: warm_rain.cu:122-154
          const float dz = fmaxf(a.layer_depth, 1.0e-3f);
          const float frac = fminf(fmaxf(a.vt * a.dt / dz, 0.0f), 1.0f);
          if (frac > 0.0f) {
            const float old_a = fmaxf(rqr, 0.0f) * dz;
            const float fall = frac * old_a;
            rqr = ((old_a - fall) + out) / dz;
            if (top) { top_kept = old_a - fall; top_f = dz; }
            out = fall;
          } else if (top) {
            top_kept = rqr;
            top_f = 0.0f;  // nothing falls: the cell keeps its water
          }
        }
        const float rt_new = MICRO ? rho * th : c_rt;
        if (MICRO) {
          store_tile(a.qv, g, kCell, gi, gj, k, rho * qv, edge);
          store_tile(a.qc, g, kCell, gi, gj, k, rho * qc, edge);
          store_tile(a.rt, g, kCell, gi, gj, k, rt_new, edge);
        }
        if ((MICRO || a.fallout_mode) && !top) store_tile(a.qr, g, kCell, gi, gj, k, rqr, edge);
        if (a.th_acc) th_sum = fx(quotient(rt_new), kFxTheta);
      }
      if (a.th_acc) {
        const long long t = warp_total_fx(th_sum);
        if (lane == 0) s_th[k][wx] = t;
      }
    }
    s_out[wid][lane] = out;
    __syncthreads();
    if (active && waits) {  // the top cell's inflow: what fell out of the warp above
      const float in = s_out[wid + WX][lane];
      const float rqr = a.fallout_mode == 1 ? (top_kept + in) * top_f : (top_f > 0.0f ? (top_kept + in) / top_f : top_kept);
      store_tile(a.qr, g, kCell, gi, gj, k1 - 1, rqr, edge);
    }
    if (wz == 0 && active && a.fallout_mode && a.precip) {  // compensated FP64 surface accumulation
      const int o = gj * g.nx + gi;
      const double s = a.precip[o], x = (double)out, t = s + x;
      a.precip_comp[o] += (fabs(s) >= fabs(x)) ? (s - t) + x : (x - t) + s;
      a.precip[o] = t;
    }
  }
  if (a.th_acc)
    for (int k = threadIdx.x; k < g.nz; k += 32 * kRW) {
      long long t = 0;
      for (int v = 0; v < WX; ++v) t += s_th[k][v];
      acc_add(a.th_acc + k, t);
    }
}

}  // namespace

cudaError_t launch_tracer_stage(const TracerArgs& a, cudaStream_t s, int tile_rows) {
  if (tile_rows == 16) {
    const dim3 grid((a.g.nx + BX - 3) / (BX - 2), (a.g.ny + 16 - 3) / (16 - 2));
    k_tracer_stage<16><<<grid, dim3(BX, 16), 0, s>>>(a);
  } else {
    const dim3 grid((a.g.nx + BX - 3) / (BX - 2), (a.g.ny + 8 - 3) / (8 - 2));
    k_tracer_stage<8><<<grid, dim3(BX, 8), 0, s>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_warm_rain(const RainArgs& a, cudaStream_t s, bool micro) {
  if (a.g.nz > kMaxNz) return cudaErrorInvalidValue;
  // enough CTAs for two waves of four per SM decide how much of the CTA goes along the row
  const int nseg = (a.g.nx + 31) / 32 * a.g.ny;
  const int wave = 8 * sm_count();
  const int wx = nseg >= 4 * wave ? 4 : nseg >= 2 * wave ? 2 : 1;
  const dim3 grid((a.g.nx + 32 * wx - 1) / (32 * wx), a.g.ny);
  if (!micro && !a.fallout_mode && !a.th_acc) return cudaSuccess;
  switch (wx) {
    case 4: micro ? k_warm_rain<true, 4><<<grid, 32 * kRW, 0, s>>>(a) : k_warm_rain<false, 4><<<grid, 32 * kRW, 0, s>>>(a); break;
    case 2: micro ? k_warm_rain<true, 2><<<grid, 32 * kRW, 0, s>>>(a) : k_warm_rain<false, 2><<<grid, 32 * kRW, 0, s>>>(a); break;
    default: micro ? k_warm_rain<true, 1><<<grid, 32 * kRW, 0, s>>>(a) : k_warm_rain<false, 1><<<grid, 32 * kRW, 0, s>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace gwmb
