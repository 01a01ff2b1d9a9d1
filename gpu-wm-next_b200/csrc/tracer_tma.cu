// tracer_tma.cu — one SSPRK3 stage of up to three passive tracers on owned tiles fed by
// TMA (flat terrain, and terrain with the per-cell inverse layer depth).
//
// Same operator and per-cell arithmetic as k_tracer_stage: the upwind mixing-ratio
// flux divergence with frozen end-of-step dry mass fluxes
// (passive_tracer_stage_kernel, src/dycore/dry_transport.cu:49-125; clip at zero) and
// the SSPRK3 blend of advance_passive_tracers_ssprk3 (:440-518).  As in fast_rows.cu a warp
// owns 32 x 4 cells, four rows per thread, an extra warp issues the TMA loads into a
// three-slot ring with full and empty barriers, and the plane loop has no block barrier:
//   rho, rho*q (up to three tracers)  40 x 18 boxes: the tile and its halo ring
//   u, v                              36 x 17 boxes: owned faces + the east/north face
//   w                                 32 x 16 box: owned Z faces (plane nz: w only)
// A thread computes the mixing ratios of its rows one plane ahead and those of the rows around
// them, and a position of the warp's two ring columns, with one reciprocal per position; all of
// a plane's come first, with one test for quotients that are not finite, so their
// chains interleave.  The Y fluxes between its rows are computed once, and the flux out of a
// plane's top is carried as the next plane's bottom flux.  Bounds: issue, close to HBM (13
// fields of 4 B per cell take 0.53 ms for 1024 x 1024 x 64, three tracers, at the copy
// bandwidth): there 0.640 ms a stage, 0.767 with a test per position and the blend decided at
// run time, 1.045 with two rows eight apart per thread, 426 instructions per cell and a block
// barrier per plane; 517 x 389 x 50 0.113 ms, 0.141, 0.191.
#include <type_traits>

#include "physics.cuh"
#include "stencil.cuh"
#include "tma.cuh"
#include "zsplit.cuh"

namespace gwmb {
namespace {

namespace tt {
constexpr int TX = 32, ROWS = 4, NW = 4, TY = ROWS * NW;  // consumer warps: 4 rows each
constexpr int NT = 32 * (NW + 1);                         // and the producer warp
constexpr int MIN_CTAS = 3, NTR = 3;
constexpr int CBW = 40, CBH = 18, FBW = 36, FBH = 17, OBW = 32, OBH = 16;
constexpr int O_RHO = 0, O_U = 736, O_V = 1376, O_W = 2016, O_Q = 2528, Q_STRIDE = 736, NSLOT = 3;
template <int N> constexpr int kSlot = O_Q + N * Q_STRIDE;  // floats, N tracers
constexpr unsigned B_CELL = CBW * CBH * 4, B_FACE = FBW * FBH * 4, B_OWN = OBW * OBH * 4;
constexpr size_t smem_bytes(int ntr) { return size_t(O_Q + ntr * Q_STRIDE) * NSLOT * sizeof(float) + 128; }
static_assert(O_U % 32 == 0 && O_V % 32 == 0 && O_W % 32 == 0 && O_Q % 32 == 0 && Q_STRIDE % 32 == 0 &&
                  O_U - O_RHO >= CBW * CBH && O_V - O_U >= FBW * FBH && O_W - O_V >= FBW * FBH &&
                  O_Q - O_W >= OBW * OBH && Q_STRIDE >= CBW * CBH,
              "128-byte aligned boxes that fit");
}  // namespace tt

template <bool TERRAIN, int N, bool BLEND>  // N: tracers; BLEND: stages 2 and 3
__global__ void __launch_bounds__(tt::NT, tt::MIN_CTAS)
    k_tracer_tma(const TracerArgs a, const __grid_constant__ TracerMaps m, ZSplit zs) {
  using namespace tt;
  constexpr int SLOT = kSlot<N>;
  extern __shared__ unsigned char s_dyn[];
  __shared__ __align__(8) uint64_t s_full[NSLOT], s_empty[NSLOT];
  __shared__ float s_q[2][NW][N][ROWS][TX + 2];  // a warp's mixing ratios with its ring columns
  float* const ring = reinterpret_cast<float*>(align_smem_128(s_dyn));

  const Geom& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  // planes kb .. ke-1 are the CTA's; it also loads plane ke and (above the ground) the plane
  // below, whose mixing ratios its lowest faces read
  const int kb = zs.first(blockIdx.z), ke = zs.last(blockIdx.z, nz), kg = kb > 0 ? kb - 1 : 0;

  if (tid == 0) {
    for (int s = 0; s < NSLOT; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], NW);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (wid == NW) {  // ---- producer
    if (lane == 0) {
      int stall = take_stall(a.err, kStallTracer);  // failure-path tests
      if (stall >= 0) stall = kg + stall % (ke - kg + 1);
      int issued = kg - 1;
      for (int kk = kg; kk <= ke; ++kk) {  // plane nz holds the top faces only
        const int q = kk - kg, s = q % NSLOT;
        if (q >= NSLOT && !mbar_wait(&s_empty[s], (q / NSLOT - 1) & 1)) {
          atomicExch(a.err, 1);
          break;
        }
        float* st = ring + s * SLOT;
        uint64_t* bar = &s_full[s];
        const bool cells = kk < nz, body = kk >= kb && kk < ke;
        mbar_arrive_expect_tx(bar, B_OWN + (cells ? (1 + N) * B_CELL : 0u) + (body ? 2 * B_FACE : 0u));
        issued = kk;
        if (kk == stall) continue;  // failure-path testing
        const int x = i0 + kXOff, y = j0 + 1;
        tma_load_3d(st + O_W, &m.w, x, y, kk, bar);
        if (cells) {
          tma_load_3d(st + O_RHO, &m.rho, x - 4, j0, kk, bar);
#pragma unroll
          for (int t = 0; t < N; ++t) tma_load_3d(st + O_Q + t * Q_STRIDE, &m.q[t], x - 4, j0, kk, bar);
        }
        if (body) {
          tma_load_3d(st + O_U, &m.u, x, y, kk, bar);
          tma_load_3d(st + O_V, &m.v, x, y, kk, bar);
        }
      }
      // the loads in flight end before the CTA's shared memory goes away
      for (int kk = max(kg, issued - NSLOT + 1); kk <= issued; ++kk) {
        const int q = kk - kg;
        mbar_wait(&s_full[q % NSLOT], (q / NSLOT) & 1);
      }
    }
    return;
  }
  // ---- consumers
  const int r0 = wid * ROWS;  // the warp's first row in the tile
  const int w = min(TX, nx - i0), h = min(TY, ny - j0);
  const int gi = i0 + lane, gj = j0 + r0;  // the thread's column and first row
  const bool edge = (g.per_x && (i0 <= 1 || i0 + w >= nx - 1)) || (g.per_y && (j0 <= 1 || j0 + h >= ny - 1));
  const float idx = g.inv_dx, idy = g.inv_dy;
  // Interior tiles (full, away from every periodic edge ring) run a copy of the plane loop
  // with plain stores instead of the periodic mirror stores; the arithmetic is the same.
  const bool interior = !edge && i0 + TX <= nx && j0 + TY <= ny;
  auto wait_full = [&](int kk) -> bool {
    const int q = kk - kg;
    const bool ok = mbar_wait(&s_full[q % NSLOT], (q / NSLOT) & 1);
    return __all_sync(0xffffffffu, ok);
  };
  auto release = [&](int kk) {  // the warp is done with plane kk's slot
    __syncwarp();
    if (lane == 0) mbar_arrive(&s_empty[(kk - kg) % NSLOT]);
  };
  auto slot_at = [&](int kk) { return ring + ((kk - kg) % NSLOT) * SLOT; };
  // mixing ratios (dry_transport.cu:91-94) at position b of a plane's cell boxes; `near` is
  // cleared where one is not finite and each is to be tested
  auto mix_near = [&](const float* st, int b, float* q, bool& near) {
    const float rr = fmaxf(st[O_RHO + b], 1.0e-6f), y = fp::recip(rr);
    float sum = 0.0f;
#pragma unroll
    for (int t = 0; t < N; ++t) {
      q[t] = fp::div_by(st[O_Q + t * Q_STRIDE + b], rr, y);
      sum += fabsf(q[t]);
    }
    near = near && fp::finite(sum);
  };
  // each quotient tested on its own: rare, so a call (128 x 128 x 64: 27 us a stage, 30 inlined)
  auto mix_each = [&](const float* st, int b, float* q) {
    const float rr = fmaxf(st[O_RHO + b], 1.0e-6f);
#pragma unroll
    for (int t = 0; t < N; ++t) q[t] = fp::quotient_far(st[O_Q + t * Q_STRIDE + b], rr);
  };
  auto mix = [&](const float* st, int b, float* q) {
    bool near = true;
    mix_near(st, b, q, near);
    if (!near) mix_each(st, b, q);
  };

  auto run = [&](auto tile_class) -> bool {  // false when a bounded wait gave up
    constexpr bool IN = decltype(tile_class)::value;  // interior tile: plain stores
    int off[ROWS];  // the owned cells of the current plane
    bool own[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      off[r] = gidx(g, gi, gj + r, kb);
      own[r] = IN || (lane < w && r0 + r < h);
    }
    const int b0 = (r0 + 1) * CBW + lane + 4;  // box position of the thread's first row
    const int ring_row = lane & 3, ring_col = (lane & 4) ? TX : -1;
    const int ring_b = (r0 + ring_row + 1) * CBW + ring_col + 4;
    float qc[ROWS][N], fz[ROWS][N];  // mixing ratios of plane k, fluxes through its bottom faces
    if (!wait_full(kg)) return false;
    {
      const float* st = slot_at(kg);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) mix(st, b0 + r * CBW, qc[r]);
    }
    if (kb > 0) {
      if (!wait_full(kb)) return false;
      const float* st = slot_at(kb);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        float qn[N];
        mix(st, b0 + r * CBW, qn);
        const float f = st[O_W + (r0 + r) * OBW + lane];
#pragma unroll
        for (int t = 0; t < N; ++t) {
          fz[r][t] = fp::upwind(f, qc[r][t], qn[t]);
          qc[r][t] = qn[t];
        }
      }
      release(kg);
    } else {
      const float* st = slot_at(0);
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int t = 0; t < N; ++t) fz[r][t] = fp::upwind(st[O_W + (r0 + r) * OBW + lane], qc[r][t], qc[r][t]);
    }
    for (int k = kb; k < ke; ++k) {
      const float* st = slot_at(k);
      const int pb = k & 1;
      // blend partner and inverse depths of the plane: used at the end
      float q0[ROWS][N], idz[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        idz[r] = TERRAIN ? (own[r] ? __ldg(a.idz_c + off[r]) : 0.f) : __ldg(a.idz_c + k);
#pragma unroll
        for (int t = 0; t < N; ++t) q0[r][t] = BLEND && own[r] ? __ldg(a.q0[t] + off[r]) : 0.f;
      }
      // the mixing ratios of the rows around the warp's and of its ring columns (a position per
      // lane), and of its rows at plane k+1: one test for quotients that are not finite
      const bool top = k + 1 == nz;
      float qs[N], qn[N], qr[N], qt[ROWS][N];
      bool near = true;
      mix_near(st, b0 - CBW, qs, near);
      mix_near(st, b0 + ROWS * CBW, qn, near);
      mix_near(st, ring_b, qr, near);
      if (!wait_full(k + 1)) return false;
      const float* sn = slot_at(k + 1);
      if (!top) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) mix_near(sn, b0 + r * CBW, qt[r], near);
      }
      if (!near) {
        mix_each(st, b0 - CBW, qs);
        mix_each(st, b0 + ROWS * CBW, qn);
        mix_each(st, ring_b, qr);
        if (!top) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) mix_each(sn, b0 + r * CBW, qt[r]);
        }
      }
      if (top) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
          for (int t = 0; t < N; ++t) qt[r][t] = qc[r][t];
      }
      // the ring columns, and the warp's rows for the neighbouring lanes
      if (lane < 2 * ROWS) {
#pragma unroll
        for (int t = 0; t < N; ++t) s_q[pb][wid][t][ring_row][ring_col + 1] = qr[t];
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int t = 0; t < N; ++t) s_q[pb][wid][t][r][lane + 1] = qc[r][t];
      __syncwarp();
      const float* su = st + O_U + r0 * FBW + lane;
      const float* sv = st + O_V + r0 * FBW + lane;
      float gy[N];  // Y fluxes below the row
#pragma unroll
      for (int t = 0; t < N; ++t) gy[t] = fp::upwind(sv[0], qs[t], qc[0][t]);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float fw = su[r * FBW], fe = su[r * FBW + 1], fn = sv[(r + 1) * FBW];
        const float ft = sn[O_W + (r0 + r) * OBW + lane];
#pragma unroll
        for (int t = 0; t < N; ++t) {
          const float c = qc[r][t];
          const float gw = fp::upwind(fw, s_q[pb][wid][t][r][lane], c);
          const float ge = fp::upwind(fe, c, s_q[pb][wid][t][r][lane + 2]);
          const float gn = fp::upwind(fn, c, r + 1 < ROWS ? qc[r + 1 < ROWS ? r + 1 : r][t] : qn[t]);
          const float gt = fp::upwind(ft, c, qt[r][t]);
          const float div = fp::divergence(ge, gw, gn, gy[t], gt, fz[r][t], idx, idy, idz[r]);
          float out = fp::update(st[O_Q + t * Q_STRIDE + b0 + r * CBW], -a.dt, div, 0.0f);
          if (BLEND) out = fp::blend(a.wa, q0[r][t], a.wb, out);
          if (IN) a.q_out[t][off[r]] = out;
          else if (own[r]) store_tile(a.q_out[t], g, kCell, gi, gj + r, k, out, edge);
          gy[t] = gn;
          fz[r][t] = gt;
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int t = 0; t < N; ++t) qc[r][t] = qt[r][t];
        off[r] += g.plane;
      }
      release(k);
    }
    return true;
  };
  const bool ok = interior ? run(std::true_type{}) : run(std::false_type{});
  if (!ok && lane == 0) atomicExch(a.err, 1);
}

template <bool TERRAIN, int N>
cudaError_t allow_smem() {
  cudaError_t e = cudaFuncSetAttribute(k_tracer_tma<TERRAIN, N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)tt::smem_bytes(N));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tracer_tma<TERRAIN, N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)tt::smem_bytes(N));
  return e;
}

template <bool TERRAIN, bool BLEND>
void launch(const TracerArgs& a, const TracerMaps& m, dim3 grid, const ZSplit& zs, cudaStream_t s) {
  const size_t smem = tt::smem_bytes(a.ntracers);
  if (a.ntracers == 1) k_tracer_tma<TERRAIN, 1, BLEND><<<grid, tt::NT, smem, s>>>(a, m, zs);
  else if (a.ntracers == 2) k_tracer_tma<TERRAIN, 2, BLEND><<<grid, tt::NT, smem, s>>>(a, m, zs);
  else k_tracer_tma<TERRAIN, 3, BLEND><<<grid, tt::NT, smem, s>>>(a, m, zs);
}

}  // namespace

cudaError_t init_tracer_tma() {
  cudaError_t e = allow_smem<false, 1>();
  if (e == cudaSuccess) e = allow_smem<false, 2>();
  if (e == cudaSuccess) e = allow_smem<false, 3>();
  if (e == cudaSuccess) e = allow_smem<true, 1>();
  if (e == cudaSuccess) e = allow_smem<true, 2>();
  if (e == cudaSuccess) e = allow_smem<true, 3>();
  return e;
}

cudaError_t launch_tracer_tma(const TracerArgs& a, const TracerMaps& m, cudaStream_t s) {
  if (a.g.nz < 1 || !a.err || a.ntracers < 1 || a.ntracers > tt::NTR) return cudaErrorInvalidValue;
  dim3 grid((a.g.nx + tt::TX - 1) / tt::TX, (a.g.ny + tt::TY - 1) / tt::TY);
  const ZSplit zs = z_split(grid.x * grid.y, a.g.nz, tt::MIN_CTAS, 1.0f);
  grid.z = zs.chunks;
  const bool blend = a.q0[0] != nullptr;
  if (a.terrain) blend ? launch<true, true>(a, m, grid, zs, s) : launch<true, false>(a, m, grid, zs, s);
  else blend ? launch<false, true>(a, m, grid, zs, s) : launch<false, false>(a, m, grid, zs, s);
  return cudaGetLastError();
}

}  // namespace gwmb
