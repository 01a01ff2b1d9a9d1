// fast_rows.cu — the acoustic substep (flat terrain) with independent warps.
//
// Same operator and per-cell arithmetic as k_fast_tma (LocalSplitExplicitFastMode::apply,
// dry_fast_modes.cu:400-656, K9-K15 on one substep), for the substeps that load p' of their
// input with its ring: all inner ones, and a stage's first one behind the TMA slow stage.
//
// What bounds the operator is HBM: 6 fields in and 5 out, 44 B per cell.  k_fast_tma reaches
// 0.69 of the copy bandwidth because it is issue-bound: about 240 instructions per cell, a
// third of them addresses, loop control and the exchange through shared memory around one
// block barrier per plane.  Here
//   - a warp owns 32 x 4 cells, four rows per thread: the Y faces between a thread's rows are
//     computed once, its two outer ones need no neighbour (the warp computes the Y face above
//     its rows itself), so warps exchange nothing and the plane loop has no block barrier;
//   - an extra warp issues the TMA loads: a plane's slot has a full barrier (the loads'
//     transaction count) and an empty one (an arrival per consumer warp);
//   - p' - p'_ref and rho - rho_ref of a level are formed once and carried up;
//   - the level sums stay in shared memory until the CTA's end: one atomic per level.
// 1024 x 1024 x 64: 0.549 ms a substep (0.82 of the copy bandwidth), 0.627 with k_fast_tma's
// split columns, 0.654 with its whole columns; 517 x 389 x 50: 98 us (100 with a test for the
// EOS's far form per row instead of one per plane), 116 with k_fast_tma.
#include <type_traits>

#include "dycore.cuh"
#include "stencil.cuh"
#include "tma.cuh"
#include "zsplit.cuh"

namespace gwmb {
namespace {

namespace fr {
constexpr int TX = 32, ROWS = 4, NW = 4, TY = ROWS * NW;  // consumer warps: 4 rows each
constexpr int NT = 32 * (NW + 1);                         // and the producer warp
constexpr int MIN_CTAS = 4;
constexpr int CBW = 40, CBH = 18;  // p' box: tile and ring
constexpr int FBW = 36, FBH = 17;  // face box: owned faces + east/north face
constexpr int OBW = 32, OBH = 16;  // owned box
constexpr unsigned B_CELL = CBW * CBH * 4, B_FACE = FBW * FBH * 4, B_OWN = OBW * OBH * 4;
constexpr int NSLOT = 3;
// Slot layout in floats, every box on a 128-byte boundary; the base momenta only in the last
// substep of a step, the increments not in a stage's first.
template <bool FIRST, bool FINAL> struct Slot {
  static constexpr int O_RHO = 0, O_TH = 512, O_P = 1024, O_DU = 1760, O_DV = 2400, O_DW = 3040,
                       O_BU = FIRST ? 1760 : 3552, O_BV = O_BU + 512, O_BW = O_BU + 1024,
                       SIZE = FINAL ? O_BU + 1536 : O_BU;
  static_assert(O_DU - O_P >= CBW * CBH && O_DV - O_DU >= FBW * FBH && O_DW - O_DV >= FBW * FBH &&
                    O_P % 32 == 0 && O_DU % 32 == 0 && O_DV % 32 == 0 && O_DW % 32 == 0 && O_BU % 32 == 0,
                "128-byte aligned boxes that fit");
};
// per level: EOS base state (2 doubles), reference means and metric columns (4 floats), the
// warps' level sums (2 long long each)
constexpr size_t kLevel = 2 * sizeof(double) + 4 * sizeof(float) + 2 * NW * sizeof(long long);
template <bool FIRST, bool FINAL>
constexpr size_t smem_bytes(int planes) {
  return size_t(Slot<FIRST, FINAL>::SIZE) * NSLOT * sizeof(float) + 128 + kLevel * size_t(planes + 2);
}
}  // namespace fr

// A level sum's warp total row by row: in a state that has blown up the total can wrap, and the
// cells that it covers show (common.cuh).  Rare, so a call.
__noinline__ __device__ long long row_totals(float v0, float v1, float v2, float v3, float scale) {
  return warp_total_fx(fx(v0, scale)) + warp_total_fx(fx(v1, scale)) + warp_total_fx(fx(v2, scale)) +
         warp_total_fx(fx(v3, scale));
}

template <bool FIRST, int KIND>  // KIND: FastArgs::final_kind
__global__ void __launch_bounds__(fr::NT, fr::MIN_CTAS)
    k_fast_rows(const FastArgs a, const __grid_constant__ FastMaps m, ZSplit zs, int planes) {  // planes: levels of the longest chunk
  using namespace fr;
  constexpr bool FINAL = KIND == 2;
  using L = Slot<FIRST, FINAL>;
  extern __shared__ unsigned char s_dyn[];
  __shared__ __align__(8) uint64_t s_full[NSLOT], s_empty[NSLOT];
  __shared__ float s_ue[2][NW][ROWS][TX + 1];  // X-face increments of a warp's rows, and the east one
  __shared__ int s_abort;
  float* const ring = reinterpret_cast<float*>(align_smem_128(s_dyn));
  double* const t_binv = reinterpret_cast<double*>(ring + L::SIZE * NSLOT);
  double* const t_bpr = t_binv + planes + 2;
  long long* const t_red = reinterpret_cast<long long*>(t_bpr + planes + 2);  // [level][warp][a, b]
  float* const t_pref = reinterpret_cast<float*>(t_red + 2 * NW * (planes + 2));
  float* const t_rref = t_pref + planes + 2;
  float* const t_idzc = t_rref + planes + 2;
  float* const t_idzf = t_idzc + planes + 2;

  const Geom& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  // planes kb .. ke-1 are the CTA's; kg .. kl are loaded (the plane below for the lowest Z
  // face, the one above for the highest)
  const int kb = zs.first(blockIdx.z), ke = zs.last(blockIdx.z, nz), kg = kb > 0 ? kb - 1 : 0, kl = min(ke, nz - 1);
  const int acc_mode = a.acc_off ? 0 : (KIND == 0 ? 1 : 2);

  if (tid == 0) {
    for (int s = 0; s < NSLOT; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], NW);
    }
    mbar_fence_init();
    s_abort = 0;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && a.clr_a)
    for (int q = tid; q < nz; q += NT) { a.clr_a[q] = 0ull; a.clr_b[q] = 0ull; }
  for (int q = kg + tid; q <= kl; q += NT) {  // K6/K7 level means; metric columns; EOS base
    t_rref[q - kg] = (float)(acc_read(a.ref_a + q, kScaleRho) * a.inv_count);
    t_pref[q - kg] = (float)(acc_read(a.ref_b + q, kScaleP) * a.inv_count);
    t_idzc[q - kg] = __ldg(a.idz_c + q);
    t_idzf[q - kg] = __ldg(a.idz_f + q);
    t_binv[q - kg] = __ldg(a.base + nz + q);
    t_bpr[q - kg] = __ldg(a.base + 2 * nz + q);
  }
  __syncthreads();

  if (wid == NW) {  // ---- producer
    if (lane == 0) {
      int stall = take_stall(a.err, FINAL ? kStallLastSubstep : kStallSubstep);  // failure-path tests
      if (stall >= 0) stall = kg + stall % (kl - kg + 1);
      int issued = kg - 1;
      for (int kk = kg; kk <= kl; ++kk) {
        const int q = kk - kg, s = q % NSLOT;
        if (q >= NSLOT && !mbar_wait(&s_empty[s], (q / NSLOT - 1) & 1)) {
          atomicExch(a.err, 1);
          break;
        }
        float* st = ring + s * L::SIZE;
        uint64_t* bar = &s_full[s];
        const bool body = kk >= kb && kk < ke, wface = kk + 1 < nz && kk < ke;
        unsigned bytes = B_OWN + B_CELL + (body ? B_OWN : 0u);
        if (!FIRST) bytes += (body ? 2 * B_FACE : 0u) + (wface ? B_OWN : 0u);
        if (FINAL && body) bytes += 3 * B_OWN;
        mbar_arrive_expect_tx(bar, bytes);
        issued = kk;
        if (kk == stall) continue;  // failure-path testing
        const int x = i0 + kXOff, y = j0 + 1;
        tma_load_3d(st + L::O_P, &m.p, x - 4, j0, kk, bar);
        tma_load_3d(st + L::O_RHO, &m.rho, x, y, kk, bar);
        if (!FIRST && wface) tma_load_3d(st + L::O_DW, &m.dw, x, y, kk + 1, bar);
        if (body) {
          if (!FIRST) {
            tma_load_3d(st + L::O_DU, &m.du, x, y, kk, bar);
            tma_load_3d(st + L::O_DV, &m.dv, x, y, kk, bar);
          }
          tma_load_3d(st + L::O_TH, &m.th, x, y, kk, bar);
          if (FINAL) {
            tma_load_3d(st + L::O_BU, &m.bu, x, y, kk, bar);
            tma_load_3d(st + L::O_BV, &m.bv, x, y, kk, bar);
            tma_load_3d(st + L::O_BW, &m.bw, x, y, kk + 1, bar);
          }
        }
      }
      // the loads in flight end before the CTA's shared memory goes away
      for (int kk = max(kg, issued - NSLOT + 1); kk <= issued; ++kk) {
        const int q = kk - kg;
        mbar_wait(&s_full[q % NSLOT], (q / NSLOT) & 1);
      }
    }
  } else {  // ---- consumers
    const int r0 = wid * ROWS;  // the warp's first row in the tile
    const int w = min(TX, nx - i0), h = min(TY, ny - j0);
    const int gi = i0 + lane, gj = j0 + r0;  // the thread's column and first row
    const float idx = g.inv_dx, idy = g.inv_dy, dtf = a.dtf, gravity = a.gravity;
    const bool edge = (g.per_x && (i0 <= 1 || i0 + w >= nx - 1)) || (g.per_y && (j0 <= 1 || j0 + h >= ny - 1));
    // Interior tiles (full, away from every periodic edge ring and open side) run a copy of
    // the plane loop compiled without the edge logic; both copies do the same arithmetic.
    const bool interior = !edge && i0 + TX <= nx && j0 + TY <= ny && (g.per_x || (i0 > 0 && i0 + TX < nx)) &&
                          (g.per_y || (j0 > 0 && j0 + TY < ny));
    int off[ROWS];  // the owned cells of the current plane
#pragma unroll
    for (int r = 0; r < ROWS; ++r) off[r] = gidx(g, gi, gj + r, kb);
    auto wait_full = [&](int kk) -> bool {
      const int q = kk - kg;
      const bool ok = mbar_wait(&s_full[q % NSLOT], (q / NSLOT) & 1);
      return __all_sync(0xffffffffu, ok);
    };
    auto release = [&](int kk) {  // the warp is done with plane kk's slot
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[(kk - kg) % NSLOT]);
    };
    auto slot_at = [&](int kk) { return ring + ((kk - kg) % NSLOT) * L::SIZE; };

    auto run = [&](auto tile_class) -> bool {  // false when a bounded wait gave up
      constexpr bool IN = decltype(tile_class)::value;
      bool own[ROWS];
      bool su = false;                    // the column's X face lies on an open side
      bool sv[ROWS + 1];                  // the rows' Y faces (and the one above) do
#pragma unroll
      for (int r = 0; r <= ROWS; ++r) sv[r] = !IN && !g.per_y && (gj + r == 0 || gj + r == ny);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) own[r] = IN || (lane < w && r0 + r < h);
      su = !IN && !g.per_x && (gi == 0 || gi == nx);
      const bool se = !IN && !g.per_x && i0 + TX == nx;  // the tile's east X face does
      // store at plane k + up of the thread's row r
      auto put = [&](float* f, int o, int r, int k, int up, float v) {
        if (IN) f[off[r] + up * g.plane] = v;
        else store_tile(f, g, o, gi, gj + r, k + up, v, edge);
      };
      // level means and perturbations of the level below the next face, carried up
      float pc[ROWS], rc[ROWS], pa[ROWS], ra[ROWS], dwc[ROWS];
      auto load_level = [&](int kk, float* p, float* rho) {
        const float* st = slot_at(kk);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          p[r] = st[L::O_P + (r0 + r + 1) * CBW + lane + 4];
          rho[r] = st[L::O_RHO + (r0 + r) * OBW + lane];
        }
      };
      // K14 vertical momentum increment of face kk+1; moves the carried level up
      auto faces_w = [&](int kk, const float* dw, float* wn) {
        float pn[ROWS], rn[ROWS];
        load_level(kk + 1, pn, rn);
        const float pru = t_pref[kk + 1 - kg], rru = t_rref[kk + 1 - kg], idzf = t_idzf[kk + 1 - kg];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float pu = fp::sub(pn[r], pru), ru = fp::sub(rn[r], rru);
          wn[r] = fp::wmom_pert(dw[r], pu, pa[r], ra[r], ru, idzf, gravity, dtf);
          pa[r] = pu;
          ra[r] = ru;
          pc[r] = pn[r];
          rc[r] = rn[r];
        }
      };
      if (!wait_full(kg)) return false;
      load_level(kg, pc, rc);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        pa[r] = fp::sub(pc[r], t_pref[0]);
        ra[r] = fp::sub(rc[r], t_rref[0]);
        dwc[r] = 0.f;  // face 0 never changes
      }
      if (kb > 0) {  // the chunk's lowest Z face, from the plane below
        if (!wait_full(kb)) return false;
        float dw[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) dw[r] = FIRST ? 0.f : slot_at(kg)[L::O_DW + (r0 + r) * OBW + lane];
        faces_w(kg, dw, dwc);
        release(kg);
      }
      for (int k = kb; k < ke; ++k) {
        const float* st = slot_at(k);
        const int pb = k & 1, kt = k - kg;
        // ---- K12/K13 horizontal momentum increments of plane k
        float un[ROWS], vn[ROWS + 1], wn[ROWS];
        {
          const float* sp = st + L::O_P + r0 * CBW + lane + 4;  // p' one row south of the warp's rows
          const float ps = sp[0], pnorth = sp[(ROWS + 1) * CBW];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            const float d = FIRST ? 0.f : st[L::O_DU + (r0 + r) * FBW + lane];
            const float pw = sp[(r + 1) * CBW - 1];
            un[r] = su ? d : fp::hmom(d, pc[r], pw, idx, dtf);
            s_ue[pb][wid][r][lane] = un[r];
          }
#pragma unroll
          for (int r = 0; r <= ROWS; ++r) {
            const float d = FIRST ? 0.f : st[L::O_DV + (r0 + r) * FBW + lane];
            vn[r] = sv[r] ? d : fp::hmom(d, r < ROWS ? pc[r] : pnorth, r > 0 ? pc[r - 1] : ps, idy, dtf);
          }
          if (lane < ROWS) {  // the tile's east X face, a row per lane
            const float d = FIRST ? 0.f : st[L::O_DU + (r0 + lane) * FBW + TX];
            const float* pe = st + L::O_P + (r0 + lane + 1) * CBW + TX + 4;
            s_ue[pb][wid][lane][TX] = se ? d : fp::hmom(d, pe[0], pe[-1], idx, dtf);
          }
        }
        float rho[ROWS], dw[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          rho[r] = rc[r];
          dw[r] = 0.f;
        }
        if (k + 1 < nz) {
          if (!FIRST) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) dw[r] = st[L::O_DW + (r0 + r) * OBW + lane];
          }
          if (!wait_full(k + 1)) return false;
          faces_w(k, dw, wn);
        } else {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) wn[r] = 0.f;  // face nz never changes
        }
        __syncwarp();  // the X-face increments of the warp's rows
        // ---- K15 density of plane k, K10 rho*theta, stores
        const float idzc = t_idzc[kt];
        const double binv = t_binv[kt], bpr = t_bpr[kt];
        long long sa = 0, sb = 0;
        // the rows' new density, rho*theta and p' first, with one test for the EOS's far form
        float nrho[ROWS], nrt[ROWS], np[ROWS];
        bool near = true;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          nrho[r] = fp::density(rho[r], s_ue[pb][wid][r][lane + 1], un[r], vn[r + 1], vn[r], wn[r], dwc[r], idx, idy,
                                idzc, dtf);
          nrt[r] = fp::mul(nrho[r], st[L::O_TH + (r0 + r) * OBW + lane]);
          if (KIND == 0) {
            bool n = true;
            np[r] = eos_pprime_near(nrho[r], nrt[r], binv, bpr, n);
            near = near && (n || !own[r]);
          }
        }
        if (KIND == 0 && !near) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) np[r] = eos_pprime_ref(nrho[r], nrt[r], binv, bpr);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          if (!own[r]) continue;
          const float rn = nrho[r], rt = nrt[r];
          if (FINAL) {
            const int ob = (r0 + r) * OBW + lane;
            put(a.f_rho, kCell, r, k, 0, rn);
            put(a.f_rt, kCell, r, k, 0, rt);
            put(a.f_u, kFaceX, r, k, 0, fp::add(st[L::O_BU + ob], un[r]));
            put(a.f_v, kFaceY, r, k, 0, fp::add(st[L::O_BV + ob], vn[r]));
            if (k == 0) put(a.f_w, kFaceZ, r, 0, 0, __ldg(a.bw + gidx(g, gi, gj + r, 0)));
            put(a.f_w, kFaceZ, r, k, 1, fp::add(st[L::O_BW + ob], wn[r]));
            // open sides: faces nx and ny belong to no tile; their step values are base + increment
            if (!IN && !g.per_x && gi == nx - 1) {
              const int o = gidx(g, nx, gj + r, k);
              a.f_u[o] = fp::add(__ldg(a.bu + o), s_ue[pb][wid][r][lane + 1]);
            }
            if (!IN && !g.per_y && gj + r == ny - 1) {
              const int o = gidx(g, gi, ny, k);
              a.f_v[o] = fp::add(__ldg(a.bv + o), vn[r + 1]);
            }
          } else {
            put(a.rho_out, kCell, r, k, 0, rn);
            put(a.du_out, kFaceX, r, k, 0, un[r]);
            put(a.dv_out, kFaceY, r, k, 0, vn[r]);
            if (k + 1 < nz) put(a.dw_out, kFaceZ, r, k, 1, wn[r]);
          }
          if (KIND == 0) {
            sa += fx(rn, kFxRho);
            sb += fx(np[r], kFxP);
            put(a.p_out, kCell, r, k, 0, np[r]);
          } else if (acc_mode == 2) {
            sa += fx(fp::theta(rn, rt), kFxTheta);
          }
        }
        release(k);
        if (acc_mode) {
          long long ta, tb = 0;
          if (!__any_sync(0xffffffffu, fx_wild(sa) || (KIND == 0 && fx_wild(sb)))) {
            ta = warp_total_fx(sa);
            if (KIND == 0) tb = warp_total_fx(sb);
          } else {
            float v[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) v[r] = !own[r] ? 0.0f : KIND == 0 ? nrho[r] : fp::theta(nrho[r], nrt[r]);
            ta = row_totals(v[0], v[1], v[2], v[3], KIND == 0 ? kFxRho : kFxTheta);
            if (KIND == 0) {
#pragma unroll
              for (int r = 0; r < ROWS; ++r) v[r] = own[r] ? np[r] : 0.0f;
              tb = row_totals(v[0], v[1], v[2], v[3], kFxP);
            }
          }
          if (lane == 0) {
            long long* red = t_red + 2 * (NW * (k - kb) + wid);
            red[0] = ta;
            if (KIND == 0) red[1] = tb;
          }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          dwc[r] = wn[r];
          off[r] += g.plane;
        }
      }
      return true;
    };
    const bool ok = interior ? run(std::true_type{}) : run(std::false_type{});
    if (!ok && lane == 0) {
      s_abort = 1;
      atomicExch(a.err, 1);
    }
  }
  __syncthreads();
  if (acc_mode && !s_abort)
    for (int q = tid; q < ke - kb; q += NT) {
      const long long* red = t_red + 2 * NW * q;
      long long sa = 0, sb = 0;
      for (int v = 0; v < NW; ++v) {
        sa += red[2 * v];
        if (KIND == 0) sb += red[2 * v + 1];
      }
      acc_add(a.acc_a + kb + q, sa);
      if (KIND == 0) acc_add(a.acc_b + kb + q, sb);
    }
}

template <bool FIRST, int KIND>
cudaError_t allow_smem() {
  return cudaFuncSetAttribute(k_fast_rows<FIRST, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)fr::smem_bytes<FIRST, KIND == 2>(kMaxNz));
}

template <bool FIRST, int KIND>
void launch(const FastArgs& a, const FastMaps& m, dim3 grid, const ZSplit& zs, cudaStream_t s) {
  const int planes = zs.longest();
  k_fast_rows<FIRST, KIND><<<grid, fr::NT, fr::smem_bytes<FIRST, KIND == 2>(planes), s>>>(a, m, zs, planes);
}

}  // namespace

cudaError_t init_fast_rows() {
  cudaError_t e = allow_smem<true, 0>();
  if (e == cudaSuccess) e = allow_smem<true, 1>();
  if (e == cudaSuccess) e = allow_smem<true, 2>();
  if (e == cudaSuccess) e = allow_smem<false, 0>();
  if (e == cudaSuccess) e = allow_smem<false, 1>();
  if (e == cudaSuccess) e = allow_smem<false, 2>();
  return e;
}

cudaError_t launch_fast_rows(const FastArgs& a, const FastMaps& m, bool first, cudaStream_t s) {
  if (a.g.nz > kMaxNz || a.g.nz < 1 || !a.err || !a.hmom || !a.dens) return cudaErrorInvalidValue;
  dim3 grid((a.g.nx + fr::TX - 1) / fr::TX, (a.g.ny + fr::TY - 1) / fr::TY);
  const ZSplit zs = z_split(grid.x * grid.y, a.g.nz, 4, 0.7f);
  grid.z = zs.chunks;
  if (first) {
    if (a.final_kind == 0) launch<true, 0>(a, m, grid, zs, s);
    else if (a.final_kind == 1) launch<true, 1>(a, m, grid, zs, s);
    else launch<true, 2>(a, m, grid, zs, s);
  } else {
    if (a.final_kind == 0) launch<false, 0>(a, m, grid, zs, s);
    else if (a.final_kind == 1) launch<false, 1>(a, m, grid, zs, s);
    else launch<false, 2>(a, m, grid, zs, s);
  }
  return cudaGetLastError();
}

}  // namespace gwmb
