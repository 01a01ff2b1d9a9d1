// fast_terrain_tma.cu — acoustic substep on terrain fed by TMA tile loads.
//
// Same operator and per-cell arithmetic as k_fast_substep<TERRAIN = true> (K9-K15 of
// LocalSplitExplicitFastMode::apply, src/dycore/dry_fast_modes.cu:160-394: the
// chain-rule horizontal pressure gradient of :160-301, perturbations about the column
// hydrostatic reference of :108-158, which k_column_reference builds before the
// substep), with the data path of k_fast_tma: one elected thread per CTA fetches every
// plane's tiles with cp.async.bulk.tensor.3d into a five-slot shared-memory ring, and a
// CTA owns a 32 x 16 tile, two adjacent rows per thread.  Per plane kk the slot holds
//   rho(kk), theta(kk)   first substep of a stage: 40 x 18 boxes (the tile and its halo
//                        ring, from which the full pressure is derived); otherwise the
//                        owned 32 x 16 box
//   z(kk)                40 x 18: cell-centre heights of the tile and its ring
//   p(kk)                40 x 18, not in a first substep: the full pressure of the input
//                        with its ring, stored by the previous substep, so the EOS runs
//                        once per owned cell instead of at every position of a tile
//   du(kk), dv(kk)       36 x 17, not in a first substep: owned faces plus the tile's
//                        east/north face
//   dw(kk+1)             32 x 16, not in a first substep
// The vertical pressure derivative of the tile and its ring takes p at three levels; it
// is derived one plane ahead (plane k+1 while plane k's faces are computed, from the
// slots of planes k, k+1, k+2), so one barrier per plane publishes it together with the
// new face increments.  A thread carries p, z and dp/dz of its rows up, so it reads each once,
// and computes the Y face between its rows itself.  The owned cells' metric columns, column
// reference and (last substep of the step) stage base momenta are per-thread coalesced loads
// issued one plane ahead.
// Bounds: the chain of a plane (dp/dz, faces, barrier, density, EOS) with 16 warps per SM, and
// issue; 16 fields of 4 B per cell would take 0.20 ms for 512 x 512 x 80 at the copy bandwidth.
// There 0.346 ms, 0.465 with every neighbour read from shared memory and no carried values;
// independent warps of four rows as in fast_rows.cu took 0.51 to 0.58 (too few warps in flight
// for these chains, at 168 registers).
#include <type_traits>

#include "dycore.cuh"
#include "stencil.cuh"
#include "tma.cuh"
#include "zsplit.cuh"

namespace gwmb {
namespace {

namespace fz {
constexpr int TX = 32, TY = 16, ROWS = 2, NT = 256, NW = NT / 32;
constexpr int CBW = 40, CBH = 18;  // cell box: tile + halo ring, x from i0-4 (16-byte aligned)
constexpr int FBW = 36, FBH = 17;  // face box: owned faces + the tile's east/north face
constexpr int OBW = 32, OBH = 16;  // owned box
constexpr unsigned B_CELL = CBW * CBH * 4, B_FACE = FBW * FBH * 4, B_OWN = OBW * OBH * 4;
// ring: planes k, k+1, k+2 are read while plane k is computed; plane k+4 is issued into
// the slot of plane k-1 after the plane's barrier
constexpr int NSLOT = 5, AHEAD = NSLOT - 1;
constexpr int ISSUER = NT - 32;  // lane 0 of the last warp: no halo role (warps 0-2 carry those)
constexpr int PW = TX + 2, PH = TY + 2;  // derived planes: tile + ring, 34 x 18
// Slot layouts in floats; every sub-buffer starts on a 128-byte boundary.
template <bool FIRST> struct Slot;
template <> struct Slot<true> {  // rho, theta with the ring (pressure derived), heights
  static constexpr int O_RHO = 0, O_TH = 736, O_Z = 1472, O_P = 0, O_DU = 0, O_DV = 0, O_DW = 0, SIZE = 2208,
                       RW = CBW, R0 = 1, C0 = 4;
};
template <> struct Slot<false> {  // owned rho, theta; heights and pressure with the ring; increments
  static constexpr int O_RHO = 0, O_TH = 512, O_Z = 1024, O_P = 1760, O_DU = 2496, O_DV = 3136, O_DW = 3776,
                       SIZE = 4288, RW = OBW, R0 = 0, C0 = 0;
};
template <bool FIRST>
constexpr bool slot_ok() {
  using L = Slot<FIRST>;
  constexpr int rb = FIRST ? CBW * CBH : OBW * OBH;
  return L::O_TH % 32 == 0 && L::O_Z % 32 == 0 && L::SIZE % 32 == 0 && L::O_TH - L::O_RHO >= rb &&
         L::O_Z - L::O_TH >= rb &&
         (FIRST ? L::SIZE - L::O_Z >= CBW * CBH
                : (L::O_P % 32 == 0 && L::O_DU % 32 == 0 && L::O_DV % 32 == 0 && L::O_DW % 32 == 0 &&
                   L::O_P - L::O_Z >= CBW * CBH && L::O_DU - L::O_P >= CBW * CBH && L::O_DV - L::O_DU >= FBW * FBH &&
                   L::O_DW - L::O_DV >= FBW * FBH && L::SIZE - L::O_DW >= OBW * OBH));
}
static_assert(slot_ok<true>() && slot_ok<false>(), "128-byte aligned sub-buffers that fit their boxes");
template <bool FIRST>
constexpr size_t dyn_smem() {
  return size_t(Slot<FIRST>::SIZE) * NSLOT * sizeof(float) + 128;
}
}  // namespace fz

// Derived planes and per-CTA state besides the ring.  p: the full pressure of the tile
// and its ring, three planes (first substep only; later substeps read it from the ring).
template <bool FIRST>
struct TerrainShared {
  float p[FIRST ? 3 : 1][fz::PH][fz::PW];
  float dz[2][fz::PH][fz::PW];               // dp/dz of the tile and its ring (column_dpdz)
  float du[2][fz::TY][fz::TX + 1];           // new X-face increments (own + east face)
  float dv[2][fz::TY / fz::ROWS + 1][fz::TX];  // new Y-face increments below each thread's rows, and the north face
  long long red[2][fz::NW];
  __align__(8) uint64_t bar[fz::NSLOT];
  int abort[2];
};

// Owned-cell columns of one row at one plane, loaded a plane ahead of their use.
struct TerrainCol {
  float idzc, idzf, pref, rref, bu, bv, bw;  // idzf, bw: face k+1; pref, rref: level k+1
};

template <bool FIRST, int KIND>  // KIND: FastArgs::final_kind
__global__ void __launch_bounds__(fz::NT, 2)
    k_fast_terrain_tma(const FastArgs a, const __grid_constant__ FastTerrainMaps m, ZSplit zs) {
  using namespace fz;
  using L = Slot<FIRST>;
  constexpr int O_RHO = L::O_RHO, O_TH = L::O_TH, O_Z = L::O_Z, O_P = L::O_P, O_DU = L::O_DU, O_DV = L::O_DV,
                O_DW = L::O_DW, RW = L::RW, R0 = L::R0, C0 = L::C0, SLOT = L::SIZE;
  constexpr bool FINAL = KIND == 2;
  extern __shared__ unsigned char s_dyn[];
  __shared__ TerrainShared<FIRST> S;
  float* const ring = reinterpret_cast<float*>(align_smem_128(s_dyn));

  const Geom& g = a.g;
  const int nz = g.nz;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nx = g.nx, ny = g.ny;
  const int w = min(TX, nx - i0), h = min(TY, ny - j0);
  const int r0 = ty * ROWS, gi = i0 + tx, gj = j0 + r0;  // the thread's column and first row
  const bool own_rt[ROWS] = {tx < w && r0 < h, tx < w && r0 + 1 < h};
  const bool edge = (g.per_x && (i0 <= 1 || i0 + w >= nx - 1)) || (g.per_y && (j0 <= 1 || j0 + h >= ny - 1));
  // halo roles (threads 0-95, whole warps): 0 west column, 1 east column, 2 south row,
  // 3 north row; (hr, hc) in derived-plane coordinates (row 0 = j0-1, column 0 = i0-1)
  int role = -1, hr = 0, hc = 0;
  if (tid < TY) { if (tid < h) { role = 0; hr = tid + 1; hc = 0; } }
  else if (tid < 2 * TY) { if (tid - TY < h) { role = 1; hr = tid - TY + 1; hc = w + 1; } }
  else if (tid < 2 * TY + TX) { if (tid - 2 * TY < w) { role = 2; hr = 0; hc = tid - 2 * TY + 1; } }
  else if (tid < 2 * TY + 2 * TX) { if (tid - 2 * TY - TX < w) { role = 3; hr = h + 1; hc = tid - 2 * TY - TX + 1; } }
  const int hi = i0 + hc - 1, hj = j0 + hr - 1;  // global cell of the halo role
  const bool h_skip = (role == 1 && hi == nx && !g.per_x) || (role == 3 && hj == ny && !g.per_y);
  const float idx = g.inv_dx, idy = g.inv_dy, dtf = a.dtf, gravity = a.gravity;
  // terrain: no reference level sums; theta level sums of a stage's result
  const bool acc = KIND != 0 && !a.acc_off;

  if (tid == 0) {
    for (int s = 0; s < NSLOT; ++s) mbar_init(&S.bar[s], 1);
    mbar_fence_init();
    S.abort[0] = 0;
    S.abort[1] = 0;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && a.clr_a)
    for (int q = tid; q < nz; q += NT) { a.clr_a[q] = 0ull; a.clr_b[q] = 0ull; }
  __syncthreads();

  int stall = tid == ISSUER ? take_stall(a.err, FINAL ? kStallLastSubstep : kStallSubstep) : -1;  // failure-path tests
  // the CTA's planes are kb .. ke-1; it also loads the planes around them: the one below for
  // its lowest Z face and dp/dz, the one above for its highest
  const int kb = zs.first(blockIdx.z), ke = zs.last(blockIdx.z, nz), kg = kb > 0 ? kb - 1 : 0, kl = min(ke, nz - 1);
  if (stall >= 0) stall = kg + stall % (kl - kg + 1);
  auto slot_of = [&](int kk) { return ring + ((kk - kg) % NSLOT) * SLOT; };
  auto issue = [&](int kk) {
    float* st = slot_of(kk);
    uint64_t* bar = &S.bar[(kk - kg) % NSLOT];
    const bool body = kk >= kb && kk < ke;
    const bool wface = kk + 1 < nz && kk < ke;
    unsigned bytes = FIRST ? 3 * B_CELL : B_OWN + 2 * B_CELL + (body ? B_OWN + 2 * B_FACE : 0u) + (wface ? B_OWN : 0u);
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(bar, bytes);
    if (kk == stall) return;  // failure-path testing: this plane's loads stay unissued
    if (FIRST) {
      tma_load_3d(st + O_RHO, &m.rho, i0 + kXOff - 4, j0, kk, bar);
      tma_load_3d(st + O_TH, &m.th, i0 + kXOff - 4, j0, kk, bar);
    } else {
      tma_load_3d(st + O_RHO, &m.rho, i0 + kXOff, j0 + 1, kk, bar);
      tma_load_3d(st + O_P, &m.p, i0 + kXOff - 4, j0, kk, bar);
      if (body) {
        tma_load_3d(st + O_TH, &m.th, i0 + kXOff, j0 + 1, kk, bar);
        tma_load_3d(st + O_DU, &m.du, i0 + kXOff, j0 + 1, kk, bar);
        tma_load_3d(st + O_DV, &m.dv, i0 + kXOff, j0 + 1, kk, bar);
      }
      if (wface) tma_load_3d(st + O_DW, &m.dw, i0 + kXOff, j0 + 1, kk + 1, bar);
    }
    tma_load_3d(st + O_Z, &m.z, i0 + kXOff - 4, j0, kk, bar);
  };
  int issued = kg - 1, waited = kg - 1;
  auto wait_plane = [&](int kk, int epoch) {
    if (!mbar_wait(&S.bar[(kk - kg) % NSLOT], ((kk - kg) / NSLOT) & 1)) {
      S.abort[epoch & 1] = 1;
      atomicExch(a.err, 1);
    } else if (waited == kk - 1) {
      waited = kk;  // a plane whose wait gave up stays in the drain below, with those after it
    }
  };
  // values of plane kk at derived-plane position (r, c)
  auto Pv = [&](int kk, int r, int c) {
    if constexpr (FIRST) return S.p[kk % 3][r][c];
    else return slot_of(kk)[O_P + r * CBW + c + 3];
  };
  auto Zv = [&](int kk, int r, int c) { return slot_of(kk)[O_Z + r * CBW + c + 3]; };
  // p and z of plane kk in the thread's rows.  First substep, K10 + K20: the full pressure is
  // derived, at the thread's halo role too, and published.
  auto load_level = [&](int kk, float* p, float* z) {
    const float* st = slot_of(kk);
    auto derive = [&](int r, int c) {
      const float rho = st[O_RHO + r * CBW + c + 3], th = st[O_TH + r * CBW + c + 3];
      return eos_pressure(rho, fp::mul(rho, th));
    };
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      z[r] = Zv(kk, r0 + r + 1, tx + 1);
      if constexpr (FIRST) {
        p[r] = derive(r0 + r + 1, tx + 1);
        if (own_rt[r]) S.p[kk % 3][r0 + r + 1][tx + 1] = p[r];
      } else {
        p[r] = Pv(kk, r0 + r + 1, tx + 1);
      }
    }
    if constexpr (FIRST) {
      if (role >= 0) S.p[kk % 3][hr][hc] = derive(hr, hc);
    }
  };
  // dp/dz of plane kk at the thread's halo role (planes kk-1 .. kk+1 resident)
  auto role_dz = [&](int kk) {
    if (role < 0) return;
    const float pm = kk > 0 ? Pv(kk - 1, hr, hc) : 0.f, zm = kk > 0 ? Zv(kk - 1, hr, hc) : 0.f;
    const float pn = kk + 1 < nz ? Pv(kk + 1, hr, hc) : 0.f, zn = kk + 1 < nz ? Zv(kk + 1, hr, hc) : 0.f;
    S.dz[kk & 1][hr][hc] = column_dpdz(kk, nz, pm, Pv(kk, hr, hc), pn, zm, Zv(kk, hr, hc), zn);
  };
  int off[ROWS];  // the owned cells of the current plane
#pragma unroll
  for (int r = 0; r < ROWS; ++r) off[r] = gidx(g, gi, gj + r, kb);
  // owned-cell columns of plane kk, `up` planes above the current one (zeros above the top)
  auto load_col = [&](int r, int kk, int up) {
    TerrainCol c{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (!own_rt[r] || kk >= nz) return c;
    const int o = off[r] + up * g.plane;
    c.idzc = __ldg(a.idz_c + o);
    if (kk + 1 < nz) {
      c.idzf = __ldg(a.idz_f + o + g.plane);
      c.pref = __ldg(a.col_pref + o + g.plane);
      c.rref = __ldg(a.col_rref + o + g.plane);
    }
    if (FINAL) {
      c.bu = __ldg(a.bu + o);
      c.bv = __ldg(a.bv + o);
      c.bw = __ldg(a.bw + o + g.plane);
    }
    return c;
  };
  auto rho_at = [&](int kk, int r) { return slot_of(kk)[O_RHO + (r0 + r + R0) * RW + tx + C0]; };

  if (tid == ISSUER)
    for (int kk = kg; kk < kb + AHEAD && kk <= kl; ++kk) { issue(kk); issued = kk; }
  // Carried up the thread's rows: p and z of planes k and k+1, dp/dz of plane k, rho and the
  // perturbations about the column reference at plane k, the increment of face k
  float p0[ROWS], z0[ROWS], p1[ROWS], z1[ROWS], dz0[ROWS], rc[ROWS], pa[ROWS], ra[ROWS], dwc[ROWS], bwz[ROWS];
  TerrainCol col[ROWS];
  float prk[ROWS], rrk[ROWS];  // the column reference at plane kb
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    prk[r] = rrk[r] = bwz[r] = dwc[r] = 0.f;  // face 0 never changes
    if (own_rt[r]) {
      prk[r] = __ldg(a.col_pref + off[r]);
      rrk[r] = __ldg(a.col_rref + off[r]);
      if (FINAL && kb == 0) bwz[r] = __ldg(a.bw + off[r]);
    }
    col[r] = load_col(r, kb, 0);
  }
  {
    float pm[ROWS] = {0.f, 0.f}, zm[ROWS] = {0.f, 0.f};
    if (kb > 0) {
      wait_plane(kg, kb);
      load_level(kg, pm, zm);
    }
    wait_plane(kb, kb);
    load_level(kb, p0, z0);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      rc[r] = rho_at(kb, r);
      pa[r] = fp::sub(p0[r], prk[r]);
      ra[r] = fp::sub(rc[r], rrk[r]);
      if (kb > 0 && own_rt[r]) {  // the chunk's lowest Z face, from the plane below
        const int o = off[r] - g.plane;
        const float dw = FIRST ? 0.f : slot_of(kg)[O_DW + (r0 + r) * OBW + tx];
        dwc[r] = fp::wmom_pert(dw, pa[r], fp::sub(pm[r], __ldg(a.col_pref + o)),
                               fp::sub(rho_at(kg, r), __ldg(a.col_rref + o)), ra[r], __ldg(a.idz_f + off[r]), gravity,
                               dtf);
      }
      p1[r] = z1[r] = 0.f;
    }
    if (kb + 1 <= kl) {
      wait_plane(kb + 1, kb);
      load_level(kb + 1, p1, z1);
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      dz0[r] = column_dpdz(kb, nz, pm[r], p0[r], p1[r], zm[r], z0[r], z1[r]);
      if (own_rt[r]) S.dz[kb & 1][r0 + r + 1][tx + 1] = dz0[r];
    }
    role_dz(kb);
  }
  __syncthreads();

  // Interior tiles (full, away from every periodic edge ring and open side) run a copy
  // of the plane loop compiled without the edge logic; both copies do the same arithmetic.
  const bool interior = !edge && i0 + TX <= nx && j0 + TY <= ny && (g.per_x || (i0 > 0 && i0 + TX < nx)) &&
                        (g.per_y || (j0 > 0 && j0 + TY < ny));
  auto plane_loop = [&](auto tile_class) -> bool {  // true when a bounded wait gave up
    constexpr bool IN = decltype(tile_class)::value;
    const bool su = !IN && !g.per_x && gi == 0, hs = !IN && h_skip;  // faces of open sides never change
    bool sv[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) sv[r] = !IN && !g.per_y && (gj + r == 0 || gj + r == ny);
    // store at plane k + up of the thread's row r
    auto put = [&](float* f, int o, int r, int k, int up, float v) {
      if (IN) f[off[r] + up * g.plane] = v;
      else store_tile(f, g, o, gi, gj + r, k + up, v, edge);
    };
    for (int k = kb; k < ke; ++k) {
      const int pb = k & 1;
      const float* st = slot_of(k);
      const bool up = k + 1 < nz;
      TerrainCol ncol[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) ncol[r] = load_col(r, k + 1, 1);
      // ---- dp/dz of plane k+1 (plane k+2 arrives first)
      float p2[ROWS] = {0.f, 0.f}, z2[ROWS] = {0.f, 0.f}, dz1[ROWS] = {0.f, 0.f};
      if (k + 2 <= kl) {
        wait_plane(k + 2, k);
        load_level(k + 2, p2, z2);
      }
      if (k + 1 < ke) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          dz1[r] = column_dpdz(k + 1, nz, p0[r], p1[r], p2[r], z0[r], z1[r], z2[r]);
          if (IN || own_rt[r]) S.dz[pb ^ 1][r0 + r + 1][tx + 1] = dz1[r];
        }
        role_dz(k + 1);
      }
      // ---- faces of plane k: K12/K13 horizontal momenta, K14 vertical momentum at face k+1
      float un[ROWS], vn[ROWS], wn[ROWS], rn[ROWS], pu[ROWS], ru[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int row = r0 + r + 1;
        const float du = FIRST ? 0.f : st[O_DU + (r0 + r) * FBW + tx];
        const float dv = FIRST ? 0.f : st[O_DV + (r0 + r) * FBW + tx];
        un[r] = su ? du
                   : fp::hmom_terrain(du, p0[r], Pv(k, row, tx), z0[r], Zv(k, row, tx), S.dz[pb][row][tx], dz0[r], idx,
                                      dtf);
        if (r == 0)
          vn[r] = sv[r] ? dv
                        : fp::hmom_terrain(dv, p0[r], Pv(k, row - 1, tx + 1), z0[r], Zv(k, row - 1, tx + 1),
                                           S.dz[pb][row - 1][tx + 1], dz0[r], idy, dtf);
        else
          vn[r] = sv[r] ? dv
                        : fp::hmom_terrain(dv, p0[r], p0[r > 0 ? r - 1 : 0], z0[r], z0[r > 0 ? r - 1 : 0],
                                           dz0[r > 0 ? r - 1 : 0], dz0[r], idy, dtf);
        if (IN || own_rt[r]) S.du[pb][r0 + r][tx] = un[r];
      }
      if (IN || own_rt[0]) S.dv[pb][ty][tx] = vn[0];
      if (role == 1) {  // the tile's east X face
        float d = FIRST ? 0.f : st[O_DU + (hr - 1) * FBW + w];
        if (!hs)
          d = fp::hmom_terrain(d, Pv(k, hr, hc), Pv(k, hr, hc - 1), Zv(k, hr, hc), Zv(k, hr, hc - 1),
                               S.dz[pb][hr][hc - 1], S.dz[pb][hr][hc], idx, dtf);
        S.du[pb][hr - 1][w] = d;
        // open east boundary: face nx belongs to no tile; its step value is base + increment
        if (FINAL && hs) {
          const int o = gidx(g, hi, hj, k);
          a.f_u[o] = fp::add(__ldg(a.bu + o), d);
        }
      } else if (role == 3) {  // the tile's north Y face
        float d = FIRST ? 0.f : st[O_DV + h * FBW + hc - 1];
        if (!hs)
          d = fp::hmom_terrain(d, Pv(k, hr, hc), Pv(k, hr - 1, hc), Zv(k, hr, hc), Zv(k, hr - 1, hc),
                               S.dz[pb][hr - 1][hc], S.dz[pb][hr][hc], idy, dtf);
        if (IN || h % ROWS == 0) S.dv[pb][h / ROWS][hc - 1] = d;  // else a thread's own second face
        if (FINAL && hs) {
          const int o = gidx(g, hi, hj, k);
          a.f_v[o] = fp::add(__ldg(a.bv + o), d);
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        wn[r] = rn[r] = pu[r] = ru[r] = 0.f;  // face nz never changes
        if (up) {
          const float dw = FIRST ? 0.f : st[O_DW + (r0 + r) * OBW + tx];
          rn[r] = rho_at(k + 1, r);
          pu[r] = fp::sub(p1[r], col[r].pref);
          ru[r] = fp::sub(rn[r], col[r].rref);
          wn[r] = fp::wmom_pert(dw, pu[r], pa[r], ra[r], ru[r], col[r].idzf, gravity, dtf);
        }
      }
      __syncthreads();  // publishes dz(k+1), p(k+2), du(k), dv(k); the slot of plane k-1 is free
      if (S.abort[pb]) return true;
      if (tid == ISSUER) {
        if (acc && k > kb) {  // level sums of plane k-1 (warp totals published above)
          long long sa = 0;
          for (int q = 0; q < NW; ++q) sa += S.red[pb ^ 1][q];
          acc_add(a.acc_a + k - 1, sa);
        }
        if (k + AHEAD <= kl) { issue(k + AHEAD); issued = k + AHEAD; }
      }
      // ---- K15 density of plane k, K10 rho*theta, stores
      long long sum[ROWS] = {0, 0};
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        if (!(IN || own_rt[r])) continue;
        const float ue = S.du[pb][r0 + r][tx + 1], vnorth = r + 1 < ROWS ? vn[r + 1 < ROWS ? r + 1 : r] : S.dv[pb][ty + 1][tx];
        const float rnew = fp::density(rc[r], ue, un[r], vnorth, vn[r], wn[r], dwc[r], idx, idy, col[r].idzc, dtf);
        const float rt = fp::mul(rnew, st[O_TH + (r0 + r + R0) * RW + tx + C0]);
        if (FINAL) {
          put(a.f_rho, kCell, r, k, 0, rnew);
          put(a.f_rt, kCell, r, k, 0, rt);
          put(a.f_u, kFaceX, r, k, 0, fp::add(col[r].bu, un[r]));
          put(a.f_v, kFaceY, r, k, 0, fp::add(col[r].bv, vn[r]));
          if (k == 0) put(a.f_w, kFaceZ, r, 0, 0, bwz[r]);
          put(a.f_w, kFaceZ, r, k, 1, fp::add(col[r].bw, wn[r]));
        } else {
          put(a.rho_out, kCell, r, k, 0, rnew);
          put(a.du_out, kFaceX, r, k, 0, un[r]);
          put(a.dv_out, kFaceY, r, k, 0, vn[r]);
          if (up) put(a.dw_out, kFaceZ, r, k, 1, wn[r]);
          // the next substep's pressure, loaded with its ring
          if (KIND == 0) put(a.p_out, kCell, r, k, 0, eos_pressure(rnew, rt));
        }
        if (acc) sum[r] = fx(fp::theta(rnew, rt), kFxTheta);
      }
      if (acc) {
        // row by row: in a state that has blown up a warp's total can wrap (common.cuh)
        long long t = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) t += warp_total_fx(sum[r]);
        if (tx == 0) S.red[pb][ty] = t;
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        dwc[r] = wn[r];
        rc[r] = rn[r];
        pa[r] = pu[r];
        ra[r] = ru[r];
        p0[r] = p1[r];
        z0[r] = z1[r];
        p1[r] = p2[r];
        z1[r] = z2[r];
        dz0[r] = dz1[r];
        col[r] = ncol[r];
        off[r] += g.plane;
      }
    }
    return false;
  };
  const bool aborted = interior ? plane_loop(std::true_type{}) : plane_loop(std::false_type{});
  if (aborted) {
    // drain the tiles still in flight (bounded) before the CTA's shared memory goes away
    if (tid == ISSUER)
      for (int kk = waited + 1; kk <= issued; ++kk) mbar_wait(&S.bar[(kk - kg) % NSLOT], ((kk - kg) / NSLOT) & 1);
    return;
  }
  if (acc) {
    __syncthreads();  // the last plane's warp totals
    if (tid == ISSUER) {
      const int pb = (ke - 1) & 1;
      long long sa = 0;
      for (int q = 0; q < NW; ++q) sa += S.red[pb][q];
      acc_add(a.acc_a + ke - 1, sa);
    }
  }
}

template <bool FIRST, int KIND>
cudaError_t allow_smem() {
  return cudaFuncSetAttribute(k_fast_terrain_tma<FIRST, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)fz::dyn_smem<FIRST>());
}

template <bool FIRST>
void launch(const FastArgs& a, const FastTerrainMaps& m, dim3 grid, const ZSplit& zs, cudaStream_t s) {
  const dim3 block(fz::TX, fz::NW);
  if (a.final_kind == 0) k_fast_terrain_tma<FIRST, 0><<<grid, block, fz::dyn_smem<FIRST>(), s>>>(a, m, zs);
  else if (a.final_kind == 1) k_fast_terrain_tma<FIRST, 1><<<grid, block, fz::dyn_smem<FIRST>(), s>>>(a, m, zs);
  else k_fast_terrain_tma<FIRST, 2><<<grid, block, fz::dyn_smem<FIRST>(), s>>>(a, m, zs);
}

}  // namespace

cudaError_t init_fast_terrain_tma() {
  cudaError_t e = allow_smem<true, 0>();
  if (e == cudaSuccess) e = allow_smem<true, 1>();
  if (e == cudaSuccess) e = allow_smem<true, 2>();
  if (e == cudaSuccess) e = allow_smem<false, 0>();
  if (e == cudaSuccess) e = allow_smem<false, 1>();
  if (e == cudaSuccess) e = allow_smem<false, 2>();
  return e;
}

cudaError_t launch_fast_terrain_tma(const FastArgs& a, const FastTerrainMaps& m, bool first, cudaStream_t s) {
  if (a.g.nz > kMaxNz || a.g.nz < 1 || !a.err || !a.hmom || !a.dens || !a.col_pref || !a.col_rref || !a.idz_c ||
      !a.idz_f || (a.final_kind == 0 && !a.p_out) || (a.final_kind == 2 && (!a.bu || !a.bv || !a.bw)))
    return cudaErrorInvalidValue;
  dim3 grid((a.g.nx + fz::TX - 1) / fz::TX, (a.g.ny + fz::TY - 1) / fz::TY);
  // a chunk derives up to three planes more than its own; 201 x 163 x 40 takes 50.9 us with 1.5
  // and 54.9 with 3.0, 512 x 512 x 80 351 with either
  const ZSplit zs = z_split(grid.x * grid.y, a.g.nz, 2, 1.5f);
  grid.z = zs.chunks;
  if (first) launch<true>(a, m, grid, zs, s);
  else launch<false>(a, m, grid, zs, s);
  return cudaGetLastError();
}

}  // namespace gwmb
