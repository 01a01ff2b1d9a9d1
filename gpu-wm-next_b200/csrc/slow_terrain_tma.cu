// slow_terrain_tma.cu — one fused slow RK stage on terrain on owned tiles fed by TMA.
//
// Same operator and per-cell arithmetic as k_slow_stage<true, R> (the K2/K3/K16-K19/
// K21/K22 tendencies of compute_slow_tendencies, src/dycore/dry_core.cu:400-539, with
// the terrain pressure gradient of dry_pressure_gradient.cu:37-240 and the hybrid-height
// metric columns; the update K4 and blend K5 of :189-205), with the data path of
// k_slow_tma: a CTA owns a 32 x 16 tile, two adjacent rows per thread, and one elected thread
// fetches each plane's boxes with cp.async.bulk.tensor.3d into a three-slot shared-memory
// ring two planes ahead:
//   rho, theta (or rho*theta), u, w, z (+ du, dw)   40 x 18 boxes: tile, halo ring, corners
//   v (+ dv)                                        40 x 19 (one more Y-face row)
// Plane nz carries only w (+ dw), the top faces.  Per plane the CTA derives, at all 34 x 18
// positions of the tile and its ring, theta, the cell velocities uc, vc, wc, the full
// pressure and dp/dz of the plane (a position's pressures of three planes stay in its thread's
// registers); one barrier publishes them, every thread computes its cells and faces, and a second barrier
// frees the derived planes for the next one (the terrain planes would not fit a CTA pair
// per SM double-buffered).  The owned columns' metric values (the cell and face inverse
// layer depths) and the blend partner q0 are per-thread coalesced loads at the top of the plane
// that uses them, so its derive phase covers them.
// Bounds: issue and the two barriers of a plane, as in the flat stage, whose shared and carried
// fluxes and shared reciprocals it has.  512 x 512 x 80: 0.68 ms a stage against 1.00 with
// separate rows, 201 x 163 x 40: 82 us against 119 (27 fields of 4 B per cell at the copy
// bandwidth: 0.35 ms and 22 us).
#include <type_traits>

#include "dycore.cuh"
#include "stencil.cuh"
#include "tma.cuh"
#include "zsplit.cuh"

namespace gwmb {
namespace {

namespace st {
constexpr int TX = 32, TY = 16, ROWS = 2, NT = 256, NW = NT / 32;  // two adjacent rows per thread
// the thread that issues the TMA loads and folds the level sums: lane 0 of the last warp
constexpr int ISSUER = NT - 32;
constexpr int BW = 40, BH = 18, BHV = 19;  // boxes: cells, X and Z faces / Y faces
constexpr int DW = TX + 2, DH = TY + 2, DN = DW * DH;  // derived plane: 34 x 18
// raw slot (floats; sub-buffers on 128-byte boundaries)
constexpr int R_RHO = 0, R_TH = 736, R_U = 1472, R_W = 2208, R_V = 2944, R_Z = 3712, R_DU = 4448, R_DW = 5184,
              R_DV = 5920, SLOT = 6688, SLOT_SHORT = 4448, NSLOT = 3;
constexpr unsigned B_BOX = BW * BH * 4, B_BOXV = BW * BHV * 4;
// derived arrays (floats): uc, vc [2][DN] (planes k-1, k); theta [2][DN] (planes k, k+1); wc, dp/dz,
// p [DN]
constexpr int D_UC = 0, D_VC = 2 * DN, D_TH = 4 * DN, D_WC = 6 * DN, D_DZ = 7 * DN, D_P = 8 * DN, DERIVED = 9 * DN;
static_assert(R_TH % 32 == 0 && R_U % 32 == 0 && R_W % 32 == 0 && R_V % 32 == 0 && R_Z % 32 == 0 &&
                  R_DU % 32 == 0 && R_DW % 32 == 0 && R_DV % 32 == 0 && SLOT % 32 == 0 && SLOT_SHORT == R_DU,
              "128-byte aligned sub-buffers");
static_assert(R_TH - R_RHO >= BW * BH && R_U - R_TH >= BW * BH && R_W - R_U >= BW * BH &&
                  R_V - R_W >= BW * BH && R_Z - R_V >= BW * BHV && R_DU - R_Z >= BW * BH &&
                  R_DW - R_DU >= BW * BH && R_DV - R_DW >= BW * BH && SLOT - R_DV >= BW * BHV,
              "boxes fit their sub-buffers");
constexpr size_t smem_bytes(bool inc) {
  return size_t((inc ? SLOT : SLOT_SHORT) * NSLOT + DERIVED) * sizeof(float) + 128;
}
}  // namespace st

// Blend partner q0 at an owned position of one plane.
struct SlowBlend {
  float rho, rt, u, v, w;
};

// Metric values of one owned column at one plane: inverse layer depth of the cell, of its
// west and south neighbours (the X and Y faces average two cells) and of the Z face.
struct TerrMetric {
  float c, w, s, f;
};

// FIRST: a step's first stage (rho*theta in, no blend); INC: acoustic increments are added to
// the momenta (stages 2 and 3 behind the fast modes).
template <bool FIRST, bool INC, bool DAMP>  // DAMP: with the Rayleigh layer
__global__ void __launch_bounds__(st::NT, 2)
    k_slow_terrain_tma(const SlowArgs a, const __grid_constant__ SlowMaps m, ZSplit zs) {
  using namespace st;
  constexpr bool BLEND = !FIRST;
  extern __shared__ unsigned char s_dyn[];
  __shared__ float s_trf[kMaxNz], s_ytrf[kMaxNz];   // theta_ref at Z face k, reciprocal of its floored value
  __shared__ long long s_red[2][NW];
  __shared__ __align__(8) uint64_t s_bar[NSLOT];
  __shared__ int s_abort[2];
  constexpr int slot = INC ? SLOT : SLOT_SHORT;
  float* const ring = reinterpret_cast<float*>(align_smem_128(s_dyn));
  float* const der = ring + NSLOT * slot;

  const Geom& g = a.g;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int w = min(TX, nx - i0), h = min(TY, ny - j0);
  const int r0 = ty * ROWS, gi = i0 + tx, gj = j0 + r0;  // the thread's column and first row
  const bool open_x = !g.per_x, open_y = !g.per_y;
  const bool edge = (g.per_x && (i0 <= 1 || i0 + w >= nx - 1)) || (g.per_y && (j0 <= 1 || j0 + h >= ny - 1));
  const float idx = g.inv_dx, idy = g.inv_dy, dt = a.dt;
  // open boundaries: X face nx and Y face ny belong to the last tiles; their tendency
  // is zero (dry_momentum_flux.cu:79-235 skips them), so they are blends of the stage
  // value.  Under periodic wrap they are the mirrors of faces 0 written by store_tile.
  const bool xf = open_x && i0 + w == nx && ty == 0 && tx < h;  // X face nx, row j0+tx
  const bool yf = open_y && j0 + h == ny && ty == 1 && tx < w;  // Y face ny, column i0+tx
  // the CTA's planes are kb .. ke-1; it also loads plane ke and (above the ground) the plane
  // below, kb-1, whose derived values its lowest faces read
  const int kb = zs.first(blockIdx.z), ke = zs.last(blockIdx.z, nz), kg = kb > 0 ? kb - 1 : 0;

  if (tid == 0) {
    for (int s = 0; s < NSLOT; ++s) mbar_init(&s_bar[s], 1);
    mbar_fence_init();
    s_abort[0] = 0;
    s_abort[1] = 0;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && a.clr_a)
    for (int q = tid; q < nz; q += NT) { a.clr_a[q] = 0ull; a.clr_b[q] = 0ull; }
  for (int q = kg + tid; q < ke; q += NT) {
    const float tu = (float)(acc_read(a.th_acc + q, kScaleTheta) * a.inv_count);
    const float tl = q > 0 ? (float)(acc_read(a.th_acc + q - 1, kScaleTheta) * a.inv_count) : tu;
    const float trf = fp::avg(tl, tu);
    s_trf[q] = trf;
    s_ytrf[q] = fp::recip(fmaxf(trf, 1.0e-6f));
  }
  __syncthreads();

  int stall = tid == ISSUER ? take_stall(a.err, kStallSlow) : -1;  // failure-path tests
  if (stall >= 0) stall = kg + stall % (ke - kg + 1);
  auto slot_at = [&](int kk) { return ring + ((kk - kg) % NSLOT) * slot; };
  auto issue = [&](int kk) {  // plane kk in [kg, ke] into its slot
    float* sr = slot_at(kk);
    uint64_t* bar = &s_bar[(kk - kg) % NSLOT];
    const bool cells = kk < nz;
    unsigned bytes = (INC ? 2u : 1u) * B_BOX;
    if (cells) bytes += 4 * B_BOX + B_BOXV + (INC ? B_BOX + B_BOXV : 0u);
    const int x = i0 + kXOff - 4, y = j0;
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(bar, bytes);
    if (kk == stall) return;  // failure-path testing: this plane's loads stay unissued
    tma_load_3d(sr + R_W, &m.w, x, y, kk, bar);
    if (INC) tma_load_3d(sr + R_DW, &m.dw, x, y, kk, bar);
    if (cells) {
      tma_load_3d(sr + R_RHO, &m.rho, x, y, kk, bar);
      tma_load_3d(sr + R_TH, &m.th, x, y, kk, bar);
      tma_load_3d(sr + R_U, &m.u, x, y, kk, bar);
      tma_load_3d(sr + R_V, &m.v, x, y, kk, bar);
      tma_load_3d(sr + R_Z, &m.z, x, y, kk, bar);
      if (INC) {
        tma_load_3d(sr + R_DU, &m.du, x, y, kk, bar);
        tma_load_3d(sr + R_DV, &m.dv, x, y, kk, bar);
      }
    }
  };
  int issued = kg - 1, waited = kg - 1;
  auto wait_plane = [&](int kk, int epoch) {
    if (!mbar_wait(&s_bar[(kk - kg) % NSLOT], ((kk - kg) / NSLOT) & 1)) {
      s_abort[epoch & 1] = 1;
      atomicExch(a.err, 1);
    } else if (waited == kk - 1) {
      waited = kk;  // a plane whose wait gave up stays in the drain below, with those after it
    }
  };
  // raw accessors: box index of derived position (r, c) is r * BW + c + 3
  auto U = [&](const float* sr, int b) { return INC ? fp::add(sr[R_U + b], sr[R_DU + b]) : sr[R_U + b]; };
  auto V = [&](const float* sr, int b) { return INC ? fp::add(sr[R_V + b], sr[R_DV + b]) : sr[R_V + b]; };
  auto W = [&](const float* sr, int b) { return INC ? fp::add(sr[R_W + b], sr[R_DW + b]) : sr[R_W + b]; };
  auto RT = [&](const float* sr, int b, float rho) {
    const float t = sr[R_TH + b];
    return FIRST ? t : fp::mul(rho, t);
  };

  int off[ROWS];  // the owned cells of the current plane
  bool own_rt[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    off[r] = gidx(g, gi, gj + r, kb);
    own_rt[r] = tx < w && r0 + r < h;
  }
  // blend partner at the current plane of the thread's row r
  auto load_q0 = [&](auto tile_class, int r) {
    constexpr bool IN = decltype(tile_class)::value;
    SlowBlend q{0.f, 0.f, 0.f, 0.f, 0.f};
    if (!BLEND || !(IN || own_rt[r])) return q;
    const int o = off[r];
    q.rho = __ldg(a.rho0 + o);
    q.rt = __ldg(a.rt0 + o);
    q.u = __ldg(a.u0 + o);
    q.v = __ldg(a.v0 + o);
    q.w = __ldg(a.w0 + o);
    return q;
  };

  if (tid == ISSUER)
    for (int kk = kg; kk <= kb + 1; ++kk) { issue(kk); issued = kk; }
  // metric values at the current plane of the thread's rows
  auto load_metric = [&](TerrMetric* t) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      t[r] = TerrMetric{0.f, 0.f, 0.f, 0.f};
      if (!own_rt[r]) continue;
      const int o = off[r];
      t[r].c = __ldg(a.idz_c + o);
      t[r].w = __ldg(a.idz_c + o - 1);
      t[r].s = r > 0 ? t[r > 0 ? r - 1 : 0].c : __ldg(a.idz_c + o - g.pitch);
      t[r].f = __ldg(a.idz_f + o);
    }
  };

  // ---- derived planes: the thread's positions of the 34 x 18 (a third one in the first
  // warps), their box indices and the reciprocal of their floored density
  constexpr int NP = (DN + NT - 1) / NT, FULL = DN / NT;  // FULL: positions every thread has
  int pos_b[NP];
  float yrho[NP], p_m[NP], p_c[NP];  // the reciprocal at plane k; the pressure at planes k-1 and k
  // positions whose theta (bit n) and whose p, dp/dz and velocities (bit 8 + n) are read: not
  // those of a partial tile's missing rows and columns, and beyond an open side only theta
  unsigned live = 0;
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const int q = tid + n * NT, r = q / DW, c = q - r * DW;
    pos_b[n] = r * BW + c + 3;
    if (q < DN && r <= h + 1 && c <= w + 1) {
      const int pi = i0 + c - 1, pj = j0 + r - 1;
      live |= 1u << n;
      if ((g.per_x || (pi >= 0 && pi < nx)) && (g.per_y || (pj >= 0 && pj < ny))) live |= 256u << n;
    }
  }
  // K20 (dry_pressure_gradient.cu:27-35): eos_pressure with theta at hand
  auto pressure = [&](float rho, float th, bool& near) {
    const float x = fp::div_by(rho * kRd * th, kP0, 1.0f / kP0);
    near = near && fp::finite(x);
    return kP0 * powf(fmaxf(x, 1.0e-6f), 1.0f / (1.0f - kKappa));
  };
  // theta and pressure of plane kk (kk < nz), and the reciprocals that derive(kk) divides by:
  // the pressure becomes p_c, the one before it p_m
  auto derive_theta = [&](auto tile_class, int kk) {
    constexpr bool IN = decltype(tile_class)::value;
    const float* sr = slot_at(kk);
    float* th = der + D_TH + (kk & 1) * DN;
    bool near = true;
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      p_m[n] = p_c[n];
      if ((IN && n < FULL) || live & (1u << n)) {
        const float rho = sr[R_RHO + pos_b[n]], rt = RT(sr, pos_b[n], rho), rr = fmaxf(rho, 1.0e-6f);
        yrho[n] = fp::recip(rr);
        const float t = fp::div_by(rt, rr, yrho[n]);
        near = near && fp::finite(t);
        th[tid + n * NT] = t;
        if ((IN && n < FULL) || live & (256u << n)) p_c[n] = pressure(rho, t, near);
      }
    }
    if (!near) {  // a value that is not finite: each one tested
#pragma unroll
      for (int n = 0; n < NP; ++n)
        if (live & (1u << n)) {
          const float rho = sr[R_RHO + pos_b[n]], rt = RT(sr, pos_b[n], rho);
          th[tid + n * NT] = fp::quotient_far(rt, fmaxf(rho, 1.0e-6f));
          if (live & (256u << n)) p_c[n] = eos_pressure(rho, rt);
        }
    }
  };
  // uc, vc, wc, p and dp/dz of plane k, with derive_theta(k) done; does derive_theta(k + 1).  grad:
  // p and dp/dz are wanted (not for the plane below a chunk)
  auto derive = [&](auto tile_class, int k, bool grad) {
    constexpr bool IN = decltype(tile_class)::value;
    const float* sm = slot_at(k > kg ? k - 1 : kg);  // plane k-1 (its slot is intact)
    const float* sr = slot_at(k);
    const float* sn = slot_at(k + 1);
    float* uc = der + D_UC + (k & 1) * DN;
    float* vc = der + D_VC + (k & 1) * DN;
    float* wc = der + D_WC;
    float* pp = der + D_P;
    float* dz = der + D_DZ;
    bool near = true;
    auto momenta = [&](int b, float& mu, float& mv, float& mw) {
      mu = fp::avg(U(sr, b), U(sr, b + 1));
      mv = fp::avg(V(sr, b), V(sr, b + BW));
      mw = fp::avg(W(sr, b), W(sn, b));
    };
#pragma unroll
    for (int n = 0; n < NP; ++n)
      if ((IN && n < FULL) || live & (256u << n)) {
        const int b = pos_b[n], q = tid + n * NT;
        // cell-centred velocities: dry_momentum_flux.cu:36-73
        const float rr = fmaxf(sr[R_RHO + b], 1.0e-6f), y = yrho[n];
        float mu, mv, mw;
        momenta(b, mu, mv, mw);
        const float cu = fp::div_by(mu, rr, y), cv = fp::div_by(mv, rr, y), cw = fp::div_by(mw, rr, y);
        near = near && fp::finite(fabsf(cu) + fabsf(cv) + fabsf(cw));
        uc[q] = cu;
        vc[q] = cv;
        wc[q] = cw;
      }
    if (!near) {  // a quotient that is not finite: each one tested
#pragma unroll 1
      for (int n = 0; n < NP; ++n) {
        if (!(live & (256u << n))) continue;
        const int q = tid + n * NT, r = q / DW, b = r * BW + (q - r * DW) + 3;
        const float rr = fmaxf(sr[R_RHO + b], 1.0e-6f);
        float mu, mv, mw;
        momenta(b, mu, mv, mw);
        uc[q] = fp::quotient_far(mu, rr);
        vc[q] = fp::quotient_far(mv, rr);
        wc[q] = fp::quotient_far(mw, rr);
      }
    }
    float below[NP];  // the pressure at plane k-1
#pragma unroll
    for (int n = 0; n < NP; ++n) below[n] = p_m[n];
    if (k + 1 < nz) {  // p_m, p_c become the pressures at planes k and k+1
      derive_theta(tile_class, k + 1);
    } else {
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        p_m[n] = p_c[n];
        p_c[n] = 0.f;
      }
    }
    if (!grad) return;
#pragma unroll
    for (int n = 0; n < NP; ++n)
      if ((IN && n < FULL) || live & (256u << n)) {
        const int b = pos_b[n], q = tid + n * NT;
        pp[q] = p_m[n];
        dz[q] = column_dpdz(k, nz, below[n], p_m[n], p_c[n], k > 0 ? sm[R_Z + b] : 0.f, sr[R_Z + b],
                            k + 1 < nz ? sn[R_Z + b] : 0.f);
      }
  };

  // Values of the thread's columns carried up: the stage input at plane k, theta and rho of
  // plane k-1, and the vertical fluxes through the faces between planes k-1 and k (the flux
  // out of a plane's top is the one into the next plane's bottom)
  float rho_c[ROWS], u_c[ROWS], v_c[ROWS], w_c[ROWS], th_l[ROWS], rho_l[ROWS];
  float fz_th[ROWS], fz_u[ROWS], fz_v[ROWS], fz_w[ROWS];
  const int d0 = (r0 + 1) * DW + tx + 1, b0 = (r0 + 1) * BW + tx + 4;  // derived and box index of row 0
  auto load_column = [&](int kk) {
    const float* sr = slot_at(kk);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      rho_c[r] = sr[R_RHO + b0 + r * BW];
      u_c[r] = U(sr, b0 + r * BW);
      v_c[r] = V(sr, b0 + r * BW);
      w_c[r] = W(sr, b0 + r * BW);
    }
  };
#pragma unroll
  for (int n = 0; n < NP; ++n) p_c[n] = 0.f;
  wait_plane(kg, kb);
  derive_theta(std::false_type{}, kg);
  load_column(kg);
  if (kb > 0) {  // the plane below the chunk: its derived values and the fluxes out of its top
    wait_plane(kb, kb);
    derive(std::false_type{}, kg, false);
    __syncthreads();
    const float* wc = der + D_WC;
    const float* tl = der + D_TH + (kg & 1) * DN;
    const float* tu = der + D_TH + (kb & 1) * DN;
    float u[ROWS], v[ROWS], ww[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      u[r] = u_c[r];
      v[r] = v_c[r];
      ww[r] = w_c[r];
      rho_l[r] = rho_c[r];
    }
    load_column(kb);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int d = d0 + r * DW;
      th_l[r] = tl[d];
      fz_th[r] = fp::upwind(w_c[r], tl[d], tu[d]);
      fz_u[r] = fp::upwind(fp::avg(wc[d - 1], wc[d]), u[r], u_c[r]);
      fz_v[r] = fp::upwind(fp::avg(wc[d - DW], wc[d]), v[r], v_c[r]);
      fz_w[r] = fp::upwind(wc[d], ww[r], w_c[r]);
    }
    __syncthreads();  // wc is derived anew for plane kb
  } else {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) th_l[r] = rho_l[r] = fz_th[r] = fz_u[r] = fz_v[r] = fz_w[r] = 0.f;
  }

  // damping constants of the plane
  struct PlaneConst {
    float damp_c, damp_f, uref, vref;
  };
  auto plane_const = [&](int k) {
    PlaneConst pc{0.0f, 0.0f, 0.0f, 0.0f};
    if (DAMP) {
      pc.damp_c = __ldg(a.damp_c + k);
      pc.damp_f = __ldg(a.damp_f + k);
      pc.uref = __ldg(a.uref + k);
      pc.vref = __ldg(a.vref + k);
    }
    return pc;
  };

  // cells, X faces, Y faces and Z faces of plane k in the thread's rows (+ the top faces)
  auto columns = [&](auto tile_class, int k, const SlowBlend* q0, const TerrMetric* mt, long long* ra,
                     const PlaneConst& kc) {
    constexpr bool IN = decltype(tile_class)::value;  // an interior tile
    // store of an owned value at plane k + up: a plain store in interior tiles, else with the
    // periodic mirrors
    auto put = [&](float* f, int o, int r, int up, float v) {
      if (IN) f[off[r] + up * g.plane] = v;
      else if (own_rt[r]) store_tile(f, g, o, gi, gj + r, k + up, v, edge);
    };
    const float* sr = slot_at(k);
    const float* sn = slot_at(k + 1);
    const float* uc = der + D_UC + (k & 1) * DN;
    const float* vc = der + D_VC + (k & 1) * DN;
    const float* wc = der + D_WC;
    const float* ucm = der + D_UC + ((k + 1) & 1) * DN;  // plane k-1
    const float* vcm = der + D_VC + ((k + 1) & 1) * DN;
    const float* th = der + D_TH + (k & 1) * DN;
    const float* thn = der + D_TH + ((k + 1) & 1) * DN;  // plane k+1
    const float* pp = der + D_P;
    const float* dz = der + D_DZ;
    const bool top = k + 1 == nz;
    const bool sx0 = !IN && gi == 0 && open_x, sx1 = !IN && gi + 1 == nx && open_x;  // no flux through the side
    bool sy[ROWS + 1];  // the Y face below row r lies on an open side
#pragma unroll
    for (int r = 0; r <= ROWS; ++r) sy[r] = !IN && open_y && (gj + r == 0 || gj + r == ny);
    // column values of plane k+1 (plane nz holds the top faces only)
    float rho_n[ROWS], u_n[ROWS], v_n[ROWS], w_n[ROWS], tc[ROWS + 2], tt[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS + 2; ++r) tc[r] = th[d0 + (r - 1) * DW];  // rows -1 .. ROWS
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int b = b0 + r * BW;
      w_n[r] = W(sn, b);
      rho_n[r] = sn[R_RHO + b];  // the top plane reads none of these
      u_n[r] = U(sn, b);
      v_n[r] = V(sn, b);
      tt[r] = top ? tc[r + 1] : thn[d0 + r * DW];
    }
    const float u_s = U(sr, b0 - BW), u_t = U(sr, b0 + ROWS * BW);  // rows -1 and ROWS
    const float v_s = V(sr, b0 - BW), v_t = V(sr, b0 + ROWS * BW);
    // the wind in the rows -1 .. ROWS-1: at the column and (vc) averaged onto its X face, (uc)
    // its two cells
    float uw[ROWS + 1], ue[ROWS + 1], vx[ROWS + 1], vv[ROWS + 1];
#pragma unroll
    for (int r = 0; r <= ROWS; ++r) {
      const int d = d0 + (r - 1) * DW;
      uw[r] = uc[d - 1];
      ue[r] = uc[d];
      vv[r] = vc[d];
      vx[r] = fp::avg(vc[d - 1], vv[r]);
    }
    // ---- cells: K2 compute_cell_tendencies_kernel (dry_core.cu:62-144)
    {
      float gy[ROWS + 1];
#pragma unroll
      for (int r = 0; r <= ROWS; ++r) gy[r] = fp::upwind(r < ROWS ? v_c[r] : v_t, tc[r], tc[r + 1]);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int d = d0 + r * DW, b = b0 + r * BW;
        const float fw = u_c[r], fe = U(sr, b + 1), fs = v_c[r], fn = r + 1 < ROWS ? v_c[r + 1] : v_t;
        const float fb = w_c[r], ft = w_n[r], rho = rho_c[r], rt = RT(sr, b, rho);
        const float t_rho = -fp::divergence(fe, fw, fn, fs, ft, fb, idx, idy, mt[r].c);
        const float gw = fp::upwind(fw, th[d - 1], tc[r + 1]), ge = fp::upwind(fe, tc[r + 1], th[d + 1]);
        const float gb = k > 0 ? fz_th[r] : fp::upwind(fb, tc[r + 1], tc[r + 1]);
        const float gt = fp::upwind(ft, tc[r + 1], tt[r]);
        fz_th[r] = gt;
        const float t_rt = -fp::divergence(ge, gw, gy[r + 1], gy[r], gt, gb, idx, idy, mt[r].c);
        float r1 = fp::update(rho, dt, t_rho, 1.0e-6f);
        float q1 = fp::update(rt, dt, t_rt, 1.0e-6f);
        if (BLEND) {
          r1 = fp::blend(a.wa, q0[r].rho, a.wb, r1);
          q1 = fp::blend(a.wa, q0[r].rt, a.wb, q1);
        }
        const float th1 = fp::theta(r1, q1);
        put(a.o_rho, kCell, r, 0, r1);
        put(a.o_th, kCell, r, 0, a.out_rt ? q1 : th1);
        if (a.acc_mode == 2 && (IN || own_rt[r])) ra[r] = fx(th1, kFxTheta);
      }
    }
    // ---- X faces: K17 (dry_momentum_flux.cu:79-156) + K21 (dry_pressure_gradient.cu:75-123)
    {
      float fy[ROWS + 1];
#pragma unroll
      for (int r = 0; r <= ROWS; ++r) {
        fy[r] = fp::upwind(vx[r], r > 0 ? u_c[r - 1] : u_s, r < ROWS ? u_c[r] : u_t);
        if (sy[r]) fy[r] = 0.0f;
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int d = d0 + r * DW, b = b0 + r * BW;
        const float qc = u_c[r];
        const float flw = fp::upwind(uw[r + 1], U(sr, b - 1), qc), fle = fp::upwind(ue[r + 1], qc, U(sr, b + 1));
        const float flt = top ? 0.0f : fp::upwind(fp::avg(wc[d - 1], wc[d]), qc, u_n[r]);
        float t_u = -fp::divergence(fle, flw, fy[r + 1], fy[r], flt, fz_u[r], idx, idy,
                                    fp::avg(mt[r].w, mt[r].c));
        fz_u[r] = flt;
        t_u = fp::add_pgf_terrain(t_u, pp[d], pp[d - 1], sr[R_Z + b], sr[R_Z + b - 1], dz[d - 1], dz[d], idx);
        if (DAMP) t_u = fp::add_damping(t_u, kc.damp_c, qc, kc.uref);
        if (sx0) t_u = 0.0f;
        float u1 = fp::update(qc, dt, t_u, -1.0e30f);
        if (BLEND) u1 = fp::blend(a.wa, q0[r].u, a.wb, u1);
        put(a.o_u, kFaceX, r, 0, u1);
      }
    }
    // ---- Y faces: K18 (dry_momentum_flux.cu:158-235) + K22 (dry_pressure_gradient.cu:125-173)
    {
      float fy[ROWS + 1];
#pragma unroll
      for (int r = 0; r <= ROWS; ++r)
        fy[r] = fp::upwind(vv[r], r > 0 ? v_c[r - 1] : v_s, r < ROWS ? v_c[r] : v_t);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int d = d0 + r * DW, b = b0 + r * BW;
        const float qc = v_c[r];
        float flw = fp::upwind(fp::avg(uw[r], uw[r + 1]), V(sr, b - 1), qc);
        float fle = fp::upwind(fp::avg(ue[r], ue[r + 1]), qc, V(sr, b + 1));
        if (sx0) flw = 0.0f;
        if (sx1) fle = 0.0f;
        const float flt = top ? 0.0f : fp::upwind(fp::avg(wc[d - DW], wc[d]), qc, v_n[r]);
        float t_v = -fp::divergence(fle, flw, fy[r + 1], fy[r], flt, fz_v[r], idx, idy,
                                    fp::avg(mt[r].s, mt[r].c));
        fz_v[r] = flt;
        t_v = fp::add_pgf_terrain(t_v, pp[d], pp[d - DW], sr[R_Z + b], sr[R_Z + b - BW], dz[d - DW], dz[d], idy);
        if (DAMP) t_v = fp::add_damping(t_v, kc.damp_c, qc, kc.vref);
        if (!IN && gj + r == 0 && open_y) t_v = 0.0f;
        float v1 = fp::update(qc, dt, t_v, -1.0e30f);
        if (BLEND) v1 = fp::blend(a.wa, q0[r].v, a.wb, v1);
        put(a.o_v, kFaceY, r, 0, v1);
      }
    }
    // ---- Z faces k: K19 (dry_momentum_flux.cu:237-312) + K3 buoyancy (dry_core.cu:146-187)
    {
      float fy[ROWS + 1];
      if (k > 0) {
        const float w_s = W(sr, b0 - BW), w_t = W(sr, b0 + ROWS * BW);
#pragma unroll
        for (int r = 0; r <= ROWS; ++r) {
          fy[r] = fp::upwind(fp::avg(vcm[d0 + (r - 1) * DW], vv[r]), r > 0 ? w_c[r - 1] : w_s, r < ROWS ? w_c[r] : w_t);
          if (sy[r]) fy[r] = 0.0f;
        }
      }
      float flt[ROWS], t_w[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        flt[r] = fp::upwind(wc[d0 + r * DW], w_c[r], w_n[r]);
        t_w[r] = 0.0f;
      }
      if (k > 0) {
        float flux[ROWS];
        bool near = true;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const int d = d0 + r * DW, b = b0 + r * BW;
          const float qc = w_c[r];
          float flw = fp::upwind(fp::avg(ucm[d - 1], uw[r + 1]), W(sr, b - 1), qc);
          float fle = fp::upwind(fp::avg(ucm[d], ue[r + 1]), qc, W(sr, b + 1));
          if (sx0) flw = 0.0f;
          if (sx1) fle = 0.0f;
          flux[r] = -fp::divergence(fle, flw, fy[r + 1], fy[r], flt[r], fz_w[r], idx, idy, mt[r].f);
          t_w[r] = fp::add_buoyancy_ref(flux[r], th_l[r], tc[r + 1], s_trf[k], s_ytrf[k], rho_l[r], rho_c[r],
                                        a.gravity, near);
        }
        if (!near) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r)
            t_w[r] = fp::add_buoyancy(flux[r], th_l[r], tc[r + 1], s_trf[k], rho_l[r], rho_c[r], a.gravity);
        }
        if (DAMP) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) t_w[r] = fp::add_damping(t_w[r], kc.damp_f, w_c[r], 0.0f);
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float qc = w_c[r];
        fz_w[r] = flt[r];
        float w1 = fp::update(qc, dt, t_w[r], -1.0e30f);
        if (BLEND) w1 = fp::blend(a.wa, q0[r].w, a.wb, w1);
        put(a.o_w, kFaceZ, r, 0, w1);
        if (top) {  // top face: zero tendency
          float wt = fmaxf(-1.0e30f, w_n[r]);
          if (BLEND && own_rt[r]) wt = fp::blend(a.wa, __ldg(a.w0 + off[r] + g.plane), a.wb, wt);
          put(a.o_w, kFaceZ, r, 1, wt);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      th_l[r] = tc[r + 1];
      rho_l[r] = rho_c[r];
      rho_c[r] = rho_n[r];
      u_c[r] = u_n[r];
      v_c[r] = v_n[r];
      w_c[r] = w_n[r];
    }
  };

  // Interior tiles (full, away from every periodic edge ring and open side) run a copy
  // of the plane loop compiled without the edge logic: plain stores, none of the
  // open-boundary flux tests.  Both copies do the same arithmetic on the same values.
  const bool interior = !edge && i0 + TX <= nx && j0 + TY <= ny && (g.per_x || (i0 > 0 && i0 + TX < nx)) &&
                        (g.per_y || (j0 > 0 && j0 + TY < ny));
  auto plane_loop = [&](auto tile_class) -> bool {  // true when a bounded wait gave up
    constexpr bool IN = decltype(tile_class)::value;
    for (int k = kb; k < ke; ++k) {
      const int pb = k & 1;
      const PlaneConst kc = plane_const(k);
      SlowBlend q0[ROWS];  // the derive phase covers the loads
#pragma unroll
      for (int r = 0; r < ROWS; ++r) q0[r] = load_q0(tile_class, r);
      TerrMetric mt[ROWS];
      load_metric(mt);
      wait_plane(k + 1, k);
      derive(tile_class, k, true);
      __syncthreads();  // publishes plane k's derived values; slot (k-1) is free
      if (s_abort[pb]) return true;
      if (tid == ISSUER) {
        if (a.acc_mode && k > kb) {
          long long sa = 0;
          for (int q = 0; q < NW; ++q) sa += s_red[pb ^ 1][q];
          acc_add(a.acc_a + k - 1, sa);
        }
        if (k + 2 <= ke) { issue(k + 2); issued = k + 2; }
      }
      // ---- cells and faces of plane k
      long long ra[ROWS] = {0, 0};
      columns(tile_class, k, q0, mt, ra, kc);
      if (!IN && xf) {  // open east boundary: X face nx of row j0+tx
        const float* sr = slot_at(k);
        const float uf = U(sr, (tx + 1) * BW + w + 4);
        float u1 = fp::update(uf, dt, 0.0f, -1.0e30f);
        if (BLEND) u1 = fp::blend(a.wa, __ldg(a.u0 + gidx(g, nx, j0 + tx, k)), a.wb, u1);
        store_tile(a.o_u, g, kFaceX, nx, j0 + tx, k, u1, edge);
      }
      if (!IN && yf) {  // open north boundary: Y face ny of column i0+tx
        const float* sr = slot_at(k);
        const float vf = V(sr, (h + 1) * BW + tx + 4);
        float v1 = fp::update(vf, dt, 0.0f, -1.0e30f);
        if (BLEND) v1 = fp::blend(a.wa, __ldg(a.v0 + gidx(g, i0 + tx, ny, k)), a.wb, v1);
        store_tile(a.o_v, g, kFaceY, i0 + tx, ny, k, v1, edge);
      }
      if (a.acc_mode) {
        // row by row: in a state that has blown up a warp's total can wrap (common.cuh)
        const long long ta = warp_total_fx(ra[0]) + warp_total_fx(ra[1]);
        if (tx == 0) s_red[pb][ty] = ta;
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) off[r] += g.plane;
      __syncthreads();  // every thread is done with plane k's derived values
    }
    return false;
  };
  const bool aborted = interior ? plane_loop(std::true_type{}) : plane_loop(std::false_type{});
  if (aborted) {
    if (tid == ISSUER)
      for (int kk = waited + 1; kk <= issued; ++kk) mbar_wait(&s_bar[(kk - kg) % NSLOT], ((kk - kg) / NSLOT) & 1);
    return;
  }
  if (a.acc_mode && tid == ISSUER) {  // the last plane's warp totals (published by the loop's last barrier)
    const int pb = (ke - 1) & 1;
    long long sa = 0;
    for (int q = 0; q < NW; ++q) sa += s_red[pb][q];
    acc_add(a.acc_a + ke - 1, sa);
  }
}

template <bool FIRST, bool INC>
cudaError_t allow_smem() {
  cudaError_t e = cudaFuncSetAttribute(k_slow_terrain_tma<FIRST, INC, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)st::smem_bytes(INC));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_slow_terrain_tma<FIRST, INC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)st::smem_bytes(INC));
  return e;
}

template <bool FIRST, bool INC>
void launch(const SlowArgs& a, const SlowMaps& m, dim3 grid, const ZSplit& zs, cudaStream_t s) {
  const dim3 block(st::TX, st::NW);
  const size_t smem = st::smem_bytes(INC);
  if (a.damp_c) k_slow_terrain_tma<FIRST, INC, true><<<grid, block, smem, s>>>(a, m, zs);
  else k_slow_terrain_tma<FIRST, INC, false><<<grid, block, smem, s>>>(a, m, zs);
}

}  // namespace

cudaError_t init_slow_terrain_tma() {
  cudaError_t e = allow_smem<true, false>();
  if (e == cudaSuccess) e = allow_smem<false, false>();
  if (e == cudaSuccess) e = allow_smem<false, true>();
  return e;
}

cudaError_t launch_slow_terrain_tma(const SlowArgs& a, const SlowMaps& m, cudaStream_t s) {
  // a step's first stage takes rho*theta and no blend, the others theta and q0
  const bool first = a.th_is_rt != 0;
  if (a.g.nz > kMaxNz || a.g.nz < 1 || !a.err || a.tend_only || a.acc_mode == 1 || !a.idz_c || !a.idz_f ||
      first != !a.rho0 || (first && a.du))
    return cudaErrorInvalidValue;
  dim3 grid((a.g.nx + st::TX - 1) / st::TX, (a.g.ny + st::TY - 1) / st::TY);
  const ZSplit zs = z_split(grid.x * grid.y, a.g.nz, 2, 1.2f);
  grid.z = zs.chunks;
  if (first) launch<true, false>(a, m, grid, zs, s);
  else if (a.du) launch<false, true>(a, m, grid, zs, s);
  else launch<false, false>(a, m, grid, zs, s);
  return cudaGetLastError();
}

}  // namespace gwmb
