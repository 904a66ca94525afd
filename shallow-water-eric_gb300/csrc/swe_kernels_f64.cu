// FP64 stage kernels in the reference's evaluation order.
//
// One thread owns one mesh row and walks its entries in the reference CSR
// order, so every sum is formed in the same order as the Fortran loops.  This
// translation unit is compiled with -fmad=false (no FMA contraction) and uses
// IEEE sqrt/div: the result equals the FP64 CPU restatement bit for bit (the
// Manning friction's x**(4/3) aside).  It is the parity path and the "plain FP64
// GPU step" of the measurements.
//
// Per stage (SOURCES/update.f90 euler, :134-289, 'fct' + 'type2'):
//   k_node   : one_over_h, velocity, entropy E, alpha_i       (flux, alpha_limit)
//   k_low    : d_ij, mu_ij (alpha-limited), low-order state,   (compute_dij, compute_muij,
//              entropy residual res_i                           smb_2_roundoff, smb_2, maxmin)
//   k_fct    : f_ij, R^-_i                                      (compute_fct_matrix, FCT_positivity)
//   k_update : limited antidiffusion, RK combination, Dirichlet (apply_viscosity, main.f90:77-90)
// Per step: k_dt (COMPUTE_DT) and the time bookkeeping kernels.
#include "swe_kernels.hpp"

namespace swe {

struct NodeF64 {        // per-row arrays of the FP64 path
  double* ovh;
  double* v1;
  double* v2;
  double* ent;
  double* alpha;        // or null: no alpha_i (swe_compute_dij)
  double* sqgh;         // sqrt(g |h|), the sql / sqr of compute_lambda_vacc
  double* w2;           // qy one_over_h (v2 unless type 13)
  double* eta;          // h + z (w2, eta, rh and flux: null without the row kernels)
  double* rh;           // 1/h
  double* flux;         // v1 u_q and v2 u_q: (2 q + a) n_rows + r
  double* pt;           // SGN pressure (type 13)
  float4* nf;           // FP32: h, sqrt(g |h|), q one_over_h
};
static NodeF64 node_of(const WorkF64& w) {
  return NodeF64{w.ovh, w.v1, w.v2, w.ent, w.alpha, w.sqgh, w.w2, w.eta, w.rh, w.flux, w.pt, w.nf};
}

// The state of row r as lambda_row takes it.
__device__ __forceinline__ LamState lam_state(const StateF64& u, const NodeF64& nd, int64_t r) {
  return LamState{u.h[r], u.q1[r], u.q2[r], nd.ovh[r], nd.sqgh[r], nd.nf[r]};
}

// SGN pressure pTilde_n and source s_n (mSGN_RHS, update.f90:505-529)
__device__ __forceinline__ void sgn_node_f64(const InstConst& c, double m, double h, double heta,
                                             double* pTilde, double* s) {
  double lms = sqrt(m);
  double pc = c.lambda_sgn * c.g / (3.0 * lms);
  double x = heta / (h * h);
  double psi = 12.0 * (x - 1.0);
  double x3 = (x * x) * x, x4 = (x * x) * (x * x);
  *pTilde = pc * ((h * h) * h) * (2.0 + 4.0 * x3 - 6.0 * x4);
  double t = heta / h;
  *s = 3.0 * pc * (t * t) * psi;
}

// ---------------------------------------------------------------------------
// k_node: flux() globals (SOURCES/condlim.f90:21-77, 79-90), the entropy
// E_i = 0.5 (g h^2 + v.q) of entropy_residual (update.f90:844-851), the
// smoothness indicator alpha_i of alpha_limit (update.f90:758-781), and every
// other quantity of one node that the entry loops would otherwise form once
// per entry: the flux products v u_q, h + z, 1/h, the SGN pressure and the
// FP32 shadow of lambda_row.  ROWS: with what only the row kernels read.
// ---------------------------------------------------------------------------
template <bool ROWS>
__global__ void k_node_f64(Graph G, const InstConst* C, const InstState* St,
                           StateF64 u, NodeF64 nd) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  int L = G.len[r];
  if (L == 0) return;
  int b = G.slice_inst[r >> 5];
  if (St[b].done) return;
  const InstConst& c = C[b];
  const int64_t n = G.n_rows;
  double h = u.h[r], qx = u.q1[r], qy = u.q2[r];
  double o = one_over_h(h, c.htiny);
  double v1 = qx * o;
  double w2 = qy * o;
  double v2 = (c.type_test == 13) ? w2 * 0.0 : w2;
  const double sq = sqrt(c.g * fabs(h));
  nd.ovh[r] = o;
  nd.v1[r] = v1;
  nd.v2[r] = v2;
  if (ROWS) nd.w2[r] = w2;
  nd.sqgh[r] = sq;
  if (ROWS) {
    nd.eta[r] = h + G.bath[r];
    nd.rh[r] = 1.0 / h;
  }
  nd.nf[r] = make_float4((float)h, (float)sq, (float)v1, (float)w2);
  const double f11 = v1 * qx, f22 = v2 * qy;
  if (ROWS) {
    nd.flux[r] = v1 * h;
    nd.flux[2 * n + r] = f11;
    nd.flux[4 * n + r] = v1 * qy;
  }
  if (c.type_test == 13) {           // v2 = 0
    const double heta = u.q3[r];
    if (ROWS) {
      nd.flux[6 * n + r] = v1 * heta;
      nd.flux[8 * n + r] = v1 * u.q4[r];
    }
    double s;
    sgn_node_f64(c, G.lumped[r], h, heta, &nd.pt[r], &s);
  } else if (ROWS) {
    nd.flux[n + r] = v2 * h;
    nd.flux[3 * n + r] = v2 * qx;
    nd.flux[5 * n + r] = f22;
  }
  double E = c.g * (h * h);
  E = E + f11;
  E = E + f22;
  nd.ent[r] = 0.5 * E;
  if (!nd.alpha) return;
  double alpha = 1.0;
  if (c.alpha_limit && !(h <= c.htiny)) {
    const int64_t base = entry_base(G, r);
    const int dp = G.dpos[r];
    double num = 0.0, denom = 0.0;
    for (int kk = 0; kk <= L; kk++) {          // reference order, diagonal at dp
      const int k = kk - (kk > dp ? 1 : 0);
      const double hj = (kk == dp) ? h : u.h[G.col[base + 32 * k]];
      num = num + hj - h;
      denom = denom + fabs(hj - h);
    }
    double a = (denom <= tabs(num)) ? 1.0 : tabs(num) / (denom);
    double a2 = a * a, a4 = a2 * a2;
    alpha = a4 * a4;
  }
  nd.alpha[r] = alpha;
}

// x**gamma of the Manning friction (update.f90:436), gamma = 4/3 rounded to 64
// bits: with c = cbrt(x), r = x - c^3 (exact products), x**(4/3) = x c + c r/3,
// and x**(gamma - 4/3) = 1 + (gamma - 4/3) ln x.  Within 0.6 units in the last
// place over [1e-8, 20] (CUDA's pow: 1.0), in 29 FP64 instructions against 99.
__device__ __forceinline__ double pow_43(double x) {
  const double c = cbrt(x), c2 = c * c, p = x * c;
  const double r = __fma_rn(-__fma_rn(c, c, -c2), c, __fma_rn(-c2, c, x));
  const float lx = __logf(fminf(fmaxf((float)x, 1.2e-38f), 3e38f));
  double t = __fma_rn(x, c, -p);
  t = __fma_rn(c * r, 1.0 / 3.0, t);
  t = __fma_rn(p, (double)(-7.4014868308343765e-17f * lx), t);
  return p + t;
}

// Source terms (SOURCES/update.f90:425-551) added to the undivided rk of one
// row.  velocity is the row's own (v1, v2).
__device__ __forceinline__ void source_f64(const InstConst& c, const InstState& st, double m, const double* ui,
                                           double v1, double v2, double* rk, double pt_sum_x, double pt_sum_y,
                                           double s_i) {
  const int S = c.S;
  if (c.type_test == 9 || c.type_test == 10) {
    const double chi = 1.0;
    double fric = c.g * c.mannings * c.mannings;
    double hstar = pow_43(tmax(ui[0], c.htiny));
    double vel = fric * sqrt(v1 * v1 + v2 * v2);
    double hloc = chi * vel * st.dt;
    for (int k = 1; k < S; k++) rk[k] = rk[k] - m * ui[k] * vel * 2 / (hstar + tmax(hstar, hloc));
  } else if (c.type_test == 11) {
    const double kappa = 0.2;
    for (int k = 1; k < S; k++) rk[k] = rk[k] - m * kappa * ui[k];
  } else if (c.type_test == 12) {
    const double f = 2.0;
    for (int j = 3; j <= S; j++) {
      rk[S - 2] = rk[S - 2] + m * f * ui[S - 1];
      rk[S - 1] = rk[S - 1] - m * f * ui[S - 2];
    }
  } else if (c.type_test == 13) {
    rk[1] = pt_sum_x;   // already accumulated in entry order by the caller
    rk[2] = pt_sum_y;
    rk[3] = rk[3] + m * ui[4];
    rk[4] = rk[4] - m * s_i;
  }
}

// Viscosities seen by the row sums: the low-order (alpha-limited) d_ij, mu_ij,
// or the entropy-viscosity d^H = MIN(d, res_ij), mu^H = MIN(mu, res_ij) of
// update.f90:232-239 (applied to the diagonal too: res_ii = res_i).
struct LowVisc {
  const double* dL;
  const double* muL;
  double dii, muii;
  __device__ void get(bool isd, int64_t e, int, double& d, double& mu) const {
    d = isd ? dii : dL[e];
    mu = isd ? muii : muL[e];
  }
};
struct HighVisc {
  const double* dL;
  const double* muL;
  const double* res;
  double dii, muii, resi;
  __device__ void get(bool isd, int64_t e, int j, double& d, double& mu) const {
    const double rij = isd ? tmax(resi, resi) : tmax(resi, res[j]);
    d = tmin(isd ? dii : dL[e], 1.0 * rij);
    mu = tmin(isd ? muii : muL[e], 1.0 * rij);
  }
};

struct RowSums {
  double rk[5] = {0, 0, 0, 0, 0};    // smb_2_roundoff (htiny tests), with fix
  double rk2[5] = {0, 0, 0, 0, 0};   // smb_2 (h <= 0 tests)
  double rk1[5] = {0, 0, 0, 0, 0};   // smb_1 ('type1')
  double fix = 0.0;                   // fix_roundoff
  double emax = 0.0, emin = 0.0;      // maxmin of the entropy over the row
};

// One row of smb_2_roundoff (update.f90:554-624), smb_2 (:626-682) and smb_1
// (:366-423), each with its source terms (:425-551), over the row's entries
// in reference order with the diagonal at dp; the entropy max/min of maxmin
// (:924-935) on the way.  Undivided by the lumped mass.
template <class V>
__device__ __forceinline__ void smb_rows_f64(const Graph& G, const InstConst& c, const InstState& st, const StateF64& u,
                                             const NodeF64& nd, int64_t r, int64_t base, int L, int dp,
                                             const double* ui, double zi, double m, const V& visc, bool want_round,
                                             bool want_plain, bool want_t1, RowSums& o) {
  const int S = c.S;
  const double g = c.g, htiny = c.htiny;
  const double v1i = nd.v1[r], v2i = nd.v2[r];
  double* rk = o.rk;
  double* rk2 = o.rk2;
  double* rk1 = o.rk1;
  o.emax = nd.ent[r];
  o.emin = o.emax;
  for (int kk = 0; kk <= L; kk++) {
    const bool isd = (kk == dp);
    const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
    const int j = isd ? (int)r : G.col[e];
    double uj[5];
    uj[0] = u.h[j]; uj[1] = u.q1[j]; uj[2] = u.q2[j];
    if (S == 5) { uj[3] = u.q3[j]; uj[4] = u.q4[j]; }
    const double zj = G.bath[j];
    const double v1j = nd.v1[j], v2j = nd.v2[j];
    double d, mu;
    visc.get(isd, e, j, d, mu);
    const double cxe = isd ? G.cxii[r] : G.cx[e], cye = isd ? G.cyii[r] : G.cy[e];
    const double ej = nd.ent[j];
    o.emax = tmax(o.emax, ej);
    o.emin = tmin(o.emin, ej);
    const double zmax = tmax(zi, zj);
    const double Hij = tmax(0.0, ui[0] + zi - zmax);
    const double Hji = tmax(0.0, uj[0] + zj - zmax);
    // H*/h, formed once for the three rows (each tests h against its own bound)
    const double qij = (ui[0] <= 0.0) ? 0.0 : Hij / ui[0];
    const double qji = (uj[0] <= 0.0) ? 0.0 : Hji / uj[0];
    if (want_round) {   // smb_2_roundoff (htiny tests)
      const double ratij = (ui[0] <= htiny) ? 0.0 : (ui[0] > 0.0 ? qij : Hij / ui[0]);   // h > htiny >= 0: qij
      const double ratji = (uj[0] <= htiny) ? 0.0 : (uj[0] > 0.0 ? qji : Hji / uj[0]);
      double xx = 0.0;
      xx = xx - cxe * (v1j);
      xx = xx - cye * (v2j);
      if (isd) {
        o.fix = o.fix + xx;
      } else {
        o.fix = o.fix - mu + (d - mu) * (-ratij);
        rk[0] = rk[0] + (xx + mu) * uj[0] + tmax((d - mu) * Hji, 0.0);
      }
      for (int q = 1; q < S; q++) {
        double x2 = 0.0;
        x2 = x2 - cxe * (v1j * uj[q]);
        x2 = x2 - cye * (v2j * uj[q]);
        rk[q] = rk[q] + x2 + d * (uj[q] * ratji - ui[q] * ratij) + mu * (uj[q] * (1.0 - ratji) - ui[q] * (1.0 - ratij));
      }
      rk[1] = rk[1] - g * ui[0] * (uj[0] + zj - ui[0] - zi) * cxe;
      rk[2] = rk[2] - g * ui[0] * (uj[0] + zj - ui[0] - zi) * cye;
    }
    if (want_plain) {   // smb_2 (h <= 0 tests)
      const double ratij = qij;
      const double ratji = qji;
      for (int q = 0; q < S; q++) {
        double x2 = 0.0;
        x2 = x2 - cxe * (v1j * uj[q]);
        x2 = x2 - cye * (v2j * uj[q]);
        rk2[q] = rk2[q] + x2 + d * (uj[q] * ratji - ui[q] * ratij) + mu * (uj[q] * (1.0 - ratji) - ui[q] * (1.0 - ratij));
      }
      rk2[1] = rk2[1] - g * ui[0] * (uj[0] + zj - ui[0] - zi) * cxe;
      rk2[2] = rk2[2] - g * ui[0] * (uj[0] + zj - ui[0] - zi) * cye;
    }
    if (want_t1) {      // smb_1 (htiny tests, flux vv = velocity u_k)
      const double ratij = (ui[0] <= htiny) ? 0.0 : (ui[0] > 0.0 ? qij : Hij / ui[0]);   // h > htiny >= 0: qij
      const double ratji = (uj[0] <= htiny) ? 0.0 : (uj[0] > 0.0 ? qji : Hji / uj[0]);
      for (int q = 0; q < S; q++) {
        double xx = 0.0;
        xx = xx - cxe * ((v1j * uj[q]) * ratji + (v1i * ui[q]) * ratij);
        xx = xx - cye * ((v2j * uj[q]) * ratji + (v2i * ui[q]) * ratij);
        rk1[q] = rk1[q] + xx + d * (uj[q] * ratji - ui[q] * ratij);
      }
      rk1[1] = rk1[1] - 0.5 * g * (Hji * Hji - Hij * Hij) * cxe;
      rk1[2] = rk1[2] - 0.5 * g * (Hji * Hji - Hij * Hij) * cye;
    }
  }
  // source terms
  if (c.type_test == 13) {
    // mSGN_RHS adds -pTilde_j c_ij after the smb loops, entry by entry, onto
    // the momentum rows: redo that accumulation in entry order on top of rk.
    double s_i, p_i;
    sgn_node_f64(c, m, ui[0], ui[3], &p_i, &s_i);
    double ax = rk[1], ay = rk[2], bx = rk2[1], by = rk2[2], tx = rk1[1], ty = rk1[2];
    for (int kk = 0; kk <= L; kk++) {
      const bool isd = (kk == dp);
      const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
      const int j = isd ? (int)r : G.col[e];
      const double cxe = isd ? G.cxii[r] : G.cx[e], cye = isd ? G.cyii[r] : G.cy[e];
      const double pj = nd.pt[j];
      ax = ax - pj * cxe; ay = ay - pj * cye;
      bx = bx - pj * cxe; by = by - pj * cye;
      tx = tx - pj * cxe; ty = ty - pj * cye;
    }
    if (want_round) source_f64(c, st, m, ui, v1i, v2i, rk, ax, ay, s_i);
    if (want_plain) source_f64(c, st, m, ui, v1i, v2i, rk2, bx, by, s_i);
    if (want_t1) source_f64(c, st, m, ui, v1i, v2i, rk1, tx, ty, s_i);
  } else {
    if (want_round) source_f64(c, st, m, ui, v1i, v2i, rk, 0, 0, 0);
    if (want_plain) source_f64(c, st, m, ui, v1i, v2i, rk2, 0, 0, 0);
    if (want_t1) source_f64(c, st, m, ui, v1i, v2i, rk1, 0, 0, 0);
  }
}

// ---------------------------------------------------------------------------
// k_low: compute_dij + compute_muij + MAX + alpha_limit (update.f90:180-187,
// 291-364, 782-798), smb_2_roundoff (:554-624) -> low-order state
// (:202-210), smb_2 + entropy residual (:825-878).  Writes dL/muL per entry,
// uL per row, res per row, fix_roundoff-free low-order h.
// ---------------------------------------------------------------------------
__global__ void k_low_f64(Graph G, const InstConst* C, const InstState* St,
                          StateF64 u, NodeF64 nd, double* __restrict__ dL, double* __restrict__ muL,
                          double* __restrict__ dLii, double* __restrict__ muLii, StateF64 uL,
                          double* __restrict__ res, const double* dij_in, unsigned* __restrict__ err) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const InstState st = St[b];
  if (st.done) return;
  const InstConst& c = C[b];
  const int S = c.S;
  const double g = c.g, htiny = c.htiny, dt = st.dt;
  const int64_t base = entry_base(G, r);
  const int dp = G.dpos[r];
  const LamState li = lam_state(u, nd, r);
  double ui[5];
  ui[0] = u.h[r]; ui[1] = u.q1[r]; ui[2] = u.q2[r];
  if (S == 5) { ui[3] = u.q3[r]; ui[4] = u.q4[r]; }
  const double ovhi = nd.ovh[r], v1i = nd.v1[r], v2i = nd.v2[r], ai = nd.alpha[r];
  const double zi = G.bath[r], m = G.lumped[r];
  bool delta_bad = false;

  // pass 1: raw d_ij (lambda_max) and mu_ij, diagonals = -row sums (the
  // diagonal's own value, 0, adds nothing to the sums).  'galerkin' sets
  // every d_ij and mu_ij to 0 (update.f90:155-158).
  double sd = 0.0, sm = 0.0;
  for (int k = 0; k < (c.visc == VISC_GALERKIN ? 0 : L); k++) {
    const int64_t e = base + 32 * k;
    const int j = G.col[e];
    double d = 0.0, mu = 0.0;
    {
      const double cxe = G.cx[e], cye = G.cy[e];
      if (dij_in) {                            // stage 1: k_dt computed this d_ij on this state
        d = dij_in[e];
      } else {
        double lam;
        if (!lambda_row(li, lam_state(u, nd, j), G.cnx[e], G.cny[e], G.cnf[e], c, &lam)) delta_bad = true;
        d = G.cnorm[e] * lam;                   // sqrt(c.c) lambda_max, normal c/sqrt(c.c)
      }
      const double sl = cxe * v1i + cye * v2i;
      // compute_muij uses q*ovh of the raw state, equal to velocity except
      // for type 13 whose velocity(2) is zeroed: recompute from q there
      double sr;
      if (c.type_test == 13) {
        const double ulx = ui[1] * ovhi, uly = ui[2] * ovhi;
        const double ox = nd.ovh[j];
        const double urx = u.q1[j] * ox, ury = u.q2[j] * ox;
        const double sl2 = cxe * ulx + cye * uly;
        sr = cxe * urx + cye * ury;
        mu = tmax(tmax(-sl2, 0.0), tmax(sr, 0.0));
      } else {
        sr = cxe * nd.v1[j] + cye * nd.v2[j];
        mu = tmax(tmax(-sl, 0.0), tmax(sr, 0.0));
      }
    }
    dL[e] = d;
    muL[e] = mu;
    sd = sd + d;
    sm = sm + mu;
  }
  const double dii_raw = -sd, muii_raw = -sm;
  // pass 2: dij = MAX(dij, muij) on every entry, then alpha limiting with the
  // reference's diagonal re-summation (the mu sum includes the old mu_ii at
  // its place in the row)
  sd = 0.0; sm = 0.0;
  double dii = tmax(dii_raw, muii_raw), muii = muii_raw;
  if (c.alpha_limit) dii = 0.0;
  if (c.visc == VISC_GALERKIN) {
    for (int k = 0; k < L; k++) { dL[base + 32 * k] = 0.0; muL[base + 32 * k] = 0.0; }
    dii = 0.0; muii = 0.0;
  }
  for (int kk = 0; kk <= (c.visc == VISC_GALERKIN ? -1 : L); kk++) {
    if (kk == dp) {
      sd = sd + dii;
      sm = sm + muii;
      continue;
    }
    const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
    double mu = muL[e];
    double d = tmax(dL[e], mu);
    if (c.alpha_limit) {
      const double s = tmax(ai, nd.alpha[G.col[e]]);
      d = d * s;
      mu = mu * s;
    }
    sd = sd + d;
    sm = sm + mu;
    dL[e] = d;
    muL[e] = mu;
  }
  if (c.alpha_limit && c.visc != VISC_GALERKIN) {
    dii = -sd;
    muii = -sm;
  }
  dLii[r] = dii;
  muLii[r] = muii;

  // pass 3: smb_2_roundoff / smb_2 / smb_1 rows and maxmin of the entropy,
  // in reference order with the diagonal at dp
  const bool galerkin = c.visc == VISC_GALERKIN;
  const bool type1 = !galerkin && c.viscous_type == 1;
  const bool need_res = c.visc == VISC_ENTROPY || c.visc == VISC_FCT;
  RowSums rs;
  const LowVisc lv{dL, muL, dii, muii};
  smb_rows_f64(G, c, st, u, nd, r, base, L, dp, ui, zi, m, lv,
               !galerkin && !type1 && c.roundoff_fix,              // smb_2_roundoff: low order
               galerkin || need_res || (!type1 && !c.roundoff_fix), // smb_2: Galerkin, residual, plain type2
               type1, rs);
  const double* rk2 = rs.rk2;
  // divide_by_lumped (:801-808) and the low-order state (:202-215)
  double ul[5];
  if (type1) {
    for (int q = 0; q < S; q++) ul[q] = ui[q] + dt * (rs.rk1[q] / m);
  } else if (!galerkin && c.roundoff_fix) {
    ul[0] = ui[0] * (1 + dt * rs.fix / m) + dt * (rs.rk[0] / m);
    for (int q = 1; q < S; q++) ul[q] = ui[q] + dt * (rs.rk[q] / m);
  } else {
    ul[0] = tmax(ui[0] + dt * (rk2[0] / m), 0.0);
    for (int q = 1; q < S; q++) ul[q] = ui[q] + dt * (rk2[q] / m);
  }
  uL.h[r] = ul[0]; uL.q1[r] = ul[1]; uL.q2[r] = ul[2];
  if (S == 5) { uL.q3[r] = ul[3]; uL.q4[r] = ul[4]; }
  if (delta_bad) atomicOr(err, ERRB_DELTA);
  if (!need_res) return;
  const double emax = rs.emax, emin = rs.emin;
  double rk2m[5];
  for (int q = 0; q < S; q++) rk2m[q] = rk2[q] / m;
  // entropy residual (update.f90:838-868), rescale hoisted
  double un_[5];
  for (int q = 0; q < S; q++) un_[q] = ui[q] + dt * rk2m[q];
  const double on = one_over_h(un_[0], htiny);
  const double vn1 = un_[1] * on, vn2 = un_[2] * on;
  double En = g * (un_[0] * un_[0]);
  En = En + vn1 * un_[1];
  En = En + vn2 * un_[2];
  En = 0.5 * En;
  const double E = nd.ent[r];
  double Ep[5] = {0, 0, 0, 0, 0};
  Ep[0] = g * ui[0];
  Ep[0] = Ep[0] - 0.5 * (v1i * v1i);
  Ep[1] = v1i;
  Ep[0] = Ep[0] - 0.5 * (v2i * v2i);
  Ep[2] = v2i;
  double rsd = m * (En - E) / dt;
  for (int q = 0; q < S; q++) rsd = rsd - m * rk2m[q] * Ep[q];
  const double rescale = tabs(emax - emin) / 2 + c.rescale_floor;
  res[r] = tabs(rsd) / rescale;
}

// ---------------------------------------------------------------------------
// k_fct: d^H = MIN(dL, res_ij), mu^H likewise (update.f90:232-239), f_ij
// (compute_fct_matrix :721-748), check_hmin of the low-order state (:271) and
// R^-_i of FCT_positivity (SOURCES/fct.f90:15-30).
// ---------------------------------------------------------------------------
__global__ void k_fct_f64(Graph G, const InstConst* C, const InstState* St,
                          StateF64 u, const double* dL, const double* muL,
                          StateF64 uL, const double* res, double* __restrict__ fct,
                          double* __restrict__ rminus, unsigned* __restrict__ err) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const InstState st = St[b];
  if (st.done) return;
  const InstConst& c = C[b];
  if (c.visc != VISC_FCT) return;
  const int64_t base = entry_base(G, r);
  const double hi = u.h[r], zi = G.bath[r], resi = res[r];
  double P = -1.e-15;
  for (int k = 0; k < L; k++) {
    const int64_t e = base + 32 * k;
    const int j = G.col[e];
    const double rij = tmax(resi, res[j]);
    const double d0 = dL[e], m0 = muL[e];
    const double dH = tmin(d0, 1.0 * rij), mH = tmin(m0, 1.0 * rij);
    const double hj = u.h[j], zj = G.bath[j];
    const double zmax = tmax(zi, zj);
    const double Hij = tmax(0.0, hi + zi - zmax);
    const double Hji = tmax(0.0, hj + zj - zmax);
    const double ratij = (hi <= 0.0) ? 0.0 : Hij / hi;
    const double ratji = (hj <= 0.0) ? 0.0 : Hji / hj;
    const double f = (dH - d0) * (hj * ratji - hi * ratij) + (mH - m0) * (hj * (1.0 - ratji) - hi * (1.0 - ratij));
    fct[e] = f;
    if (f < 0.0) P = P + f;
  }
  const double hL = uL.h[r];
  if (hL < 0.0) atomicOr(err, ERRB_NEG_H);
  const double scaled = (G.lumped[r] / st.dt) * hL;
  const double Q = 0.0 - scaled;
  double R = tmin(Q / P, 1.0);
  if (scaled <= c.htiny) R = 0.0;
  rminus[r] = R;
}

// Component q of a state at row r (no local arrays of pointers: the row's
// values stay in registers).
__device__ __forceinline__ double comp_f64(const StateF64& s, int q, int64_t r) {
  switch (q) {
    case 0: return s.h[r];
    case 1: return s.q1[r];
    case 2: return s.q2[r];
    case 3: return s.q3[r];
    default: return s.q4[r];
  }
}
__device__ __forceinline__ void store_f64(const StateF64& s, int q, int64_t r, double v) {
  switch (q) {
    case 0: s.h[r] = v; break;
    case 1: s.q1[r] = v; break;
    case 2: s.q2[r] = v; break;
    case 3: s.q3[r] = v; break;
    default: s.q4[r] = v; break;
  }
}

// End of a stage for one row: check_hmin (when the mode has it), non-finite
// check, the SSP-RK combination and bdy of the time loop (main.f90:77-90)
// when rk_stage > 0, and the store.
__device__ __forceinline__ void finish_row_f64(const Graph& G, const InstConst& c, const InstState& st, int64_t r,
                                               int S, double (&un)[5], bool check_hmin, int rk_stage,
                                               const StateF64& u0, const StateF64& out, unsigned* err) {
  if (check_hmin && un[0] < 0.0) atomicOr(err, ERRB_NEG_H);
  if (!(un[0] == un[0]) || !(un[1] == un[1]) || !(un[2] == un[2])) atomicOr(err, ERRB_NAN);
  const unsigned msk = (rk_stage >= 1 && G.dir_mask) ? G.dir_mask[r] : 0u;
#pragma unroll
  for (int q = 0; q < 5; q++) {
    if (q >= S) break;
    double v = un[q];
    if (rk_stage == 2) v = (3 * comp_f64(u0, q, r) + v) * 0.25;
    else if (rk_stage == 3) v = div_known(__fma_rn(2.0, v, comp_f64(u0, q, r)), 3.0, 1.0 / 3.0);   // 2 v is exact
    if (msk & (1u << q)) v = dirichlet_value(G, c, st, rk_stage, q, r);
    store_f64(out, q, r, v);
  }
}

// ---------------------------------------------------------------------------
// k_update: l_ij (fct.f90:31-41), (d^H-d^L) l_ij and (mu^H-mu^L) l_ij
// (update.f90:278-279), apply_viscosity (:684-718), unext = u^L + dt rk/m
// (:281-282), check_hmin (:285), then the SSP-RK combination and bdy of the
// time loop (main.f90:77-90) when rk_stage > 0.
//   rk_stage 0: out = unext                       (plain euler call)
//   rk_stage 1: out = unext, Dirichlet
//   rk_stage 2: out = (3 u0 + unext)/4, Dirichlet
//   rk_stage 3: out = (u0 + 2 unext)/3, Dirichlet
// ---------------------------------------------------------------------------
__global__ void k_update_f64(Graph G, const InstConst* C, const InstState* St,
                             StateF64 u, const double* dL, const double* muL,
                             StateF64 uL, const double* res, const double* fct,
                             const double* rminus, StateF64 u0, StateF64 out, int rk_stage,
                             double* __restrict__ lij_out, unsigned* __restrict__ err) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const InstState st = St[b];
  if (st.done) return;
  const InstConst& c = C[b];
  if (c.visc == VISC_ENTROPY) return;          // k_entropy_f64 writes these rows
  const bool fct_mode = c.visc == VISC_FCT;
  const int S = c.S;
  const int64_t base = entry_base(G, r);
  double ui[5];
  ui[0] = u.h[r]; ui[1] = u.q1[r]; ui[2] = u.q2[r];
  if (S == 5) { ui[3] = u.q3[r]; ui[4] = u.q4[r]; }
  const double zi = G.bath[r], resi = res[r], Ri = fct_mode ? rminus[r] : 0.0;
  double xx[5] = {0, 0, 0, 0, 0};
  for (int k = 0; k < (fct_mode ? L : 0); k++) {   // 'galerkin' / 'viscous': u^L is the result
    const int64_t e = base + 32 * k;
    const int j = G.col[e];
    const double f = fct[e];
    const double l = (f >= 0.0) ? rminus[j] : Ri;
    if (lij_out) lij_out[e] = l;
    const double rij = tmax(resi, res[j]);
    const double d0 = dL[e], m0 = muL[e];
    const double dd = (tmin(d0, 1.0 * rij) - d0) * l;
    const double dm = (tmin(m0, 1.0 * rij) - m0) * l;
    double uj[5];
    uj[0] = u.h[j]; uj[1] = u.q1[j]; uj[2] = u.q2[j];
    if (S == 5) { uj[3] = u.q3[j]; uj[4] = u.q4[j]; }
    const double zj = G.bath[j];
    const double zmax = tmax(zi, zj);
    const double Hij = tmax(0.0, ui[0] + zi - zmax);
    const double Hji = tmax(0.0, uj[0] + zj - zmax);
    const double ratij = (ui[0] <= 0.0) ? 0.0 : Hij / ui[0];
    const double ratji = (uj[0] <= 0.0) ? 0.0 : Hji / uj[0];
    for (int q = 0; q < S; q++)
      xx[q] = xx[q] + dd * (uj[q] * ratji - ui[q] * ratij) + dm * (uj[q] * (1.0 - ratji) - ui[q] * (1.0 - ratij));
  }
  const double m = G.lumped[r], dt = st.dt;
  double un[5] = {0, 0, 0, 0, 0};
  const double* ulp[5] = {uL.h, uL.q1, uL.q2, uL.q3, uL.q4};
  for (int q = 0; q < S; q++) un[q] = ulp[q][r] + dt * (xx[q] / m);
  // check_hmin follows 'fct' (update.f90:285); 'viscous' and 'galerkin' return
  // before it (:219-222, :155-176)
  finish_row_f64(G, c, st, r, S, un, fct_mode, rk_stage, u0, out, err);
}

// ---------------------------------------------------------------------------
// k_entropy: 'entropy_visc' (update.f90:225-262): the smb_2_roundoff (or
// smb_2) rows with d^H = MIN(d, res_ij), mu^H = MIN(mu, res_ij), the update
// u = u(1 + dt fix/m) + dt rk/m, check_hmin (:285), then the RK combination
// and bdy like k_update.
// ---------------------------------------------------------------------------
__global__ void k_entropy_f64(Graph G, const InstConst* C, const InstState* St,
                              StateF64 u, NodeF64 nd, const double* dL, const double* muL,
                              const double* dLii, const double* muLii,
                              const double* res, StateF64 u0, StateF64 out, int rk_stage,
                              unsigned* __restrict__ err) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const InstState st = St[b];
  if (st.done) return;
  const InstConst& c = C[b];
  if (c.visc != VISC_ENTROPY) return;
  const int S = c.S;
  const int64_t base = entry_base(G, r);
  const int dp = G.dpos[r];
  double ui[5];
  ui[0] = u.h[r]; ui[1] = u.q1[r]; ui[2] = u.q2[r];
  if (S == 5) { ui[3] = u.q3[r]; ui[4] = u.q4[r]; }
  const double zi = G.bath[r], m = G.lumped[r], dt = st.dt;
  const HighVisc hv{dL, muL, res, dLii[r], muLii[r], res[r]};
  RowSums rs;
  smb_rows_f64(G, c, st, u, nd, r, base, L, dp, ui, zi, m, hv, c.roundoff_fix != 0, c.roundoff_fix == 0, false, rs);
  double un[5] = {0, 0, 0, 0, 0};
  if (c.roundoff_fix) {
    un[0] = ui[0] * (1 + dt * rs.fix / m) + dt * (rs.rk[0] / m);
    for (int q = 1; q < S; q++) un[q] = ui[q] + dt * (rs.rk[q] / m);
  } else {
    un[0] = tmax(ui[0] + dt * (rs.rk2[0] / m), 0.0);
    for (int q = 1; q < S; q++) un[q] = ui[q] + dt * (rs.rk2[q] / m);
  }
  finish_row_f64(G, c, st, r, S, un, true, rk_stage, u0, out, err);
}

// ---------------------------------------------------------------------------
// The 'fct' row kernels (every instance of the context runs 'fct', 'viscous'
// 'type2' or 'entropy_visc' with the roundoff fix; others take the general
// kernels above).  A 'viscous' instance stops at the low-order state;
// 'entropy_visc' walks its rows once more (k_entropy_rows).  The FP64 unit bounds
// them: an SM retires a warp's FP64 instruction in 16 cycles, so they spend
// memory (idle at 1-3% of its rate in the general kernels) to form every
// FP64 value once:
//   * k_low_fct walks the row once (d_ij, mu_ij, both right-hand sides) and
//     stores, per entry and component, the two row differences
//       A_q = u_j rat_ji - u_i rat_ij,  B_q = u_j (1 - rat_ji) - u_i (1 - rat_ij)
//     that compute_fct_matrix and apply_viscosity form again;
//   * the diagonal contributes only -c_ii.F_i and the rounding residue of
//     (h_i + z_i) - h_i - z_i: both are formed once per row and added at the
//     diagonal's place in the row;
//   * where both depths exceed htiny the two right-hand sides add the same
//     products, and where both rats are 1 (flat bottom) B_q = 0;
//   * the diagonals of d and mu enter nothing ('fct' multiplies them by
//     u_i rat_ii - u_i rat_ii = 0): only swe_euler, which hands them out, forms
//     them.
// Wet/dry basin of 250k nodes, general kernels -> row kernels with lambda_row:
// k_low 942 -> 436 us (stage 1, d_ij from k_dt) and 576 (stages 2, 3), 836 and
// 1007 FP64 instructions per 32 rows, the unit 82-83% busy; k_fct 191 -> 37;
// k_update 258 -> 78 (75% busy).
// ---------------------------------------------------------------------------

// H / h for H >= 0, h > 0 (rh = 1/h): 1 where they are equal
__device__ __forceinline__ double rat_f64(double H, double h, double rh) {
  if (bits64(h) <= 0) return 0.0;
  return bits64(H) == bits64(h) ? 1.0 : div_known(H, h, rh);
}

// FCT: every instance runs 'fct' (no mode tests in the loop, which would cost
// registers).
template <int S, bool FCT, bool HIGH>
__device__ __forceinline__ void fct_row_f64(const Graph& G, const InstConst* C, const InstState* St, const StateF64& u,
                                            const NodeF64& nd, double* __restrict__ dL, double* __restrict__ muL,
                                            double* __restrict__ dLii, double* __restrict__ muLii, const StateF64& uL,
                                            double* res, double* __restrict__ ab, const double* dij_in, int want_diag,
                                            int64_t n_entries, unsigned* err, const StateF64& u0, const StateF64& out,
                                            int rk_stage) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  if (St[b].done) return;
  const InstConst& c = C[b];
  if (HIGH && c.visc != VISC_ENTROPY) return;
  const int64_t base = entry_base(G, r), nr = G.n_rows;
  const int dp = G.dpos[r];
  const double g = c.g, htiny = c.htiny;
  const LamState li = lam_state(u, nd, r);
  double ui[S];
  ui[0] = li.h; ui[1] = li.q1; ui[2] = li.q2;
  if (S == 5) { ui[3] = u.q3[r]; ui[4] = u.q4[r]; }
  const double zi = G.bath[r], etai = nd.eta[r], rhi = nd.rh[r], ai = nd.alpha[r];
  const double w1i = nd.v1[r], w2i = nd.w2[r], ghi = g * ui[0];
  const bool wet_i = !le_nn(ui[0], htiny);
  const bool fct = FCT || (!HIGH && c.visc == VISC_FCT);                    // keep the row differences
  const bool full = fct || (!HIGH && c.visc == VISC_ENTROPY);     // the right-hand side of smb_2 too, for the residual
  const double resi = HIGH ? own_res(res[r]) : 0.0;
  // the diagonal's terms: -c_ii.F_i and the topography residue
  double Dq[S], Dfix, tdx, tdy;
  {
    const double cxd = G.cxii[r], cyd = G.cyii[r];
    const double td = ghi * (etai - ui[0] - zi);
    tdx = td * cxd; tdy = td * cyd;
#pragma unroll
    for (int q = 0; q < S; q++) {
      Dq[q] = cxd * nd.flux[(int64_t)(2 * q) * nr + r];
      if (S == 3) Dq[q] = Dq[q] + cyd * nd.flux[(int64_t)(2 * q + 1) * nr + r];
    }
    Dfix = cxd * w1i;
    if (S == 3) Dfix = Dfix + cyd * w2i;
    if (HIGH && bits64(res[r]) < 0) {            // a NaN residual: d_ii, which multiplies a zero, is one too
#pragma unroll
      for (int q = 1; q < S; q++) Dq[q] = res[r];
    }
  }
  double fix = 0.0, rk[S], rk2[S];
#pragma unroll
  for (int q = 0; q < S; q++) rk[q] = rk2[q] = 0.0;
  double emax = nd.ent[r], emin = emax, sd = 0.0, sm = 0.0;
  bool bad = false;
  for (int k = 0; k <= L; k++) {
    if (k == dp) {                              // the diagonal's place in the row
      fix = fix - Dfix;
#pragma unroll
      for (int q = 1; q < S; q++) rk[q] = rk[q] - Dq[q];
      rk[1] = rk[1] - tdx; rk[2] = rk[2] - tdy;
      if (full) {
#pragma unroll
        for (int q = 0; q < S; q++) rk2[q] = rk2[q] - Dq[q];
        rk2[1] = rk2[1] - tdx; rk2[2] = rk2[2] - tdy;
      }
    }
    if (k == L) break;
    const int64_t e = base + 32 * k;
    const int j = G.col[e];
    const double cxe = G.cx[e], cye = G.cy[e];
    const LamState lj = lam_state(u, nd, j);
    // d_ij, mu_ij (compute_dij, compute_muij, MAX, alpha_limit)
    double d, mu;
    if (!HIGH) {
      if (dij_in) {
        d = dij_in[e];
      } else {
        double lam;
        if (!lambda_row(li, lj, G.cnx[e], G.cny[e], G.cnf[e], c, &lam)) bad = true;
        d = G.cnorm[e] * lam;
      }
    }
    const double w1j = nd.v1[j];
    double sr = cxe * w1j, srf = sr;             // c.v_j: the viscosity's velocity, the flux's (type 13: v2 = 0)
    sr = sr + cye * nd.w2[j];
    if (S == 3) srf = sr;
    if (HIGH) {                                  // d^H = MIN(d, res_ij), mu^H = MIN(mu, res_ij) (update.f90:232-239)
      const double rij = max_res(resi, res[j]);
      d = min_nn(dL[e], rij);
      mu = min_nn(muL[e], rij);
    } else {
      mu = max_nn(pos_part(-(cxe * w1i + cye * w2i)), pos_part(sr));
      if (want_diag) { sd = sd + d; sm = sm + mu; }
      d = max_nn(d, mu);
      const double s = max_nn(ai, nd.alpha[j]);  // 1 without alpha_limit
      d = d * s;
      mu = mu * s;
      dL[e] = d;
      muL[e] = mu;
    }
    if (full) {
      const double ej = nd.ent[j];
      emax = max_any(emax, ej);
      emin = min_any(emin, ej);
    }
    // hydrostatic reconstruction
    const double zj = G.bath[j], etaj = nd.eta[j];
    const double zmax = max_any(zi, zj);
    const double Hij = pos_part(etai - zmax), Hji = pos_part(etaj - zmax);
    const double qij = rat_f64(Hij, ui[0], rhi), qji = rat_f64(Hji, lj.h, nd.rh[j]);
    const bool wet_j = !le_nn(lj.h, htiny);
    const double dmu = d - mu;
    // smb_2_roundoff mass row
    fix = fix - mu - (wet_i ? dmu * qij : 0.0);
    rk[0] = rk[0] + (mu - srf) * lj.h + pos_part(dmu * Hji);
    // the momenta of both right-hand sides and the mass row of smb_2
    double uj[S];
    uj[0] = lj.h; uj[1] = lj.q1; uj[2] = lj.q2;
    if (S == 5) { uj[3] = u.q3[j]; uj[4] = u.q4[j]; }
    const bool flat = bits64(qij) == 0x3ff0000000000000ll && bits64(qji) == 0x3ff0000000000000ll;
    const bool wet = wet_i && wet_j;
    const double tp = ghi * (etaj - ui[0] - zi);
    const double tx = tp * cxe, ty = tp * cye;
    const double pij = 1.0 - qij, pji = 1.0 - qji;
#pragma unroll
    for (int q = 0; q < S; q++) {
      if (q == 0 && !full) continue;
      double x2 = cxe * nd.flux[(int64_t)(2 * q) * nr + j];
      if (S == 3) x2 = x2 + cye * nd.flux[(int64_t)(2 * q + 1) * nr + j];
      double A, B = 0.0, mB = 0.0;
      if (flat) {
        A = uj[q] - ui[q];
      } else {
        real_branch();
        A = uj[q] * qji - ui[q] * qij;
        B = uj[q] * pji - ui[q] * pij;
        mB = mu * B;
      }
      const double dA = d * A;
      if (fct) {
        ab[(int64_t)(2 * q) * n_entries + e] = A;
        ab[(int64_t)(2 * q + 1) * n_entries + e] = B;
      }
      if (full) {
        rk2[q] = rk2[q] - x2 + dA;
        if (!flat) { real_branch(); rk2[q] = rk2[q] + mB; }
      }
      if (q > 0) {
        rk[q] = rk[q] - x2;
        if (wet) {
          rk[q] = rk[q] + dA;
          if (!flat) { real_branch(); rk[q] = rk[q] + mB; }
        } else {                                // rats are 0 where h <= htiny
          real_branch();
          const double ti = wet_i ? qij : 0.0, tj = wet_j ? qji : 0.0;
          rk[q] = rk[q] + d * (uj[q] * tj - ui[q] * ti) + mu * (uj[q] * (1.0 - tj) - ui[q] * (1.0 - ti));
        }
      }
      if (q == 1) { rk[1] = rk[1] - tx; rk2[1] = rk2[1] - tx; }
      if (q == 2) { rk[2] = rk[2] - ty; rk2[2] = rk2[2] - ty; }
    }
  }
  if (!HIGH && want_diag) {   // the diagonals of the viscosities (update.f90:315-323, 782-798), as k_low_f64 forms them
    const double dii_raw = -sd, muii_raw = -sm;
    double dii = tmax(dii_raw, muii_raw), muii = muii_raw;
    if (c.alpha_limit) {
      sd = sm = 0.0;
      for (int kk = 0; kk <= L; kk++) {
        if (kk == dp) { sm = sm + muii; continue; }
        const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
        sd = sd + dL[e];
        sm = sm + muL[e];
      }
      dii = -sd;
      muii = -sm;
    }
    dLii[r] = dii;
    muLii[r] = muii;
  }
  const double m = G.lumped[r], im = G.inv_lumped[r], dt = St[b].dt;
  const double v1i = w1i, v2i = nd.v2[r];
  // source terms (:425-551), the same for both right-hand sides
  if (S == 5) {      // mSGN_RHS subtracts pTilde_j c_ij after the loops, entry by entry
    double p_i, s_i;
    sgn_node_f64(c, m, ui[0], ui[3], &p_i, &s_i);
    const double pdx = p_i * G.cxii[r], pdy = p_i * G.cyii[r];
    for (int k = 0; k <= L; k++) {
      if (k == dp) { rk[1] = rk[1] - pdx; rk[2] = rk[2] - pdy; rk2[1] = rk2[1] - pdx; rk2[2] = rk2[2] - pdy; }
      if (k == L) break;
      const int64_t e = base + 32 * k;
      const double pj = nd.pt[G.col[e]];
      const double px = pj * G.cx[e], py = pj * G.cy[e];
      rk[1] = rk[1] - px; rk[2] = rk[2] - py;
      rk2[1] = rk2[1] - px; rk2[2] = rk2[2] - py;
    }
    const double a3 = m * ui[S - 1], a4 = m * s_i;
    rk[S - 2] = rk[S - 2] + a3; rk2[S - 2] = rk2[S - 2] + a3;
    rk[S - 1] = rk[S - 1] - a4; rk2[S - 1] = rk2[S - 1] - a4;
  } else if (c.type_test == 9 || c.type_test == 10) {
    const double fric = c.g * c.mannings * c.mannings;
    const double hstar = pow_43(max_any(ui[0], htiny));
    const double vel = fric * sqrt(v1i * v1i + v2i * v2i);
    const double den = hstar + max_nn(hstar, vel * dt), y = 1.0 / den;
#pragma unroll
    for (int q = 1; q < 3; q++) {
      const double x = div_known(m * ui[q] * vel * 2.0, den, y);
      rk[q] = rk[q] - x;
      rk2[q] = rk2[q] - x;
    }
  } else if (c.type_test == 11) {
    const double kappa = 0.2;
#pragma unroll
    for (int q = 1; q < 3; q++) {
      const double x = m * kappa * ui[q];
      rk[q] = rk[q] - x;
      rk2[q] = rk2[q] - x;
    }
  } else if (c.type_test == 12) {
    const double f = 2.0, x1 = m * f * ui[2], x2 = m * f * ui[1];
    rk[1] = rk[1] + x1; rk2[1] = rk2[1] + x1;
    rk[2] = rk[2] - x2; rk2[2] = rk2[2] - x2;
  }
  // divide_by_lumped (:801-808) and the low-order state (:202-215)
  double ul[S];
  ul[0] = ui[0] * (1.0 + div_known(dt * fix, m, im)) + dt * div_known(rk[0], m, im);
#pragma unroll
  for (int q = 1; q < S; q++) ul[q] = ui[q] + dt * div_known(rk[q], m, im);
  if (HIGH) {        // 'entropy_visc': this is the stage's result
    double un[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < S; q++) un[q] = ul[q];
    finish_row_f64(G, c, St[b], r, S, un, true, rk_stage, u0, out, err);
    return;
  }
  uL.h[r] = ul[0]; uL.q1[r] = ul[1]; uL.q2[r] = ul[2];
  if (S == 5) { uL.q3[r] = ul[3]; uL.q4[r] = ul[4]; }
  if (bad) atomicOr(err, ERRB_DELTA);
  if (!full) return;
  // entropy residual (update.f90:838-868); Entprime(4:5) are 0
  double rm[3], un_[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    rm[q] = div_known(rk2[q], m, im);
    un_[q] = ui[q] + dt * rm[q];
  }
  const double on = one_over_h(un_[0], htiny);
  const double vn1 = un_[1] * on, vn2 = un_[2] * on;
  double En = g * (un_[0] * un_[0]);
  En = En + vn1 * un_[1];
  En = En + vn2 * un_[2];
  En = 0.5 * En;
  const double E = nd.ent[r];
  const double Ep0 = ghi - 0.5 * (v1i * v1i) - 0.5 * (v2i * v2i);
  double rsd = div_known(m * (En - E), dt, St[b].inv_dt);
  rsd = rsd - m * rm[0] * Ep0;
  rsd = rsd - m * rm[1] * v1i;
  rsd = rsd - m * rm[2] * v2i;
  const double rescale = __fma_rn(fabs(emax - emin), 0.5, c.rescale_floor);   // the product is exact
  res[r] = keep_res(fabs(rsd) / rescale);
}

template <int S, bool FCT>
__global__ void __launch_bounds__(128, 4)
k_low_fct(Graph G, const InstConst* C, const InstState* St, StateF64 u, NodeF64 nd, double* __restrict__ dL,
          double* __restrict__ muL, double* __restrict__ dLii, double* __restrict__ muLii, StateF64 uL,
          double* __restrict__ res, double* __restrict__ ab, const double* dij_in, int want_diag, int64_t n_entries,
          unsigned* __restrict__ err) {
  fct_row_f64<S, FCT, false>(G, C, St, u, nd, dL, muL, dLii, muLii, uL, res, ab, dij_in, want_diag, n_entries, err, u, u, 0);
}

// ---------------------------------------------------------------------------
// Small meshes: four warps per 32 rows.  The FP64 unit of an SM quarter takes 64
// cycles per warp instruction however few warps there are, so below about two
// slices per SM a row's chain of instructions is the kernel's time and most
// quarters idle.  Warp w forms the terms of entries w, w + 4, ... of the slice's
// rows and leaves them in shared memory; the warps then add them up in the
// reference's order, each its own sums (independent chains), and share the
// tail the same way.  Same operations and order as fct_row_f64.
// ---------------------------------------------------------------------------
template <int S>
struct SplitTerms {
  enum { MU, F, A0, B0, E, TX, TY, DRAW, MRAW, Q, N = Q + 5 * S };   // Q + 5 q: x2, d A, mu B, and those of smb_2_roundoff
};

template <int S>
__global__ void __launch_bounds__(128)
k_low_split(Graph G, const InstConst* C, const InstState* St, StateF64 u, NodeF64 nd, double* __restrict__ dL,
            double* __restrict__ muL, double* __restrict__ dLii, double* __restrict__ muLii, StateF64 uL,
            double* __restrict__ res, double* __restrict__ ab, const double* dij_in, int want_diag, int64_t n_entries,
            unsigned* __restrict__ err) {
  using T = SplitTerms<S>;
  __shared__ double term[4][T::N][32];
  __shared__ double tail[6][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.x * 32 + lane;     // n_rows is a multiple of 32
  const int b = G.slice_inst[blockIdx.x];
  if (St[b].done) return;                               // the whole block
  const InstConst& c = C[b];
  const int L = G.len[r], width = (int)((G.slice_ptr[blockIdx.x + 1] - G.slice_ptr[blockIdx.x]) >> 5);
  const int64_t base = entry_base(G, r), nr = G.n_rows;
  const int dp = G.dpos[r];
  const double g = c.g, htiny = c.htiny;
  const LamState li = lam_state(u, nd, r);
  double ui[S];
  ui[0] = li.h; ui[1] = li.q1; ui[2] = li.q2;
  if (S == 5) { ui[3] = u.q3[r]; ui[4] = u.q4[r]; }
  const double zi = G.bath[r], etai = nd.eta[r], rhi = nd.rh[r], ai = nd.alpha[r];
  const double w1i = nd.v1[r], w2i = nd.w2[r], ghi = g * ui[0];
  const bool wet_i = !le_nn(ui[0], htiny);
  // this warp's sums: warp 0 fix and rk[0], warp 1 rk2[0] and the entropy's
  // maximum and minimum; the pair rk[p], rk2[p] of one momentum component each
  const int p = w == 2 ? 1 : w == 3 ? 2 : (S == 5 ? (w == 0 ? 3 : 4) : 0);
  const double cxd = G.cxii[r], cyd = G.cyii[r];
  auto diag = [&](int q) {                              // c_ii.F_i
    double x = cxd * nd.flux[(int64_t)(2 * q) * nr + r];
    if (S == 3) x = x + cyd * nd.flux[(int64_t)(2 * q + 1) * nr + r];
    return x;
  };
  const double Dp = p ? diag(p) : 0.0;
  double D0 = 0.0, td = 0.0;
  if (w == 0) {
    D0 = cxd * w1i;
    if (S == 3) D0 = D0 + cyd * w2i;
  } else if (w == 1) {
    D0 = diag(0);
  } else {
    td = ghi * (etai - ui[0] - zi) * (w == 2 ? cxd : cyd);
  }
  double s0 = 0.0, s1 = 0.0, rk = 0.0, rk2 = 0.0;       // warp 0: fix, rk[0]; warp 1: rk2[0]; the pair
  double emax = nd.ent[r], emin = emax, sd = 0.0, sm = 0.0;
  auto add_diag = [&]() {
    if (w <= 1) s0 = s0 - D0;
    if (p) { rk = rk - Dp; rk2 = rk2 - Dp; }
    if (w >= 2) { rk = rk - td; rk2 = rk2 - td; }
  };
  bool bad = false;
  for (int k0 = 0; k0 < width; k0 += 4) {
    if (k0 + w < L) {
      const int64_t e = base + 32 * (k0 + w);
      const int j = G.col[e];
      const double cxe = G.cx[e], cye = G.cy[e];
      const LamState lj = lam_state(u, nd, j);
      double d;
      if (dij_in) {
        d = dij_in[e];
      } else {
        double lam;
        if (!lambda_row(li, lj, G.cnx[e], G.cny[e], G.cnf[e], c, &lam)) bad = true;
        d = G.cnorm[e] * lam;
      }
      double sr = cxe * nd.v1[j], srf = sr;
      sr = sr + cye * nd.w2[j];
      if (S == 3) srf = sr;
      double mu = max_nn(pos_part(-(cxe * w1i + cye * w2i)), pos_part(sr));
      term[w][T::DRAW][lane] = d;
      term[w][T::MRAW][lane] = mu;
      d = max_nn(d, mu);
      const double s = max_nn(ai, nd.alpha[j]);
      d = d * s;
      mu = mu * s;
      dL[e] = d;
      muL[e] = mu;
      term[w][T::E][lane] = nd.ent[j];
      const double zj = G.bath[j], etaj = nd.eta[j], zmax = max_any(zi, zj);
      const double Hij = pos_part(etai - zmax), Hji = pos_part(etaj - zmax);
      const double qij = rat_f64(Hij, ui[0], rhi), qji = rat_f64(Hji, lj.h, nd.rh[j]);
      const bool wet_j = !le_nn(lj.h, htiny);
      const double dmu = d - mu;
      term[w][T::MU][lane] = mu;
      term[w][T::F][lane] = wet_i ? dmu * qij : 0.0;
      term[w][T::A0][lane] = (mu - srf) * lj.h;
      term[w][T::B0][lane] = pos_part(dmu * Hji);
      const double tp = ghi * (etaj - ui[0] - zi);
      term[w][T::TX][lane] = tp * cxe;
      term[w][T::TY][lane] = tp * cye;
      double uj[S];
      uj[0] = lj.h; uj[1] = lj.q1; uj[2] = lj.q2;
      if (S == 5) { uj[3] = u.q3[j]; uj[4] = u.q4[j]; }
      const bool flat = bits64(qij) == 0x3ff0000000000000ll && bits64(qji) == 0x3ff0000000000000ll;
      const double pij = 1.0 - qij, pji = 1.0 - qji;
      const double ti = wet_i ? qij : 0.0, tj = wet_j ? qji : 0.0;
#pragma unroll
      for (int q = 0; q < S; q++) {
        double x2 = cxe * nd.flux[(int64_t)(2 * q) * nr + j];
        if (S == 3) x2 = x2 + cye * nd.flux[(int64_t)(2 * q + 1) * nr + j];
        double A, B = 0.0, mB = 0.0;
        if (flat) {
          A = uj[q] - ui[q];
        } else {
          real_branch();
          A = uj[q] * qji - ui[q] * qij;
          B = uj[q] * pji - ui[q] * pij;
          mB = mu * B;
        }
        const double dA = d * A;
        ab[(int64_t)(2 * q) * n_entries + e] = A;
        ab[(int64_t)(2 * q + 1) * n_entries + e] = B;
        term[w][T::Q + 5 * q][lane] = x2;
        term[w][T::Q + 5 * q + 1][lane] = dA;
        term[w][T::Q + 5 * q + 2][lane] = mB;
        if (q > 0) {
          double dAr = dA, mBr = mB;
          if (!(wet_i && wet_j)) {
            real_branch();
            dAr = d * (uj[q] * tj - ui[q] * ti);
            mBr = mu * (uj[q] * (1.0 - tj) - ui[q] * (1.0 - ti));
          }
          term[w][T::Q + 5 * q + 3][lane] = dAr;
          term[w][T::Q + 5 * q + 4][lane] = mBr;
        }
      }
    }
    __syncthreads();
    for (int k = k0; k < k0 + 4; k++) {
      if (k == dp && k < L) add_diag();
      if (k >= L) continue;
      const auto& t = term[k - k0];
      if (w == 0) {
        s0 = s0 - t[T::MU][lane] - t[T::F][lane];
        s1 = s1 + t[T::A0][lane] + t[T::B0][lane];
      } else if (w == 1) {
        s0 = s0 - t[T::Q][lane] + t[T::Q + 1][lane];
        s0 = s0 + t[T::Q + 2][lane];
        emax = max_any(emax, t[T::E][lane]);
        emin = min_any(emin, t[T::E][lane]);
        if (want_diag) { sd = sd + t[T::DRAW][lane]; sm = sm + t[T::MRAW][lane]; }
      }
      if (p) {
        const double x2 = t[T::Q + 5 * p][lane];
        rk = rk - x2 + t[T::Q + 5 * p + 3][lane] + t[T::Q + 5 * p + 4][lane];
        rk2 = rk2 - x2 + t[T::Q + 5 * p + 1][lane] + t[T::Q + 5 * p + 2][lane];
      }
      if (w >= 2) {
        const double tp = t[w == 2 ? T::TX : T::TY][lane];
        rk = rk - tp;
        rk2 = rk2 - tp;
      }
    }
    __syncthreads();
  }
  if (dp == L) add_diag();
  const double m = G.lumped[r], im = G.inv_lumped[r], dt = St[b].dt;
  const double v1i = w1i, v2i = nd.v2[r];
  if (want_diag && w == 1 && L > 0) {    // as in fct_row_f64
    const double dii_raw = -sd, muii_raw = -sm;
    double dii = tmax(dii_raw, muii_raw), muii = muii_raw;
    if (c.alpha_limit) {
      sd = sm = 0.0;
      for (int kk = 0; kk <= L; kk++) {
        if (kk == dp) { sm = sm + muii; continue; }
        const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
        sd = sd + dL[e];
        sm = sm + muL[e];
      }
      dii = -sd;
      muii = -sm;
    }
    dLii[r] = dii;
    muLii[r] = muii;
  }
  // source terms (:425-551)
  if (S == 5) {
    double p_i, s_i;
    sgn_node_f64(c, m, ui[0], ui[3], &p_i, &s_i);
    if (w >= 2) {
      const double pd = p_i * (w == 2 ? cxd : cyd);
      for (int k = 0; k <= L; k++) {
        if (k == dp) { rk = rk - pd; rk2 = rk2 - pd; }
        if (k == L) break;
        const int64_t e = base + 32 * k;
        const double px = nd.pt[G.col[e]] * (w == 2 ? G.cx[e] : G.cy[e]);
        rk = rk - px;
        rk2 = rk2 - px;
      }
    } else if (w == 0) {
      const double x = m * ui[S - 1];
      rk = rk + x; rk2 = rk2 + x;
    } else {
      const double x = m * s_i;
      rk = rk - x; rk2 = rk2 - x;
    }
  } else if (w >= 2) {
    const double up = w == 2 ? ui[1] : ui[2];
    if (c.type_test == 9 || c.type_test == 10) {
      const double fric = c.g * c.mannings * c.mannings;
      const double hstar = pow_43(max_any(ui[0], htiny));
      const double vel = fric * sqrt(v1i * v1i + v2i * v2i);
      const double den = hstar + max_nn(hstar, vel * dt);
      const double x = m * up * vel * 2.0 / den;
      rk = rk - x; rk2 = rk2 - x;
    } else if (c.type_test == 11) {
      const double kappa = 0.2, x = m * kappa * up;
      rk = rk - x; rk2 = rk2 - x;
    } else if (c.type_test == 12) {
      const double f = 2.0, x = m * f * (w == 2 ? ui[2] : ui[1]);
      rk = w == 2 ? rk + x : rk - x;
      rk2 = w == 2 ? rk2 + x : rk2 - x;
    }
  }
  // divide_by_lumped (:801-808), the low-order state (:202-215), and what the
  // residual takes of the smb_2 rows
  if (w == 0 && L > 0) uL.h[r] = ui[0] * (1.0 + div_known(dt * s0, m, im)) + dt * div_known(s1, m, im);
  if (p) {
    const double up = p == 1 ? ui[1] : p == 2 ? ui[2] : p == 3 ? ui[S - 2] : ui[S - 1];
    const double ul = up + dt * div_known(rk, m, im);
    if (L > 0) store_f64(uL, p, r, ul);
    if (w >= 2) {
      const double rm = div_known(rk2, m, im);
      tail[2 * p][lane] = rm;
      tail[2 * p + 1][lane] = up + dt * rm;
    }
  }
  if (w == 1) {
    const double rm = div_known(s0, m, im);
    tail[0][lane] = rm;
    tail[1][lane] = ui[0] + dt * rm;
  }
  if (bad) atomicOr(err, ERRB_DELTA);
  __syncthreads();
  if (w != 1 || L == 0) return;
  // entropy residual (update.f90:838-868)
  const double un0 = tail[1][lane], un1 = tail[3][lane], un2 = tail[5][lane];
  const double on = one_over_h(un0, htiny);
  double En = g * (un0 * un0);
  En = En + un1 * on * un1;
  En = En + un2 * on * un2;
  En = 0.5 * En;
  const double Ep0 = ghi - 0.5 * (v1i * v1i) - 0.5 * (v2i * v2i);
  double rsd = div_known(m * (En - nd.ent[r]), dt, St[b].inv_dt);
  rsd = rsd - m * tail[0][lane] * Ep0;
  rsd = rsd - m * tail[2][lane] * v1i;
  rsd = rsd - m * tail[4][lane] * v2i;
  res[r] = keep_res(fabs(rsd) / __fma_rn(fabs(emax - emin), 0.5, c.rescale_floor));
}

// 'entropy_visc' (update.f90:225-262): the smb_2_roundoff rows again, with
// d^H and mu^H, are the stage's result.
template <int S>
__global__ void __launch_bounds__(128, 4)
k_entropy_rows(Graph G, const InstConst* C, const InstState* St, StateF64 u, NodeF64 nd, double* dL, double* muL,
               double* res, StateF64 u0, StateF64 out, int rk_stage, unsigned* err) {
  fct_row_f64<S, false, true>(G, C, St, u, nd, dL, muL, nullptr, nullptr, u, res, nullptr, nullptr, 0, 0, err, u0, out,
                       rk_stage);
}

// f_ij and R^-_i from the stored differences: five FP64 instructions per
// entry (the general k_fct_f64 forms the rats again: 42).
__global__ void k_fct_fct(Graph G, const InstConst* C, const InstState* St,
                          const double* dL, const double* muL, const double* hL,
                          const double* res, const double* ab, double* __restrict__ fct,
                          double* __restrict__ rminus, int64_t n_entries, unsigned* __restrict__ err) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  if (St[b].done) return;
  if (C[b].visc != VISC_FCT) return;
  const int64_t base = entry_base(G, r);
  const double resi = own_res(res[r]);
  double P = -1.e-15;
#pragma unroll 2
  for (int k = 0; k < L; k++) {
    const int64_t e = base + 32 * k;
    const double rij = max_res(resi, res[G.col[e]]);
    const double d0 = dL[e], m0 = muL[e];
    const double f = (min_nn(d0, rij) - d0) * ab[e] + (min_nn(m0, rij) - m0) * ab[n_entries + e];
    fct[e] = f;
    if (__double2hiint(f) <= (int)0xfff00000) P = P + f;   // f < 0 and not NaN; -0 adds nothing
  }
  const double h = hL[r];
  if (__double2hiint(h) < 0 && h < 0.0) atomicOr(err, ERRB_NEG_H);
  const double scaled = div_known(G.lumped[r], St[b].dt, St[b].inv_dt) * h;
  double R = 0.0;
  if (!le_nn(scaled, C[b].htiny)) {
    R = 1.0;                                      // Q^-/P^- >= 1: most rows
    if (bits64(scaled) < bits64(-P)) {
      real_branch();
      R = scaled / -P;
    }
  }
  rminus[r] = R;
}

// l_ij, the limited antidiffusion from the stored differences, and the end of
// the stage (see k_update_f64 for rk_stage).
template <int S>
__global__ void k_update_fct(Graph G, const InstConst* C, const InstState* St,
                             const double* dL, const double* muL, StateF64 uL,
                             const double* res, const double* fct,
                             const double* rminus, const double* ab, StateF64 u0,
                             StateF64 out, int rk_stage, double* __restrict__ lij_out, int64_t n_entries,
                             unsigned* __restrict__ err) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const InstState& st = St[b];
  if (st.done) return;
  const InstConst& c = C[b];
  if (c.visc == VISC_ENTROPY) return;          // k_entropy_rows writes these rows
  const int64_t base = entry_base(G, r);
  const bool fct_mode = c.visc == VISC_FCT;
  const double resi = fct_mode ? own_res(res[r]) : 0.0, Ri = fct_mode ? rminus[r] : 0.0;
  double xx[S];
#pragma unroll
  for (int q = 0; q < S; q++) xx[q] = 0.0;
  for (int k = 0; k < (fct_mode ? L : 0); k++) {
    const int64_t e = base + 32 * k;
    const int j = G.col[e];
    const double l = (bits64(fct[e]) << 1) == 0 || bits64(fct[e]) > 0 ? rminus[j] : Ri;   // f >= 0
    if (lij_out) lij_out[e] = l;
    const double rij = max_res(resi, res[j]);
    const double d0 = dL[e], m0 = muL[e];
    const double dd = (min_nn(d0, rij) - d0) * l;
    const double dm = (min_nn(m0, rij) - m0) * l;
#pragma unroll
    for (int q = 0; q < S; q++)
      xx[q] = xx[q] + dd * ab[(int64_t)(2 * q) * n_entries + e] + dm * ab[(int64_t)(2 * q + 1) * n_entries + e];
  }
  const double m = G.lumped[r], im = G.inv_lumped[r], dt = st.dt;
  double un[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int q = 0; q < S; q++) un[q] = comp_f64(uL, q, r) + dt * div_known(xx[q], m, im);
  finish_row_f64(G, c, st, r, S, un, fct_mode, rk_stage, u0, out, err);
}

// Maximum over a warp of values >= 0 (NaN counts as 0, as in fmax), lane 0:
// compared as integers, off the FP64 unit.
__device__ __forceinline__ double warp_max(double v) {
  long long m = bits64(v) <= 0x7ff0000000000000ll ? bits64(v) : 0;
  for (int off = 16; off > 0; off >>= 1) {
    const long long o = __shfl_down_sync(0xffffffffu, m, off);
    m = o > m ? o : m;
  }
  return __longlong_as_double(m);
}

// ---------------------------------------------------------------------------
// k_dt: compute_dij (update.f90:291-326) diagonal and COMPUTE_DT's
// max |d_ii|/m_i (main.f90:166-174), per instance.  d_out (nullable)
// receives every d_ij.  The FP64 unit (67% busy at 250k nodes, the slices along
// the shoreline end last): 554 -> 159 us with lambda_row, 182 FP64 instructions
// per 32 rows.
// ---------------------------------------------------------------------------
__global__ void k_dt_f64(Graph G, const InstConst* C, InstState* St, StateF64 u, NodeF64 nd,
                         double* __restrict__ d_out, double* __restrict__ dii_out, unsigned* __restrict__ err,
                         StepTurn turn) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double val = 0.0;
  if (r < G.n_rows && G.len[r] > 0 && !St[G.slice_inst[r >> 5]].done) {
    const InstConst& c = C[G.slice_inst[r >> 5]];
    const int L = G.len[r];
    const int64_t base = entry_base(G, r);
    const LamState li = lam_state(u, nd, r);
    double s = 0.0;
    bool bad = false;
    for (int k = 0; k < L; k++) {
      const int64_t e = base + 32 * k;
      double lam;
      if (!lambda_row(li, lam_state(u, nd, G.col[e]), G.cnx[e], G.cny[e], G.cnf[e], c, &lam)) bad = true;
      const double d = G.cnorm[e] * lam;                                   // sqrt(c.c) lambda_max
      if (d_out) d_out[e] = d;
      s = s + d;
    }
    if (dii_out) dii_out[r] = -s;
    val = div_known(fabs(-s), G.lumped[r], G.inv_lumped[r]);
    if (bad) atomicOr(err, ERRB_DELTA);
  }
  // warp-level max per instance: a warp covers one 32-row slice and a slice
  // never straddles two instances
  val = warp_max(val);
  const int64_t r0 = r & ~(int64_t)31;
  if ((threadIdx.x & 31) == 0 && r0 < G.n_rows) {
    const int bw = G.slice_inst[r0 >> 5];
    if (!St[bw].done && val > 0.0) atomicMax(&St[bw].maxd_bits, (unsigned long long)__double_as_longlong(val));
  }
  step_turn(turn, C, St);
}

// k_dt, four warps per 32 rows (see k_low_split; measured at split_dt)
__global__ void __launch_bounds__(128) k_dt_split(Graph G, const InstConst* C, InstState* St, StateF64 u, NodeF64 nd,
                                                  double* __restrict__ d_out, double* __restrict__ dii_out,
                                                  unsigned* __restrict__ err, StepTurn turn) {
  __shared__ double dk[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.x * 32 + lane;
  const int b = G.slice_inst[blockIdx.x];
  if (!St[b].done) {                                    // the whole block
    const InstConst& c = C[b];
    const int L = G.len[r], width = (int)((G.slice_ptr[blockIdx.x + 1] - G.slice_ptr[blockIdx.x]) >> 5);
    const int64_t base = entry_base(G, r);
    const LamState li = lam_state(u, nd, r);
    double s = 0.0;
    bool bad = false;
    for (int k0 = 0; k0 < width; k0 += 8) {
      for (int q = w; q < 8 && k0 + q < L; q += 4) {
        const int64_t e = base + 32 * (k0 + q);
        double lam;
        if (!lambda_row(li, lam_state(u, nd, G.col[e]), G.cnx[e], G.cny[e], G.cnf[e], c, &lam)) bad = true;
        const double d = G.cnorm[e] * lam;
        if (d_out) d_out[e] = d;
        dk[q][lane] = d;
      }
      __syncthreads();
      if (w == 0)
        for (int q = 0; q < 8 && k0 + q < L; q++) s = s + dk[q][lane];
      __syncthreads();
    }
    if (bad) atomicOr(err, ERRB_DELTA);
    if (w == 0) {
      double val = 0.0;
      if (L > 0) {
        if (dii_out) dii_out[r] = -s;
        val = div_known(s, G.lumped[r], G.inv_lumped[r]);
      }
      val = warp_max(val);
      if (lane == 0 && val > 0.0) atomicMax(&St[b].maxd_bits, (unsigned long long)__double_as_longlong(val));
    }
  }
  step_turn(turn, C, St);
}

// The turn between two steps as a kernel of its own
__global__ void k_step_turn(StepTurn t, const InstConst* C, InstState* St) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < t.n_inst) turn_instance(t, C[b], St[b]);
}

// Start of a swe_rk3_steps call: step counters and the lambda_max maximum
// restart (the instances' time, dt and done flags carry over)
__global__ void k_reset_counters(InstState* St, int n_inst) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_inst) return;
  St[b].steps = 0;
  St[b].maxd_bits = 0ull;
}

// End of a time step: time = to + dt (main.f90:91)
__global__ void k_step_end(InstState* St, int n_inst) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_inst) return;
  InstState& s = St[b];
  if (s.done) return;
  s.time = s.time + s.dt;
  s.steps += 1;
}

// FCT_positivity as a stand-alone operator on one instance (fct.f90:5-42)
__global__ void k_fct_positivity_f64(Graph G, const InstConst* __restrict__ C, const double* __restrict__ unext,
                                     const double* __restrict__ mat, const double* __restrict__ matii,
                                     double* __restrict__ rtmp, double* __restrict__ lij, int pass) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int b = G.slice_inst[r >> 5];
  const int64_t base = entry_base(G, r);
  if (pass == 0) {
    const int dp = G.dpos[r];
    double P = -1.e-15;
    for (int kk = 0; kk <= L; kk++) {         // reference order, diagonal at dp
      const double f = (kk == dp) ? matii[r] : mat[base + 32 * (kk - (kk > dp ? 1 : 0))];
      if (f < 0.0) P = P + f;
    }
    double R = tmin((0.0 - unext[r]) / P, 1.0);
    if (unext[r] <= C[b].htiny) R = 0.0;
    rtmp[r] = R;
  } else {
    for (int k = 0; k < L; k++) {
      const int64_t e = base + 32 * k;
      lij[e] = (mat[e] >= 0.0) ? rtmp[G.col[e]] : rtmp[r];
    }
  }
}

// FCT_generic (SOURCES/SAFE/fct.f90:3-43) as a stand-alone operator: the
// two-sided Zalesak limiter with local bounds maxn/minn.  Pass 0: P+-, Q+-,
// R+- per row (entries in reference order, the diagonal at dpos); pass 1:
// sum_j l_ij f_ij with l_ij = MIN(R+_i, R-_j) (f >= 0) or MIN(R-_i, R+_j), and
// u_i += x / dg_i.
__global__ void k_fct_generic_f64(Graph G, double* __restrict__ unext, const double* __restrict__ maxn,
                                  const double* __restrict__ minn, const double* __restrict__ dg,
                                  const double* __restrict__ mat, const double* __restrict__ matii,
                                  double* __restrict__ rplus, double* __restrict__ rminus, int pass) {
  int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= G.n_rows) return;
  const int L = G.len[r];
  if (L == 0) return;
  const int64_t base = entry_base(G, r);
  const int dp = G.dpos[r];
  if (pass == 0) {
    const double Qplus = dg[r] * (maxn[r] - unext[r]);
    const double Qminus = dg[r] * (minn[r] - unext[r]);
    double Pplus = 1.e-15, Pminus = -1.e-15;
    for (int kk = 0; kk <= L; kk++) {
      const double f = (kk == dp) ? matii[r] : mat[base + 32 * (kk - (kk > dp ? 1 : 0))];
      if (f >= 0.0) Pplus = Pplus + f;
      else Pminus = Pminus + f;
    }
    rplus[r] = tmin(Qplus / Pplus, 1.0);
    rminus[r] = tmin(Qminus / Pminus, 1.0);
  } else {
    double x = 0.0;
    for (int kk = 0; kk <= L; kk++) {
      const int64_t e = base + 32 * (kk - (kk > dp ? 1 : 0));
      const double f = (kk == dp) ? matii[r] : mat[e];
      const int64_t j = (kk == dp) ? r : (int64_t)G.col[e];
      const double l = (f >= 0.0) ? tmin(rplus[r], rminus[j]) : tmin(rminus[r], rplus[j]);
      x = x + l * f;
    }
    unext[r] = unext[r] + x / dg[r];
  }
}


// ----------------------------- launchers -----------------------------------
static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

#define EV_BEGIN(k) if (kev) cudaEventRecord(kev->ev[2 * (k)], s)
#define EV_END(k) if (kev) cudaEventRecord(kev->ev[2 * (k) + 1], s)

// Ordinary launches: with programmatic dependent launch the next kernel's
// blocks are placed while this one's still hold their SMs, and the FP64 unit of
// an SM that got two is the step's time (10k nodes: 357 us against 253).
template <typename... KArgs, typename... Args>
static void launch_full(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  kern<<<grid, block, smem, s>>>(static_cast<KArgs>(args)...);
}

static int64_t sm_count() {
  static const int64_t sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return (int64_t)n;
  }();
  return sms;
}

// Where k_low runs four warps per slice: up to one wave of its blocks, 4 slices per
// SM (registers), 2.5 for 5-component systems.  Per step, four warps against
// one: 2k nodes 153 against 244 us, 10k 179 / 248, 16k 244 / 250, 20k 268 /
// 332, 29k 360 / 346; SGN 2k 171 / 248, 12k 231 / 249, 16k 299 / 256.
static bool split_rows(int64_t n_rows, int S) { return n_rows <= (S == 5 ? 80 : 128) * sm_count(); }
// k_dt adds one sum per row, so its four warps cost nothing in throughput, and
// they shorten the slices along a shoreline, whose general evaluations are its
// time on meshes of ordinary size: wet/dry basin of 20k / 50k / 102k / 200k / 1M
// nodes 65 / 76 / 93 / 134 / 499 us, one warp 103 / 115 / 130 / 187 / 499; dam
// break of 102k / 200k / 1M 75 / 114 / 450 against 91 / 136 / 424; SGN of 36k /
// 102k / 200k 33 / 59 / 93 against 27 / 57 / 89.
static bool split_dt(int64_t n_rows, int S) { return n_rows <= (S == 5 ? 80 : 1400) * sm_count(); }
// One slice per block in k_dt and k_low: neighbouring slices are alike, and four
// expensive ones (a shoreline) in one block wait for one SM.  k_dt 512 -> 499
// and k_low 1840 -> 1832 us on the basin of 1M nodes, 122 -> 115 and 192 -> 185
// at 50k, SGN of 20k nodes k_low 82 -> 62.
constexpr int kRowBlock = 32;

void launch_node_f64(const StageArgs& a, cudaStream_t s) {
  const NodeF64 nd = node_of(a.w);
  const unsigned nb = nblk(a.G.n_rows, a.block);
  if (nd.flux) launch_full(k_node_f64<true>, nb, a.block, 0, s, a.G, a.C, a.St, a.u, nd);
  else launch_full(k_node_f64<false>, nb, a.block, 0, s, a.G, a.C, a.St, a.u, nd);
}

void launch_stage_f64(const StageArgs& a, cudaStream_t s, const KernelEvents* kev) {
  const int bs = a.block;
  const NodeF64 nd = node_of(a.w);
  EV_BEGIN(1);
  if (!a.skip_node) launch_node_f64(a, s);
  EV_END(1); EV_BEGIN(2);
  const unsigned nb = nblk(a.G.n_rows, bs);
  if (a.fused) {
    const int64_t ne = a.w.n_entries;
    const int diag = a.rk_stage == 0;            // swe_euler_intermediates hands out the diagonals
    if (a.all_fct && split_rows(a.G.n_rows, a.S)) {
      const unsigned ns = (unsigned)(a.G.n_rows / 32);
      if (a.S == 5)
        launch_full(k_low_split<5>, ns, 128, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.dLii, a.w.muLii, a.w.uL,
                    a.w.res, a.w.ab, a.dij_in, diag, ne, a.err);
      else
        launch_full(k_low_split<3>, ns, 128, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.dLii, a.w.muLii, a.w.uL,
                    a.w.res, a.w.ab, a.dij_in, diag, ne, a.err);
    } else
#define SWE_LOWF(S, F)                                                                                              \
    launch_full(k_low_fct<S, F>, nblk(a.G.n_rows, kRowBlock), kRowBlock, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL,       \
                a.w.muL, a.w.dLii, a.w.muLii, a.w.uL, a.w.res, a.w.ab, a.dij_in, diag, ne, a.err)
    if (a.S == 5) { if (a.all_fct) SWE_LOWF(5, true); else SWE_LOWF(5, false); }
    else { if (a.all_fct) SWE_LOWF(3, true); else SWE_LOWF(3, false); }
#undef SWE_LOWF
    EV_END(2); EV_BEGIN(3);
    if (a.any_fct)
      launch_full(k_fct_fct, nb, bs, 0, s, a.G, a.C, a.St, a.w.dL, a.w.muL, a.w.uL.h, a.w.res, a.w.ab, a.w.fct, a.w.rminus, ne,
                                a.err);
    EV_END(3); EV_BEGIN(4);
    if (a.S == 5)
      launch_full(k_update_fct<5>, nb, bs, 0, s, a.G, a.C, a.St, a.w.dL, a.w.muL, a.w.uL, a.w.res, a.w.fct, a.w.rminus, a.w.ab,
                                        a.u0, a.out, a.rk_stage, a.lij_out, ne, a.err);
    else
      launch_full(k_update_fct<3>, nb, bs, 0, s, a.G, a.C, a.St, a.w.dL, a.w.muL, a.w.uL, a.w.res, a.w.fct, a.w.rminus, a.w.ab,
                                        a.u0, a.out, a.rk_stage, a.lij_out, ne, a.err);
    if (a.entropy) {
      if (a.S == 5)
        launch_full(k_entropy_rows<5>, nb, bs, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.res, a.u0, a.out,
                    a.rk_stage, a.err);
      else
        launch_full(k_entropy_rows<3>, nb, bs, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.res, a.u0, a.out,
                    a.rk_stage, a.err);
    }
    EV_END(4);
    return;
  }
  launch_full(k_low_f64, nb, bs, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.dLii, a.w.muLii, a.w.uL, a.w.res, a.dij_in,
                              a.err);
  EV_END(2); EV_BEGIN(3);
  if (a.any_fct)
    launch_full(k_fct_f64, nb, bs, 0, s, a.G, a.C, a.St, a.u, a.w.dL, a.w.muL, a.w.uL, a.w.res, a.w.fct, a.w.rminus, a.err);
  EV_END(3); EV_BEGIN(4);
  launch_full(k_update_f64, nb, bs, 0, s, a.G, a.C, a.St, a.u, a.w.dL, a.w.muL, a.w.uL, a.w.res, a.w.fct, a.w.rminus, a.u0, a.out,
                                 a.rk_stage, a.lij_out, a.err);
  if (a.entropy)
    launch_full(k_entropy_f64, nb, bs, 0, s, a.G, a.C, a.St, a.u, nd, a.w.dL, a.w.muL, a.w.dLii, a.w.muLii, a.w.res, a.u0, a.out,
                                    a.rk_stage, a.err);
  EV_END(4);
}

void launch_dt_f64(const Graph& G, const InstConst* C, InstState* St, const StateF64& u, const WorkF64& node,
                   double* d_out, double* dii_out, unsigned* err, const StepTurn& turn, cudaStream_t s) {
  if (split_dt(G.n_rows, u.q3 ? 5 : 3)) {
    launch_full(k_dt_split, (unsigned)(G.n_rows / 32), 128, 0, s, G, C, St, u, node_of(node), d_out, dii_out, err, turn);
    return;
  }
  launch_full(k_dt_f64, nblk(G.n_rows, kRowBlock), kRowBlock, 0, s, G, C, St, u, node_of(node), d_out, dii_out, err, turn);
}

void launch_step_turn(const StepTurn& t, const InstConst* C, InstState* St, cudaStream_t s) {
  k_step_turn<<<nblk(t.n_inst, 128), 128, 0, s>>>(t, C, St);
}
void launch_step_end(InstState* St, int n_inst, cudaStream_t s) {
  k_step_end<<<nblk(n_inst, 128), 128, 0, s>>>(St, n_inst);
}
void launch_reset_counters(InstState* St, int n_inst, cudaStream_t s) {
  k_reset_counters<<<nblk(n_inst, 128), 128, 0, s>>>(St, n_inst);
}

void launch_fct_positivity_f64(const Graph& G, const InstConst* C, const double* unext, const double* mat,
                               const double* matii, double* rtmp, double* lij, cudaStream_t s) {
  k_fct_positivity_f64<<<nblk(G.n_rows, 128), 128, 0, s>>>(G, C, unext, mat, matii, rtmp, lij, 0);
  k_fct_positivity_f64<<<nblk(G.n_rows, 128), 128, 0, s>>>(G, C, unext, mat, matii, rtmp, lij, 1);
}

void launch_fct_generic_f64(const Graph& G, double* unext, const double* maxn, const double* minn, const double* dg,
                            const double* mat, const double* matii, double* rplus, double* rminus, cudaStream_t s) {
  k_fct_generic_f64<<<nblk(G.n_rows, 128), 128, 0, s>>>(G, unext, maxn, minn, dg, mat, matii, rplus, rminus, 0);
  k_fct_generic_f64<<<nblk(G.n_rows, 128), 128, 0, s>>>(G, unext, maxn, minn, dg, mat, matii, rplus, rminus, 1);
}


}  // namespace swe
