// Device-side data layout and per-edge physics shared by the FP64 and the
// mixed-precision kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace swe {

// Error bits raised by kernels (never a trap); the host maps them to
// SWE_ERR_* after each launch sequence.
enum : unsigned { ERRB_NEG_H = 1u, ERRB_DELTA = 2u, ERRB_NAN = 4u };

// inputs%viscosity_type (the values of SWE_VISC_* in the C ABI header)
enum : int { VISC_GALERKIN = 0, VISC_VISCOUS = 1, VISC_ENTROPY = 2, VISC_FCT = 3 };

// Per-instance constants (one record per mesh of a batch).  The FP32 copies
// are rounded once on the host: the mixed kernels never convert per row
// (a float<->double conversion issues on GB300's narrow FP64 pipe).
struct InstConst {
  double g, htiny, cfl, mannings, lambda_sgn, max_water_h, rescale_floor;
  int type_test, S, visc, viscous_type, alpha_limit, roundoff_fix;
  float gf, htinyf, htiny_lo;      // htiny = htinyf + htiny_lo (double-float)
  float fricf;                     // g n^2 (friction)
  float lambda_sgnf, rescale_floorf;
  double inv_16g;                  // 1 / (16 g), rounded once
};

// Per-instance time-loop state, device resident.
struct InstState {
  double dt, inv_dt, time, t_final;
  unsigned long long maxd_bits;   // max |d_ii|/m_i of the current step (double bits)
  int done, steps;
  float dtf, inv_dtf;             // FP32 copies of dt and inv_dt
};

__host__ __device__ inline void inst_set_dt(InstState& s, double dt) {
  s.dt = dt;
  s.inv_dt = dt > 0.0 ? 1.0 / dt : 0.0;
  s.dtf = (float)s.dt;
  s.inv_dtf = (float)s.inv_dt;
}

// The turn between two time steps: it closes the step before (end_prev: time
// = to + dt, main.f90:91) and opens the next (DO WHILE(time < Tfinal), dt =
// CFL / max, main.f90:61, 173; the fixed dt = 2.5e-2 of the Malpasset case,
// main.f90:67-69).  The last block of k_dt runs it where k_dt is a few waves
// (ticket not null: the count of its blocks that are done); the fence and the
// ticket cost a block more than a launch of its own costs a large grid (2k
// nodes: 46 -> 43 us per step; 4M nodes: k_dt 161 -> 192 us).
struct StepTurn {
  unsigned* ticket;
  int n_inst, end_prev;
};
__device__ __forceinline__ void turn_instance(const StepTurn& t, const InstConst& c, InstState& s) {
  if (s.done) return;
  if (t.end_prev) {
    s.time = s.time + s.dt;
    s.steps += 1;
  }
  if (!(s.time < s.t_final)) {
    s.done = 1;
    return;
  }
  const double mx = __longlong_as_double((long long)__ldcg(&s.maxd_bits));   // other SMs' atomics: from L2
  inst_set_dt(s, c.type_test == 9 ? 2.5e-2 : c.cfl * 1 / mx);
  s.maxd_bits = 0ull;
}
__device__ __forceinline__ void step_turn(const StepTurn& t, const InstConst* C, InstState* St) {
  if (!t.ticket) return;
  __shared__ bool last;
  __syncthreads();                               // this block's maxima ...
  if (threadIdx.x == 0) {
    __threadfence();                             // ... before its ticket
    last = atomicAdd(t.ticket, 1u) == gridDim.x - 1;
    if (last) __threadfence();
  }
  __syncthreads();
  if (!last) return;
  for (int b = threadIdx.x; b < t.n_inst; b += blockDim.x) turn_instance(t, C[b], St[b]);
  if (threadIdx.x == 0) *t.ticket = 0u;
}

// Programmatic dependent launch: a kernel launched so may start while the
// previous kernel's last blocks still run; pdl_trigger lets its dependents
// start, pdl_wait waits until the previous grid has completed and its writes
// are visible.  Completion is transitive (every kernel waits before it can
// exit), so outputs of any earlier kernel are visible after the wait.  Without
// the launch attribute both do nothing.  What an earlier kernel writes is read
// through pointers without __restrict__: a restrict pointer's loads may be moved
// above the wait.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The SELL-32 edge graph (see swe_setup.hpp).  Entry k of row r is at
// slice_ptr[r>>5] + 32*k + (r&31); entries are the off-diagonal CSR entries
// in reference order, the diagonal (c_ii) is stored per row and belongs
// between entries dpos-1 and dpos of the reference row.
struct Graph {
  int64_t n_rows;
  const int64_t* __restrict__ slice_ptr;
  const int* __restrict__ slice_inst;
  const int* __restrict__ col;
  const uint8_t* __restrict__ len;       // off-diagonal entries (0: padding row)
  const uint8_t* __restrict__ dpos;
  const double* __restrict__ cx;
  const double* __restrict__ cy;
  const double* __restrict__ cxii;
  const double* __restrict__ cyii;
  const float2* __restrict__ cf;          // mixed path, per entry: c_ij in FP32, (x, y) interleaved
  const float* __restrict__ cxiif;
  const float* __restrict__ cyiif;
  const double* __restrict__ cnorm;       // FP64 path, per entry: |c_ij| and c_ij/|c_ij|
  const double* __restrict__ cnx;         // (compute_dij's norm and normal, formed once)
  const double* __restrict__ cny;
  const float2* __restrict__ cnf;         // FP64 path, per entry: the normal in FP32
  const double* __restrict__ lumped;
  const double* __restrict__ inv_lumped;
  const float* __restrict__ lumpedf;      // FP32 copies (mixed path)
  const float* __restrict__ inv_lumpedf;
  const double* __restrict__ bath;
  const float2* __restrict__ bathdf;     // mixed path: bathymetry as a double-float pair
  const uint8_t* __restrict__ dir_mask;   // bit k: component k is Dirichlet
  const double* __restrict__ dir_val;     // (S, n_rows) SoA, read where masked
  const uint8_t* __restrict__ dir_anal;   // bit k: component k's value is sol_anal(t) (or null)
  const double* __restrict__ rr_row;      // node coordinates (x, y) per row, where dir_anal is set
};

// sol_anal(k, rr, t) (SOURCES/condlim.f90:421-456, 751-791) of the analytic
// cases whose boundary data change with time, components 1-3 (h, qx, qy):
// type 5 (Thacker's planar oscillation, with the current reference's +htiny
// film) and type 13 (the SGN solitary wave).  The operations follow the
// reference's expressions in its order; cos, sin and cosh are CUDA's.
__device__ inline double sol_anal_dev(int type_test, int k, double x, double y, double t, double g, double htiny) {
  if (type_test == 5) {
    const double a = 1.0, h0 = 0.1, hL = 4.0, eta = 0.5;
    const double omega = sqrt(2 * g * h0) / a;
    const double dx = x - hL / 2.0, dy = y - hL / 2.0;
    const double bathi = -h0 * (1.0 - (dx * dx + dy * dy) / (a * a));
    const double v = (eta * h0 / (a * a)) * (2.0 * dx * cos(omega * t) + 2.0 * dy * sin(omega * t)) - bathi;
    const double base = v > 0.0 ? v : 0.0;
    if (k == 1) return base + htiny;
    if (k == 2) return -eta * omega * sin(omega * t) * base;
    return eta * omega * cos(omega * t) * base;
  }
  // type 13
  const double h1 = 10.0 / 100.0, h2 = 11.0 / 100.0, x0 = 2.75;
  const double D = sqrt(g * h2);
  const double z = sqrt((3.0 * (h2 - h1)) / (h2 * (h1 * h1)));
  const double arg = 1.0 / 2.0 * z * (x - x0 - D * t);
  const double se = 1.0 / cosh(arg);
  const double hv = h1 + (h2 - h1) * (se * se);
  const double ht = hv > 0.0 ? hv : 0.0;
  if (k == 1) return ht;
  if (k == 2) return ht * D - h1 * D;
  return ht * 0.0;
}

// Value bdy (main.f90:176-188) writes into component q of row r after RK
// stage rk_stage of the device loop: the fixed value, or sol_anal at the
// reference's bdy time of that stage (main.f90:78, 84, 90: to + dt, then
// (to + dt) + dt/2, then (to + dt/2) + dt).
__device__ inline double dirichlet_value(const Graph& G, const InstConst& c, const InstState& st, int rk_stage, int q,
                                         int64_t r) {
  if (G.dir_anal && ((G.dir_anal[r] >> q) & 1u)) {
    const double to = st.time, dt = st.dt;
    const double t = rk_stage == 1 ? to + dt : (rk_stage == 2 ? (to + dt) + dt / 2 : (to + dt / 2) + dt);
    return sol_anal_dev(c.type_test, q + 1, G.rr_row[2 * r], G.rr_row[2 * r + 1], t, c.g, c.htiny);
  }
  return G.dir_val[(int64_t)q * G.n_rows + r];
}

__device__ __forceinline__ int64_t entry_base(const Graph& G, int64_t r) {
  return G.slice_ptr[r >> 5] + (r & 31);
}

// FP32 shadow of an FP64 depth that keeps the sign of (h - htiny) and of h:
// the mixed kernels branch on h <= htiny and h <= 0 (SOURCES/update.f90:572-582,
// 644-655) with the shadow, so both branch decisions must match the FP64 depth.
__device__ __forceinline__ float shadow_depth(double h, double htiny) {
  float f = (float)h;
  const float ft = (float)htiny;
  if (h > htiny && !(f > ft)) f = nextafterf(ft, 3.4e38f);
  if (h > 0.0 && !(f > 0.0f)) f = 1.17549435e-38f;   // smallest normal (FTZ-safe)
  return f;
}

// ---- double-float arithmetic (value = x + y, two FP32 words, |y| <= ulp(x)/2)
// Knuth's two-sum and the FMA two-product, written with explicit roundings so
// that no contraction changes them.  About 48 significant bits; every
// operation issues on the FP32 pipes.
__device__ __forceinline__ float2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return make_float2(s, e);
}
__device__ __forceinline__ float2 df_from_double(double v) {
  const float hi = __double2float_rn(v);
  return make_float2(hi, __double2float_rn(v - (double)hi));
}
__device__ __forceinline__ double df_to_double(float2 a) { return (double)a.x + (double)a.y; }
__device__ __forceinline__ float2 df_add_f(float2 a, float b) {     // a + b
  const float2 t = two_sum(a.x, b);
  return two_sum(t.x, __fadd_rn(t.y, a.y));
}
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {      // a + b
  const float2 t = two_sum(a.x, b.x);
  return two_sum(t.x, __fadd_rn(t.y, __fadd_rn(a.y, b.y)));
}
__device__ __forceinline__ float2 df_mul_f(float2 a, float b) {     // a * b
  const float p = __fmul_rn(a.x, b);
  const float e = __fmaf_rn(a.y, b, __fmaf_rn(a.x, b, -p));
  return two_sum(p, e);
}
__device__ __forceinline__ float2 df_scale(float2 a, float pow2) {  // a * 2^k, exact
  return make_float2(__fmul_rn(a.x, pow2), __fmul_rn(a.y, pow2));
}
__device__ __forceinline__ float2 df_div3(float2 a) {               // a / 3
  const float q1 = __fdiv_rn(a.x, 3.0f);
  const float r = __fadd_rn(__fmaf_rn(-3.0f, q1, a.x), a.y);      // a.x - 3 q1 is exact
  return two_sum(q1, __fdiv_rn(r, 3.0f));
}
// a > (hi + lo) for normalised pairs
__device__ __forceinline__ bool df_gt(float2 a, float hi, float lo) { return a.x > hi || (a.x == hi && a.y > lo); }

template <typename T> __device__ __forceinline__ T tmax(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T tmin(T a, T b) { return a < b ? a : b; }
template <typename T> __device__ __forceinline__ T tabs(T a) { return a < T(0) ? -a : a; }

// compute_one_over_h (SOURCES/condlim.f90:79-90): 2h/(h^2 + max(h,htiny)^2)
template <typename T> __device__ __forceinline__ T one_over_h(T h, T htiny) {
  T mh = tmax(h, htiny);
  return T(2) * h / (h * h + mh * mh);
}

// Per-call constants of compute_lambda_vacc, formed once per thread with the
// reference's own expressions (so every use sees the value the reference
// forms at that point).
template <typename T>
struct LamConstF64 {
  T x0;              // (2 sqrt2 - 1)^2
  T a, two_a;        // 1/(2 sqrt2), 2 a
  T sixteen_g;       // 16 g
  T two_sqrt_g;      // 2 sqrt(g)
  T sqrt_2_over_g;   // sqrt(2/g)
  T g_half;          // g/2
};
template <typename T>
__device__ __forceinline__ LamConstF64<T> lam_const_f64(T g, T sqrt2) {
  LamConstF64<T> k;
  const T t0 = T(2) * sqrt2 - T(1);
  k.x0 = t0 * t0;
  k.a = T(1) / (T(2) * sqrt2);
  k.two_a = T(2) * k.a;
  k.sixteen_g = T(16) * g;
  k.two_sqrt_g = T(2) * sqrt(g);
  k.sqrt_2_over_g = sqrt(T(2) / g);
  k.g_half = g / T(2);
  return k;
}

// phi (SOURCES/condlim.f90:960-981).  The node terms one_over_h(hl),
// one_over_h(hr) and sqrt(g hl), sqrt(g hr) are the nodes' per-node values
// (ovhl, ovhr; sqghl = sqrt(g |hl|) equals sqrt(g hl) for hl > 0, and is
// recomputed otherwise), so each is formed once per node instead of per
// entry and per call; one_over_h(h) and sqrt(g h) are formed once per call.
template <typename T>
__device__ __forceinline__ T phi_fn(T h, T ul, T hl, T ur, T hr, T g, T htiny, T ovhl, T ovhr, T sqghl, T sqghr,
                                    T g_half) {
  const bool shock_l = h > hl, shock_r = h > hr;
  const T ovh = (shock_l || shock_r) ? one_over_h(h, htiny) : T(0);
  const T sgh = (!shock_l || !shock_r) ? sqrt(g * h) : T(0);
  T fl, fr;
  if (shock_l) fl = (h - hl) * sqrt(g_half * (ovh + ovhl));
  else fl = T(2) * (sgh - (hl > T(0) ? sqghl : sqrt(g * hl)));
  if (shock_r) fr = (h - hr) * sqrt(g_half * (ovh + ovhr));
  else fr = T(2) * (sgh - (hr > T(0) ? sqghr : sqrt(g * hr)));
  return fl + fr + ur - ul;
}

// compute_lambda_vacc (SOURCES/condlim.f90:879-957) with the node values
// ovhl/ovhr (one_over_h) and sqghl/sqghr (sqrt(g |h|), the reference's
// sql/sqr) passed in; they equal what the reference forms bit for bit.
// Returns false where the reference STOPs (Delta < 0).
template <typename T>
__device__ __forceinline__ bool lambda_vacc(T hl, T qxl, T qyl, T ovhl, T sqghl, T hr, T qxr, T qyr, T ovhr, T sqghr,
                                            T nx, T ny, T g, T htiny, const LamConstF64<T>& k, T* lambda) {
  T vl = (qxl * nx + qyl * ny) * ovhl;
  T vr = (qxr * nx + qyr * ny) * ovhr;
  const T sql = sqghl, sqr = sqghr;
  T hmin, hmax;
  if (hl <= hr) { hmin = hl; hmax = hr; } else { hmin = hr; hmax = hl; }
  T ht;
  bool ok = true;
  T fh = phi_fn(k.x0 * hmin, vl, hl, vr, hr, g, htiny, ovhl, ovhr, sql, sqr, k.g_half);
  if (T(0) <= fh) {
    T s = tmax(vl - vr + T(2) * sql + T(2) * sqr, T(0));
    ht = tmin(k.x0 * hmin, s * s / k.sixteen_g);
  } else {
    fh = phi_fn(k.x0 * hmax, vl, hl, vr, hr, g, htiny, ovhl, ovhr, sql, sqr, k.g_half);
    T sqrmin = sqrt(hmin), sqrmax = sqrt(hmax);
    if (T(0) <= fh) {
      T c = -(hmin * k.a) - sqrmin * sqrmax + sqrmin * (vr - vl) / k.two_sqrt_g;
      T Delta = hmin - T(4) * k.a * c;
      if (Delta < T(0)) { ok = false; Delta = T(0); }
      T s = (-sqrmin + sqrt(Delta)) / k.two_a;
      ht = tmin(k.x0 * hmax, s * s);
    } else {
      ht = sqrmin * sqrmax * (T(1) + k.sqrt_2_over_g * (vl - vr) / (sqrmin + sqrmax));
    }
  }
  T lbdl = vl - sql * sqrt((T(1) + tmax((ht - hl) * ovhl / T(2), T(0))) * (T(1) + tmax((ht - hl) * ovhl, T(0))));
  T lbdr = vr + sqr * sqrt((T(1) + tmax((ht - hr) * ovhr / T(2), T(0))) * (T(1) + tmax((ht - hr) * ovhr, T(0))));
  *lambda = tmax(tabs(lbdl), tabs(lbdr));
  return ok;
}

// ---- FP64 arithmetic on GB300: an FP64 instruction (add, multiply, compare,
// conversion) holds an SM's FP64 unit for 16 cycles per warp, an integer or
// FP32 one a quarter to half a cycle.  The FP64 kernels therefore compare and
// select with integer instructions on the bits, divide by values whose
// reciprocal is known with three FP64 instructions instead of about seven,
// and decide in FP32, with error bounds, which of the reference's branches
// can matter before they evaluate one in FP64.  Every result keeps the
// reference's bits (the sign of a zero aside).
__device__ __forceinline__ long long bits64(double x) { return __double_as_longlong(x); }
// Marks a block that a warp skips when none of its lanes need it: without side
// effects the compiler forms both sides of a short branch and selects, which
// costs FP64 instructions.
__device__ __forceinline__ void real_branch() { asm volatile("" ::); }
// MAX(x, 0)
__device__ __forceinline__ double pos_part(double x) { return bits64(x) > 0 ? x : 0.0; }
// MAX, MIN of non-negative values
__device__ __forceinline__ double max_nn(double a, double b) { return bits64(a) > bits64(b) ? a : b; }
__device__ __forceinline__ double min_nn(double a, double b) { return bits64(a) < bits64(b) ? a : b; }
// Entropy residuals, not negative or NaN (0/0 at rest with max_water_h = 0).  A
// NaN is kept with its sign bit set: above every residual as an unsigned
// integer and below as a signed one, so that MAX(res_i, res_j) and MIN(d, res_ij)
// in the general kernels' comparisons (a > b ? a : b, a < b ? a : b) pass on a
// NaN of the neighbour at no instruction per entry.  own_res: the row's own, whose
// NaN the comparison drops.
__device__ __forceinline__ double keep_res(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) > 0x7ff00000u ? __longlong_as_double(0xfff8000000000000ll) : x;
}
__device__ __forceinline__ double own_res(double res) { return bits64(res) < 0 ? 0.0 : res; }
__device__ __forceinline__ double max_res(double own, double res) {
  return (unsigned long long)bits64(own) > (unsigned long long)bits64(res) ? own : res;
}
// h <= t for t >= 0 and any h
__device__ __forceinline__ bool le_nn(double h, double t) { return bits64(h) <= bits64(t); }
// integers in the order of the doubles
__device__ __forceinline__ long long order_key(double x) {
  const long long b = bits64(x);
  return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
__device__ __forceinline__ double max_any(double a, double b) { return order_key(a) > order_key(b) ? a : b; }
__device__ __forceinline__ double min_any(double a, double b) { return order_key(a) < order_key(b) ? a : b; }

// a / b correctly rounded, given y = 1/b correctly rounded: q = RN(a y) is
// within 1.5 units in the last place of a/b, r = a - b q is exact, and
// RN(q + r y) is RN(a / b) (Markstein, IBM J. Res. Dev. 34(1), 1990;
// Brisebarre, Muller and Raina, IEEE Trans. Comput. 53(8), 2004) while no
// intermediate leaves the normal range: a is 0 or within 2^+-600 and y within
// 2^+-400, else the ordinary division.
__host__ __device__ __forceinline__ bool div_range(unsigned hi_a, unsigned lo_a, unsigned hi_y) {
  const unsigned ea = (hi_a >> 20) & 0x7ffu, ey = (hi_y >> 20) & 0x7ffu;
  return (ea - 423u <= 1200u || ((hi_a << 1) | lo_a) == 0u) && ey - 623u <= 800u;
}
__device__ __forceinline__ double div_known(double a, double b, double y) {
  if (div_range((unsigned)__double2hiint(a), (unsigned)__double2loint(a), (unsigned)__double2hiint(y))) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
  }
  return a / b;
}

// The general evaluation, out of line: the states the FP32 tests of
// lambda_row cannot settle (thin films, depth ratios above 3.34, strong
// compression).
static __device__ __noinline__ double lambda_general(double hl, double qxl, double qyl, double ovhl, double sqghl,
                                                     double hr, double qxr, double qyr, double ovhr, double sqghr,
                                                     double nx, double ny, double g, double htiny, bool* ok) {
  const LamConstF64<double> k = lam_const_f64(g, sqrt(2.0));
  double lam;
  *ok = lambda_vacc(hl, qxl, qyl, ovhl, sqghl, hr, qxr, qyr, ovhr, sqghr, nx, ny, g, htiny, k, &lam);
  return lam;
}

// A state as compute_lambda_vacc sees it, and its FP32 shadow
// (h, sqrt(g |h|), q one_over_h).
struct LamState {
  double h, q1, q2, ovh, sq;
  float4 f;
};

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float one_over_h_f(float h, float htiny) {
  const float m = fmaxf(h, htiny);
  return __fdividef(2.f * h, h * h + m * m);
}

// phi(x0 hmin) >= 0 for certain, from phi in FP32 (within 2e-6 M): a dam front
// or a bank, where the depths differ by more than x0
__device__ __forceinline__ bool rarefactions_f(const LamState& l, const LamState& r, float lv, float rv, float hmin,
                                               float hmax, float M, const InstConst& c) {
  const float hx = 3.3431458f * hmin, ox = one_over_h_f(hx, c.htinyf), cx = sqrt_approx(c.gf * hx), hg = 0.5f * c.gf;
  const float fl = hx > l.f.x ? (hx - l.f.x) * sqrt_approx(hg * (ox + one_over_h_f(l.f.x, c.htinyf)))
                              : 2.f * (cx - l.f.y);
  const float fr = hx > r.f.x ? (hx - r.f.x) * sqrt_approx(hg * (ox + one_over_h_f(r.f.x, c.htinyf)))
                              : 2.f * (cx - r.f.y);
  return fl + fr + (rv - lv) > 1e-5f * M && hmin > 1e-18f && hmax < 1e18f && bits64(l.h) > 0 && bits64(r.h) > 0;
}

// compute_lambda_vacc (SOURCES/condlim.f90:879-957) with the same bits and
// about a third of the FP64 instructions (the bound of k_dt_f64 and
// k_low_fct).  With c = sqrt(g h):
//  * a node with h = 0 makes ht = 0 in every branch and has v = c = 0 itself:
//    lambda is the other node's |v -+ c|.
//  * phi(x0 hmin) >= 0, the two-rarefaction branch, is certain when
//    x0 hmin > hmax (both terms of phi are shocks, so >= 0) and vl - vr is at
//    most the term of hmin alone: (x0 - 1) sqrt((1 + 1/x0) / 2) c_min =
//    1.8884 c_min for hmin >= htiny, at least (x0 - 1) / sqrt(2 x0) c_min =
//    0.9061 c_min where only x0 hmin >= htiny.  phi's square roots and
//    division are not formed.
//    Else FP32 forms phi(x0 hmin) itself (rarefactions_f): dam break of 10k
//    nodes, first steps, k_dt 32 -> 17 and k_low 46 -> 38 us.
//  * sqrt((1 + max(x/2, 0)) (1 + max(x, 0))) is 1 exactly where ht <= h.
//  * only the larger of |lambda_l| and |lambda_r| is formed where FP32 tells
//    them apart.
// FP32 bounds: with V = sum |v| and M = V + 2 (c_l + c_r) the FP32 velocities
// are within 5e-7 V, c and s within 5e-7 M and the two speeds within 2e-6 M;
// the tests use 2e-6 V, 2e-6 M and 1e-5 M.  What is not certain is evaluated
// in full.
__device__ __forceinline__ bool lambda_row(const LamState& l, const LamState& r, double nx, double ny, float2 nf,
                                           const InstConst& c, double* lambda) {
  const float lv = nf.x * l.f.z + nf.y * l.f.w, rv = nf.x * r.f.z + nf.y * r.f.w;
  const float V = fabsf(l.f.z) + fabsf(l.f.w) + fabsf(r.f.z) + fabsf(r.f.w);
  const float M = V + 2.f * (l.f.y + r.f.y);
  const float tol = 2e-6f * M;
  const float hmin = fminf(l.f.x, r.f.x), hmax = fmaxf(l.f.x, r.f.x);
  const float kmin = hmin > 1.00001f * c.htinyf ? 1.888f : (3.3431f * hmin > 1.00001f * c.htinyf ? 0.906f : 0.f);
  if (!(3.3431f * hmin > hmax && (lv - rv) + 2e-6f * V <= kmin * fminf(l.f.y, r.f.y) && hmin > 1e-18f &&
        hmax < 1e18f) &&
      !rarefactions_f(l, r, lv, rv, hmin, hmax, M, c)) {
    const bool dry_l = (bits64(l.h) << 1) == 0, dry_r = (bits64(r.h) << 1) == 0;
    if ((dry_l || dry_r) && bits64(l.h) >= 0 && bits64(r.h) >= 0 && bits64(c.htiny) > 0 && V < 1e30f) {
      const double qx = dry_l ? r.q1 : l.q1, qy = dry_l ? r.q2 : l.q2, o = dry_l ? r.ovh : l.ovh;
      const double v = __dmul_rn(__dadd_rn(__dmul_rn(qx, nx), __dmul_rn(qy, ny)), o);
      *lambda = fabs(dry_l ? __dadd_rn(v, r.sq) : __dsub_rn(v, l.sq));
      return true;
    }
    bool ok;
    *lambda = lambda_general(l.h, l.q1, l.q2, l.ovh, l.sq, r.h, r.q1, r.q2, r.ovh, r.sq, nx, ny, c.g, c.htiny, &ok);
    return ok;
  }
  const float s = (lv - rv) + 2.f * (l.f.y + r.f.y);
  const float i16g = 0.0625f / c.gf;
  const float su = fmaxf(s + tol, 0.f), sm = fmaxf(s, 0.f);
  const float hup = su * su * i16g * 1.000002f;                         // ht <= hup
  const float hst = fminf(sm * sm * i16g, 3.3431458f * hmin);
  const bool triv_l = hup <= l.f.x * 0.999998f, triv_r = hup <= r.f.x * 0.999998f;
  const float xl = fmaxf((hst - l.f.x) * one_over_h_f(l.f.x, c.htinyf), 0.f);
  const float xr = fmaxf((hst - r.f.x) * one_over_h_f(r.f.x, c.htinyf), 0.f);
  const float al = fabsf(lv - l.f.y * sqrt_approx((1.f + 0.5f * xl) * (1.f + xl)));
  const float ar = fabsf(rv + r.f.y * sqrt_approx((1.f + 0.5f * xr) * (1.f + xr)));
  const float tl = 1e-5f * M;
  const bool need_l = !(ar > al + tl), need_r = !(al > ar + tl);
  // the side evaluated first: l unless r is the larger for certain
  const bool both = need_l && need_r;
  const bool tr1 = need_l ? triv_l : triv_r;
  const double h1 = need_l ? l.h : r.h, o1 = need_l ? l.ovh : r.ovh, c1 = need_l ? l.sq : r.sq;
  const double v1 = __dmul_rn(__dadd_rn(__dmul_rn(need_l ? l.q1 : r.q1, nx), __dmul_rn(need_l ? l.q2 : r.q2, ny)), o1);
  double f1 = 1.0, v2 = 0.0, ht = 0.0;
  const bool nt = !tr1 || (both && !triv_r);
  if (nt || both) {
    real_branch();
    const double o2 = need_l ? r.ovh : l.ovh;
    v2 = __dmul_rn(__dadd_rn(__dmul_rn(need_l ? r.q1 : l.q1, nx), __dmul_rn(need_l ? r.q2 : l.q2, ny)), o2);
  }
  if (nt) {
    real_branch();
    const double vl = need_l ? v1 : v2, vr = need_l ? v2 : v1;
    // ((vl - vr) + 2 sql) + 2 sqr, each product by 2 exact
    const double sd = pos_part(__fma_rn(2.0, r.sq, __fma_rn(2.0, l.sq, __dsub_rn(vl, vr))));
    ht = div_known(__dmul_rn(sd, sd), 16.0 * c.g, c.inv_16g);
    if (!(hup < 3.3431f * hmin)) {
      const double t0 = 2.0 * sqrt(2.0) - 1.0;
      ht = tmin((t0 * t0) * tmin(l.h, r.h), ht);
    }
    if (!tr1) {
      real_branch();
      const double x = pos_part(__dmul_rn(__dsub_rn(ht, h1), o1));
      f1 = sqrt(__dmul_rn(__fma_rn(x, 0.5, 1.0), __dadd_rn(1.0, x)));   // x/2 is exact
    }
  }
  double cf = tr1 ? c1 : __dmul_rn(c1, f1);
  double lam = fabs(need_l ? __dsub_rn(v1, cf) : __dadd_rn(v1, cf));
  if (both) {
    real_branch();
    double f2 = f1;
    if (bits64(l.h) != bits64(r.h)) {                     // equal depths: equal factors
      f2 = 1.0;
      if (!triv_r) {
        const double x = pos_part(__dmul_rn(__dsub_rn(ht, r.h), r.ovh));
        f2 = sqrt(__dmul_rn(__fma_rn(x, 0.5, 1.0), __dadd_rn(1.0, x)));
      }
    }
    lam = max_nn(lam, fabs(__dadd_rn(v2, __dmul_rn(r.sq, f2))));
  }
  *lambda = lam;
  return true;
}

}  // namespace swe
