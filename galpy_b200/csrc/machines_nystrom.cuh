// galpy_b200/csrc/machines_nystrom.cuh
//
// The Runge-Kutta machines of orbits (machines.cuh's RKMachine, Dopr54Machine
// and Dop853Machine on OrbitSystem) in Nystrom form.  An orbit's equation is
// of second order, x'' = a(x, t), and every scheme's stage positions are
// combinations of the stage accelerations alone (dop853_nystrom.cuh):
//
//   * half the stage values are kept and a little over half of the stage
//     arithmetic is left;
//   * the position of stage i does not depend on the acceleration of stage
//     i - 1, so a machine asks for TWO forces at a time,
//
//         m.point2(q1, q2, slot);            // two positions
//         eval_force2<...>(..., a1, a2);     // the kernel's one call site
//         m.consume2(q1, q2, a1, a2, out, slot);
//
//     whose dependent chains overlap in one thread.  The schemes split into
//     pairs without a gap: rk4 (1,2)(3,4); dopr54 (2,3)(4,5)(6,7); dop853
//     (2,3)(4,5)(6,7)(8,9)(10,11)(12,13), the 13th being the derivative at
//     the new state; its dense output (14,15)(16).  rk6 has seven stages and
//     evaluates its last one twice.
//
// The chain of one force is what bounds a thread (a DOP853 step of a lone
// warp took 35,800 cycles at one force a time), so pairing is worth more than
// what it wastes: the 13th force of a rejected dop853 attempt, rk6's eighth.
// Measured on a B200, first-order form -> this one: dop853, 1,048,576 orbits
// with their own end times 908 -> 569 ms, one orbit of 1,165 steps 21.5 ->
// 14.6 ms, 262,143 orbits in 96 parameter groups 64.4 -> 51.0 ms; rk4,
// 100,001 orbits x 2,000 steps 38.6 -> 25.3 ms; dopr54 in the full run-time
// list, which pairs the usual components and the Dehnen bar (potentials.cuh,
// sum2), 3,000 orbits in MWPotential2014 with a bar 65.8 -> 36.9 ms.
//
// The steps are the first-order form's up to rounding: same error estimates,
// controller, step estimators, force times, dense output and status codes
// (references in machines.cuh).  Surfaces of section are first-order systems
// and stay with machines.cuh, and so does dop853 in the full run-time list
// (orbit_kernels_dop853.cu).
#pragma once
#include <type_traits>
#include <utility>

#include "dop853_nystrom.cuh"
#include "machines.cuh"

namespace gpc {

template <int... K>
using Ints = std::integer_sequence<int, K...>;
template <int N>
using Count = std::make_integer_sequence<int, N>;

// a b + c as one fused operation in device code.  A sum of two products leaves
// the compiler a choice of which to fuse; where the same step is compiled more
// than once (register variants, the queued and the plain loop) it is spelled
// out, so that all give the same bits.
GPC_HD GPC_FI double mad(double a, double b, double c)
{
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return a * b + c;
#endif
}

// (x, v[, dx, dv]) rows <-> the second-order system's position and velocity
// vectors x = (x[, dx]), v = (v[, dv])
template <int D, bool VAR>
GPC_HD GPC_FI void split_row(const double* w, double* x, double* v)
{
#pragma unroll
  for (int k = 0; k < D; k++) {
    x[k] = w[k];
    v[k] = w[D + k];
    if (VAR) {
      x[D + k] = w[2 * D + k];
      v[D + k] = w[3 * D + k];
    }
  }
}
template <int D, bool VAR>
GPC_HD GPC_FI void join_row(const double* x, const double* v, double* w)
{
#pragma unroll
  for (int k = 0; k < D; k++) {
    w[k] = x[k];
    w[D + k] = v[k];
    if (VAR) {
      w[2 * D + k] = x[D + k];
      w[3 * D + k] = v[D + k];
    }
  }
}

// est_scale over a split state (the maximum does not depend on the order)
template <int NQ>
GPC_HD GPC_FI double est_scale2(const double* x, const double* v, double rtol, double atol)
{
  double w[2 * NQ];
#pragma unroll
  for (int k = 0; k < NQ; k++) {
    w[k] = x[k];
    w[NQ + k] = v[k];
  }
  return est_scale(w, 2 * NQ, 1, rtol, atol);
}

// The common part of the machines below.
template <int D, bool VAR>
struct PairMachine : OrbitCommon {
  static constexpr int NQ = VAR ? 2 * D : D;  // positions of the second-order system
  static constexpr int N = 2 * NQ;
  static constexpr int NY = NQ;  // one force argument
  static constexpr int NV = N;
  static constexpr int NA = NQ;
  static constexpr int kRow = ROW_ORBIT;
  static constexpr bool kPair = true;

  GPC_HD GPC_FI void reset(const double* tt, int nt_, long long max_att)
  {
    t = tt;
    nt = nt_;
    iout = 0;
    err = E_OK;
    done = false;
    nsteps = 0;
    attempts = 0;
    max_attempts = max_att;
  }
};

// ------------------------------------------------------------------------
// rk4
// ------------------------------------------------------------------------
// One step of bovy_rk4_onestep (bovy_rk.c:142-170) from (x, v): round 0 the
// forces a1, a2 at x and x + h v / 2, round 1 a3, a4 at x + h v / 2 +
// h^2 a1 / 4 and x + h v + h^2 a2 / 2.
template <int NQ>
struct Rk4Nystrom {
  static constexpr int kRounds = 2;
  double a[2][NQ];
  GPC_HD GPC_FI void point2(int r, double h, const double* x, const double* v, double* q1,
                            double* q2) const
  {
    const double h2 = 0.5 * h, g1 = r ? h2 * h2 : 0.0, g2 = r ? h * h2 : 0.0;
    const double c1 = r ? h2 : 0.0, c2 = r ? h : h2;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      q1[k] = x[k] + (c1 * v[k] + g1 * a[0][k]);
      q2[k] = x[k] + (c2 * v[k] + g2 * a[1][k]);
    }
  }
  // the step's last round: (x1, v1)
  GPC_HD GPC_FI void finish(double h, const double* x, const double* v, const double* a3,
                            const double* a4, double* x1, double* v1) const
  {
    const double h6 = h / 6., hh6 = h * h6;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      const double s = a[0][k] + a[1][k] + a3[k];
      x1[k] = x[k] + (h * v[k] + hh6 * s);
      v1[k] = v[k] + h6 * (s + (a[1][k] + a3[k]) + a4[k]);
    }
  }
  GPC_HD GPC_FI void start()
  {
#pragma unroll
    for (int k = 0; k < NQ; k++) a[0][k] = a[1][k] = 0.0;
  }
  GPC_HD GPC_FI void keep(int, const double* a1, const double* a2)
  {
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      a[0][k] = a1[k];
      a[1][k] = a2[k];
    }
  }
  GPC_HD GPC_FI static void times(int r, double tb, double h, double& t1, double& t2)
  {
    t1 = r ? tb + h / 2. : tb;
    t2 = r ? tb + h : tb + h / 2.;
  }
};

// ------------------------------------------------------------------------
// rk6
// ------------------------------------------------------------------------
// bovy_rk6_onestep (bovy_rk.c:256-327): its tableau's square gives the stage
// positions x + c_i h v + h^2 sum X_ik a_k; the seventh stage's acceleration
// enters the velocity only.
namespace rk6n {
constexpr double A[8][6] = {{0, 0, 0, 0, 0, 0},
                            {1. / 3, 0, 0, 0, 0, 0},
                            {0, 2. / 3, 0, 0, 0, 0},
                            {1. / 12, 1. / 3, -1. / 12, 0, 0, 0},
                            {-1. / 16, 9. / 8, -3. / 16, -3. / 8, 0, 0},
                            {0, 9. / 8, -3. / 8, -3. / 4, 1. / 2, 0},
                            {9. / 44, -9. / 11, 63. / 44, 18. / 11, 0, -16. / 11},
                            {11. / 120, 0, 27. / 40, 27. / 40, -4. / 15, -4. / 15}};
constexpr double C[7] = {0, 1. / 3, 2. / 3, 1. / 3, 1. / 2, 1. / 2, 1};
constexpr double kB7 = 11. / 120;
// X_ik, i = 0..6 the stages' positions, i = 7 the new state's (whose seventh
// weight multiplies row 6)
GPC_HD constexpr double X(int i, int k)
{
  double s = 0.0;
  for (int j = 0; j < 6; j++) s += A[i][j] * A[j][k];
  if (i == 7) s += kB7 * A[6][k];
  return s > -1e-15 && s < 1e-15 ? 0.0 : s;
}
}  // namespace rk6n

template <int NQ>
struct Rk6Nystrom {
  static constexpr int kRounds = 4;
  double a[6][NQ];
  GPC_HD GPC_FI void start() {}

  template <int I, int K>
  GPC_HD GPC_FI void term(double* s) const
  {
    constexpr double w = rk6n::X(I, K);
    if constexpr (w != 0.0) {
#pragma unroll
      for (int k = 0; k < NQ; k++) s[k] += w * a[K][k];
    }
  }
  template <int I, int... K>
  GPC_HD GPC_FI void stage(double h, const double* x, const double* v, double* q, Ints<K...>) const
  {
    double s[NQ];
#pragma unroll
    for (int k = 0; k < NQ; k++) s[k] = 0.0;
    (term<I, K>(s), ...);
    constexpr double c = I < 7 ? rk6n::C[I < 7 ? I : 0] : 1.0;
#pragma unroll
    for (int k = 0; k < NQ; k++) q[k] = x[k] + h * (c * v[k] + h * s[k]);
  }
  GPC_HD GPC_FI void point2(int r, double h, const double* x, const double* v, double* q1,
                            double* q2) const
  {
    using S = Count<6>;
    switch (r) {
      case 0:
        stage<0>(h, x, v, q1, S());
        stage<1>(h, x, v, q2, S());
        break;
      case 1:
        stage<2>(h, x, v, q1, S());
        stage<3>(h, x, v, q2, S());
        break;
      case 2:
        stage<4>(h, x, v, q1, S());
        stage<5>(h, x, v, q2, S());
        break;
      default:
        stage<6>(h, x, v, q1, S());
#pragma unroll
        for (int k = 0; k < NQ; k++) q2[k] = q1[k];
    }
  }
  GPC_HD GPC_FI void keep(int r, const double* a1, const double* a2)
  {
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      if (r == 0) {
        a[0][k] = a1[k];
        a[1][k] = a2[k];
      } else if (r == 1) {
        a[2][k] = a1[k];
        a[3][k] = a2[k];
      } else {
        a[4][k] = a1[k];
        a[5][k] = a2[k];
      }
    }
  }
  GPC_HD GPC_FI void finish(double h, const double* x, const double* v, const double* a7,
                            const double*, double* x1, double* v1) const
  {
    stage<7>(h, x, v, x1, Count<6>());
#pragma unroll
    for (int k = 0; k < NQ; k++)
      v1[k] = v[k] + h * (11. / 120. * (a[0][k] + a7[k]) + 27. / 40. * (a[2][k] + a[3][k]) -
                          4. / 15. * (a[4][k] + a[5][k]));
  }
  GPC_HD GPC_FI static void times(int r, double tb, double h, double& t1, double& t2)
  {
    t1 = r == 0 ? tb : (r == 1 ? tb + 2. * h / 3. : (r == 2 ? tb + h / 2. : tb + h));
    t2 = r <= 1 ? tb + h / 3. : (r == 2 ? tb + h / 2. : tb + h);
  }
};

// rk4 / rk6 with galpy's step estimators (RKMachine of machines.cuh)
template <int D, bool VAR, int ORD>
struct RKMachine<D, VAR, ORD, OrbitSystem<D, VAR>> : PairMachine<D, VAR> {
  using B = PairMachine<D, VAR>;
  using B::NQ;
  using Step = std::conditional_t<ORD == 4, Rk4Nystrom<NQ>, Rk6Nystrom<NQ>>;
  static constexpr int kRadialBlocks = ORD == 4 ? 4 : 3;  // orbit_kernel.cuh, default_blocks
  static constexpr int kSlotDoubles = 0;
  GPC_HD GPC_FI void bind(double*) {}
  GPC_HD GPC_FI bool wants_dense() const { return false; }
  GPC_HD GPC_FI static int next_slot(int slot, bool) { return slot; }
  enum { EST_A = 0, EST_B = 1, EST_C = 2, MAIN = 3 };
  double xo[NQ], vo[NQ];  // the last completed step's state
  double xs[NQ], vs[NQ];  // start of the running step (the estimator's second half step)
  double y1[2 * NQ];      // estimator: the one-step result
  Step st;
  double dt, init_dt, h, s, rtol, atol;
  double tk;  // the reference's `to` of the main loop (bovy_rk.c: += dt per step)
  long long nrun, step;
  int round, phase;

  GPC_HD GPC_FI void times2(double& t1, double& t2, int /*slot*/) const
  {
    const double tb = phase == MAIN ? tk : (phase == EST_C ? this->t[0] + dt / 2. : this->t[0]);
    Step::times(round, tb, h, t1, t2);
  }

  GPC_HD GPC_FI void start(const double* x, const double* v, double hh)
  {
    h = hh;
    round = 0;
    st.start();
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      xs[k] = x[k];
      vs[k] = v[k];
    }
  }

  GPC_HD GPC_FI void begin_main()
  {
    const long long ndt = (long long)(init_dt / dt);
    nrun = ndt < 1 ? 1 : ndt;
    step = 0;
    phase = MAIN;
    tk = this->t[0];
    start(xo, vo, dt);
  }

  template <class W>
  GPC_HD GPC_FI void row_out(W& out) const
  {
    double w[B::NV];
    join_row<D, VAR>(xo, vo, w);
    out(this->iout, w);
  }

  template <class W>
  GPC_HD void init(const double* w, const double* tt, int nt_, double dt_in, double rtol_,
                   double atol_, long long max_att, W& out)
  {
    this->reset(tt, nt_, max_att);
    rtol = rtol_;
    atol = atol_;
    split_row<D, VAR>(w, xo, vo);
    row_out(out);
    if (nt_ < 2) {
      this->done = true;
      return;
    }
    init_dt = tt[1] - tt[0];
    if (dt_in == kDtSentinel) {
      dt = init_dt;
      s = est_scale2<NQ>(xo, vo, rtol, atol);
      phase = EST_A;
      start(xo, vo, dt);
    } else {
      dt = dt_in;
      begin_main();
    }
  }

  GPC_HD GPC_FI void point2(double* q1, double* q2, int /*slot*/) const
  {
    st.point2(round, h, xs, vs, q1, q2);
  }

  template <class W>
  GPC_HD void consume2(const double*, const double*, const double* a1, const double* a2, W& out,
                       int /*slot*/)
  {
    if (round < Step::kRounds - 1) {
      st.keep(round, a1, a2);
      round++;
      return;
    }
    double x1[NQ], v1[NQ];
    st.finish(h, xs, vs, a1, a2, x1, v1);
    // rk4_estimate_step / rk6_estimate_step (bovy_rk.c:328-480): one step of
    // dt against two of dt/2
    if (phase == EST_A) {
#pragma unroll
      for (int k = 0; k < NQ; k++) {
        y1[k] = x1[k];
        y1[NQ + k] = v1[k];
      }
      phase = EST_B;
      start(xo, vo, dt / 2.);
      return;
    }
    if (phase == EST_B) {
      phase = EST_C;
      start(x1, v1, dt / 2.);
      return;
    }
    if (phase == EST_C) {
      double e = 0.;
#pragma unroll
      for (int k = 0; k < NQ; k++) {
        e += exp(2. * log(fabs(y1[k] - x1[k])) - 2. * s);
        e += exp(2. * log(fabs(y1[NQ + k] - v1[k])) - 2. * s);
      }
      e = sqrt(e / B::N);
      const double c = ceil(pow(e, ORD == 4 ? 1. / 5. : 1. / 7.));
      if (c > 1. && init_dt / dt * c < kMaxDtReduce) {
        dt /= c;
        phase = EST_A;
        start(xo, vo, dt);
      } else {
        begin_main();
      }
      return;
    }
    bool fin = true;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      xo[k] = x1[k];
      vo[k] = v1[k];
      fin = fin && isfinite(x1[k]) && isfinite(v1[k]);
    }
    tk += dt;
    this->nsteps++;
    this->attempts++;
    if (++step < nrun) {
      if (!fin) {
        this->err = E_NONFINITE;
        this->done = true;
        return;
      }
      start(xo, vo, dt);
      return;
    }
    step = 0;
    this->iout++;
    row_out(out);
    if (!fin) {
      this->err = E_NONFINITE;
      this->done = true;
    } else if (this->iout == this->nt - 1) {
      this->done = true;
    } else if (this->max_attempts > 0 && this->attempts >= this->max_attempts) {
      this->err = E_BUDGET;
      this->done = true;
    } else {
      start(xo, vo, dt);
    }
  }
};

// ------------------------------------------------------------------------
// dopr54
// ------------------------------------------------------------------------
namespace dp5n {
using namespace dp5;
constexpr double A[7][6] = {{0, 0, 0, 0, 0, 0},      {a21, 0, 0, 0, 0, 0},
                            {a31, a32, 0, 0, 0, 0},  {a41, a42, a43, 0, 0, 0},
                            {a51, a52, a53, a54, 0, 0}, {a61, a62, a63, a64, a65, 0},
                            {b1, 0, b3, b4, b5, b6}};
constexpr double E[7] = {e1, 0, e3, e4, e5, e6, e7};
// position weights of stage i (0-based; 6: the new state) and of the error
// estimate, products with A
GPC_HD constexpr double X(int i, int k)
{
  double s = 0.0;
  for (int j = 0; j < 6; j++) s += A[i][j] * A[j][k];
  return s > -1e-14 && s < 1e-14 ? 0.0 : s;
}
GPC_HD constexpr double EX(int k)
{
  double s = 0.0;
  for (int j = 0; j < 7; j++) s += E[j] * A[j][k];
  return s > -1e-14 && s < 1e-14 ? 0.0 : s;
}
constexpr double C[7] = {0, 0.2, 0.3, 0.8, 8. / 9., 1, 1};
}  // namespace dp5n

// Dopr54Machine of machines.cuh: rounds (2,3), (4,5), (6,7) of an attempt.
// The step estimation is rk4_estimate_step's; its first force is the one at
// the initial state, which the first attempt needs again, so no round is
// spent on it (a run with a given step evaluates it in a start-up of three
// rounds, which keeps the lanes of a warp on the same round of an attempt).
template <int D, bool VAR>
struct Dopr54Machine<D, VAR, OrbitSystem<D, VAR>> : PairMachine<D, VAR> {
  using B = PairMachine<D, VAR>;
  using B::NQ;
  static constexpr int kSlotDoubles = 0;
  static constexpr int kRadialBlocks = 4;
  GPC_HD GPC_FI void bind(double*) {}
  GPC_HD GPC_FI bool wants_dense() const { return false; }
  GPC_HD GPC_FI static int next_slot(int slot, bool) { return slot; }
  enum { EST_A = 0, EST_B = 1, EST_C = 2, FSAL0 = 3, MAIN = 4 };
  double xo[NQ], vo[NQ];  // state at time `to`
  double a1[NQ];          // acceleration there
  // accelerations 2..5 of an attempt; during the step estimation the rk4
  // step's two kept ones (ac[0], ac[1]), its start (ac[2], ac[3])
  double ac[4][NQ];
  double y1[2 * NQ];      // estimator: the one-step result
  double to, dtout, init_to, dt_one, init_dt_one, h, s, rtol, atol, est_dt, est_init;
  double eatol, ertol;  // exp(atol), exp(rtol)
  int round, phase;
  bool forced;

  template <int I, int K>
  GPC_HD GPC_FI double coef(double w, int k) const
  {
    return w * (K == 0 ? a1[k] : ac[K > 0 ? K - 1 : 0][k]);
  }
  template <int I, int K>
  GPC_HD GPC_FI void term(double* sum) const
  {
    constexpr double w = dp5n::X(I, K);
    if constexpr (w != 0.0) {
#pragma unroll
      for (int k = 0; k < NQ; k++) sum[k] += coef<I, K>(w, k);
    }
  }
  template <int I, int... K>
  GPC_HD GPC_FI void stage(double* q, Ints<K...>) const
  {
    double sum[NQ];
#pragma unroll
    for (int k = 0; k < NQ; k++) sum[k] = 0.0;
    (term<I, K>(sum), ...);
    constexpr double c = dp5n::C[I];
#pragma unroll
    for (int k = 0; k < NQ; k++) q[k] = xo[k] + h * (c * vo[k] + h * sum[k]);
  }

  // the rk4 trial steps of the estimation, over this machine's arrays
  GPC_HD GPC_FI Rk4Nystrom<NQ> est() const
  {
    Rk4Nystrom<NQ> e;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      e.a[0][k] = ac[0][k];
      e.a[1][k] = ac[1][k];
    }
    return e;
  }

  GPC_HD GPC_FI void times2(double& t1, double& t2, int /*slot*/) const
  {
    if (phase < FSAL0) {
      Rk4Nystrom<NQ>::times(round, phase == EST_C ? to + est_dt / 2. : to, h, t1, t2);
    } else if (phase == FSAL0) {
      t1 = t2 = to;
    } else {
      t1 = round == 0 ? to + 0.2 * h : (round == 1 ? to + 0.8 * h : to + h);
      t2 = round == 0 ? to + 0.3 * h : (round == 1 ? to + 8. / 9. * h : to + h);
    }
  }

  GPC_HD GPC_FI void est_start(const double* x, const double* v, double hh)
  {
    h = hh;
    round = 0;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      ac[0][k] = ac[1][k] = 0.0;
      ac[2][k] = x[k];
      ac[3][k] = v[k];
    }
  }

  template <class W>
  GPC_HD GPC_FI void row_out(W& out) const
  {
    double w[B::NV];
    join_row<D, VAR>(xo, vo, w);
    out(this->iout, w);
  }

  template <class W>
  GPC_HD void init(const double* w, const double* tt, int nt_, double dt_in, double rtol_,
                   double atol_, long long max_att, W& out)
  {
    this->reset(tt, nt_, max_att);
    rtol = rtol_;
    atol = atol_;
    split_row<D, VAR>(w, xo, vo);
    row_out(out);
    if (nt_ < 2) {
      this->done = true;
      return;
    }
    dtout = tt[1] - tt[0];
    to = tt[0];
    round = 0;
    eatol = exp(atol);
    ertol = exp(rtol);
    if (dt_in == kDtSentinel) {
      est_dt = est_init = dtout;
      s = est_scale2<NQ>(xo, vo, rtol, atol);
      phase = EST_A;
      est_start(xo, vo, est_dt);
    } else {
      dt_one = dt_in;
      phase = FSAL0;
    }
  }

  GPC_HD GPC_FI void point2(double* q1, double* q2, int /*slot*/) const
  {
    if (phase < FSAL0) {
      est().point2(round, h, ac[2], ac[3], q1, q2);
      return;
    }
    if (phase == FSAL0) {
#pragma unroll
      for (int k = 0; k < NQ; k++) q1[k] = q2[k] = xo[k];
      return;
    }
    using S = Count<5>;
    if (round == 0) {
      stage<1>(q1, S());
      stage<2>(q2, S());
    } else if (round == 1) {
      stage<3>(q1, S());
      stage<4>(q2, S());
    } else {
      stage<5>(q1, S());
      stage<6>(q2, S());
    }
  }

  template <class W>
  GPC_HD void consume2(const double*, const double* q2, const double* f1, const double* f2, W& out,
                       int /*slot*/)
  {
    if (phase < FSAL0) {
      if (round == 0) {
        if (phase == EST_A) {  // the force at the initial state
#pragma unroll
          for (int k = 0; k < NQ; k++) a1[k] = f1[k];
        }
#pragma unroll
        for (int k = 0; k < NQ; k++) {
          ac[0][k] = f1[k];
          ac[1][k] = f2[k];
        }
        round = 1;
        return;
      }
      est_step_done(f1, f2, out);
      return;
    }
    if (phase == FSAL0) {
      if (round < 2) {
        round++;
        return;
      }
#pragma unroll
      for (int k = 0; k < NQ; k++) a1[k] = f1[k];
      begin_main(out);
      return;
    }
    if (round < 2) {
#pragma unroll
      for (int k = 0; k < NQ; k++) {
        if (round == 0) {
          ac[0][k] = f1[k];
          ac[1][k] = f2[k];
        } else {
          ac[2][k] = f1[k];
          ac[3][k] = f2[k];
        }
      }
      round++;
      return;
    }
    attempt_done(q2, f1, f2, out);
  }

  template <class W>
  GPC_HD GPC_FI void begin_main(W& out)
  {
    phase = MAIN;
    init_dt_one = dt_one;
    init_to = to;
    next_attempt(out);
  }

  // rk4_estimate_step (bovy_rk.c:328-395)
  template <class W>
  GPC_HD void est_step_done(const double* f3, const double* f4, W& out)
  {
    double x1[NQ], v1[NQ];
    est().finish(h, ac[2], ac[3], f3, f4, x1, v1);
    if (phase == EST_A) {
#pragma unroll
      for (int k = 0; k < NQ; k++) {
        y1[k] = x1[k];
        y1[NQ + k] = v1[k];
      }
      phase = EST_B;
      est_start(xo, vo, est_dt / 2.);
      return;
    }
    if (phase == EST_B) {
      phase = EST_C;
      est_start(x1, v1, est_dt / 2.);
      return;
    }
    double e = 0.;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      e += exp(2. * log(fabs(y1[k] - x1[k])) - 2. * s);
      e += exp(2. * log(fabs(y1[NQ + k] - v1[k])) - 2. * s);
    }
    e = sqrt(e / B::N);
    const double c = ceil(pow(e, 1. / 5.));
    if (c > 1. && est_init / est_dt * c < kMaxDtReduce) {
      est_dt /= c;
      phase = EST_A;
      est_start(xo, vo, est_dt);
      return;
    }
    dt_one = est_dt;
    begin_main(out);
  }

  // bovy_dopr54_onestep's loop (bovy_rk.c:584-616): output the intervals
  // that are complete, then set up the next attempt
  template <class W>
  GPC_HD void next_attempt(W& out)
  {
    for (;;) {
      const bool more = (dtout >= 0. && to < (init_to + dtout)) ||
                        (dtout < 0. && to > (init_to + dtout));
      if (more) break;
      this->iout++;
      row_out(out);
      if (this->iout == this->nt - 1) {
        this->done = true;
        return;
      }
      init_dt_one = dt_one;
      init_to = to;
    }
    if (this->max_attempts > 0 && this->attempts >= this->max_attempts) {
      this->err = E_BUDGET;
      this->done = true;
      return;
    }
    forced = false;
    if (init_dt_one / dt_one > kMaxDtReduce || dt_one != dt_one) {
      dt_one = init_dt_one / kMaxDtReduce;
      forced = true;
      this->err = E_MINSTEP;
    }
    if (dtout >= 0. && dt_one > (init_to + dtout - to)) dt_one = (init_to + dtout - to);
    if (dtout < 0. && dt_one < (init_to + dtout - to)) dt_one = (init_to + dtout - to);
    h = dt_one;
    round = 0;
  }

  // the sixth acceleration f6 and the seventh f7 (at the new state x7):
  // error norm, controller, accept
  template <class W>
  GPC_HD void attempt_done(const double* x7, const double* f6, const double* f7, W& out)
  {
    // the reference's norm sqrt(sum_i exp(2 ln|e_i| - 2 s) / N) as
    // sqrt(sum_i e_i^2 exp(-2 s) / N) (machines.cuh)
    double ymax = fabs(xo[0]), e = 0.;
    double v7[NQ];
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      using namespace dp5;
      const double A1 = a1[k], A3 = ac[1][k], A4 = ac[2][k], A5 = ac[3][k];
      v7[k] = vo[k] + h * (b1 * A1 + b3 * A3 + b4 * A4 + b5 * A5 + b6 * f6[k]);
      const double ev = h * (e1 * A1 + e3 * A3 + e4 * A4 + e5 * A5 + e6 * f6[k] + e7 * f7[k]);
      constexpr double x0 = dp5n::EX(0), x1 = dp5n::EX(1), x2 = dp5n::EX(2), x3 = dp5n::EX(3),
                       x4 = dp5n::EX(4), x5 = dp5n::EX(5);
      double ex = x0 * A1 + x2 * A3 + x3 * A4 + x4 * A5;
      if constexpr (x1 != 0.0) ex += x1 * ac[0][k];
      if constexpr (x5 != 0.0) ex += x5 * f6[k];
      ex *= h * h;
      ymax = fmax(ymax, fmax(fabs(xo[k]), fabs(vo[k])));
      e += ex * ex + ev * ev;
    }
    // exp(-s) = 1 / (exp(atol) + exp(rtol) ymax): the scale s is the logarithm
    // of that sum
    const double p2 = step_power(sqrt(e / B::N) / (eatol + ertol * ymax));
    this->attempts++;
    if (p2 >= 0. || forced) {
      bool fin = true;
#pragma unroll
      for (int k = 0; k < NQ; k++) {
        a1[k] = f7[k];
        xo[k] = x7[k];
        vo[k] = v7[k];
        fin = fin && isfinite(x7[k]) && isfinite(v7[k]);
      }
      const double to_before = to;
      to += h;
      this->nsteps++;
      if (!fin) {
        this->err = E_NONFINITE;
        this->done = true;
        return;
      }
      // a step below half an ulp of `to` leaves it unchanged: the reference
      // would loop forever here; the orbit stops as out of budget instead
      if (to == to_before) {
        this->err = E_BUDGET;
        this->done = true;
        return;
      }
    }
    dt_one = p2 == p2 ? ldexp(h, (int)p2) : h * p2;  // h 2^p2 (NaN stays NaN)
    next_attempt(out);
  }

  // The controller's power of two, round(log2(0.85 e^(-1/5))) in [-3, 3].
  // A single-precision logarithm decides (error < 1e-4 in the rounded number)
  // but where it comes within 1e-3 of a rounding boundary; there, and for a
  // norm that is not an ordinary number, the reference's own expression does.
  // Powers and logarithms of every attempt were a third of its time.
  GPC_HD GPC_FI static double step_power(double e)
  {
    const float ef = (float)e;
    if (ef > 1e-30f && ef < 1e30f) {
      const float x = -0.23446525f - 0.2f * log2f(ef), r = rintf(x);
      if (fabsf(x - r) < 0.499f) return (double)fminf(fmaxf(r, -3.f), 3.f);
    }
    const double corr = 0.85 * pow(e, -.2);
    double p2 = ::round(log(corr) / log(2.));
    if (p2 > 3.)
      p2 = 3.;
    else if (p2 < -3.)
      p2 = -3.;
    return p2;
  }
};

// ------------------------------------------------------------------------
// dop853
// ------------------------------------------------------------------------
// e^(-1/8) for the step controller, e clamped to [1e-9, 1e6] (outside, the
// factor 0.9 e^(-1/8) is beyond the controller's limits 0.333 and 6 anyway):
// a single-precision seed (1e-6) and one third-order Newton correction of
// y^-8 = e, y <- y (1 + r/8 + 9 r^2/128 + 51 r^3/1024), r = 1 - e y^8.  Three
// square roots and a division, or pow, are a long chain at every attempt.
GPC_HD GPC_FI double root8_inv(double e)
{
  e = dmin(dmax(e, 1e-9), 1e6);
#if defined(__CUDA_ARCH__)
  const double y = (double)exp2f(-0.125f * __log2f((float)e));
#else
  const double y = (double)exp2f(-0.125f * log2f((float)e));
#endif
  const double y2 = y * y, y4 = y2 * y2, r = 1.0 - e * y4 * y4;
  return y + y * r * (0.125 + r * (9.0 / 128.0 + r * (51.0 / 1024.0)));
}

// Without a force (a Null potential) both error estimates vanish, but the
// reference's are the rounding of sum_j er_j v and of its b - bhh sum, and
// that rounding is what its step sizes follow: the same sums here.
template <int NQ>
GPC_HD inline void dop853_force_free(const double* x0, const double* v0, double h, double rtol,
                                     double atol, double& e, double& e2)
{
  using namespace dp;
#pragma unroll
  for (int i = 0; i < NQ; i++) {
    const double v = v0[i];
    const double k4 = b1 * v + b6 * v + b7 * v + b8 * v + b9 * v + b10 * v + b11 * v + b12 * v;
    const double sk = atol + rtol * dmax(fabs(x0[i]), fabs(x0[i] + h * k4));
    double sqr = (k4 - bhh1 * v - bhh2 * v - bhh3 * v) / sk;
    e2 += sqr * sqr;
    sqr = (er1 * v + er6 * v + er7 * v + er8 * v + er9 * v + er10 * v + er11 * v + er12 * v) / sk;
    e += sqr * sqr;
  }
}

// Component i of the velocity's increment of a step over its size, sum_k b_k
// a_k; one function, so that every pass that repeats a step (the adjoint's
// replay and its segments) rounds it alike.
template <class G>
GPC_HD GPC_FI double dop853_increment(const G& g, int i)
{
  const auto& b = GPC_NY.b;
  return mad(b[0], g.template a<1>(i), b[5] * g.template a<6>(i)) + b[6] * g.template a<7>(i) +
         b[7] * g.template a<8>(i) + b[8] * g.template a<9>(i) + b[9] * g.template a<10>(i) +
         b[10] * g.template a<11>(i) + b[11] * g.template a<12>(i);
}

// The new velocity vn of a step of size h from (x0, v0) to the position x13,
// and the step's error norm (leung_dop853.c:390-418); g gives component i of
// the accelerations a1, a4..a12.
template <int NQ, class G>
GPC_HD GPC_FI double dop853_error(const G& g, const double* x0, const double* v0,
                                  const double* x13, double h, double rtol, double atol,
                                  double* vn)
{
  double e = 0.0, e2 = 0.0;
#pragma unroll
  for (int i = 0; i < NQ; i++) {
    const double A1 = g.template a<1>(i), A4 = g.template a<4>(i), A5 = g.template a<5>(i);
    const double A6 = g.template a<6>(i), A7 = g.template a<7>(i), A8 = g.template a<8>(i);
    const double A9 = g.template a<9>(i), A10 = g.template a<10>(i), A11 = g.template a<11>(i);
    const double A12 = g.template a<12>(i);
    const auto& ev = GPC_NY.ev;
    const auto& ex = GPC_NY.ex;
    const auto& hx = GPC_NY.hx;
    const double inc = dop853_increment(g, i);
    vn[i] = v0[i] + h * inc;
    const double isv = rcp_nr(atol + rtol * dmax(fabs(v0[i]), fabs(vn[i])));
    const double isx = rcp_nr(atol + rtol * dmax(fabs(x0[i]), fabs(x13[i])));
    double sqr = (inc - GPC_NY.bhh[0] * A1 - GPC_NY.bhh[1] * A9 - GPC_NY.bhh[2] * A12) * isv;
    e2 += sqr * sqr;
    sqr = (mad(ev[5], A6, ev[0] * A1) + ev[6] * A7 + ev[7] * A8 + ev[8] * A9 + ev[9] * A10 +
           ev[10] * A11 + ev[11] * A12) * isv;
    e += sqr * sqr;
    sqr = (mad(hx[3], A4, hx[0] * A1) + hx[4] * A5 + hx[5] * A6 + hx[6] * A7 + hx[7] * A8 +
           hx[8] * A9 + hx[9] * A10 + hx[10] * A11) * h * isx;
    e2 += sqr * sqr;
    sqr = (mad(ex[3], A4, ex[0] * A1) + ex[4] * A5 + ex[5] * A6 + ex[6] * A7 + ex[7] * A8 +
           ex[8] * A9 + ex[9] * A10 + ex[10] * A11) * h * isx;
    e += sqr * sqr;
  }
  if (e + e2 <= 0.0) dop853_force_free<NQ>(x0, v0, h, rtol, atol, e, e2);
  // (the floor only keeps the root of a vanishing estimate finite)
  return fabs(h) * e * rsqrt_nr(dmax(e + 0.01 * e2, 1e-280) * (double)(2 * NQ));
}

// The lanes of a warp run the rounds of their (different) orbits in lock
// step: an attempt is slots 0..5, a dense output slots 6 and 7 (run when
// some lane of the warp asks, or for 32 queued requests at a time).  A lane
// with nothing to compute in a slot (a new orbit waiting for slot 0)
// evaluates the force at its own position and discards it; the two start-up
// forces of a new orbit run in whatever slots follow its pick-up.
template <int D, bool VAR>
struct Dop853Machine<D, VAR, OrbitSystem<D, VAR>> : PairMachine<D, VAR> {
  using B = PairMachine<D, VAR>;
  using B::N;
  using B::NQ;
  static constexpr int kFsalSlot = 5, kDenseSlot = 6, kLastSlot = 7;
  static constexpr int kRadialBlocks = 1;
  enum { ST_INIT1 = -2, ST_INIT2 = -1 };  // otherwise `stage` is the slot the lane waits for
  // The accelerations a2..a11 and the new state live in a per-thread slot
  // store (shared memory in the kernel, strided by kSlotStride threads:
  // bank-conflict free; half a first-order store, so that three blocks fit a
  // multiprocessor); x, v and a1 stay in registers.  a12 takes a2's place
  // (free after stage 5), a13 a3's (free after stage 12), the dense stages
  // a14 and a15 those of a4 and a5 (free after the error estimate).
  static constexpr int XN = 10, VN = 11, kSlots = 12;
  static constexpr int kSlotDoubles = kSlots * NQ;
  GPC_HD static constexpr int slot_of(int k) { return k >= 12 ? k - 12 : k - 2; }
  double x0[NQ], v0[NQ], a1[NQ];
  double* ks;
  GPC_HD GPC_FI void bind(double* base, bool /*queue*/ = false) { ks = base; }
  GPC_HD GPC_FI double& K(int s, int i) const { return ks[(s * NQ + i) * kSlotStride]; }
  // a_k, k = 1..15
  template <int Kk>
  GPC_HD GPC_FI double acc(int i) const
  {
    if constexpr (Kk == 1)
      return a1[i];
    else
      return K(slot_of(Kk), i);
  }
  double h, hnew, hmax, pos_neg, rtol, atol;
  double t_current, t_old;
  int stage;
  bool reject;

  GPC_HD GPC_FI bool active_in(int slot) const { return stage < 0 || stage == slot; }
  GPC_HD GPC_FI bool wants_dense() const { return !this->done && stage == kDenseSlot; }
  GPC_HD GPC_FI static int next_slot(int slot, bool any_dense)
  {
    if (slot == kFsalSlot) return any_dense ? kDenseSlot : 0;
    return slot >= kLastSlot ? 0 : slot + 1;
  }

  GPC_HD GPC_FI void begin_attempt()
  {
    h = pos_neg * dmax(fabs(h), 1e3 * 2.3e-16);
    stage = 0;
  }

  template <class W>
  GPC_HD void init(const double* w, const double* tt, int nt_, double /*dt*/, double rtol_,
                   double atol_, long long max_att, W& out)
  {
    this->reset(tt, nt_, max_att);
    rtol = exp(rtol_);
    atol = exp(atol_);
    split_row<D, VAR>(w, x0, v0);
    out(0, w);
    if (nt_ < 2) {
      this->done = true;
      return;
    }
    hmax = tt[nt_ - 1] - tt[0];
    pos_neg = csign(1.0, hmax);
    reject = false;
    t_current = t_old = tt[0];
    stage = ST_INIT1;
  }

  // position of stage I (1-based, 13: the new state) from the accelerations
  template <int I, int Kk>
  GPC_HD GPC_FI void term(double* s) const
  {
    constexpr bool nz = kNy.x[I - 1][Kk - 1] != 0.0;
    if constexpr (nz) {
      const double w = GPC_NY.x[I - 1][Kk - 1];
#pragma unroll
      for (int i = 0; i < NQ; i++) s[i] += w * acc<Kk>(i);
    }
  }
  template <int I, int... Kk>
  GPC_HD GPC_FI void stage_x(double* q, Ints<Kk...>) const
  {
    double s[NQ];
#pragma unroll
    for (int i = 0; i < NQ; i++) s[i] = 0.0;
    (term<I, Kk + 1>(s), ...);
    // the new state is the old one plus its rounded increment
    const double ch = GPC_NY.c[I - 1] * h, h2 = h * h;
#pragma unroll
    for (int i = 0; i < NQ; i++)
      q[i] = I == 13 ? x0[i] + mad(h2, s[i], h * v0[i]) : mad(h2, s[i], mad(ch, v0[i], x0[i]));
  }
  template <int I>
  GPC_HD GPC_FI void two_stages(double* q1, double* q2) const
  {
    stage_x<I>(q1, Count<13>());
    stage_x<I + 1>(q2, Count<13>());
  }

  GPC_HD GPC_FI void point2(double* q1, double* q2, int slot) const
  {
    if (!active_in(slot) || stage < 0) {
      const double e = stage == ST_INIT2 ? h : 0.0;  // explicit Euler step (leung_dop853.c:310)
#pragma unroll
      for (int i = 0; i < NQ; i++) q1[i] = q2[i] = x0[i] + e * v0[i];
      return;
    }
    switch (slot) {
      case 0: two_stages<2>(q1, q2); break;
      case 1: two_stages<4>(q1, q2); break;
      case 2: two_stages<6>(q1, q2); break;
      case 3: two_stages<8>(q1, q2); break;
      case 4: two_stages<10>(q1, q2); break;
      case 5: two_stages<12>(q1, q2); break;
      case 6: two_stages<14>(q1, q2); break;
      default:
        stage_x<16>(q1, Count<14>());
#pragma unroll
        for (int i = 0; i < NQ; i++) q2[i] = q1[i];
    }
  }

  // times of the forces as the reference passes them: t0 and t0 + h for the
  // start-up, t_current + c_s h for stages 2..11, t_current + h for stage 12
  // and the new t_current (the same sum) for the 13th, t_old + c_s h for the
  // dense stages (an idle lane: any time)
  GPC_HD GPC_FI static double at(double tb, int stage1, double h)
  {
    return stage1 == 12 || stage1 == 13 ? tb + h : tb + GPC_NY.c[stage1 - 1] * h;
  }
  GPC_HD GPC_FI void times2(double& t1, double& t2, int slot) const
  {
    if (!active_in(slot) || stage < 0) {
      t1 = t2 = stage == ST_INIT2 ? t_current + h : t_current;
      return;
    }
    const double tb = slot >= kDenseSlot ? t_old : t_current;
    const int s1 = slot == kLastSlot ? 16 : 2 * slot + 2;
    t1 = at(tb, s1, h);
    t2 = slot == kLastSlot ? t1 : at(tb, s1 + 1, h);
  }

  GPC_HD GPC_FI bool output_pending() const
  {
    return this->iout < this->nt - 1 && pos_neg * this->t[this->iout + 1] < pos_neg * t_current;
  }

  GPC_HD GPC_FI void put(int k1, const double* f1, int k2, const double* f2)
  {
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      K(k1, i) = f1[i];
      K(k2, i) = f2[i];
    }
  }

  // the start-up forces: f1 at the initial state, then at the Euler step
  GPC_HD GPC_FI void start_first(const double* f1)  // leung_dop853.c:296-308
  {
    double dny = 0.0, dnf = 0.0;
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      a1[i] = f1[i];
      const double sx = atol + rtol * fabs(x0[i]), sv = atol + rtol * fabs(v0[i]);
      double sqr = v0[i] / sx;
      dnf += sqr * sqr;
      sqr = f1[i] / sv;
      dnf += sqr * sqr;
      sqr = x0[i] / sx;
      dny += sqr * sqr;
      sqr = v0[i] / sv;
      dny += sqr * sqr;
    }
    h = csign(dmin(sqrt(dny / dnf) * 0.01, fabs(hmax)), pos_neg);
    hnew = dnf;  // kept for the second start-up evaluation (hnew is free until the first step)
    stage = ST_INIT2;
  }
  // leung_dop853.c:309-324: f(y0 + h f0) - f0 = (h a1, a - a1)
  GPC_HD GPC_FI void start_second(const double* f1)
  {
    double der2 = 0.0;
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      const double sx = atol + rtol * fabs(x0[i]), sv = atol + rtol * fabs(v0[i]);
      double sqr = h * a1[i] / sx;
      der2 += sqr * sqr;
      sqr = (f1[i] - a1[i]) / sv;
      der2 += sqr * sqr;
    }
    der2 = sqrt(der2) / h;
    const double der12 = dmax(fabs(der2), sqrt(hnew));  // hnew: dnf of the first evaluation
    const double h1 = pow(0.01 / der12, 1.0 / 8.0);
    h = csign(dmin(100.0 * fabs(h), dmin(fabs(h1), fabs(hmax))), pos_neg);
    begin_attempt();
  }

  template <class W>
  GPC_HD void consume2(const double* /*q1*/, const double* q2, const double* f1, const double* f2,
                       W& out, int slot)
  {
    if (!active_in(slot)) return;
    if (stage == ST_INIT1) {
      start_first(f1);
      return;
    }
    if (stage == ST_INIT2) {
      start_second(f1);
      return;
    }
    if (slot < kFsalSlot) {
      // a2, a3 in slots 0, 1; a4, a5 in 2, 3; ...
      put(2 * slot, f1, 2 * slot + 1, f2);
      stage = slot + 1;
      return;
    }
    if (slot == kFsalSlot) {
      double vn[NQ];
      if (!attempt_end(q2, f1, f2, vn)) return;
      if (!output_pending()) {
        finish_step(q2, vn, f2);
        return;
      }
      keep_step(f1, f2, q2, vn);  // the rows need the dense stages first
      return;
    }
    if (slot == kDenseSlot) {
      put(slot_of(14), f1, slot_of(15), f2);
      stage = kLastSlot;
      return;
    }
    own_rows(f1, out);
  }

  // An accepted step whose rows wait for the lane's own dense stages (slots
  // kDenseSlot, kLastSlot): its last forces and new state go to the slots.
  GPC_HD GPC_FI void keep_step(const double* f12, const double* f13, const double* x13,
                               const double* vn)
  {
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      K(slot_of(12), i) = f12[i];
      K(slot_of(13), i) = f13[i];
      K(XN, i) = x13[i];
      K(VN, i) = vn[i];
    }
    stage = kDenseSlot;
  }
  // its rows (leung_dop853.c:441-474), f16 the last dense stage's force
  template <class W>
  GPC_HD GPC_FI void own_rows(const double* f16, W& out)
  {
    while (output_pending()) {
      const double sv = (this->t[this->iout + 1] - t_old) / h;
      double x[NQ], v[NQ], w[B::NV];
      const Dense d = dense_at(sv);
#pragma unroll
      for (int i = 0; i < NQ; i++) {
        const Own g{this, f16, i};
        dense_value(d, h, g, x[i], v[i]);
      }
      join_row<D, VAR>(x, v, w);
      this->iout++;
      out(this->iout, w);
    }
    finish_kept();
  }

  // The rows that an accepted step completes, first and last.
  GPC_HD GPC_FI void rows_of_step(int& first, int& last)
  {
    first = this->iout + 1;
    while (output_pending()) this->iout++;
    last = this->iout;
  }

  // One attempt's end (leung_dop853.c:390-440): f12, f13 = f(x13) the last
  // two forces.  Returns whether the step is accepted; vn receives its
  // velocity.
  struct SlotAcc {
    const Dop853Machine* m;
    const double* f12;
    template <int Kk>
    GPC_HD GPC_FI double a(int i) const
    {
      if constexpr (Kk == 12)
        return f12[i];
      else
        return m->template acc<Kk>(i);
    }
  };
  GPC_HD GPC_FI bool attempt_end(const double* x13, const double* f12, const double* f13,
                                 double* vn)
  {
    this->attempts++;
    const double e = dop853_error<NQ>(SlotAcc{this, f12}, x0, v0, x13, h, rtol, atol, vn);
    if (!isfinite(e)) {
      this->err = E_NONFINITE;
      this->done = true;
      return false;
    }
    const double fac = 0.9 * root8_inv(e);
    // Lund stabilisation with beta = 0 divides by pow(facold, 0) == 1, so the
    // reference's facold (max(e, 1e-4) of the last accepted step) drops out
    if (e <= 1.0) {
      // accepted: the step runs from t_old to t_current (the reference
      // advances both before the test and restores them on rejection)
      hnew = h * dmin(6.0, dmax(0.333, fac));
      t_old = t_current;
      t_current = t_current + h;
      this->nsteps++;
      return true;
    } else {
      // an attempt rejected at the smallest step (begin_attempt's floor)
      // repeats exactly -- same state, same step, same error -- so the
      // reference rejects it forever; the orbit stops as out of budget
      if (fabs(h) <= 1e3 * 2.3e-16) {
        this->err = E_BUDGET;
        this->done = true;
        return false;
      }
      hnew = h * dmax(0.333, fac);
      reject = true;
      h = hnew;
      if (this->max_attempts > 0 && this->attempts >= this->max_attempts) {
        this->err = E_BUDGET;
        this->done = true;
        return false;
      }
      begin_attempt();
      return false;
    }
  }

  // from the new state kept in the slots
  GPC_HD GPC_FI void finish_kept()
  {
    double x13[NQ], vn[NQ], f13[NQ];
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      x13[i] = K(XN, i);
      vn[i] = K(VN, i);
      f13[i] = K(slot_of(13), i);
    }
    finish_step(x13, vn, f13);
  }
  GPC_HD GPC_FI void finish_step(const double* x13, const double* vn, const double* f13)
  {
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      x0[i] = x13[i];
      v0[i] = vn[i];
      a1[i] = f13[i];
    }
    hnew = (fabs(hnew) > fabs(hmax)) ? pos_neg * hmax : hnew;
    if (reject) hnew = pos_neg * dmin(fabs(hnew), fabs(h));
    reject = false;
    h = hnew;
    if (this->iout == this->nt - 1) {
      this->done = true;
      return;
    }
    if (this->max_attempts > 0 && this->attempts >= this->max_attempts) {
      this->err = E_BUDGET;
      this->done = true;
      return;
    }
    begin_attempt();
  }

  // ---- dense output -------------------------------------------------------
  // Hairer's continuous extension at s in (0, 1) (leung_dop853.c:441-474),
  //   y + s (dy + s' (bspl + s (r4 + s' (r5 + s (r6 + s' (r7 + s r8))))))
  // with s' = 1 - s, dy = y1 - y, bspl = h f0 - dy, r4 = dy - h f1 - bspl,
  // r_m = h sum_j d_mj k_j: for the velocities k_j = a_j, for the positions
  // sum_j d_mj v_j = h sum_k DX_mk a_k.  The source g gives component i of
  // the step's vectors.
  struct Dense {
    double s, s1;
  };
  GPC_HD GPC_FI static Dense dense_at(double s) { return {s, 1.0 - s}; }
  template <int M, bool X, int Kk, class G>
  GPC_HD GPC_FI static void dense_term(const G& g, double& sum)
  {
    if constexpr (X) {
      constexpr bool nz = kNy.dx[M][Kk < 16 ? Kk - 1 : 0] != 0.0 && Kk < 16;
      if constexpr (nz) sum += GPC_NY.dx[M][Kk - 1] * g.template a<Kk>();
    } else {
      constexpr bool nz = kNy.d[M][Kk - 1] != 0.0;
      if constexpr (nz) sum += GPC_NY.d[M][Kk - 1] * g.template a<Kk>();
    }
  }
  template <int M, bool X, class G, int... Kk>
  GPC_HD GPC_FI static double dense_sum(const G& g, Ints<Kk...>)
  {
    double sum = 0.0;
    (dense_term<M, X, Kk + 1>(g, sum), ...);
    return sum;
  }
  GPC_HD GPC_FI static double dense_poly(const Dense& d, double h, double y0, double y1, double f0,
                                         double f1, double r5, double r6, double r7, double r8)
  {
    const double ydiff = y1 - y0, bspl = h * f0 - ydiff, r4 = ydiff - h * f1 - bspl;
    return y0 + d.s * (ydiff +
                       d.s1 * (bspl + d.s * (r4 + d.s1 * (r5 + d.s * (r6 + d.s1 * (r7 + d.s * r8))))));
  }
  template <class G>
  GPC_HD GPC_FI static void dense_value(const Dense& d, double h, const G& g, double& x, double& v)
  {
    using S = Count<16>;
    const double h2 = h * h;
    x = dense_poly(d, h, g.x0(), g.xn(), g.v0(), g.vn(), h2 * dense_sum<0, true>(g, S()),
                   h2 * dense_sum<1, true>(g, S()), h2 * dense_sum<2, true>(g, S()),
                   h2 * dense_sum<3, true>(g, S()));
    v = dense_poly(d, h, g.v0(), g.vn(), g.template a<1>(), g.template a<13>(),
                   h * dense_sum<0, false>(g, S()), h * dense_sum<1, false>(g, S()),
                   h * dense_sum<2, false>(g, S()), h * dense_sum<3, false>(g, S()));
  }
  // the lane's own step (f16: the last dense stage's force)
  struct Own {
    const Dop853Machine* m;
    const double* f16;
    int i;
    GPC_HD GPC_FI double x0() const { return m->x0[i]; }
    GPC_HD GPC_FI double v0() const { return m->v0[i]; }
    GPC_HD GPC_FI double xn() const { return m->K(XN, i); }
    GPC_HD GPC_FI double vn() const { return m->K(VN, i); }
    template <int Kk>
    GPC_HD GPC_FI double a() const
    {
      if constexpr (Kk == 16)
        return f16[i];
      else
        return m->template acc<Kk>(i);
    }
  };

  // ---- queued dense output ------------------------------------------------
  // With a request queue (the kernel's per-warp ring in global memory,
  // pair_loop), a step that contains output times does not run the dense
  // stages in the warp's slot cycle, where the other lanes would sit idle for
  // them: the lane writes the step's data to the queue and goes on with its
  // next step, and the warp later runs the dense stages of 32 queued requests
  // side by side (one per lane).  Same arithmetic, same rows.
  //
  // Request record, field-major with kQueueSlots slots per field (component
  // i of vector field f of slot p at q[(f * NQ + i) * kQueueSlots + p]):
  // vector fields 0 x, 1 v, 2 a1, 3..10 a6..a13, 11 the new x, 12 the new v;
  // then h, t_old, the output position and the row range (first << 32 | last)
  // at q[(13 NQ + k) * kQueueSlots + p].
  static constexpr int kQueueSlots = 64;
  static constexpr int kQueueVecs = 13;
  static constexpr int kQueueFields = kQueueVecs * NQ + 4;  // doubles per slot
  static constexpr bool kQueue = !VAR;
  GPC_HD static constexpr int rec_of(int k) { return k == 1 ? 2 : k - 3; }

  template <int... Kk>
  GPC_HD GPC_FI void write_accs(double* q, int p, Ints<Kk...>) const
  {
#pragma unroll
    for (int i = 0; i < NQ; i++)
      ((q[(rec_of(Kk + 6) * NQ + i) * kQueueSlots + p] = acc<Kk + 6>(i)), ...);
  }
  // the accepted step's request for rows jf..jl (before finish_step)
  GPC_HD GPC_FI void write_request(double* q, int p, long long orbit, int jf, int jl,
                                   const double* f12, const double* f13, const double* x13,
                                   const double* vn) const
  {
    constexpr int QS = kQueueSlots;
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      q[(0 * NQ + i) * QS + p] = x0[i];
      q[(1 * NQ + i) * QS + p] = v0[i];
      q[(2 * NQ + i) * QS + p] = a1[i];
      q[(rec_of(12) * NQ + i) * QS + p] = f12[i];
      q[(rec_of(13) * NQ + i) * QS + p] = f13[i];
      q[(11 * NQ + i) * QS + p] = x13[i];
      q[(12 * NQ + i) * QS + p] = vn[i];
    }
    write_accs(q, p, Count<6>());
    q[(kQueueVecs * NQ + 0) * QS + p] = h;
    q[(kQueueVecs * NQ + 1) * QS + p] = t_old;
    long long* qi = reinterpret_cast<long long*>(q);
    qi[(kQueueVecs * NQ + 2) * QS + p] = orbit;
    qi[(kQueueVecs * NQ + 3) * QS + p] = ((long long)jf << 32) | (long long)(unsigned)jl;
  }
  GPC_HD GPC_FI static long long req_orbit(const double* q, int p)
  {
    return reinterpret_cast<const long long*>(q)[(kQueueVecs * NQ + 2) * kQueueSlots + p];
  }

  // Request p's step, component i; the dense stages a14, a15 are in this
  // lane's own slots (free between its attempts), f16 in a register.
  struct Rec {
    const Dop853Machine* m;
    const double* q;
    int p, i;
    double f16;
    GPC_HD GPC_FI double f(int field) const { return q[(field * NQ + i) * kQueueSlots + p]; }
    GPC_HD GPC_FI double x0() const { return f(0); }
    GPC_HD GPC_FI double v0() const { return f(1); }
    GPC_HD GPC_FI double xn() const { return f(11); }
    GPC_HD GPC_FI double vn() const { return f(12); }
    template <int Kk>
    GPC_HD GPC_FI double a() const
    {
      if constexpr (Kk == 16)
        return f16;
      else if constexpr (Kk >= 14)
        return m->K(slot_of(Kk), i);
      else
        return f(rec_of(Kk));
    }
  };
  template <int I, int Kk>
  GPC_HD GPC_FI void req_term(const double* q, int p, double* s) const
  {
    constexpr bool nz = kNy.x[I - 1][Kk - 1] != 0.0;
    if constexpr (nz) {
      const double w = GPC_NY.x[I - 1][Kk - 1];
#pragma unroll
      for (int i = 0; i < NQ; i++) s[i] += w * Rec{this, q, p, i, 0.0}.template a<Kk>();
    }
  }
  template <int I, int... Kk>
  GPC_HD GPC_FI void req_stage(const double* q, int p, double* pos, Ints<Kk...>) const
  {
    double s[NQ];
#pragma unroll
    for (int i = 0; i < NQ; i++) s[i] = 0.0;
    (req_term<I, Kk + 1>(q, p, s), ...);
    const double hq = q[kQueueVecs * NQ * kQueueSlots + p], ch = GPC_NY.c[I - 1] * hq, h2 = hq * hq;
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      const Rec g{this, q, p, i, 0.0};
      pos[i] = g.x0() + ch * g.v0() + h2 * s[i];
    }
  }
  // ---- one round of the kernel's pair_loop ---------------------------------
  // Slots 0..5 are an attempt, 6 and 7 the dense stages of request p, 8 and 9
  // the start-up of a new orbit, 10 and 11 the lane's own dense stages (a
  // launch without a queue).
  static constexpr int kInitSlot = 8, kOwnSlot = 10;
  GPC_HD GPC_FI void slot_point(double* q1, double* q2, int slot, const double* q, int p) const
  {
    switch (slot) {
      case 0: two_stages<2>(q1, q2); break;
      case 1: two_stages<4>(q1, q2); break;
      case 2: two_stages<6>(q1, q2); break;
      case 3: two_stages<8>(q1, q2); break;
      case 4: two_stages<10>(q1, q2); break;
      case 5: two_stages<12>(q1, q2); break;
      case 6:
        req_stage<14>(q, p, q1, Count<13>());
        req_stage<15>(q, p, q2, Count<13>());
        break;
      case 7:
        req_stage<16>(q, p, q1, Count<14>());
#pragma unroll
        for (int i = 0; i < NQ; i++) q2[i] = q1[i];
        break;
      case kOwnSlot: two_stages<14>(q1, q2); break;
      case kOwnSlot + 1:
        stage_x<16>(q1, Count<14>());
#pragma unroll
        for (int i = 0; i < NQ; i++) q2[i] = q1[i];
        break;
      default: {
        const double e = slot == kInitSlot ? 0.0 : h;  // explicit Euler step (leung_dop853.c:310)
#pragma unroll
        for (int i = 0; i < NQ; i++) q1[i] = q2[i] = x0[i] + e * v0[i];
      }
    }
  }
  GPC_HD GPC_FI void slot_times(double& t1, double& t2, int slot, const double* q, int p) const
  {
    if (slot >= kOwnSlot) {
      t1 = at(t_old, slot == kOwnSlot ? 14 : 16, h);
      t2 = slot == kOwnSlot ? at(t_old, 15, h) : t1;
    } else if (slot >= kInitSlot) {
      t1 = t2 = slot == kInitSlot ? t_current : t_current + h;
    } else if (slot >= kDenseSlot) {
      const double hq = q[kQueueVecs * NQ * kQueueSlots + p];
      const double told = q[(kQueueVecs * NQ + 1) * kQueueSlots + p];
      t1 = at(told, slot == kLastSlot ? 16 : 14, hq);
      t2 = slot == kLastSlot ? t1 : at(told, 15, hq);
    } else {
      t1 = at(t_current, 2 * slot + 2, h);
      t2 = at(t_current, 2 * slot + 3, h);
    }
  }
  // (the last forces of an attempt and of a dense round stay with the caller)
  GPC_HD GPC_FI void slot_keep(const double* f1, const double* f2, int slot)
  {
    if (slot <= kDenseSlot) {
      if (slot != kFsalSlot) {  // a2, a3; ...; a10, a11; the dense a14, a15
        const int k = slot == kDenseSlot ? slot_of(14) : 2 * slot;
        put(k, f1, k + 1, f2);
      }
    } else if (slot == kInitSlot) {
      start_first(f1);
    } else if (slot == kInitSlot + 1) {
      start_second(f1);
    } else if (slot == kOwnSlot) {
      put(slot_of(14), f1, slot_of(15), f2);
    }
  }
  // the rows of request p, f1 = a16
  template <class W>
  GPC_HD GPC_FI void req_rows(const double* f1, const double* q, int p, const double* tt,
                              W& out) const
  {
    constexpr int QS = kQueueSlots;
    const double hq = q[kQueueVecs * NQ * QS + p], told = q[(kQueueVecs * NQ + 1) * QS + p];
    const long long rr = reinterpret_cast<const long long*>(q)[(kQueueVecs * NQ + 3) * QS + p];
    const int j0 = (int)(rr >> 32), j1 = (int)(unsigned)(rr & 0xffffffffLL);
    for (int j = j0; j <= j1; j++) {
      const Dense d = dense_at((tt[j] - told) / hq);
      double x[NQ], v[NQ], w[B::NV];
#pragma unroll
      for (int k = 0; k < NQ; k++) x[k] = v[k] = 0.0;
      // one component at a time: unrolled, the compiler would issue all of
      // the record's loads at once and hold them in registers.  The
      // component index of this loop is a run-time value, so f1, x and v are
      // read and written through selects over compile-time indices: indexed
      // by it they would live in local memory.
#pragma unroll 1
      for (int i = 0; i < NQ; i++) {
        double di = f1[0], xi, vi;
#pragma unroll
        for (int k = 1; k < NQ; k++) di = i == k ? f1[k] : di;
        const Rec g{this, q, p, i, di};
        dense_value(d, hq, g, xi, vi);
#pragma unroll
        for (int k = 0; k < NQ; k++) {
          x[k] = i == k ? xi : x[k];
          v[k] = i == k ? vi : v[k];
        }
      }
      join_row<D, VAR>(x, v, w);
      out(j, w);
    }
  }
};

// The dop853 machine of a component list.
// The full run-time list keeps the first-order machine, whose sums are in
// the reference's order.  It carries the potentials whose second
// derivative jumps (the Dehnen bar at its radius): there the error
// estimate of many steps is near 1, and the pair machine's rounding
// decides some of them otherwise, which moves an orbit by 7e-10 where the
// first-order machine keeps to 30 times its one-ulp response
// (tests/test_gpu_timedep.py).  Pairs would take 21.2 ms instead of 38.4
// for 3,000 orbits in MWPotential2014 with a bar, 4.54 instead of 4.77 in
// an ellipsoidal halo, and 153 instead of 146 in a nonaxisymmetric SCF
// expansion.
template <int D, bool VAR, class POT>
using Dop853For = std::conditional_t<POT::kFullList && !VAR,
                                     Dop853Machine<D, VAR, FirstOrderOrbit<D>>, Dop853Machine<D, VAR>>;

}  // namespace gpc
