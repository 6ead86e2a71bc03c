// galpy_b200/csrc/adjoint.cuh
//
// Reverse-mode differentiation of DOP853 orbit integration: gradients of a
// loss on the final states y(T) with respect to the initial conditions and
// the potential parameters.  The reference has no adjoint; its gradient
// information comes from the variational equations (integrate_dxdv,
// galpy/orbit/orbit_c_ext/integratePlanarOrbit.c:940-1014), one tangent
// vector per input direction.  The adjoint gives the whole gradient of a
// scalar loss in one backward sweep per orbit.
//
// What is differentiated: the discrete map that the forward integrator
// applies, with its accepted step sizes held fixed (they are not
// differentiated; this is the standard discrete adjoint of an adaptive
// method and is exact for the frozen step sequence).
//
//   * Forward: galpy's DOP853 (same tableau, initial step, controller and
//     dense output as Dop853Machine, leung_dop853.c:231-517) from t0 to T;
//     y(T) is the dense-output value inside the step that passes T, as in
//     the reference (it does not shorten the last step).  Every 64 accepted
//     steps the state (y, t) is saved, a checkpoint, together with the
//     segment's 64 accepted step sizes.
//   * Backward, per orbit, segment by segment from the last: restore the
//     segment's checkpoint, recompute the start state of each of its steps
//     with the recorded step sizes (no step-size control runs again, so a
//     marginal accept/reject decision cannot come out differently), then
//     sweep the steps in reverse.  Each step recomputes its stages and
//     applies the adjoint of an explicit Runge-Kutta step:
//         kappa_i = h W_i lambda + h sum_{j>i} A_ji mu_j
//         mu_i    = J(Y_i)^T kappa_i = (K(q_i) kappa_v, kappa_q)
//         lambda <- lambda + sum_i mu_i,   g_theta += sum_i (da/dtheta)^T kappa_v
//     with K the tidal tensor (potentials.cuh, accel_tidal) and da/dtheta
//     the analytic parameter derivatives below.  W = b (8th-order weights)
//     for full steps; the last step is the 16-stage dense-output map with
//     weights W(s), s = (T - t_n) / h_n.
//
// Both sweeps use the scheme's Nystrom form (dop853_nystrom.cuh): only stage
// positions and accelerations, x1 = x + h v + h^2 sum Xb_k a_k, v1 = v + h sum
// b_k a_k, and backward
//         kappa_k = h^2 Xb_k lx + h b_k lv + h^2 sum_{i>k+1} X_ik mu_i,
//         mu_k    = K(q_k) kappa_k,      g_theta += (da/dtheta)^T kappa_k,
//         lv <- lv + h lx + h sum c_k mu_k,   lx <- lx + sum mu_k.
// Forward a stage's position, backward its kappa, does not depend on its
// neighbour, so forces and products are formed two at a time, their chains
// overlapping: latency at 8 warps per multiprocessor is what bounds both.
//
// All functions are host/device portable so that the CPU test harness runs
// the same code against finite differences and the reference's variational
// integration.
#pragma once
#include "dop853_tableau.cuh"
#include "gpc_common.cuh"
#include "machines.cuh"
#include "potentials.cuh"

namespace gpc {
namespace adj {

constexpr int kCkptEvery = 64;              // accepted steps per checkpointed segment
constexpr int kMaxParam = 3 * kMaxComp;     // differentiable parameters per group
constexpr int kMaxRejects = 1000;           // consecutive rejected attempts per step

// ------------------------------------------------------- parameters ---
// Differentiable parameters of a component, in this order:
//   PowerSphericalPotentialwCutoff: amp, rc        (galpy args 0, 2)
//   MiyamotoNagai:                  amp, a, b      (args 0, 1, 2)
//   NFW, Hernquist:                 amp, a         (args 0, 1)
//   LogarithmicHalo:                amp, q, core^2 (args 0, 1, 2)
GPC_HD GPC_FI int comp_nparam(int type)
{
  switch (type) {
    case T_PSWC: return 2;
    case T_MN: return 3;
    case T_NFW: return 2;
    case T_HERNQUIST: return 2;
    case T_LOGHALO: return 3;
    default: return 0;
  }
}
inline int comp_param_arg(int type, int p) { return (type == T_PSWC && p == 1) ? 2 : p; }

GPC_HD GPC_FI int group_nparam(const GpComp* comp, int ncomp)
{
  int n = 0;
  for (int k = 0; k < ncomp; k++) n += comp_nparam(ldg(&comp[k].type));
  return n;
}

// g[p] += lambda . d a(x) / d theta_p for the parameters of one group
// (a = the acceleration; lambda = (lx, ly, lz), lz unused when PLANAR).
template <bool PLANAR>
GPC_HD void accel_param_vjp(const GpComp* __restrict__ comp, int ncomp, double x, double y,
                            double z, double lx, double ly, double lz, double* g)
{
  if (PLANAR) z = lz = 0.0;
  const double R2 = x * x + y * y, z2 = z * z, r2 = R2 + z2;
  const double xl = x * lx + y * ly + z * lz;  // x . lambda: spherical terms a = f(r) x
  int p = 0;
  for (int k = 0; k < ncomp; k++) {
    const GpComp* cp = comp + k;
    const double amp = ldg(&cp->c[0]);
    switch (ldg(&cp->type)) {
      case T_PSWC: {
        // f = -amp M(r)/r^3, M = 2 pi rc^(3-alpha) gamma(a, r^2/rc^2):
        // dM/drc = ((3 - alpha) M - 4 pi r^(3-alpha) e^(-u)) / rc
        const double u = r2 * ldg(&cp->c[1]);
        const double pw = exp(ldg(&cp->c[3]) * log(r2));  // (r^2)^(-alpha/2)
        double Mr3;
        if (u < ldg(&cp->c[5])) {
          Mr3 = ldg(&cp->c[2]) * pw * gamma_star<double>(tables(cp), u, ldg(&cp->c[6]));
        } else {
          const double ir = rsq(r2);
          Mr3 = ldg(&cp->c[4]) * ir * ir * ir;
        }
        const double alpha = -2.0 * ldg(&cp->c[3]), rc = ldg(&cp->c[9]);
        g[p] -= Mr3 * xl;
        g[p + 1] -= amp * ((3.0 - alpha) * Mr3 - ldg(&cp->c[7]) * pw * exp(-u)) / rc * xl;
        p += 2;
        break;
      }
      case T_MN: {
        // a = (x gR, y gR, z gz): gR = -amp D^-3/2, gz = -amp (s/zeta) D^-3/2,
        // zeta = sqrt(z^2 + b^2), s = a + zeta, D = R^2 + s^2
        const double a = ldg(&cp->c[1]), b2 = ldg(&cp->c[2]), b = sqrt(b2);
        const double zb2 = z2 + b2, izb = rsq(zb2), zeta = zb2 * izb, s = a + zeta;
        const double iD = rsq(R2 + s * s), iD3 = iD * iD * iD, iD5 = iD3 * iD * iD;
        const double xyl = x * lx + y * ly, zl = z * lz;
        g[p] += -iD3 * xyl - s * izb * iD3 * zl;
        g[p + 1] += 3.0 * amp * s * iD5 * xyl - amp * (iD3 - 3.0 * s * s * iD5) * izb * zl;
        const double bz = b * izb;  // d zeta / d b = d s / d b
        g[p + 2] += 3.0 * amp * s * iD5 * bz * xyl -
                    amp * bz * (iD3 * izb - s * iD3 * izb * izb - 3.0 * s * s * iD5 * izb) * zl;
        p += 3;
        break;
      }
      case T_NFW: {
        // f = amp / r^2 (1/(a+r) - ln(1+r/a)/r);  df/da = amp / (r a (a+r)^2)
        const double a = ldg(&cp->c[1]);
        const double ir = rsq(r2), r = r2 * ir, iar = 1.0 / (a + r);
        g[p] += ir * ir * (iar - log1p(r * ldg(&cp->c[2])) * ir) * xl;
        g[p + 1] += amp * ir * ldg(&cp->c[2]) * iar * iar * xl;
        p += 2;
        break;
      }
      case T_HERNQUIST: {
        // f = -amp / (2 r (r+a)^2);  df/da = amp / (r (r+a)^3)
        const double a = ldg(&cp->c[1]);
        const double ir = rsq(r2), ira = 1.0 / (r2 * ir + a);
        g[p] -= 0.5 * ir * ira * ira * xl;
        g[p + 1] += amp * ir * ira * ira * ira * xl;
        p += 2;
        break;
      }
      case T_LOGHALO: {
        // a = g (x, e y, z/q^2), g = -amp / D, D = x^2 + e y^2 + z^2/q^2 + core^2
        const double iq2 = ldg(&cp->c[1]), ye = ldg(&cp->c[3]);
        const double D = x * x + ye * y * y + z2 * iq2 + ldg(&cp->c[2]);
        const double iDl = 1.0 / D, gl = -amp * iDl;
        const double vl = x * lx + ye * y * ly + iq2 * z * lz;
        const double diq2 = -2.0 * iq2 * sqrt(iq2);  // d(1/q^2)/dq
        g[p] -= iDl * vl;
        g[p + 1] += amp * iDl * iDl * z2 * diq2 * vl + gl * diq2 * z * lz;
        g[p + 2] += amp * iDl * iDl * vl;
        p += 3;
        break;
      }
      default:
        break;
    }
  }
}

// The per-point force and vector-Jacobian functions are called, not
// inlined, in device code: a DOP853 step unrolls 12-16 stages, and inlining
// a force or tidal evaluation into every one of them made the kernels too
// large for the instruction cache (warps stalled on instruction fetch).
// Arguments and results travel in registers (scalars and a small struct).
#if defined(__CUDACC__)
#define GPC_NI __noinline__
#else
#define GPC_NI
#endif

struct V3 {
  double x, y, z;
};

// mu_q = K(q) lv (K the symmetric tidal tensor); g += (da/dtheta)^T lv.
template <bool PLANAR>
GPC_HD GPC_NI V3 vjp_at(const GpComp* __restrict__ comp, int ncomp, double x, double y, double z,
                        double lx, double ly, double lz, double* g)
{
  double ax, ay, az, K[6];
  if (PLANAR) z = lz = 0.0;
  accel_tidal<PLANAR>(comp, ncomp, x, y, z, ax, ay, az, K);
  V3 r;
  r.x = K[0] * lx + K[1] * ly + K[3] * lz;
  r.y = K[1] * lx + K[2] * ly + K[4] * lz;
  r.z = K[3] * lx + K[4] * ly + K[5] * lz;
  accel_param_vjp<PLANAR>(comp, ncomp, x, y, z, lx, ly, lz, g);
  return r;
}

template <int D>
GPC_HD GPC_FI void accel_vjp(const GpComp* __restrict__ comp, int ncomp, const double* q,
                             const double* lv, double* Kv, double* g)
{
  const V3 r = vjp_at<D == 2>(comp, ncomp, q[0], q[1], D == 3 ? q[D - 1] : 0.0, lv[0], lv[1],
                              D == 3 ? lv[D - 1] : 0.0, g);
  Kv[0] = r.x;
  Kv[1] = r.y;
  if (D == 3) Kv[D - 1] = r.z;
}

// ---------------------------------------------------------- tableau ---
// The DOP853 stages as one 16-stage explicit scheme (0-based stage index;
// stage 12 is the evaluation at the new state, whose input weights are the
// 8th-order solution weights b; stages 13-15 are the dense-output stages).
// A(i, j) is the weight of stage j in the input of stage i (Hairer's a_ij).
GPC_HD constexpr double A(int i, int j)
{
  using namespace dp;
  switch (i * 16 + j) {
    case 1 * 16 + 0: return a21;
    case 2 * 16 + 0: return a31;
    case 2 * 16 + 1: return a32;
    case 3 * 16 + 0: return a41;
    case 3 * 16 + 2: return a43;
    case 4 * 16 + 0: return a51;
    case 4 * 16 + 2: return a53;
    case 4 * 16 + 3: return a54;
    case 5 * 16 + 0: return a61;
    case 5 * 16 + 3: return a64;
    case 5 * 16 + 4: return a65;
    case 6 * 16 + 0: return a71;
    case 6 * 16 + 3: return a74;
    case 6 * 16 + 4: return a75;
    case 6 * 16 + 5: return a76;
    case 7 * 16 + 0: return a81;
    case 7 * 16 + 3: return a84;
    case 7 * 16 + 4: return a85;
    case 7 * 16 + 5: return a86;
    case 7 * 16 + 6: return a87;
    case 8 * 16 + 0: return a91;
    case 8 * 16 + 3: return a94;
    case 8 * 16 + 4: return a95;
    case 8 * 16 + 5: return a96;
    case 8 * 16 + 6: return a97;
    case 8 * 16 + 7: return a98;
    case 9 * 16 + 0: return a101;
    case 9 * 16 + 3: return a104;
    case 9 * 16 + 4: return a105;
    case 9 * 16 + 5: return a106;
    case 9 * 16 + 6: return a107;
    case 9 * 16 + 7: return a108;
    case 9 * 16 + 8: return a109;
    case 10 * 16 + 0: return a111;
    case 10 * 16 + 3: return a114;
    case 10 * 16 + 4: return a115;
    case 10 * 16 + 5: return a116;
    case 10 * 16 + 6: return a117;
    case 10 * 16 + 7: return a118;
    case 10 * 16 + 8: return a119;
    case 10 * 16 + 9: return a1110;
    case 11 * 16 + 0: return a121;
    case 11 * 16 + 3: return a124;
    case 11 * 16 + 4: return a125;
    case 11 * 16 + 5: return a126;
    case 11 * 16 + 6: return a127;
    case 11 * 16 + 7: return a128;
    case 11 * 16 + 8: return a129;
    case 11 * 16 + 9: return a1210;
    case 11 * 16 + 10: return a1211;
    case 12 * 16 + 0: return b1;
    case 12 * 16 + 5: return b6;
    case 12 * 16 + 6: return b7;
    case 12 * 16 + 7: return b8;
    case 12 * 16 + 8: return b9;
    case 12 * 16 + 9: return b10;
    case 12 * 16 + 10: return b11;
    case 12 * 16 + 11: return b12;
    case 13 * 16 + 0: return a141;
    case 13 * 16 + 6: return a147;
    case 13 * 16 + 7: return a148;
    case 13 * 16 + 8: return a149;
    case 13 * 16 + 9: return a1410;
    case 13 * 16 + 10: return a1411;
    case 13 * 16 + 11: return a1412;
    case 13 * 16 + 12: return a1413;
    case 14 * 16 + 0: return a151;
    case 14 * 16 + 5: return a156;
    case 14 * 16 + 6: return a157;
    case 14 * 16 + 7: return a158;
    case 14 * 16 + 10: return a1511;
    case 14 * 16 + 11: return a1512;
    case 14 * 16 + 12: return a1513;
    case 14 * 16 + 13: return a1514;
    case 15 * 16 + 0: return a161;
    case 15 * 16 + 5: return a166;
    case 15 * 16 + 6: return a167;
    case 15 * 16 + 7: return a168;
    case 15 * 16 + 8: return a169;
    case 15 * 16 + 12: return a1613;
    case 15 * 16 + 13: return a1614;
    case 15 * 16 + 14: return a1615;
    default: return 0.0;
  }
}

// Dense-output coefficient d_{m+4, j} of stage j (m = 0..3).
GPC_HD constexpr double Dc(int m, int j)
{
  using namespace dp;
  switch (m * 16 + j) {
    case 0 * 16 + 0: return d41;
    case 0 * 16 + 5: return d46;
    case 0 * 16 + 6: return d47;
    case 0 * 16 + 7: return d48;
    case 0 * 16 + 8: return d49;
    case 0 * 16 + 9: return d410;
    case 0 * 16 + 10: return d411;
    case 0 * 16 + 11: return d412;
    case 0 * 16 + 12: return d413;
    case 0 * 16 + 13: return d414;
    case 0 * 16 + 14: return d415;
    case 0 * 16 + 15: return d416;
    case 1 * 16 + 0: return d51;
    case 1 * 16 + 5: return d56;
    case 1 * 16 + 6: return d57;
    case 1 * 16 + 7: return d58;
    case 1 * 16 + 8: return d59;
    case 1 * 16 + 9: return d510;
    case 1 * 16 + 10: return d511;
    case 1 * 16 + 11: return d512;
    case 1 * 16 + 12: return d513;
    case 1 * 16 + 13: return d514;
    case 1 * 16 + 14: return d515;
    case 1 * 16 + 15: return d516;
    case 2 * 16 + 0: return d61;
    case 2 * 16 + 5: return d66;
    case 2 * 16 + 6: return d67;
    case 2 * 16 + 7: return d68;
    case 2 * 16 + 8: return d69;
    case 2 * 16 + 9: return d610;
    case 2 * 16 + 10: return d611;
    case 2 * 16 + 11: return d612;
    case 2 * 16 + 12: return d613;
    case 2 * 16 + 13: return d614;
    case 2 * 16 + 14: return d615;
    case 2 * 16 + 15: return d616;
    case 3 * 16 + 0: return d71;
    case 3 * 16 + 5: return d76;
    case 3 * 16 + 6: return d77;
    case 3 * 16 + 7: return d78;
    case 3 * 16 + 8: return d79;
    case 3 * 16 + 9: return d710;
    case 3 * 16 + 10: return d711;
    case 3 * 16 + 11: return d712;
    case 3 * 16 + 12: return d713;
    case 3 * 16 + 13: return d714;
    case 3 * 16 + 14: return d715;
    case 3 * 16 + 15: return d716;
    default: return 0.0;
  }
}

// Weights W_j(s) of the dense output y(t_n + s h) = y_n + h sum_j W_j k_j.
// Hairer's continuous extension
//   y + s (dy + s' (bspl + s (r4 + s' (r5 + s (r6 + s' (r7 + s r8))))))
// (s' = 1 - s, dy = h sum b_j k_j, bspl = h k_0 - dy,
// r4 = dy - h k_12 - bspl, r_{m} = h sum_j d_{m,j} k_j) is linear in the
// stages; expanding the products gives these weights.
GPC_HD GPC_FI void dense_weights(double s, double* W)
{
  const double s1 = 1.0 - s;
  const double P1 = s, P2 = s * s1, P3 = s * P2, P4 = P3 * s1, P5 = P4 * s, P6 = P5 * s1,
               P7 = P6 * s;
  const double cb = P1 - P2 + 2.0 * P3;
#pragma unroll
  for (int j = 0; j < 16; j++)
    W[j] = cb * A(12, j) + P4 * Dc(0, j) + P5 * Dc(1, j) + P6 * Dc(2, j) + P7 * Dc(3, j);
  W[0] += P2 - P3;
  W[12] -= P3;
}

// ------------------------------------------------------------ field ---
template <class POT>
struct Field {
  const GpComp* comp;
  int ncomp;
  const double* scal;
};

// ------------------------------------------- Nystrom stages, in pairs ---
// Two accelerations at once: compile-time lists side by side, run-time lists
// component by component.
template <int D, class POT>
GPC_HD GPC_FI void accel_pair(const Field<POT>& F, const double* q1, const double* q2, double* a1,
                              double* a2)
{
  eval_force2<D, PREC_FP64, false, POT>(F.comp, F.ncomp, q1, q2, a1, a2, F.scal, 0.0, 0.0);
}

// A step's accelerations a_1..a_16 (a[k - 1]; a NQ = D system), indexed at
// compile time only so that they live in registers.
template <int D, int S>
struct Accs {
  double v[S][D];
  template <int Kk>
  GPC_HD GPC_FI double a(int i) const
  {
    return v[Kk - 1][i];
  }
};
template <int D, int I, int Kk, int S>
GPC_HD GPC_FI void pos_term(const Accs<D, S>& a, double* s)
{
  constexpr bool nz = Kk <= S && kNy.x[I - 1][Kk - 1] != 0.0;
  if constexpr (nz) {
    const double w = GPC_NY.x[I - 1][Kk - 1];
#pragma unroll
    for (int i = 0; i < D; i++) s[i] += w * a.v[Kk - 1][i];
  }
}
template <int D, int I, int S, int... Kk>
GPC_HD GPC_FI void stage_pos(const Accs<D, S>& a, const double* x, const double* v, double h,
                             double* q, Ints<Kk...>)
{
  double s[D];
#pragma unroll
  for (int i = 0; i < D; i++) s[i] = 0.0;
  (pos_term<D, I, Kk + 1>(a, s), ...);
  const double ch = GPC_NY.c[I - 1] * h, h2 = h * h;
#pragma unroll
  for (int i = 0; i < D; i++)
    q[i] = I == 13 ? x[i] + mad(h, v[i], h2 * s[i]) : mad(h2, s[i], mad(ch, v[i], x[i]));
}
template <int D, int I, int S>
GPC_HD GPC_FI void stage_pos(const Accs<D, S>& a, const double* x, const double* v, double h,
                             double* q)
{
  stage_pos<D, I>(a, x, v, h, q, Count<14>());
}
template <int D>
GPC_HD GPC_FI void copy(const double* from, double* to)
{
#pragma unroll
  for (int i = 0; i < D; i++) to[i] = from[i];
}

// Rounds 0..5 of a step (stages 2, 3; ...; 12, 13) from (x, v) with a_1
// given; x13 receives the new position.
template <int D, class POT, int S>
GPC_HD GPC_FI void step_rounds(const Field<POT>& F, const double* x, const double* v, double h,
                               Accs<D, S>& a, double* x13)
{
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int r = 0; r < 6; r++) {
    double q1[D], q2[D], f1[D], f2[D];
    switch (r) {
      case 0: stage_pos<D, 2>(a, x, v, h, q1); stage_pos<D, 3>(a, x, v, h, q2); break;
      case 1: stage_pos<D, 4>(a, x, v, h, q1); stage_pos<D, 5>(a, x, v, h, q2); break;
      case 2: stage_pos<D, 6>(a, x, v, h, q1); stage_pos<D, 7>(a, x, v, h, q2); break;
      case 3: stage_pos<D, 8>(a, x, v, h, q1); stage_pos<D, 9>(a, x, v, h, q2); break;
      case 4: stage_pos<D, 10>(a, x, v, h, q1); stage_pos<D, 11>(a, x, v, h, q2); break;
      default: stage_pos<D, 12>(a, x, v, h, q1); stage_pos<D, 13>(a, x, v, h, q2);
    }
    accel_pair<D, POT>(F, q1, q2, f1, f2);
    switch (r) {
      case 0: copy<D>(f1, a.v[1]); copy<D>(f2, a.v[2]); break;
      case 1: copy<D>(f1, a.v[3]); copy<D>(f2, a.v[4]); break;
      case 2: copy<D>(f1, a.v[5]); copy<D>(f2, a.v[6]); break;
      case 3: copy<D>(f1, a.v[7]); copy<D>(f2, a.v[8]); break;
      case 4: copy<D>(f1, a.v[9]); copy<D>(f2, a.v[10]); break;
      default: copy<D>(f1, a.v[11]); copy<D>(f2, a.v[12]); copy<D>(q2, x13);
    }
  }
}
// The dense-output stages 14..16.
template <int D, class POT>
GPC_HD GPC_FI void dense_rounds(const Field<POT>& F, const double* x, const double* v, double h,
                                Accs<D, 16>& a)
{
  double q1[D], q2[D];
  stage_pos<D, 14>(a, x, v, h, q1);
  stage_pos<D, 15>(a, x, v, h, q2);
  accel_pair<D, POT>(F, q1, q2, a.v[13], a.v[14]);
  stage_pos<D, 16>(a, x, v, h, q1);
  accel_pair<D, POT>(F, q1, q1, a.v[15], q2);
}

// Weights of the dense output for the accelerations: v(T) = v + h sum W_j
// a_j (dense_weights), x(T) = x + h s v + h^2 sum Wx_k a_k with Wx = W A.
GPC_HD GPC_FI void dense_weights2(double s, double* W, double* Wx)
{
  dense_weights(s, W);
#pragma unroll
  for (int k = 0; k < 16; k++) {
    double w = 0.0;
#pragma unroll
    for (int j = k + 1; j < 16; j++) {
      const double a = A(j, k);
      if (a != 0.0) w += W[j] * a;
    }
    Wx[k] = w;
  }
}

// ------------------------------------------------------- controller ---
struct Ctl {
  double h, hnew, hmax, pos_neg, rtol, atol, t;
  bool reject;
};

GPC_HD GPC_FI void begin_attempt(Ctl& c) { c.h = c.pos_neg * dmax(fabs(c.h), 1e3 * 2.3e-16); }

// Initial step (leung_dop853.c:296-324); leaves a1 = a(x).
template <int D, class POT>
GPC_HD void hinit(const Field<POT>& F, const double* x, const double* v, double* a1, Ctl& c)
{
  double q[D], f[D], g[D];
  accel_pair<D, POT>(F, x, x, a1, g);
  double dnf = 0.0, dny = 0.0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const double sx = c.atol + c.rtol * fabs(x[i]), sv = c.atol + c.rtol * fabs(v[i]);
    dnf += (v[i] / sx) * (v[i] / sx) + (a1[i] / sv) * (a1[i] / sv);
    dny += (x[i] / sx) * (x[i] / sx) + (v[i] / sv) * (v[i] / sv);
  }
  c.h = csign(dmin(sqrt(dny / dnf) * 0.01, fabs(c.hmax)), c.pos_neg);
#pragma unroll
  for (int i = 0; i < D; i++) q[i] = x[i] + c.h * v[i];
  accel_pair<D, POT>(F, q, q, f, g);
  double der2 = 0.0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const double sx = c.atol + c.rtol * fabs(x[i]), sv = c.atol + c.rtol * fabs(v[i]);
    const double dx = c.h * a1[i] / sx, dv = (f[i] - a1[i]) / sv;
    der2 += dx * dx + dv * dv;
  }
  der2 = sqrt(der2) / c.h;
  const double der12 = dmax(fabs(der2), sqrt(dnf));
  const double h1 = pow(0.01 / der12, 1.0 / 8.0);
  c.h = csign(dmin(100.0 * fabs(c.h), dmin(fabs(h1), fabs(c.hmax))), c.pos_neg);
  begin_attempt(c);
}

// The controller's decision on an attempt with error norm e
// (leung_dop853.c:419-440): 1 accepted (c.hnew proposed), 0 rejected (c.h
// reduced for the next attempt), -1 non-finite.
GPC_HD GPC_FI int decide(double e, Ctl& c)
{
  if (!isfinite(e)) return -1;
  const double fac = 0.9 * root8_inv(e);
  if (e <= 1.0) {
    c.hnew = c.h * dmin(6.0, dmax(0.333, fac));
    return 1;
  }
  c.hnew = c.h * dmax(0.333, fac);
  c.reject = true;
  c.h = c.hnew;
  begin_attempt(c);
  return 0;
}

// Step size of the next step after an accepted one (leung_dop853.c:476-500).
GPC_HD GPC_FI void next_step(Ctl& c)
{
  double hnew = (fabs(c.hnew) > fabs(c.hmax)) ? c.pos_neg * c.hmax : c.hnew;
  if (c.reject) hnew = c.pos_neg * dmin(fabs(hnew), fabs(c.h));
  c.reject = false;
  c.h = hnew;
  begin_attempt(c);
}

GPC_HD GPC_FI void init_ctl(Ctl& c, double t0, double T, double rtol_ln, double atol_ln)
{
  c.rtol = exp(rtol_ln);
  c.atol = exp(atol_ln);
  c.hmax = T - t0;
  c.pos_neg = csign(1.0, c.hmax);
  c.t = t0;
  c.reject = false;
  c.h = c.hnew = 0.0;
}

// y(T) from the start of the step that contains T (a_1..a_13 given; s = (T -
// t_n) / h): the dense-output stages and their weights.
template <int D, class POT>
GPC_HD GPC_FI void final_rows(const Field<POT>& F, const double* x, const double* v, double h,
                              double s, Accs<D, 16>& a, double* yT)
{
  dense_rounds<D, POT>(F, x, v, h, a);
  double W[16], Wx[16];
  dense_weights2(s, W, Wx);
#pragma unroll
  for (int i = 0; i < D; i++) {
    double sx = 0.0, sv = 0.0;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      sx += Wx[j] * a.v[j][i];
      sv += W[j] * a.v[j][i];
    }
    yT[i] = x[i] + h * (s * v[i] + h * sx);
    yT[D + i] = v[i] + h * sv;
  }
}

// Checkpoint record of a segment: y[N] and t at its start, then the step
// sizes of its (up to) kCkptEvery accepted steps.
template <int D>
struct Ckpt {
  static constexpr int H = 2 * D + 1;  // offset of the step sizes
  static constexpr int W = H + kCkptEvery;
};

// ---------------------------------------------------------- forward ---
// Integrate one orbit from t0 to T.  Checkpoints go to ck[(c*W + f)*cs]
// (c < ccap); the accepted step sizes, if hrec is not null, to
// hrec[n*hs] (n < hcap).  Returns the status (E_OK, E_BUDGET when the
// attempt budget, checkpoint or step capacity is exhausted, E_NONFINITE).
template <int D, class POT>
GPC_HD int forward_orbit(const Field<POT>& F, const double* w0, double t0, double T,
                         double rtol_ln, double atol_ln, long long max_att, double* ck,
                         long long cs, int ccap, double* hrec, long long hs, long long hcap,
                         double* yT, long long* nsteps)
{
  constexpr int N = 2 * D, CW = Ckpt<D>::W;
  double x[D], v[D], xn[D], vn[D];
  Accs<D, 16> a;
  copy<D>(w0, x);
  copy<D>(w0 + D, v);
  *nsteps = 0;
  if (T == t0) {
    copy<D>(x, yT);
    copy<D>(v, yT + D);
    return E_OK;
  }
  Ctl c;
  init_ctl(c, t0, T, rtol_ln, atol_ln);
  hinit<D, POT>(F, x, v, a.v[0], c);
  long long n = 0, att = 0;
  int rej = 0;
  for (;;) {
    if (n % kCkptEvery == 0 && rej == 0) {
      const long long seg = n / kCkptEvery;
      if (seg >= ccap) return E_BUDGET;
      double* p = ck + seg * CW * cs;
#pragma unroll
      for (int i = 0; i < D; i++) {
        p[i * cs] = x[i];
        p[(D + i) * cs] = v[i];
      }
      p[N * cs] = c.t;
    }
    // one attempt: the lanes of a warp run theirs together, whether the last
    // one was accepted or not
    step_rounds<D, POT>(F, x, v, c.h, a, xn);
    const double e = dop853_error<D>(a, x, v, xn, c.h, c.rtol, c.atol, vn);
    const int r = decide(e, c);
    att++;
    if (r < 0) return E_NONFINITE;
    if (r == 0) {
      // every rejection shrinks h by at least 1/1.11 down to the floor of
      // begin_attempt; an orbit still rejected long after that is stopped
      if (++rej >= kMaxRejects || (max_att > 0 && att >= max_att)) return E_BUDGET;
      continue;
    }
    rej = 0;
    ck[((n / kCkptEvery) * CW + Ckpt<D>::H + n % kCkptEvery) * cs] = c.h;
    if (hrec) {
      if (n >= hcap) return E_BUDGET;
      hrec[n * hs] = c.h;
    }
    const double t_start = c.t;
    c.t = t_start + c.h;
    n++;
    if (c.pos_neg * T < c.pos_neg * c.t) {  // T lies in this step
      final_rows<D, POT>(F, x, v, c.h, (T - t_start) / c.h, a, yT);
      *nsteps = n;
      return E_OK;
    }
    copy<D>(xn, x);
    copy<D>(vn, v);
    copy<D>(a.v[12], a.v[0]);  // FSAL: the force at the new state starts the next step
    next_step(c);
    if (max_att > 0 && att >= max_att) return E_BUDGET;
  }
}

// ------------------------------------------------ replay (fixed steps) ---
// The forward map with the step sizes held at recorded values h[n*hs],
// n < nsteps (the function the adjoint differentiates; finite differences
// of it check the gradients).
template <int D, class POT>
GPC_HD void replay_orbit(const Field<POT>& F, const double* w0, double t0, double T,
                         const double* hrec, long long hs, long long nsteps, double* yT)
{
  double x[D], v[D], xn[D];
  Accs<D, 16> a;
  copy<D>(w0, x);
  copy<D>(w0 + D, v);
  if (nsteps <= 0) {
    copy<D>(x, yT);
    copy<D>(v, yT + D);
    return;
  }
  double t = t0;
  accel_pair<D, POT>(F, x, x, a.v[0], xn);
  for (long long n = 0;; n++) {
    const double h = hrec[n * hs];
    step_rounds<D, POT>(F, x, v, h, a, xn);
    if (n == nsteps - 1) {
      final_rows<D, POT>(F, x, v, h, (T - t) / h, a, yT);
      return;
    }
#pragma unroll
    for (int i = 0; i < D; i++) v[i] = v[i] + h * dop853_increment(a, i);
    copy<D>(xn, x);
    copy<D>(a.v[12], a.v[0]);
    t = t + h;
  }
}

// --------------------------------------------------------- backward ---
// mu = K(q) l and g += (da/dtheta)^T l at one point.  MWPotential2014's list
// in one pass: the spherical components' K l = -c (x . l) x - (Phi'/r) l needs
// no tensor, and the force's table functions serve both (the general form,
// vjp_at, evaluates them again through the library's logarithm and power).
template <bool PLANAR>
GPC_HD GPC_FI void mw14_vjp(const GpComp* __restrict__ comp, const double* q, const double* l,
                            double* mu, double* g)
{
  const double x = q[0], y = q[1], z = PLANAR ? 0.0 : q[PLANAR ? 0 : 2];
  const double lx = l[0], ly = l[1], lz = PLANAR ? 0.0 : l[PLANAR ? 0 : 2];
  const double R2 = x * x + y * y, z2 = z * z, r2 = R2 + z2;
  const double xyl = x * lx + y * ly, zl = z * lz, xl = xyl + zl;
  const double ir = rsqrt_nr(r2), ir2 = ir * ir, ir3 = ir2 * ir;
  const Mw14Sphere S = mw14_sphere(comp, r2, ir, ir2, ir3);
  const double dpr = S.dpr, c = S.c;
  {  // bulge
    const double rc = ldg(&comp->c[9]);
    g[0] -= S.Mr3 * xl;
    g[1] -= ldg(&comp->c[0]) * ((3.0 + 2.0 * ldg(&comp->c[3])) * S.Mr3 - S.rho) *
            (rc * ldg(&comp->c[1])) * xl;
  }
  {  // halo
    const GpComp* cp = comp + 2;
    g[5] -= S.f * xl;
    g[6] += ldg(&cp->c[0]) * ir * ldg(&cp->c[2]) * S.iar * S.iar * xl;
  }
  const double cx = c * xl;
  mu[0] = -cx * x - dpr * lx;
  mu[1] = -cx * y - dpr * ly;
  if (!PLANAR) mu[PLANAR ? 0 : 2] = -cx * z - dpr * lz;
  {  // disk: s = a + zeta, zeta = sqrt(z^2 + b^2), D = R^2 + s^2
    const GpComp* cp = comp + 1;
    const double amp = ldg(&cp->c[0]), a = ldg(&cp->c[1]), b2 = ldg(&cp->c[2]);
    const double zb2 = z2 + b2, izb = rsqrt_nr(zb2), s = a + zb2 * izb, sz = fma(a, izb, 1.0);
    const double iD = rsqrt_nr(fma(s, s, R2)), iD2 = iD * iD, iD3 = iD2 * iD;
    const double B = xyl + sz * zl, w = 3.0 * iD3 * iD2 * B;
    mu[0] += amp * (w * x - iD3 * lx);
    mu[1] += amp * (w * y - iD3 * ly);
    if (!PLANAR)
      mu[PLANAR ? 0 : 2] += amp * (w * sz * z - (sz - a * z2 * izb * izb * izb) * iD3 * lz);
    // da/ds: dD^(-3/2)/ds = -3 s D^(-5/2); ds/da = 1, ds/db = b / zeta
    const double ds = amp * (s * w - iD3 * izb * zl), bz = sqrt(b2) * izb;
    g[2] -= iD3 * B;
    g[3] += ds;
    g[4] += bz * (ds + amp * iD3 * s * izb * izb * zl);
  }
}
template <int D, class POT>
GPC_HD GPC_FI void vjp_pair(const Field<POT>& F, const double* q1, const double* l1, double* mu1,
                            const double* q2, const double* l2, double* mu2, double* g)
{
  if constexpr (IsMw14<POT>::value) {
    mw14_vjp<D == 2>(F.comp, q1, l1, mu1, g);
    mw14_vjp<D == 2>(F.comp, q2, l2, mu2, g);
  } else {
    accel_vjp<D>(F.comp, F.ncomp, q1, l1, mu1, g);
    accel_vjp<D>(F.comp, F.ncomp, q2, l2, mu2, g);
  }
}
// Parameters of a list: at most the fixed list's seven in registers, else any.
template <class POT>
GPC_HD constexpr int param_capacity()
{
  return IsMw14<POT>::value ? 7 : kMaxParam;
}

// Stage positions and, once a stage's adjoint is known, mu in its place.
template <int D, int S>
struct Stages {
  double v[S][D];
};
template <int D, int K1, int I, int S>
GPC_HD GPC_FI void kappa_term(const Stages<D, S>& m, double* s)
{
  if constexpr (I <= S && I >= K1 + 2 && K1 <= 14) {
    constexpr bool nz = kNy.x[I - 1][K1 <= 14 ? K1 - 1 : 0] != 0.0;
    if constexpr (nz) {
      const double w = GPC_NY.x[I - 1][K1 <= 14 ? K1 - 1 : 0];
#pragma unroll
      for (int i = 0; i < D; i++) s[i] += w * m.v[I - 1][i];
    }
  }
}
// kappa of stage K1 (1-based) with output weights (wx, wv) of its
// acceleration in x and v.
template <int D, int K1, int S, int... I>
GPC_HD GPC_FI void kappa(const Stages<D, S>& m, double h, double wx, double wv, const double* lx,
                         const double* lv, double* k, Ints<I...>)
{
  double s[D];
#pragma unroll
  for (int i = 0; i < D; i++) s[i] = wx * lx[i];
  (kappa_term<D, K1, I + 1>(m, s), ...);
#pragma unroll
  for (int i = 0; i < D; i++) k[i] = h * (wv * lv[i] + h * s[i]);
}
// Stages K1 and K1 + 1 of the reverse sweep.
template <int D, int K1, class POT, int S>
GPC_HD GPC_FI void kappa_pair(Stages<D, S>& m, double h, const double* Wx, const double* W,
                              const double* lx, const double* lv, double* q1, double* l1,
                              double* q2, double* l2)
{
  kappa<D, K1>(m, h, Wx[K1 - 1], W[K1 - 1], lx, lv, l1, Count<S>());
  kappa<D, K1 + 1>(m, h, Wx[K1], W[K1], lx, lv, l2, Count<S>());
  copy<D>(m.v[K1 - 1], q1);
  copy<D>(m.v[K1], q2);
}

// Adjoint of one step from (x, v) with step h and a_1 = a(x): (lx, lv) (dL/d
// output) becomes dL/d(x, v); g accumulates dL/dtheta.  LAST: the step is the
// dense-output map to s = (T - t_n)/h.
template <int D, class POT, bool LAST>
GPC_HD GPC_FI void step_vjp(const Field<POT>& F, const double* x, const double* v,
                            const double* a1, double h, double s, double* lx, double* lv,
                            double* g)
{
  constexpr int S = LAST ? 16 : 12;
  Stages<D, S> m;
  {  // the positions of the stages (a full step's last two need no force)
    Accs<D, LAST ? 14 : 10> a;
    copy<D>(a1, a.v[0]);
    copy<D>(x, m.v[0]);
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int r = 0; r < (LAST ? 7 : 5); r++) {
      double q1[D], q2[D], f1[D], f2[D];
      switch (r) {
        case 0: stage_pos<D, 2>(a, x, v, h, q1); stage_pos<D, 3>(a, x, v, h, q2); break;
        case 1: stage_pos<D, 4>(a, x, v, h, q1); stage_pos<D, 5>(a, x, v, h, q2); break;
        case 2: stage_pos<D, 6>(a, x, v, h, q1); stage_pos<D, 7>(a, x, v, h, q2); break;
        case 3: stage_pos<D, 8>(a, x, v, h, q1); stage_pos<D, 9>(a, x, v, h, q2); break;
        case 4: stage_pos<D, 10>(a, x, v, h, q1); stage_pos<D, 11>(a, x, v, h, q2); break;
        default:
          if constexpr (LAST) {
            if (r == 5) {
              stage_pos<D, 12>(a, x, v, h, q1);
              stage_pos<D, 13>(a, x, v, h, q2);
            } else {
              stage_pos<D, 14>(a, x, v, h, q1);
              stage_pos<D, 15>(a, x, v, h, q2);
            }
          }
      }
      accel_pair<D, POT>(F, q1, q2, f1, f2);
      switch (r) {
#define GPC_ADJ_KEEP(i)                                                    \
  copy<D>(q1, m.v[i]), copy<D>(q2, m.v[i + 1]), copy<D>(f1, a.v[i]);       \
  if constexpr (i + 1 < (LAST ? 14 : 10)) copy<D>(f2, a.v[i + 1])
        case 0: GPC_ADJ_KEEP(1); break;
        case 1: GPC_ADJ_KEEP(3); break;
        case 2: GPC_ADJ_KEEP(5); break;
        case 3: GPC_ADJ_KEEP(7); break;
        case 4: GPC_ADJ_KEEP(9); break;
        default:
          if constexpr (LAST) {
            if (r == 5) {
              GPC_ADJ_KEEP(11);
            } else {
              GPC_ADJ_KEEP(13);
            }
          }
#undef GPC_ADJ_KEEP
      }
    }
    if constexpr (LAST)
      stage_pos<D, 16>(a, x, v, h, m.v[S - 1]);
    else
      stage_pos<D, 12>(a, x, v, h, m.v[S - 1]);
  }
  double W[S], Wx[S];
  if constexpr (LAST) {
    dense_weights2(s, W, Wx);
  } else {
#pragma unroll
    for (int j = 0; j < S; j++) {
      W[j] = GPC_NY.b[j];
      Wx[j] = GPC_NY.x[12][j];
    }
  }
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int r = S / 2 - 1; r >= 0; r--) {
    double q1[D], q2[D], l1[D], l2[D], u1[D], u2[D];
    switch (r) {
#define GPC_ADJ_KAPPA(r) \
  case r: kappa_pair<D, 2 * r + 1, POT>(m, h, Wx, W, lx, lv, q1, l1, q2, l2); break;
      GPC_ADJ_KAPPA(0)
      GPC_ADJ_KAPPA(1)
      GPC_ADJ_KAPPA(2)
      GPC_ADJ_KAPPA(3)
      GPC_ADJ_KAPPA(4)
      GPC_ADJ_KAPPA(5)
      default:
        if constexpr (LAST) {
          if (r == 6)
            kappa_pair<D, 13, POT>(m, h, Wx, W, lx, lv, q1, l1, q2, l2);
          else
            kappa_pair<D, 15, POT>(m, h, Wx, W, lx, lv, q1, l1, q2, l2);
        }
#undef GPC_ADJ_KAPPA
    }
    vjp_pair<D, POT>(F, q1, l1, u1, q2, l2, u2, g);
    switch (r) {
#define GPC_ADJ_MU(r) \
  case r: copy<D>(u1, m.v[2 * r]), copy<D>(u2, m.v[2 * r + 1]); break;
      GPC_ADJ_MU(0)
      GPC_ADJ_MU(1)
      GPC_ADJ_MU(2)
      GPC_ADJ_MU(3)
      GPC_ADJ_MU(4)
      GPC_ADJ_MU(5)
      default:
        if constexpr (LAST) {
          if (r == 6)
            copy<D>(u1, m.v[12]), copy<D>(u2, m.v[13]);
          else
            copy<D>(u1, m.v[14]), copy<D>(u2, m.v[15]);
        }
#undef GPC_ADJ_MU
    }
  }
  const double span = LAST ? s * h : h;
#pragma unroll
  for (int i = 0; i < D; i++) {
    double sx = 0.0, sv = 0.0;
#pragma unroll
    for (int k = 0; k < S; k++) {
      sx += m.v[k][i];
      sv += GPC_NY.c[k] * m.v[k][i];
    }
    lv[i] += span * lx[i] + h * sv;
    lx[i] += sx;
  }
}

// Backward sweep of one orbit: lam = dL/dy(T) on entry, dL/dy(t0) on exit;
// g (group_nparam entries, zeroed by the caller) accumulates dL/dtheta.
// ck/cs: the forward pass's checkpoints; nsteps its accepted steps.
template <int D, class POT>
GPC_HD void backward_orbit(const Field<POT>& F, double T, const double* ck, long long cs,
                           long long nsteps, double* lam, double* g)
{
  constexpr int CW = Ckpt<D>::W;
  if (nsteps <= 0) return;
  double xs[kCkptEvery][D], vs[kCkptEvery][D], as[kCkptEvery][D];
  double lx[D], lv[D];
  copy<D>(lam, lx);
  copy<D>(lam + D, lv);
  const long long nseg = (nsteps + kCkptEvery - 1) / kCkptEvery;
  for (long long seg = nseg - 1; seg >= 0; seg--) {
    // recompute the start states of the segment's steps
    const double* p = ck + seg * CW * cs;
    const double* hs = p + Ckpt<D>::H * cs;
    const long long n0 = seg * kCkptEvery;
    const int m1 = (int)((n0 + kCkptEvery < nsteps ? n0 + kCkptEvery : nsteps) - n0);
    double t = p[2 * D * cs];
    {
      double x[D], v[D], xn[D], q[D];
      Accs<D, 13> a;
#pragma unroll
      for (int i = 0; i < D; i++) {
        x[i] = p[i * cs];
        v[i] = p[(D + i) * cs];
      }
      accel_pair<D, POT>(F, x, x, a.v[0], q);
      for (int m = 0; m < m1; m++) {
        copy<D>(x, xs[m]);
        copy<D>(v, vs[m]);
        copy<D>(a.v[0], as[m]);
        if (m == m1 - 1) break;
        const double h = hs[m * cs];
        step_rounds<D, POT>(F, x, v, h, a, xn);
#pragma unroll
        for (int i = 0; i < D; i++) {
          v[i] = v[i] + h * dop853_increment(a, i);
          x[i] = xn[i];
          a.v[0][i] = a.v[12][i];
        }
        t = t + h;
      }
    }
    // reverse sweep over the segment's steps (t: the last one's start)
    for (int m = m1 - 1; m >= 0; m--) {
      const double h = hs[m * cs];
      if (n0 + m == nsteps - 1)
        step_vjp<D, POT, true>(F, xs[m], vs[m], as[m], h, (T - t) / h, lx, lv, g);
      else
        step_vjp<D, POT, false>(F, xs[m], vs[m], as[m], h, 0.0, lx, lv, g);
    }
  }
  copy<D>(lx, lam);
  copy<D>(lv, lam + D);
}

}  // namespace adj
}  // namespace gpc
