// Element kernels: residual, hand-derived tangent, QoI and DWR error chain of
// goal's stabilized mixed u-p mechanics on linear tets. By default one launch
// evaluates all elements into a buffer (a thread each: k_elem in FP64; k_elem_fix,
// the tangent of an overwriting Jacobian chain in 64-bit fixed point, with up to
// four threads to an element of a small mesh) and a second sums each matrix block
// and nodal row over its elements. Coloured chains accumulate in place, elements
// of one colour per launch (no two of them share a node). Neither needs atomics;
// both are deterministic.
//
// Reference chain (one integration point, src/goal_assembly.cpp:65-88):
//   Kinematics F = I + grad u, J = det F                   src/goal_kinematics.cpp:18-25
//   Neohookean sigma = mu J^-5/3 dev(F F^T) + k/2 (J-1/J) I  src/goal_neohookean.cpp:59-86
//   J2 trial be = J^-2/3 F Cp^-1 F^T, s = mu dev(be), radial return with linear
//      hardening, eqps/Fp/sigma state writes                src/goal_J2.cpp:71-156
//   Mixed sigma_ii += p - tr(sigma)/3                       src/goal_mixed.cpp:33-46
//   MResidual R^u_ai += P_ij dphi_a/dx_j w dv, P = J sigma F^-T   src/goal_mresidual.cpp:25-32
//   PResidual R^p_a += (p/kappa - (J-1/J)/2) phi_a w dv     src/goal_presidual.cpp:53-59
//   Stabilization R^p_a += tau J C^-1_ij dp/dx_i dphi_a/dx_j w dv, tau = c0 h^2/(2 mu)
//                                                            src/goal_stabilization.cpp:59-80
//   scatter PRIMAL (row-wise) / ADJOINT (transposed)        src/goal_displacement.cpp:177-214
//   QoI avg disp, KS max von Mises                          src/goal_avg_disp.cpp:16-21, src/goal_ks_vm.cpp:88-98
//   DWR weights z_diff phi_a, stabilization with z_coarse   src/goal_displacement_adjoint.cpp:37-53,
//                                                            src/goal_pressure_adjoint.cpp:38-49,
//                                                            src/goal_mechanics.cpp:169-218
//
// Tangent (replaces Sacado FAD). With G_a = grad phi_a, H = F^-T, h_a = H G_a,
// C = Cp^-1 (identity for neo-Hookean), B = F C F^T, Ic = tr B, m_a = F C G_a,
// q_a = m_a - Ic/3 h_a, alpha = mu J^-2/3, s = alpha dev B, the deviatoric
// Kirchhoff stress is S = gamma s (gamma = 1 when elastic) and
//   P G_a = S h_a + p J h_a.
// Its derivative in direction u_bk (dF = e_k (x) G_b) is
//   K^uu_{ai,bk} = V [ gamma alpha c_ab d_ik + h_ai X_bk + q_ai Y_bk + h_bi Z_ak ]
//   c_ab = G_a.C G_b,  X_b = -2/3 gamma alpha m_b + pJ h_b,
//   Y_b = -2/3 gamma alpha h_b + alpha dgamma_b,  Z_a = (gamma alpha Ic/3 - pJ) h_a,
// and for the plastic return (X = f / (2 mubar + kh), kh = 2K/3, or kh = 0 when
// goal's Newton loop stops after its first iterate)
//   dgamma_b = -A1 dmubar_b - A2 dsmag_b,  dmubar_b = 2 alpha/3 q_b,
//   dsmag_b = -2/3 smag h_b + 2 alpha/smag s m_b,
//   A1 = 2 f kh / (c^2 smag), A2 = 2 mubar k0 / (c smag^2).
// The pressure rows and columns:
//   K^up_{ai,b} = V J h_ai / 4
//   K^pu_{a,bk} = V [ h_bk (tau J w_a - (J+1/J)/8) - tau J e_ab v_k - tau J w_b h_ak ]
//   K^pp_{ab}   = V [ 1/(16 kappa) + tau J e_ab ]
// with v = H grad p, w_a = v.h_a, e_ab = h_a.h_b.
#include <type_traits>

#include "fixed.cuh"
#include "mechanics.cuh"

namespace goal {

namespace {

struct ElemArgs {
  DiscView d;
  const double* mats;
  const double* U;
  const double* Fp_old;
  const double* eqps_old;
  const double* Cpinv;
  double* sigma;
  double* Fp;
  double* eqps;
  double* Apend;   // 6 x E deferred plastic increments (see StatesDev)
  int* pend;
  double* R;
  double* A;
  double* dMdu;
  double* qoi_elem;
  const double* Zd;
  const double* Zc;
  int* failed;     // host memory: set when a return map fails
  double* ebuf;    // two-phase mode: per element [R (16) | 16 blocks x 16] (stride estride)
  double* dbuf;    // two-phase mode: per element dM/du (16)
  int estride;
  int ebase;       // element slot of the buffers' first entry (a chunk's first element)
  int begin, end;
  int stab, save, overwrite, qoi;
  int fp_reset;    // also write Fp = Fp_old at elastic points (goal leaves Fp as it was)
  double rho, ks_max, ks_scale;
};

__device__ __forceinline__ void ld4(const double* p, double& a, double& b, double& c, double& d) {
  double4_32a v = *reinterpret_cast<const double4_32a*>(p);
  a = v.x; b = v.y; c = v.z; d = v.w;
}
__device__ __forceinline__ void st4(double* p, double a, double b, double c, double d) {
  double4_32a v;
  v.x = a; v.y = b; v.z = c; v.w = d;
  *reinterpret_cast<double4_32a*>(p) = v;
}
__device__ __forceinline__ void acc4(double* p, bool first, double a, double b, double c, double d) {
  if (!first) {
    double x, y, z, w;
    ld4(p, x, y, z, w);
    a += x; b += y; c += z; d += w;
  }
  st4(p, a, b, c, d);
}

constexpr int kMatStride = 8;  // kappa, mu, K, Y, c0, 1/kappa, c0/(2 mu), 1/(16 kappa)
constexpr double kThird = 1.0 / 3.0;

// 1/(k+1) for the exponential series
__constant__ double c_inv_k[80];

// exp(A) for a symmetric traceless 3x3 A (A = dgam N) by the power series
// reduced with Cayley-Hamilton: A^3 = I2 A + I3 I, I2 = tr(A^2)/2, I3 = det A.
// Returns false if the series did not settle in 80 terms.
__device__ bool exp_traceless_sym(const double A[3][3], double out[3][3]) {
  double A2[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) A2[i][j] = A[i][0] * A[0][j] + A[i][1] * A[1][j] + A[i][2] * A[2][j];
  double I2 = 0.5 * (A2[0][0] + A2[1][1] + A2[2][2]);
  double I3 = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) - A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
              A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
  // term_k = A^k/k! = x I + y A + z A^2
  double x = 0.0, y = 0.0, z = 1.0 / 2.0;  // k = 2
  double s0 = 1.0, s1 = 1.0, s2 = 0.5;
  bool ok = false;
  for (int k = 2; k < 80; ++k) {
    double nx = z * I3, ny = x + z * I2, nz = y;
    const double inv = c_inv_k[k];
    x = nx * inv; y = ny * inv; z = nz * inv;
    s0 += x; s1 += y; s2 += z;
    double mag = fabs(x) + fabs(y) + fabs(z);
    if (mag < 1e-20 * (fabs(s0) + fabs(s1) + fabs(s2))) { ok = true; break; }
  }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) out[i][j] = s1 * A[i][j] + s2 * A2[i][j] + (i == j ? s0 : 0.0);
  return ok;
}

// What the integration point of an element gives the residual and the tangent.
struct Point {
  double V, inv_kappa, tau_coef, pp_coef;
  double un[4][3], pval, gp[3];           // nodal displacements, pressure and its gradient
  double J, Jinv, cof[3][3], H[3][3], C[6], FC[3][3];  // cof = J H, H = F^-T
  double alpha, Ic3, s[6];                // s: trial deviatoric Kirchhoff stress xx yy zz xy yz xz
  double gamma, smag, mubar, fyield, k0, cc, kh, rsmag, rcc;
  bool plastic;
  double sg[3][3];                        // Cauchy stress after Mixed
};

// Gather, kinematics, constitutive model with its state writes, and Mixed.
template <int MODEL>
__device__ __forceinline__ void eval_point(const ElemArgs& a, bool save, int s, const int (&v)[4],
                                           const double (&G)[4][3], Point& p) {
  const int E = a.d.num_elems;
  const double V = __ldg(a.d.vol + s);
  const int es = __ldg(a.d.elem_set + s);
  const double* mrow = a.mats + kMatStride * es;
  const double mu = __ldg(mrow + 1);
  const double Kh = __ldg(mrow + 2);
  const double Yld = __ldg(mrow + 3);
  const double inv_kappa = __ldg(mrow + 5);   // 1 / kappa
  const double tau_coef = __ldg(mrow + 6);    // c0 / (2 mu)
  const double pp_coef = __ldg(mrow + 7);     // 1 / (16 kappa)

  // gather + interpolation (Displacement/Pressure at_point)
  double un[4][3], pn[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) ld4(a.U + 4 * v[q], un[q][0], un[q][1], un[q][2], pn[q]);
  double F[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double t = un[0][i] * G[0][j];
      t += un[1][i] * G[1][j];
      t += un[2][i] * G[2][j];
      t += un[3][i] * G[3][j];
      F[i][j] = t;
    }
  F[0][0] += 1.0; F[1][1] += 1.0; F[2][2] += 1.0;
  const double pval = ((pn[0] * 0.25 + pn[1] * 0.25) + pn[2] * 0.25) + pn[3] * 0.25;
  double gp[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) gp[i] = ((pn[0] * G[0][i] + pn[1] * G[1][i]) + pn[2] * G[2][i]) + pn[3] * G[3][i];

  // kinematics: J and H = F^-T
  double cof[3][3];
  cof[0][0] = F[1][1] * F[2][2] - F[1][2] * F[2][1];
  cof[0][1] = F[1][2] * F[2][0] - F[1][0] * F[2][2];
  cof[0][2] = F[1][0] * F[2][1] - F[1][1] * F[2][0];
  cof[1][0] = F[0][2] * F[2][1] - F[0][1] * F[2][2];
  cof[1][1] = F[0][0] * F[2][2] - F[0][2] * F[2][0];
  cof[1][2] = F[0][1] * F[2][0] - F[0][0] * F[2][1];
  cof[2][0] = F[0][1] * F[1][2] - F[0][2] * F[1][1];
  cof[2][1] = F[0][2] * F[1][0] - F[0][0] * F[1][2];
  cof[2][2] = F[0][0] * F[1][1] - F[0][1] * F[1][0];
  const double J = F[0][0] * cof[0][0] + F[0][1] * cof[0][1] + F[0][2] * cof[0][2];
  const double Jinv = 1.0 / J;
  double H[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) H[i][j] = cof[i][j] * Jinv;

  // right Cauchy-Green of the plastic part (identity for neo-Hookean)
  double C[6] = {1.0, 1.0, 1.0, 0.0, 0.0, 0.0};  // xx yy zz xy yz xz
  double FC[3][3];  // F C
  if constexpr (MODEL == MODEL_J2) {
#pragma unroll
    for (int q = 0; q < 6; ++q) C[q] = __ldg(a.Cpinv + q * E + s);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      FC[i][0] = F[i][0] * C[0] + F[i][1] * C[3] + F[i][2] * C[5];
      FC[i][1] = F[i][0] * C[3] + F[i][1] * C[1] + F[i][2] * C[4];
      FC[i][2] = F[i][0] * C[5] + F[i][1] * C[4] + F[i][2] * C[2];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) FC[i][j] = F[i][j];
  }
  // B = F C F^T (symmetric)
  double B00 = FC[0][0] * F[0][0] + FC[0][1] * F[0][1] + FC[0][2] * F[0][2];
  double B11 = FC[1][0] * F[1][0] + FC[1][1] * F[1][1] + FC[1][2] * F[1][2];
  double B22 = FC[2][0] * F[2][0] + FC[2][1] * F[2][1] + FC[2][2] * F[2][2];
  double B01 = FC[0][0] * F[1][0] + FC[0][1] * F[1][1] + FC[0][2] * F[1][2];
  double B12 = FC[1][0] * F[2][0] + FC[1][1] * F[2][1] + FC[1][2] * F[2][2];
  double B02 = FC[0][0] * F[2][0] + FC[0][1] * F[2][1] + FC[0][2] * F[2][2];
  const double Ic = B00 + B11 + B22;
  const double Jm13 = rcbrt(J);
  const double alpha = mu * (Jm13 * Jm13);
  const double Ic3 = Ic * kThird;
  // trial deviatoric Kirchhoff stress s = alpha dev(B)
  const double s00 = alpha * (B00 - Ic3), s11 = alpha * (B11 - Ic3), s22 = alpha * (B22 - Ic3);
  const double s01 = alpha * B01, s12 = alpha * B12, s02 = alpha * B02;

  // J2 radial return (closed form of goal's scalar Newton loop)
  double gamma = 1.0;
  bool plastic = false;
  double smag = 0.0, mubar = 0.0, fyield = 0.0, k0 = 0.0, cc = 1.0, kh = 0.0, Xr = 0.0, rsmag = 0.0, rcc = 1.0;
  const double sq23 = 0.81649658092772603273;  // sqrt(2/3)
  if (MODEL == MODEL_J2 || (a.qoi == QOI_KS_VM)) {
    smag = sqrt(s00 * s00 + s11 * s11 + s22 * s22 + 2.0 * (s01 * s01 + s12 * s12 + s02 * s02));
  }
  if (MODEL == MODEL_J2) {
    mubar = alpha * Ic3;
    const double eq_old = __ldg(a.eqps_old + s);
    k0 = sq23 * (Yld + Kh * eq_old);
    fyield = smag - k0;
    if (fyield > 1.0e-12) {
      plastic = true;
      // reciprocals formed once (a division costs several FP64 instructions)
      rsmag = 1.0 / smag;
      // Newton iterates of src/goal_J2.cpp:101-121. The first has H = 0 in its
      // slope, X1 = f / (2 mubar), and leaves the residual -2/3 K X1; goal stops
      // there if |R| < 1e-11, |R|/Y < 1e-11 or |R|/f < 1e-11 (Y, f > 0).
      const double m2 = 2.0 * mubar, K23 = (2.0 / 3.0) * Kh;
      const bool conv1 = fabs(K23 * fyield) < 1.0e-11 * m2 * fmax(1.0, fmax(Yld, fyield));
      kh = conv1 ? 0.0 : K23;
      cc = m2 + kh;
      rcc = 1.0 / cc;
      Xr = fyield * rcc;
      gamma = 1.0 - 2.0 * mubar * Xr * rsmag;
      if (!(Xr >= 0.0) || !isfinite(Xr)) *a.failed = 1;
      if (save) {
        a.eqps[s] = eq_old + sq23 * Xr;
        // Fp = exp(dgam N) Fp_old (stored only at plastic points): the
        // increment dgam N is stored here, Fp formed when it is read
        const double is = Xr * rsmag;
        a.Apend[0 * E + s] = s00 * is;
        a.Apend[1 * E + s] = s11 * is;
        a.Apend[2 * E + s] = s22 * is;
        a.Apend[3 * E + s] = s01 * is;
        a.Apend[4 * E + s] = s12 * is;
        a.Apend[5 * E + s] = s02 * is;
        a.pend[s] = 1;
      }
    } else if (save) {
      a.eqps[s] = eq_old;
      if (a.fp_reset) {
        a.pend[s] = 0;
#pragma unroll
        for (int q = 0; q < 9; ++q) a.Fp[q * E + s] = __ldg(a.Fp_old + q * E + s);
      }
    }
  }

  // Cauchy stress of the model, then Mixed
  // (the model's pressure 1/2 kappa (J - 1/J) is what Mixed takes out again,
  // and with it what rounding left of the mean of s)
  const double gJ = gamma * Jinv;
  double sg[3][3];
  sg[0][0] = s00 * gJ; sg[1][1] = s11 * gJ; sg[2][2] = s22 * gJ;
  sg[0][1] = sg[1][0] = s01 * gJ;
  sg[1][2] = sg[2][1] = s12 * gJ;
  sg[0][2] = sg[2][0] = s02 * gJ;
  const double dp = fma(-kThird, (sg[0][0] + sg[1][1]) + sg[2][2], pval);
  sg[0][0] += dp; sg[1][1] += dp; sg[2][2] += dp;
  if (save) {
#pragma unroll
    for (int q = 0; q < 9; ++q) a.sigma[q * E + s] = sg[q / 3][q % 3];
  }


  p.V = V; p.inv_kappa = inv_kappa; p.tau_coef = tau_coef; p.pp_coef = pp_coef;
  p.pval = pval; p.J = J; p.Jinv = Jinv; p.alpha = alpha; p.Ic3 = Ic3;
  p.s[0] = s00; p.s[1] = s11; p.s[2] = s22; p.s[3] = s01; p.s[4] = s12; p.s[5] = s02;
  p.gamma = gamma; p.smag = smag; p.mubar = mubar; p.fyield = fyield; p.k0 = k0; p.cc = cc; p.kh = kh;
  p.rsmag = rsmag; p.rcc = rcc; p.plastic = plastic;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p.gp[i] = gp[i];
#pragma unroll
    for (int j = 0; j < 3; ++j) { p.cof[i][j] = cof[i][j]; p.H[i][j] = H[i][j]; p.FC[i][j] = FC[i][j]; p.sg[i][j] = sg[i][j]; }
#pragma unroll
    for (int q = 0; q < 4; ++q) p.un[q][i] = un[q][i];
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) p.C[q] = C[q];
}

// The gather's launch overlaps the element phase: its blocks may be on the chip
// by the time that phase ends, and wait there for its end and its stores. Chains
// of 384 elements: Jacobian 42 us -> 39, residual 31 -> 28; J2 Jacobian of 384,000
// 661 -> 658. A small element phase lets them come while it runs; waiting blocks
// cost a chip full of element blocks more than they save (Jacobian of 48k 117 us
// -> 126, of 384k 663 -> 753, residual of 48k 51 -> 60).
__device__ __forceinline__ void gather_may_start() { asm volatile("griddepcontrol.launch_dependents;"); }
// The address that loads after the wait use, so that none can move ahead of it.
// They are not read-only loads: the blocks are on the chip while the element phase
// writes, and that path is for what stays as it is for the whole kernel.
template <typename T>
__device__ __forceinline__ const T* wait_for_elements(const T* buffer) {
  asm volatile("griddepcontrol.wait;" : "+l"(buffer)::"memory");
  return buffer;
}

template <typename... P, typename... A>
void launch_gather(void (*kernel)(P...), int grid, int block, cudaStream_t st, A... args) {
  cudaLaunchAttribute overlap;
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  GOAL_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  GOAL_CHECK_LAUNCH();
}

// Element record of the default Jacobian assembly, kRecord 8-byte words:
//   [0, 16)    R (FP64)
//   [16, 32)   per block (a, b) four 16-bit exponents: of K^uu, K^up, K^pu, K^pp
//   [32, 48)   column 3 (K^up_a, K^pp_aa) of the diagonal blocks
//   [48, 240)  the twelve off-diagonal blocks, row-major
// with every block entry S 2^x in the fixed point of fixed.cuh, or in FP64 where
// the exponent is kFxFloat.
constexpr int kRecord = 240;
constexpr int kRecExp = 16, kRecDiag = 32, kRecOff = 48;
__device__ __forceinline__ int off_index(int a, int b) { return 3 * a + b - (b > a ? 1 : 0); }

// One element in FP64. BUF: its outputs go to the per-element buffer (phase 1 of
// the two-phase assembly) instead of being accumulated in place by one colour at
// a time. REC: the buffer holds records (JAC && BUF).
template <int MODEL, int MODE, bool JAC, bool ERR, bool BUF, bool REC>
__device__ __forceinline__ void elem_fp64(const ElemArgs& a, bool save, int s) {
  const int E = a.d.num_elems;

  int v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = __ldg(a.d.tets + q * E + s);
  double G[4][3];
#pragma unroll
  for (int q = 0; q < 12; ++q) G[q / 3][q % 3] = __ldg(a.d.grads + q * E + s);
  Point pt;
  eval_point<MODEL>(a, save, s, v, G, pt);
  const double V = pt.V, inv_kappa = pt.inv_kappa, tau_coef = pt.tau_coef, pp_coef = pt.pp_coef;
  const double pval = pt.pval, J = pt.J, Jinv = pt.Jinv, alpha = pt.alpha, Ic3 = pt.Ic3;
  const double s00 = pt.s[0], s11 = pt.s[1], s22 = pt.s[2], s01 = pt.s[3], s12 = pt.s[4], s02 = pt.s[5];
  const double gamma = pt.gamma, smag = pt.smag, mubar = pt.mubar, fyield = pt.fyield, k0 = pt.k0, cc = pt.cc;
  const double kh = pt.kh, rsmag = pt.rsmag, rcc = pt.rcc;
  const bool plastic = pt.plastic;
  const double(&H)[3][3] = pt.H;
  const double(&FC)[3][3] = pt.FC;
  const double(&sg)[3][3] = pt.sg;
  const double(&C)[6] = pt.C;
  const double(&gp)[3] = pt.gp;
  const double(&un)[4][3] = pt.un;

  // h_a = H G_a
  double hv[4][3];
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 3; ++i) hv[n][i] = H[i][0] * G[n][0] + H[i][1] * G[n][1] + H[i][2] * G[n][2];
  // v = H grad p, w_a = v.h_a
  double vv[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) vv[i] = H[i][0] * gp[0] + H[i][1] * gp[1] + H[i][2] * gp[2];
  double wv[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) wv[n] = vv[0] * hv[n][0] + vv[1] * hv[n][1] + vv[2] * hv[n][2];
  double tau = 0.0;
  if (a.stab) {
    const double hh = __ldg(a.d.h + s);
    tau = tau_coef * (hh * hh);
  }
  const double tauJ = tau * J;
  const double dUdJ = 0.5 * (J - Jinv);
  double T[3][3];  // J sigma
#pragma unroll
  for (int q = 0; q < 9; ++q) T[q / 3][q % 3] = J * sg[q / 3][q % 3];

  // ---------------------------------------------------------------- residual
  if (MODE != MODE_NONE && !REC) {
    double Ru[4][3], Rp[4];
    if constexpr (!JAC && !ERR) {
      // A residual alone, which the FP64 pipe bounds (all of its time): V J sigma
      // F^-T = V sigma cof F, in the stabilization v . h_a with the cofactors on
      // one side: 102 FP64 instructions against 118 from h_a and J sigma, to the
      // same error. (V gamma alpha (F C - Ic/3 F^-T) + p cof F would be 15 fewer,
      // but the difference loses digits: error 1.3e-13 against 7e-14. The last
      // node's row as the negated sum of the others', whose digits it would have,
      // gains nothing.) A chain of 384,000 elements, J2, with the point's own 22
      // instructions fewer: 292 us -> 257.
      const double rp0 = ((pval * inv_kappa) - dUdJ) * 0.25 * V;
      double P[3][3], z[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
          P[i][k] = (V * sg[i][0]) * pt.cof[0][k] + (V * sg[i][1]) * pt.cof[1][k] + (V * sg[i][2]) * pt.cof[2][k];
      if (a.stab) {
        const double f = tau * (V * Jinv);
        double cg[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
          cg[i] = f * (pt.cof[i][0] * gp[0] + pt.cof[i][1] * gp[1] + pt.cof[i][2] * gp[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) z[k] = pt.cof[0][k] * cg[0] + pt.cof[1][k] * cg[1] + pt.cof[2][k] * cg[2];
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int i = 0; i < 3; ++i) Ru[n][i] = fma(P[i][0], G[n][0], fma(P[i][1], G[n][1], P[i][2] * G[n][2]));
        Rp[n] = fma(z[0], G[n][0], fma(z[1], G[n][1], fma(z[2], G[n][2], rp0)));
      }
    } else if constexpr (!ERR) {
      double TV[3][3];  // V J sigma
#pragma unroll
      for (int q = 0; q < 9; ++q) TV[q / 3][q % 3] = V * T[q / 3][q % 3];
      const double rp0 = ((pval * inv_kappa) - dUdJ) * 0.25 * V;
      const double rpw = a.stab ? tauJ * V : 0.0;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int i = 0; i < 3; ++i) Ru[n][i] = fma(TV[i][0], hv[n][0], fma(TV[i][1], hv[n][1], TV[i][2] * hv[n][2]));
        Rp[n] = fma(rpw, wv[n], rp0);
      }
    } else {
      // DWR weights: z_diff phi_a (momentum, pressure), z_coarse phi_a (stabilization)
      double zn[4][4], zcn[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ld4(a.Zd + 4 * v[q], zn[q][0], zn[q][1], zn[q][2], zn[q][3]);
        zcn[q] = __ldg(a.Zc + 4 * v[q] + 3);
      }
      double z[3], gz[3][3], zp, zc, gzc[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        z[i] = 0.25 * (zn[0][i] + zn[1][i] + zn[2][i] + zn[3][i]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
          gz[i][j] = zn[0][i] * G[0][j] + zn[1][i] * G[1][j] + zn[2][i] * G[2][j] + zn[3][i] * G[3][j];
      }
      zp = 0.25 * (zn[0][3] + zn[1][3] + zn[2][3] + zn[3][3]);
      zc = 0.25 * (zcn[0] + zcn[1] + zcn[2] + zcn[3]);
#pragma unroll
      for (int j = 0; j < 3; ++j) gzc[j] = zcn[0] * G[0][j] + zcn[1] * G[1][j] + zcn[2] * G[2][j] + zcn[3] * G[3][j];
      double P[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) P[i][j] = T[i][0] * H[0][j] + T[i][1] * H[1][j] + T[i][2] * H[2][j];
      double Pg[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) Pg[i] = P[i][0] * gz[i][0] + P[i][1] * gz[i][1] + P[i][2] * gz[i][2];
      double hz[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) hz[i] = H[i][0] * gzc[0] + H[i][1] * gzc[1] + H[i][2] * gzc[2];
      const double vhz = vv[0] * hz[0] + vv[1] * hz[1] + vv[2] * hz[2];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          double PGa = T[i][0] * hv[n][0] + T[i][1] * hv[n][1] + T[i][2] * hv[n][2];
          Ru[n][i] = V * (0.25 * Pg[i] + z[i] * PGa);
        }
        Rp[n] = ((pval * inv_kappa) - dUdJ) * (zp * 0.25) * V + (a.stab ? tauJ * (0.25 * vhz + zc * wv[n]) * V : 0.0);
      }
    }
    if constexpr (BUF) {
      double* eb = a.ebuf + (size_t)(s - a.ebase) * a.estride;
#pragma unroll
      for (int n = 0; n < 4; ++n) st4(eb + 4 * n, Ru[n][0], Ru[n][1], Ru[n][2], Rp[n]);
    } else {
      const unsigned fm = a.overwrite ? __ldg(a.d.first + s) : 0u;
#pragma unroll
      for (int n = 0; n < 4; ++n) acc4(a.R + 4 * v[n], (fm >> (16 + n)) & 1u, Ru[n][0], Ru[n][1], Ru[n][2], Rp[n]);
    }
  }

  // ---------------------------------------------------------------- QoI
  double ks_w = 0.0;
  if (a.qoi == QOI_AVG_DISP) {
    double uval[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) uval[i] = ((un[0][i] * 0.25 + un[1][i] * 0.25) + un[2][i] * 0.25) + un[3][i] * 0.25;
    double ev = 0.0;
    ev += uval[0] * V;
    ev += uval[1] * V;
    ev += uval[2] * V;
    a.qoi_elem[s] = ev * kThird;
  } else if (a.qoi == QOI_KS_VM) {
    double d1 = sg[0][0] - sg[1][1], d2 = sg[1][1] - sg[2][2], d3 = sg[2][2] - sg[0][0];
    double s7 = 0.5 * (d1 * d1 + d2 * d2 + d3 * d3 + 6.0 * (sg[0][1] * sg[0][1] + sg[1][2] * sg[1][2] + sg[2][0] * sg[2][0]));
    double vm = sqrt(s7);
    double ex = exp(a.rho * (vm - a.ks_max));
    a.qoi_elem[s] = (1.0 / (a.rho * a.ks_scale)) * ex * V;
    ks_w = (V / a.ks_scale) * ex;  // d(elem value)/d(vm)
  }

  if constexpr (JAC) {
  // ---------------------------------------------------------------- tangent
  // m_a = F C G_a, q_a = m_a - Ic/3 h_a
  double mv[4][3], qv[4][3];
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      mv[n][i] = FC[i][0] * G[n][0] + FC[i][1] * G[n][1] + FC[i][2] * G[n][2];
      qv[n][i] = mv[n][i] - Ic3 * hv[n][i];
    }
  const double pJ = pval * J;
  const double ga = gamma * alpha;
  // dgamma_b = yq q_b + yh h_b + yn (s m_b) ; Y_b = -2/3 ga h_b + alpha dgamma_b
  double yq = 0.0, yh = 0.0, yn = 0.0;
  // d(gamma smag) = dq q_b + dh h_b + dn (s m_b)   (KS derivative)
  double vq = 0.0, vh = 0.0, vn = 0.0;
  const bool need_n = plastic || (a.qoi == QOI_KS_VM);
  if (plastic) {
    const double A1 = 2.0 * fyield * kh * (rcc * rcc) * rsmag;
    const double A2 = 2.0 * mubar * k0 * rcc * (rsmag * rsmag);
    yq = -A1 * (2.0 * alpha / 3.0);
    yh = A2 * (2.0 / 3.0) * smag;
    yn = -A2 * (2.0 * alpha * rsmag);
  }
  if (a.qoi == QOI_KS_VM) {
    // dsmag_b = -2/3 smag h_b + 2 alpha/smag n_b ; dmubar_b = 2 alpha/3 q_b
    double fs = 1.0, fmu = 0.0;
    if (plastic) { fs = kh / cc; fmu = -2.0 * fyield * kh / (cc * cc); }
    vh = fs * (-(2.0 / 3.0) * smag);
    vn = fs * (2.0 * alpha / smag);
    vq = fmu * (2.0 * alpha / 3.0);
  }
  double Xp[4][3], Yp[4][3], nv[4][3];
  // X_b = V(-2/3 ga m_b + pJ h_b), Y_b = V(-2/3 ga h_b + alpha (yq q_b + yh h_b + yn n_b)),
  // with the coefficients folded once per element
  const double xm = V * (-(2.0 / 3.0) * ga), xh = V * pJ;
  const double yhc = V * (-(2.0 / 3.0) * ga + alpha * yh), yqc = V * (alpha * yq), ync = V * (alpha * yn);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    if (need_n) {
      nv[b][0] = s00 * mv[b][0] + s01 * mv[b][1] + s02 * mv[b][2];
      nv[b][1] = s01 * mv[b][0] + s11 * mv[b][1] + s12 * mv[b][2];
      nv[b][2] = s02 * mv[b][0] + s12 * mv[b][1] + s22 * mv[b][2];
    } else {
      nv[b][0] = nv[b][1] = nv[b][2] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      Xp[b][k] = fma(xm, mv[b][k], xh * hv[b][k]);
      Yp[b][k] = need_n ? fma(yhc, hv[b][k], fma(yqc, qv[b][k], ync * nv[b][k])) : yhc * hv[b][k];
    }
  }
  // dM/du (QoI derivative) for the u dofs; pressure dofs do not enter the QoIs
  if (a.qoi != QOI_NONE) {
    const unsigned fm = (!BUF && a.overwrite) ? __ldg(a.d.first + s) : 0u;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      double d[3];
      if (a.qoi == QOI_AVG_DISP) {
        d[0] = d[1] = d[2] = V * (1.0 / 12.0);
      } else {
        const double c1 = ks_w * 1.22474487139158904909 * Jinv;  // sqrt(3/2)/J
        const double gs = gamma * smag;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          d[k] = c1 * (vq * qv[b][k] + vh * hv[b][k] + vn * nv[b][k] - gs * hv[b][k]);
      }
      if constexpr (BUF) st4(a.dbuf + 16ll * (s - a.ebase) + 4 * b, d[0], d[1], d[2], 0.0);
      else acc4(a.dMdu + 4 * v[b], (fm >> (16 + b)) & 1u, d[0], d[1], d[2], 0.0);
    }
  }

  const double zs = V * (ga * Ic3 - pJ);
  const double gaV = ga * V;
  const double upf = V * J * 0.25;
  const double tJV = tauJ * V;
  const double ppc = V * pp_coef;
  const double pu0 = V * ((J + Jinv) * 0.125);
  // stabilization coefficients of the p-u rows, folded once per element
  double tvv[3], twv[4];
#pragma unroll
  for (int k = 0; k < 3; ++k) tvv[k] = a.stab ? tJV * vv[k] : 0.0;
#pragma unroll
  for (int b = 0; b < 4; ++b) twv[b] = a.stab ? tJV * wv[b] : 0.0;
  const double tJVs = a.stab ? tJV : 0.0;
  // ga V C G_a and Z_a = zs h_a
  double CG[4][3], Zv[4][3];
#pragma unroll
  for (int ai = 0; ai < 4; ++ai) {
    if constexpr (MODEL == MODEL_J2) {
      CG[ai][0] = gaV * (C[0] * G[ai][0] + C[3] * G[ai][1] + C[5] * G[ai][2]);
      CG[ai][1] = gaV * (C[3] * G[ai][0] + C[1] * G[ai][1] + C[4] * G[ai][2]);
      CG[ai][2] = gaV * (C[5] * G[ai][0] + C[4] * G[ai][1] + C[2] * G[ai][2]);
    } else {
      CG[ai][0] = gaV * G[ai][0]; CG[ai][1] = gaV * G[ai][1]; CG[ai][2] = gaV * G[ai][2];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) Zv[ai][k] = zs * hv[ai][k];
  }
  const unsigned fm = (!BUF && a.overwrite) ? __ldg(a.d.first + s) : 0u;
  // Element block (ai, b) from Pc[i][k] = h_bi Z_ak + c_ab d_ik (TP: Pc
  // transposed), written to the element buffer or accumulated into the matrix.
  auto block = [&](int ai, int b, const double (&Pc)[3][3], bool TP, double eab) {
    double K[4][4];
    const double pu1 = twv[ai] - pu0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int k = 0; k < 3; ++k) K[i][k] = fma(hv[ai][i], Xp[b][k], fma(qv[ai][i], Yp[b][k], TP ? Pc[k][i] : Pc[i][k]));
      K[i][3] = upf * hv[ai][i];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) K[3][k] = fma(pu1, hv[b][k], -fma(eab, tvv[k], twv[b] * hv[ai][k]));
    K[3][3] = fma(tJVs, eab, ppc);
    if constexpr (REC) {
      double* rec = a.ebuf + (size_t)(s - a.ebase) * kRecord;
      if (ai == b) {
        st4(rec + kRecDiag + 4 * ai, K[0][3], K[1][3], K[2][3], K[3][3]);
      } else {
        double* blk = rec + kRecOff + 16 * off_index(ai, b);
#pragma unroll
        for (int r = 0; r < 4; ++r) st4(blk + 4 * r, K[r][0], K[r][1], K[r][2], K[r][3]);
      }
      reinterpret_cast<short4*>(rec + kRecExp)[4 * ai + b] = make_short4(kFxFloat, kFxFloat, kFxFloat, kFxFloat);
    } else if constexpr (BUF) {
      double* eb = a.ebuf + (size_t)(s - a.ebase) * a.estride + 16 + 16 * (4 * ai + b);
#pragma unroll
      for (int r = 0; r < 4; ++r) st4(eb + 4 * r, K[r][0], K[r][1], K[r][2], K[r][3]);
    } else if (MODE == MODE_PRIMAL) {
      const int q = 4 * ai + b;
      double* blk = a.A + 16ll * __ldg(a.d.blk + q * E + s);
      const bool f1 = (fm >> q) & 1u;
#pragma unroll
      for (int r = 0; r < 4; ++r) acc4(blk + 4 * r, f1, K[r][0], K[r][1], K[r][2], K[r][3]);
    } else if (MODE == MODE_ADJOINT) {
      const int q = 4 * b + ai;
      double* blk = a.A + 16ll * __ldg(a.d.blk + q * E + s);
      const bool f1 = (fm >> q) & 1u;
#pragma unroll
      for (int r = 0; r < 4; ++r) acc4(blk + 4 * r, f1, K[0][r], K[1][r], K[2][r], K[3][r]);
    }
  };
  // The off-diagonal blocks in pairs: c_ab and e_ab are symmetric in (a, b)
  // and the term h_bi Z_ak = zs h_bi h_ak of block (a, b) is the term
  // (k, i) of block (b, a), so each pair forms them once.
#pragma unroll
  for (int ai = 0; ai < 4; ++ai) {
#pragma unroll
    for (int b = ai + 1; b < 4; ++b) {
      const double eab = hv[ai][0] * hv[b][0] + hv[ai][1] * hv[b][1] + hv[ai][2] * hv[b][2];
      const double cab = fma(CG[ai][0], G[b][0], fma(CG[ai][1], G[b][1], CG[ai][2] * G[b][2]));
      double Pc[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) Pc[i][k] = (i == k) ? fma(hv[b][i], Zv[ai][k], cab) : hv[b][i] * Zv[ai][k];
      block(ai, b, Pc, false, eab);
      block(b, ai, Pc, true, eab);
    }
  }
  // the diagonal blocks (a, a)
#pragma unroll
  for (int ai = 0; ai < 4; ++ai) {
    const double eaa = hv[ai][0] * hv[ai][0] + hv[ai][1] * hv[ai][1] + hv[ai][2] * hv[ai][2];
    const double caa = fma(CG[ai][0], G[ai][0], fma(CG[ai][1], G[ai][1], CG[ai][2] * G[ai][2]));
    double Pc[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) Pc[i][k] = (i == k) ? fma(hv[ai][i], Zv[ai][k], caa) : hv[ai][i] * Zv[ai][k];
    block(ai, ai, Pc, false, eaa);
  }
  }  // JAC
}

template <int MODEL, int MODE, bool JAC, bool ERR, bool BUF>
__global__ void __launch_bounds__(128) k_elem(const ElemArgs a) {
  if (BUF && gridDim.x * blockDim.x <= 128 * kSMs) gather_may_start();
  const int s = a.begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (s < a.end) elem_fp64<MODEL, MODE, JAC, ERR, BUF, false>(a, a.save, s);
}

// ------------------------------------------------------------------ fixed-point element phase
// The record of an element that fixed point would hold to fewer digits than FP64
// (see k_elem_fix). R, the QoI value and the states are written.
template <int MODEL>
__device__ __noinline__ void record_fp64(const ElemArgs& a, int s) {
  elem_fp64<MODEL, MODE_PRIMAL, true, false, true, true>(a, false, s);
}

// Residual and tangent of one element per thread into its record, for both
// Jacobian modes (the gather transposes).
//
// The 144 entries of the off-diagonal element blocks are sums of two or three
// products and took 450 of the 1,014 FP64 instructions per element; here they
// are formed in fixed point on the integer pipes (see fixed.cuh), and so are
// the vectors that enter them (m, q, n, X, Y, Z: another 210). The blocks come
// in pairs as c_ab, e_ab and h_b Z_a are shared by (a, b) and (b, a).
//
// Of the diagonal element blocks only column 3 is formed: the u columns of a
// matrix row sum to zero over the row's blocks (the gradients of a linear
// tet's shape functions sum to zero, and every u column of K^uu and K^pu is
// linear in them), so k_gather_rows forms the diagonal blocks' u columns as
// negated sums of the off-diagonal blocks.
//
// Every vector has its own exponent per node, so that its largest component
// keeps 55 bits and more whatever the deformation: with one exponent for F C and
// F^-T a block was off by 2e-12 of its largest entry at a dilation of 10 and by
// all of it at 10,000 (now 2e-15 and 1e-14, as in FP64). What the exponents
// cannot hold is left to FP64 (record_fp64): elements with an infinity or a NaN;
// those whose F C G has fewer than kFixHeld bits, as |F C| |G| is far larger
// (uniaxial stretches above 5); and those whose h differ by more than kFxSpread
// exponents between the axes (flat elements, stretches above 30), as entries
// that much smaller than the block's largest would lose digits of their own.
// Against 113-bit arithmetic, over 60,000 random elements (sizes 1e-6 to 100,
// strains 1e-9 to 1, dilations 0.1 to 1,000, stretches and flattenings to 100),
// a block's largest error over its largest entry is at most 4 times FP64's, in
// single blocks where those roundings happened to cancel, and the same over all.
//
// The factors wait in shared memory (a column of kFixSlots words per thread)
// and the loops over nodes and pairs are not unrolled: unrolled, the kernel
// was 12,800 instructions long and waited for instruction fetches 43% of the
// time. J2 at 384,000 elements: 740 us in FP64 throughout, 1,208 unrolled, 498
// with FP64 vectors m, q, n, X, Y, Z, 422 with one exponent for all factors, now
// 427 (neo-Hookean 327, 324). What bounds it is latency at three warps per
// scheduler (registers and shared memory); the FP64 pipe is 65% busy.
//
// SPLIT threads in different warps share an element of a small mesh, where one
// thread's chain of dependent instructions is all the time there is (36 us with
// a warp alone on an SM): each forms the integration point, as the FP64 pipe
// has room for that, its share of the four nodes and its share of the six block
// pairs, to the same bits.
constexpr int kFixC = 48, kFixW = 54, kFixNode = 58, kFixSlots = 62;  // factors of h, q, X, Y; c_ab; w_a; units of a node
constexpr int kFixPart = 62, kFixSlotsSplit = 74;                     // scales and largest words of a part
constexpr int kFixHeld = 55;
template <int ELEMS, int SPLIT>
constexpr int kFixSmem = (SPLIT > 1 ? kFixSlotsSplit : kFixSlots) * ELEMS * (int)sizeof(long long);

template <int MODEL, int ELEMS, int SPLIT>
__global__ void __launch_bounds__(ELEMS * SPLIT, 384 / (ELEMS * SPLIT)) k_elem_fix(const __grid_constant__ ElemArgs a) {
  extern __shared__ long long fix_slots[];
  if (SPLIT > 1) gather_may_start();
  const int part = SPLIT > 1 ? threadIdx.x / ELEMS : 0;
  const int s = a.begin + blockIdx.x * ELEMS + threadIdx.x % ELEMS;
  if (s >= a.end) return;
  const int E = a.d.num_elems;
  long long* slot = fix_slots + threadIdx.x % ELEMS;
  auto factor = [&](int i) {
    const long long r = slot[i * ELEMS];
    Fx f;
    f.lo = (int)r;
    f.hi = (int)(r >> 32);
    return f;
  };
  auto put_factor = [&](int i, const Fx& f) {
    slot[i * ELEMS] = ((long long)f.hi << 32) | (unsigned)f.lo;
  };
  auto at = [](int v, int n, int k) { return 12 * v + 3 * n + k; };  // v: h q X Y
  double* rec_r = a.ebuf + (size_t)(s - a.ebase) * kRecord;
  long long* rec = reinterpret_cast<long long*>(rec_r);

  int v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = __ldg(a.d.tets + q * E + s);
  Point pt;
  {
    double G[4][3];
#pragma unroll
    for (int q = 0; q < 12; ++q) G[q / 3][q % 3] = __ldg(a.d.grads + q * E + s);
    eval_point<MODEL>(a, a.save && part == 0, s, v, G, pt);
  }
  const double V = pt.V, J = pt.J, Jinv = pt.Jinv, alpha = pt.alpha, Ic3 = pt.Ic3, gamma = pt.gamma;
  const double(&H)[3][3] = pt.H;
  const double(&FC)[3][3] = pt.FC;

  // residual coefficients, as in k_elem
  double vv[3], TV[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    vv[i] = H[i][0] * pt.gp[0] + H[i][1] * pt.gp[1] + H[i][2] * pt.gp[2];
#pragma unroll
    for (int j = 0; j < 3; ++j) TV[i][j] = V * (J * pt.sg[i][j]);
  }
  double tau = 0.0;
  if (a.stab) {
    const double hh = __ldg(a.d.h + s);
    tau = pt.tau_coef * (hh * hh);
  }
  const double tauJ = tau * J;
  const double rp0 = ((pt.pval * pt.inv_kappa) - 0.5 * (J - Jinv)) * 0.25 * V;
  const double tJV = a.stab ? tauJ * V : 0.0;

  // QoI value and the weight of its derivative
  double ks_w = 0.0;
  if (a.qoi == QOI_AVG_DISP) {
    double ev = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      ev += (((pt.un[0][i] * 0.25 + pt.un[1][i] * 0.25) + pt.un[2][i] * 0.25) + pt.un[3][i] * 0.25) * V;
    if (part == 0) a.qoi_elem[s] = ev * kThird;
  } else if (a.qoi == QOI_KS_VM) {
    const double(&sg)[3][3] = pt.sg;
    double d1 = sg[0][0] - sg[1][1], d2 = sg[1][1] - sg[2][2], d3 = sg[2][2] - sg[0][0];
    double s7 = 0.5 * (d1 * d1 + d2 * d2 + d3 * d3 + 6.0 * (sg[0][1] * sg[0][1] + sg[1][2] * sg[1][2] + sg[2][0] * sg[2][0]));
    double ex = exp(a.rho * (sqrt(s7) - a.ks_max));
    if (part == 0) a.qoi_elem[s] = (1.0 / (a.rho * a.ks_scale)) * ex * V;
    ks_w = (V / a.ks_scale) * ex;
  }

  // tangent coefficients, as in k_elem
  const double pJ = pt.pval * J, ga = gamma * alpha;
  double yq = 0.0, yh = 0.0, yn = 0.0;
  const bool need_n = pt.plastic || (a.qoi == QOI_KS_VM);
  if (pt.plastic) {
    const double A1 = 2.0 * pt.fyield * pt.kh * (pt.rcc * pt.rcc) * pt.rsmag;
    const double A2 = 2.0 * pt.mubar * pt.k0 * pt.rcc * (pt.rsmag * pt.rsmag);
    yq = -A1 * (2.0 * alpha / 3.0);
    yh = A2 * (2.0 / 3.0) * pt.smag;
    yn = -A2 * (2.0 * alpha * pt.rsmag);
  }
  double vq = 0.0, vh = 0.0, vn = 0.0;  // dM/du (KS): c1 (vq q + vh h + vn n)
  if (a.qoi == QOI_KS_VM) {
    double fs = 1.0, fmu = 0.0;
    if (pt.plastic) { fs = pt.kh / pt.cc; fmu = -2.0 * pt.fyield * pt.kh / (pt.cc * pt.cc); }
    const double c1 = ks_w * 1.22474487139158904909 * Jinv;  // sqrt(3/2)/J
    vh = c1 * (fs * (-(2.0 / 3.0) * pt.smag) - gamma * pt.smag);
    vn = c1 * (fs * (2.0 * alpha / pt.smag));
    vq = c1 * (fmu * (2.0 * alpha / 3.0));
  }
  const double xm = V * (-(2.0 / 3.0) * ga), xh = V * pJ;
  const double yhc = V * (-(2.0 / 3.0) * ga + alpha * yh), yqc = V * (alpha * yq), ync = V * (alpha * yn);
  const double zs = V * (ga * Ic3 - pJ), gaV = ga * V;
  const double upf = V * J * 0.25, ppc = V * pt.pp_coef, pu0 = V * ((J + Jinv) * 0.125);

  // Fixed point from here on. Every factor has the exponent of its own kind: bF of
  // F C, bS of s, bI of Ic/3, one for each coefficient, and per node bG and bh of
  // the gradient and of h.
  int lF = 0, lS = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) lF = max(lF, fx_high(FC[i][k]));
#pragma unroll
  for (int q = 0; q < 6; ++q) lS = max(lS, fx_high(pt.s[q]));
  int all = max(max(lF, lS), max(max(fx_high(xm), fx_high(xh)), max(fx_high(zs), fx_high(Ic3))));
  all = max(all, max(fx_high(yhc), max(fx_high(yqc), fx_high(ync))));
  const int bF = fx_exp(lF), bS = fx_exp(lS), bI = fx_exp(fx_high(Ic3));
  const int bm = fx_exp(fx_high(xm)), bp = fx_exp(fx_high(xh)), bz = fx_exp(fx_high(zs));
  const int byh = fx_exp(fx_high(yhc)), byq = fx_exp(fx_high(yqc)), byn = fx_exp(fx_high(ync));
  Fx fFC[3][3], fS[6];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) fFC[i][k] = fx_factor(FC[i][k], bF);
#pragma unroll
  for (int q = 0; q < 6; ++q) fS[q] = fx_factor(pt.s[q], bS);
  const Fx fI = fx_factor62(Ic3, bI), fxm = fx_factor62(xm, bm), fxh = fx_factor62(xh, bp);
  const Fx fyh = fx_factor62(yhc, byh), fyq = fx_factor62(yqc, byq), fyn = fx_factor62(ync, byn);

  // Per node n: h = F^-T G to 62 bits (from FP64, which R needs too), at the unit
  // xh = bh - 1084; m = F C G at um; q = m - Ic/3 h, n = s m, X and Y each at the
  // larger unit of its terms, so that none holds less of a term than FP64 would.
  // The units less xh wait in 16 bits a node. F, FY, up: see below.
  unsigned long long bhs = 0;
  int axis[3] = {0, 0, 0};  // exponent of the largest h per axis
  int F = bz - 1022, FY = -32768, up = 32767, held = 64;
#pragma unroll 1
  for (int n = part; n < 4; n += SPLIT) {
    double G[3], hv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) G[k] = __ldg(a.d.grads + (3 * n + k) * E + s);
#pragma unroll
    for (int i = 0; i < 3; ++i) hv[i] = H[i][0] * G[0] + H[i][1] * G[1] + H[i][2] * G[2];
    const double w = vv[0] * hv[0] + vv[1] * hv[1] + vv[2] * hv[2];
    double Ru[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) Ru[i] = fma(TV[i][0], hv[0], fma(TV[i][1], hv[1], TV[i][2] * hv[2]));
    st4(rec_r + 4 * n, Ru[0], Ru[1], Ru[2], fma(tJV, w, rp0));
    if (a.qoi == QOI_AVG_DISP) {
      const double d = V * (1.0 / 12.0);
      st4(a.dbuf + 16ll * (s - a.ebase) + 4 * n, d, d, d, 0.0);
    }
    const int lG = max(fx_high(G[0]), max(fx_high(G[1]), fx_high(G[2]))), bG = fx_exp(lG);
    const int lh = max(fx_high(hv[0]), max(fx_high(hv[1]), fx_high(hv[2]))), bh = fx_exp(lh);
    all = max(all, max(lG, lh));
#pragma unroll
    for (int k = 0; k < 3; ++k) axis[k] = max(axis[k], fx_high(hv[k]) >> 20);
    const int um = bF + bG - 2103, uP = bI + bh - 2104, uq = max(um, uP), un = um + bS - 1021;
    const int uX = max(bm + um - 1021, bp + bh - 2105);
    const int uY = max(byh + bh - 2105, need_n ? max(byq + uq - 1021, byn + un - 1021) : -32768);
    Fx fG[3], fm[3], fh[3], fq[3], fn[3];
    double dM[3];  // d (KS) / du = vq q + vh h + vn n
#pragma unroll
    for (int k = 0; k < 3; ++k) fG[k] = fx_factor(G[k], bG);
    unsigned long long mm = 0, mq = 0, mX = 0, mY = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      FxSum m;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        m.add(fFC[i][k], fG[k]);
        m.add_low(fFC[i][k], fG[k]);
      }
      const long long mi = (m.value<5>() + 2) >> 2;
      fm[i] = fx_split(mi);
      fh[i] = fx_factor62(hv[i], bh);
      const long long qi = (mi >> fx_shift(uq - um)) - (fx_mul(fI, fh[i]) >> fx_shift(uq - uP));
      fq[i] = fx_split(qi);
      if (a.qoi == QOI_KS_VM) dM[i] = vq * fx_double(qi, uq) + vh * hv[i];
      put_factor(at(0, n, i), fh[i]);
      slot[at(1, n, i) * ELEMS] = qi;
      mm |= fx_abs(mi);
      mq |= fx_abs(qi);
    }
    if (need_n) {
      FxSum n0, n1, n2;
      n0.add(fS[0], fm[0]); n0.add(fS[3], fm[1]); n0.add(fS[5], fm[2]);
      n1.add(fS[3], fm[0]); n1.add(fS[1], fm[1]); n1.add(fS[4], fm[2]);
      n2.add(fS[5], fm[0]); n2.add(fS[4], fm[1]); n2.add(fS[2], fm[2]);
      const long long nv[3] = {n0.value<4>() >> 1, n1.value<4>() >> 1, n2.value<4>() >> 1};
#pragma unroll
      for (int k = 0; k < 3; ++k) fn[k] = fx_split(nv[k]);
      if (a.qoi == QOI_KS_VM)
        st4(a.dbuf + 16ll * (s - a.ebase) + 4 * n, dM[0] + vn * fx_double(nv[0], un),
            dM[1] + vn * fx_double(nv[1], un), dM[2] + vn * fx_double(nv[2], un), 0.0);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long long x = (fx_mul1(fxm, fm[k]) >> fx_shift(uX - (bm + um - 1021))) +
                          (fx_mul1(fxh, fh[k]) >> fx_shift(uX - (bp + bh - 2105)));
      long long y = fx_mul1(fyh, fh[k]) >> fx_shift(uY - (byh + bh - 2105));
      if (need_n)
        y += (fx_mul1(fyq, fq[k]) >> fx_shift(uY - (byq + uq - 1021))) +
             (fx_mul1(fyn, fn[k]) >> fx_shift(uY - (byn + un - 1021)));
      slot[at(2, n, k) * ELEMS] = x;
      slot[at(3, n, k) * ELEMS] = y;
      mX |= fx_abs(x);
      mY |= fx_abs(y);
    }
    const int unit = bh - 1084, rq = uq - unit, rX = uX - unit, rY = uY - unit;
    held = min(held, fx_bits(mm));
    up = min(up, 62 - rq - fx_bits(mq));
    F = max(F, rX + fx_bits(mX) - 62);
    FY = max(FY, rY + fx_bits(mY) - 62);
    bhs |= (unsigned long long)bh << (16 * n);
    slot[(kFixNode + n) * ELEMS] =
        (long long)rY << 48 | (long long)(rX & 0xffff) << 32 | (long long)(rq & 0xffff) << 16 | bh;
  }
  if (SPLIT > 1) {
    __syncthreads();
    bhs = 0;
#pragma unroll
    for (int n = 0; n < 4; ++n) bhs |= (unsigned long long)(slot[(kFixNode + n) * ELEMS] & 0xffff) << (16 * n);
  }

  // The final scales. X_n, Z_n: unit xh_n + F. q_n is far smaller than h_n near the
  // undeformed state and a plastic Y_n far larger than X_n, so they have their own:
  // q_n unit xh_n - up, Y_n unit xh_n + FY; their products come `down` bits finer
  // than the others.
  auto of16 = [](long long w, int n) { return (int)(short)(w >> (16 * n)); };
  auto xh_of = [&](int n) { return of16(bhs, n) - 1084; };
  // c_ab = ga V G_a . C G_b of the pairs (in FP64: two numbers to quantize for
  // each would cost more)
#pragma unroll 1
  for (int n = 0, p = 0; n < 3; ++n) {
    if (SPLIT > 1 && n % SPLIT != part) {  // the pairs (n, b) are this node's
      p += 3 - n;
      continue;
    }
    double G[3], CG[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) G[k] = __ldg(a.d.grads + (3 * n + k) * E + s);
    if constexpr (MODEL == MODEL_J2) {
      CG[0] = gaV * (pt.C[0] * G[0] + pt.C[3] * G[1] + pt.C[5] * G[2]);
      CG[1] = gaV * (pt.C[3] * G[0] + pt.C[1] * G[1] + pt.C[4] * G[2]);
      CG[2] = gaV * (pt.C[5] * G[0] + pt.C[4] * G[1] + pt.C[2] * G[2]);
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k) CG[k] = gaV * G[k];
    }
#pragma unroll 1
    for (int b = n + 1; b < 4; ++b, ++p) {
#pragma unroll
      for (int k = 0; k < 3; ++k) G[k] = __ldg(a.d.grads + (3 * b + k) * E + s);
      const double c = fma(CG[0], G[0], fma(CG[1], G[1], CG[2] * G[2]));
      all = max(all, fx_high(c));
      F = max(F, fx_exp(fx_high(c)) - 1146 - xh_of(n) - xh_of(b));
      slot[(kFixC + p) * ELEMS] = __double_as_longlong(c);
    }
  }

  if (SPLIT > 1) {
    slot[(kFixPart + part) * ELEMS] = ((long long)held << 32) | (unsigned)all;
    slot[(kFixPart + 4 + part) * ELEMS] = ((long long)F << 32) | ((long long)(FY & 0xffff) << 16) | (up & 0xffff);
    slot[(kFixPart + 8 + part) * ELEMS] = ((long long)axis[0] << 32) | ((long long)axis[1] << 16) | axis[2];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SPLIT; ++k) {
      const long long z = slot[(kFixPart + k) * ELEMS], f = slot[(kFixPart + 4 + k) * ELEMS];
      held = min(held, (int)(z >> 32));
      all = max(all, (int)z);
      F = max(F, (int)(f >> 32));
      FY = max(FY, (int)(short)(f >> 16));
      up = min(up, (int)(short)f);
      const long long x = slot[(kFixPart + 8 + k) * ELEMS];
      axis[0] = max(axis[0], (int)(x >> 32));
      axis[1] = max(axis[1], (int)(x >> 16 & 0xffff));
      axis[2] = max(axis[2], (int)(x & 0xffff));
    }
  }
  F = max(F, FY - up);

  // scales of the other entries, and the factors
  double tvv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) tvv[k] = tJV * vv[k];
  const int lt = max(fx_high(tvv[0]), max(fx_high(tvv[1]), fx_high(tvv[2])));
  const int bT = fx_exp(lt), bJ = fx_exp(fx_high(tJV)), bU = fx_exp(fx_high(upf));
  const int bP = fx_exp(fx_high(pu0)), xc = fx_exp(fx_high(ppc)) - 1082;
  all = max(max(all, lt), max(max(fx_high(tJV), fx_high(upf)), max(fx_high(pu0), fx_high(ppc))));
  const bool wide = all >= 0x7ff00000 || held < kFixHeld || fx_spread(axis) > kFxSpread;
  const Fx fz = fx_factor62(zs, bz), fJ = fx_factor62(tJV, bJ), fU = fx_factor62(upf, bU), fP = fx_factor62(pu0, bP);
  const long long mass = fx_at(ppc, xc);
  Fx ft[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) ft[k] = fx_factor62(tvv[k], bT);
  const int down = F + up - FY;
  // h_n is in units 2^(exp_of(n) - 1082)
  auto exp_of = [&](int n) { return of16(bhs, n) - 2; };
#pragma unroll 1
  for (int n = part; n < 4; n += SPLIT) {
    const long long units = slot[(kFixNode + n) * ELEMS];
    const int dq = of16(units, 1) + up, dX = of16(units, 2) - F, dY = of16(units, 3) - FY;
    long long w = 0;  // tau J V v . h_n
#pragma unroll
    for (int q = 0; q < 3; ++q) w += fx_mul(ft[q], factor(at(0, n, q)));
#pragma unroll
    for (int q = 3; q < 12; ++q) {
      const int i = at(q / 3, n, q % 3);
      put_factor(i, fx_split(fx_scale(slot[i * ELEMS], q < 6 ? dq : q < 9 ? dX : dY)));
    }
    put_factor(kFixW + n, fx_split(w));
  }
  if (SPLIT > 1) __syncthreads();
  if (wide) {
    if (part == 0) record_fp64<MODEL>(a, s);
    return;
  }

  auto store_row = [&](long long* p, long long x0, long long x1, long long x2, long long x3) {
    st4(reinterpret_cast<double*>(p), __longlong_as_double(x0), __longlong_as_double(x1), __longlong_as_double(x2),
        __longlong_as_double(x3));
  };
  auto store_exps = [&](int r, int c, int uu, int up, int pu, int pp) {
    reinterpret_cast<short4*>(rec + kRecExp)[4 * r + c] = make_short4((short)uu, (short)up, (short)pu, (short)pp);
  };
  // e_ab = h_a . h_b, and K^pp: the pressure mass term and tau J e_ab at a common scale
  auto pp_block = [&](const Fx& e, int er, int ec, int& x) {
    const int xj = bJ + er + ec - 3120;
    long long r = mass;
    fx_acc(r, xc, fx_mul(e, fJ), xj);
    x = max(xc, xj);
    return r;
  };
#pragma unroll 1
  for (int r = 0, p = 0; r < 4; ++r) {
    const int er = exp_of(r);
    Fx hr[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) hr[k] = factor(at(0, r, k));
    Fx Z[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) Z[k] = fx_split(fx_scale(fx_mul1(fz, hr[k]), bz - 1021 - F));
    if (SPLIT == 1 || r % SPLIT == part) {  // column 3 of the diagonal block
      const Fx e = fx_split(fx_mul(hr[0], hr[0]) + fx_mul(hr[1], hr[1]) + fx_mul(hr[2], hr[2]));
      int xpp;
      const long long pp = pp_block(e, er, er, xpp);
      store_row(rec + kRecDiag + 4 * r, fx_mul1(fU, hr[0]), fx_mul1(fU, hr[1]), fx_mul1(fU, hr[2]), pp);
      store_exps(r, r, 0, bU + er - 2103, 0, xpp);
    }
#pragma unroll 1
    for (int c = r + 1; c < 4; ++c, ++p) {
      if (SPLIT > 1 && p % SPLIT != SPLIT - 1 - part) continue;
      const int ec = exp_of(c);
      const int x = er + ec + F - 2100;
      const long long cab =
          fx_at(__longlong_as_double(slot[(kFixC + p) * ELEMS]), x);
      Fx hc[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) hc[k] = factor(at(0, c, k));
      long long P[3][3];  // h_c Z_r + c_ab I: shared by the pair
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) P[i][k] = fx_mul(hc[i], Z[k]) + (i == k ? cab : 0);
      const Fx e = fx_split(fx_mul(hr[0], hc[0]) + fx_mul(hr[1], hc[1]) + fx_mul(hr[2], hc[2]));
      const Fx wr = factor(kFixW + r), wc = factor(kFixW + c);
      int xpp;
      const long long pp = pp_block(e, er, ec, xpp);
      // K^pu, stabilization: w_r h_c - w_c h_r - e v at xs, and the term with the other node's h
      const int xs = bT + er + ec - 3120;
      long long D[3], T3[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        D[k] = fx_mul(wr, hc[k]) - fx_mul(wc, hr[k]);
        T3[k] = fx_mul(e, ft[k]);
      }
      auto block = [&](int row, int col, const Fx(&hrow)[3], const Fx(&hcol)[3], int erow, int ecol, bool flip) {
        long long* blk = rec + kRecOff + 16 * off_index(row, col);
        Fx X[3], Y[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          X[k] = factor(at(2, col, k));
          Y[k] = factor(at(3, col, k));
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const Fx q = factor(at(1, row, i));
          long long K[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            K[k] = fx_mul(hrow[i], X[k]) + (fx_mul(q, Y[k]) >> min(down, 63)) + (flip ? P[k][i] : P[i][k]);
          }
          store_row(blk + 4 * i, K[0], K[1], K[2], fx_mul1(fU, hrow[i]));
        }
        const int xp = bP + ecol - 2102;
        long long K3[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          K3[k] = -fx_mul(fP, hcol[k]);
          fx_acc(K3[k], xp, (flip ? -D[k] : D[k]) - T3[k], xs);
        }
        store_row(blk + 12, K3[0], K3[1], K3[2], pp);
        store_exps(row, col, x, bU + erow - 2103, max(xp, xs), xpp);
      };
      block(r, c, hr, hc, er, ec, false);
      block(c, r, hc, hr, ec, er, true);
    }
  }
}

// ------------------------------------------------------------------ reductions
// True in all threads of the block that finishes last; part is then complete.
// The ticket is zero again for the next reduction.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) {
      *ticket = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}
__device__ __forceinline__ void put_sum(KSum acc, double* part, unsigned* ticket, double* out) {
  acc = block_reduce(acc);
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = acc.s; part[2 * blockIdx.x + 1] = acc.c; }
  if (!last_block(ticket)) return;
  KSum all;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    KSum t;
    t.s = __ldcg(part + 2 * i);
    t.c = __ldcg(part + 2 * i + 1);
    all.add(t);
  }
  all = block_reduce(all);
  if (threadIdx.x == 0) *out = all.value();
}

// The sum of x, to host memory.
__global__ void k_sum(const double* x, int n, double* part, unsigned* ticket, double* out) {
  KSum acc;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc.add(x[i]);
  put_sum(acc, part, ticket, out);
}

__device__ __forceinline__ double vm_of(const double* sig, int E, int s) {
  double a00 = sig[0 * E + s], a11 = sig[4 * E + s], a22 = sig[8 * E + s];
  double a01 = sig[1 * E + s], a12 = sig[5 * E + s], a20 = sig[6 * E + s];
  double d1 = a00 - a11, d2 = a11 - a22, d3 = a22 - a00;
  return sqrt(0.5 * (d1 * d1 + d2 * d2 + d3 * d3 + 6.0 * (a01 * a01 + a12 * a12 + a20 * a20)));
}

// The largest stored von Mises stress, to device memory (for the sum) and to
// host memory.
__global__ void k_vm_max(const double* sig, int E, double* part, unsigned* ticket, double* out, double* host) {
  double m = 0.0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < E; s += gridDim.x * blockDim.x) m = fmax(m, vm_of(sig, E, s));
  m = block_max(m);
  if (threadIdx.x == 0) part[blockIdx.x] = m;
  if (!last_block(ticket)) return;
  m = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) m = fmax(m, __ldcg(part + i));
  m = block_max(m);
  if (threadIdx.x == 0) {
    *out = m;
    *host = m;
  }
}
// sum of exp(rho (vm - max vm)) w dv, to host memory
__global__ void k_ks_sum(const double* sig, const double* vol, int E, double rho, const double* mx, double* part,
                         unsigned* ticket, double* host) {
  const double m = *mx;
  KSum acc;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < E; s += gridDim.x * blockDim.x)
    acc.add(exp(rho * (vm_of(sig, E, s) - m)) * vol[s]);
  put_sum(acc, part, ticket, host);
}

__global__ void k_cpinv(int E, const double* Fp_old, double* Cpinv) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < E; s += gridDim.x * blockDim.x) {
    double A[3][3];
    for (int q = 0; q < 9; ++q) A[q / 3][q % 3] = Fp_old[q * E + s];
    double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
    double c01 = A[1][0] * A[2][2] - A[1][2] * A[2][0];
    double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
    double d = A[0][0] * c00 - A[0][1] * c01 + A[0][2] * c02;
    double I[3][3];
    I[0][0] = c00 / d;
    I[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) / d;
    I[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) / d;
    I[1][0] = (A[1][2] * A[2][0] - A[1][0] * A[2][2]) / d;
    I[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) / d;
    I[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) / d;
    I[2][0] = (A[1][0] * A[2][1] - A[1][1] * A[2][0]) / d;
    I[2][1] = (A[0][1] * A[2][0] - A[0][0] * A[2][1]) / d;
    I[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) / d;
    // Cp^-1 = Fp^-1 Fp^-T
    auto cc = [&](int i, int j) { return I[i][0] * I[j][0] + I[i][1] * I[j][1] + I[i][2] * I[j][2]; };
    Cpinv[0 * E + s] = cc(0, 0);
    Cpinv[1 * E + s] = cc(1, 1);
    Cpinv[2 * E + s] = cc(2, 2);
    Cpinv[3 * E + s] = cc(0, 1);
    Cpinv[4 * E + s] = cc(1, 2);
    Cpinv[5 * E + s] = cc(0, 2);
  }
}

// Fp = exp(A) Fp_old at points with a pending plastic write (pend), then
// pend = 0. Sets *failed where the exponential series did not settle.
__global__ void k_materialize_fp(int E, const double* __restrict__ Apend, int* __restrict__ pend,
                                 const double* __restrict__ Fp_old, double* __restrict__ Fp, int* failed) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < E; s += gridDim.x * blockDim.x) {
    if (!pend[s]) continue;
    const double a00 = Apend[0 * E + s], a11 = Apend[1 * E + s], a22 = Apend[2 * E + s];
    const double a01 = Apend[3 * E + s], a12 = Apend[4 * E + s], a02 = Apend[5 * E + s];
    const double Am[3][3] = {{a00, a01, a02}, {a01, a11, a12}, {a02, a12, a22}};
    double Ex[3][3];
    if (!exp_traceless_sym(Am, Ex)) *failed = 1;
    double Fo[3][3];
    for (int q = 0; q < 9; ++q) Fo[q / 3][q % 3] = Fp_old[q * E + s];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) Fp[(3 * i + j) * E + s] = Ex[i][0] * Fo[0][j] + Ex[i][1] * Fo[1][j] + Ex[i][2] * Fo[2][j];
    pend[s] = 0;
  }
}

__global__ void k_fill_identity(int E, double* Fp) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < E; s += gridDim.x * blockDim.x)
    for (int q = 0; q < 9; ++q) Fp[q * E + s] = (q % 4 == 0) ? 1.0 : 0.0;
}

template <int MODEL, int MODE, bool JAC, bool ERR>
void launch_colours(const Disc& d, ElemArgs args, cudaStream_t st, bool buffered) {
  const int block = 64;  // 128 spreads less evenly: residual of 48k elements 44 us against 40, of 384k 256 both
  if (MODE == MODE_NONE || buffered) {
    // elements [args.begin, args.end) into the buffer (all of them, or a chunk)
    const int n = args.end - args.begin;
    if (n <= 0) return;
    k_elem<MODEL, MODE, JAC, ERR, true><<<(n + block - 1) / block, block, 0, st>>>(args);
    GOAL_CHECK_LAUNCH();
  } else {
  for (int c = 0; c < d.num_colors; ++c) {
    args.begin = d.color_ptr[c];
    args.end = d.color_ptr[c + 1];
    int n = args.end - args.begin;
    if (n <= 0) continue;
    k_elem<MODEL, MODE, JAC, ERR, false><<<(n + block - 1) / block, block, 0, st>>>(args);
    GOAL_CHECK_LAUNCH();
  }
  }
}

template <int MODEL, int ELEMS, int SPLIT>
void launch_fix(const ElemArgs& args, int n, cudaStream_t st) {
  constexpr int smem = kFixSmem<ELEMS, SPLIT>;
  GOAL_CUDA(cudaFuncSetAttribute(k_elem_fix<MODEL, ELEMS, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_elem_fix<MODEL, ELEMS, SPLIT><<<(n + ELEMS - 1) / ELEMS, ELEMS * SPLIT, smem, st>>>(args);
  GOAL_CHECK_LAUNCH();
}

template <int MODEL>
void dispatch(const Disc& d, const Chain& c, const ElemArgs& args, cudaStream_t st, bool buf, bool fix) {
  if (c.error_chain) {
    GOAL_REQUIRE(!c.jacobian && c.mode == MODE_PRIMAL, GOAL_ERR_ARG, "the error chain is a residual (PRIMAL) chain");
    launch_colours<MODEL, MODE_PRIMAL, false, true>(d, args, st, buf);
    return;
  }
  if (fix) {
    // Four or two threads to an element while that is four warps to an SM (their
    // FP64 work is repeated, so more would wait for its pipe: 10k elements with
    // four 52 us, 16.5k with two 44); then blocks of 64 until there are two waves
    // of 128, as they spread more evenly. J2, us, blocks of 128 -> now: 384 to
    // 4.4k elements 40 -> 25, 6k 40 -> 29, 10k 40 -> 39.5, 25k 60 -> 51, 48k
    // 82 -> 73; at 384k blocks of 64 take 435 against 432.
    const int n = args.end - args.begin;
    if (n <= 32 * kSMs) launch_fix<MODEL, 32, 4>(args, n, st);
    else if (n <= 64 * kSMs) launch_fix<MODEL, 32, 2>(args, n, st);
    else if (n <= 100000) launch_fix<MODEL, 64, 1>(args, n, st);
    else launch_fix<MODEL, 128, 1>(args, n, st);
    return;
  }
  if (c.mode == MODE_NONE) {
    if (c.jacobian) launch_colours<MODEL, MODE_NONE, true, false>(d, args, st, true);
    else launch_colours<MODEL, MODE_NONE, false, false>(d, args, st, true);
  } else if (c.mode == MODE_PRIMAL) {
    if (c.jacobian) launch_colours<MODEL, MODE_PRIMAL, true, false>(d, args, st, buf);
    else launch_colours<MODEL, MODE_PRIMAL, false, false>(d, args, st, buf);
  } else {
    GOAL_REQUIRE(c.jacobian, GOAL_ERR_ARG, "ADJOINT mode is a Jacobian (FADT) chain");
    launch_colours<MODEL, MODE_ADJOINT, true, false>(d, args, st, buf);
  }
}

// Row r of contribution v (element slot v >> 4, element block v & 15) of the
// element buffer; TRANSPOSE reads column r of the transposed element block.
template <bool TRANSPOSE>
__device__ __forceinline__ void load_contrib(const double* __restrict__ ebuf, int estride, int v, int r, double& x0,
                                             double& x1, double& x2, double& x3, int lo = 0) {
  const int s = (v >> 4) - lo, lb = v & 15;
  if (TRANSPOSE) {
    const int lt = ((lb & 3) << 2) | (lb >> 2);
    const double* p = ebuf + (size_t)s * estride + 16 + 16 * lt + r;
    x0 = __ldg(p); x1 = __ldg(p + 4); x2 = __ldg(p + 8); x3 = __ldg(p + 12);
  } else {
    ld4(ebuf + (size_t)s * estride + 16 + 16 * lb + 4 * r, x0, x1, x2, x3);
  }
}

// Phase 2 of the two-phase assembly: every matrix block sums its element
// blocks in element order (4 threads per block, one per row); TRANSPOSE
// accumulates the element blocks transposed (ADJOINT mode stores dR/du^T).
// Contributions are fetched four at a time (independent loads in flight),
// then added in element order. The blocks come from a list (ks[0..count)):
// one launch for the off-diagonal blocks (a few contributions each) and one
// for the diagonal blocks (one per incident element), so that the threads of
// a warp do equal work.
template <bool TRANSPOSE>
__global__ void __launch_bounds__(256) k_gather_blocks(int count, const int* __restrict__ ks,
                                                       const int* __restrict__ bptr, const int* __restrict__ blist,
                                                       const double* __restrict__ ebuf, int estride,
                                                       double* __restrict__ A, int accumulate) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 4ll * count;
       t += (long long)gridDim.x * blockDim.x) {
    const int k = __ldg(ks + (t >> 2)), r = (int)(t & 3);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (accumulate) ld4(A + 16ll * k + 4 * r, a0, a1, a2, a3);
    const int c1 = __ldg(bptr + k + 1);
    int c = __ldg(bptr + k);
    for (; c + 4 <= c1; c += 4) {
      double x[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        load_contrib<TRANSPOSE>(ebuf, estride, __ldg(blist + c + q), r, x[q][0], x[q][1], x[q][2], x[q][3]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a0 += x[q][0]; a1 += x[q][1]; a2 += x[q][2]; a3 += x[q][3];
      }
    }
    for (; c < c1; ++c) {
      double x0, x1, x2, x3;
      load_contrib<TRANSPOSE>(ebuf, estride, __ldg(blist + c), r, x0, x1, x2, x3);
      a0 += x0; a1 += x1; a2 += x2; a3 += x3;
    }
    st4(A + 16ll * k + 4 * r, a0, a1, a2, a3);
  }
}

// k_gather_blocks for one chunk of elements [lo, hi) (the element buffer
// holds that chunk only): the contributions of the chunk, in element order,
// are added to the block as it stands, so chunk after chunk the additions
// are the ones of the one-pass gather, in the same order.
template <bool TRANSPOSE>
__global__ void __launch_bounds__(256) k_gather_blocks_chunk(int count, const int* __restrict__ ks,
                                                             const int* __restrict__ bptr,
                                                             const int* __restrict__ blist,
                                                             const double* __restrict__ ebuf, int estride,
                                                             double* __restrict__ A, int accumulate, int lo, int hi) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 4ll * count;
       t += (long long)gridDim.x * blockDim.x) {
    const int k = __ldg(ks + (t >> 2)), r = (int)(t & 3);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (accumulate) ld4(A + 16ll * k + 4 * r, a0, a1, a2, a3);
    const int c1 = __ldg(bptr + k + 1);
    for (int c = __ldg(bptr + k); c < c1; ++c) {
      const int v = __ldg(blist + c), e = v >> 4;
      if (e < lo || e >= hi) continue;
      double x0, x1, x2, x3;
      load_contrib<TRANSPOSE>(ebuf, estride, v, r, x0, x1, x2, x3, lo);
      a0 += x0; a1 += x1; a2 += x2; a3 += x3;
    }
    st4(A + 16ll * k + 4 * r, a0, a1, a2, a3);
  }
}

// Phase 2 for nodal vectors: node n, row q sums the element rows of its
// incident elements (entries 4*s + a of nlist) in element order.
// [lo, hi): the element slots the buffer holds (a chunk; the buffer's first
// entry is slot lo); the one-pass gather has lo = 0, hi = E.
__global__ void __launch_bounds__(256) k_gather_nodes(int N, const int* __restrict__ nptr,
                                                      const int* __restrict__ nlist, const double* ebuf,
                                                      int estride, double* __restrict__ out, int accumulate, int lo,
                                                      int hi) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 4ll * N;
       t += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(t >> 2), q = (int)(t & 3);
    const int c0 = __ldg(nptr + n), c1 = __ldg(nptr + n + 1);
    const double* buf = wait_for_elements(ebuf);
    double acc = accumulate ? out[t] : 0.0;
    for (int c = c0; c < c1; ++c) {
      const int v = __ldg(nlist + c), e = v >> 2;
      if (e < lo || e >= hi) continue;
      acc += buf[(size_t)(e - lo) * estride + 4 * (v & 3) + q];
    }
    out[t] = acc;
  }
}

// One lane's share of a diagonal block's row: the sum of the row's
// off-diagonal blocks, 96 bits at a common exponent.
struct RowSum {
  long long h[3] = {0, 0, 0}, l[3] = {0, 0, 0};  // h 2^32 + l
  int x = -32768;
  __device__ __forceinline__ void raise(int to) {  // to the larger exponent `to`
    const int d = min(to - x, 95);
    if (d > 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const long long hh = h[k] + (l[k] >> 32);
        const unsigned ll = (unsigned)l[k];
        const unsigned h0 = (unsigned)hh;
        l[k] = d < 32 ? (unsigned)((((unsigned long long)h0 << 32) | ll) >> d) : (unsigned)(hh >> min(d - 32, 63));
        h[k] = hh >> min(d, 63);
      }
    }
    x = max(x, to);
  }
  __device__ __forceinline__ void add(const long long (&v)[4], int xv) {
    raise(xv);
    const int d = fx_shift(x - xv);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long long s = v[k] >> d;
      h[k] += s >> 32;
      l[k] += (unsigned)s;
    }
  }
};

// Phase 2 after a FIX element phase. The first row_blocks blocks of the grid
// take one matrix block row to a warp: a quad of lanes sums the contributions
// of one off-diagonal block (a lane per row of it) in integers aligned to the
// largest exponent met, and the warp then forms the diagonal block: its u
// columns as the negated sum of the row's off-diagonal blocks, column 3 from
// the elements' diagonal records. ADJ stores the transpose (dR/du^T): block
// (n, m) goes to block (m, n). The remaining blocks sum the nodal vectors, as
// k_gather_nodes does (four threads per node, element order): R from the
// records, and dM/du from dbuf, or zero without one.
// The sums need no FP64 instruction but one conversion per matrix entry. At
// 384,000 elements 230 us (4.1 TB/s; latency and the integer pipes, 47% busy)
// against 268 us for the FP64 gathers, which the shorter element phase and the
// single launch come on top of; with the lists fetched where they are used the
// kernel took 257 us, with the lists of two passes in registers 283 us.
// A row with an element whose record is in FP64 is summed again in FP64
// (384,000 elements, all of them such: 1.34 ms a neo-Hookean chain, J2 1.53;
// 0.1% of them: 0.56 -> 0.62 and 0.62 -> 0.69).

// Row of a record's block. Each is read once, and leaves L1 to the lists and
// exponents (gather of 384,000 elements: 237 us through L1, 230 past it; exponents
// past it too 229, but the chain of 384 elements 39.3 -> 40.0).
__device__ __forceinline__ longlong4_32a ld_row(const long long* p) {
  longlong4_32a v;
  asm volatile("ld.global.L1::no_allocate.v4.s64 {%0, %1, %2, %3}, [%4];"
               : "=l"(v.x), "=l"(v.y), "=l"(v.z), "=l"(v.w)
               : "l"(p));
  return v;
}

// The 4x4 block whose row r a lane of the quad holds, transposed.
template <bool ADJ>
__device__ __forceinline__ void transpose_quad(double (&d)[4], int r) {
  if (!ADJ) return;
  const unsigned full = 0xffffffffu;
  const bool hi = (r & 2) != 0, odd = (r & 1) != 0;
  const double s0 = __shfl_xor_sync(full, hi ? d[0] : d[2], 2), s1 = __shfl_xor_sync(full, hi ? d[1] : d[3], 2);
  const double a0 = hi ? s0 : d[0], a1 = hi ? s1 : d[1], a2 = hi ? d[2] : s0, a3 = hi ? d[3] : s1;
  const double t0 = __shfl_xor_sync(full, odd ? a0 : a1, 1), t1 = __shfl_xor_sync(full, odd ? a2 : a3, 1);
  d[0] = odd ? t0 : a0; d[1] = odd ? a1 : t0; d[2] = odd ? t1 : a2; d[3] = odd ? a3 : t1;
}
// Row [k0, k0 + nk) of the matrix by one warp, diagonal block kd: the terms in
// list order, the diagonal's u columns as negated sums of the row's blocks.
template <bool ADJ>
__device__ __noinline__ void gather_row_fp64(int k0, int nk, int kd, const int* btr, const int* bptr, const int* blist,
                                             const long long* rec, double* A) {
  const int lane = threadIdx.x & 31, q = lane >> 2, r = lane & 3;
  const unsigned full = 0xffffffffu;
  auto value = [](long long v, int e) { return e == kFxFloat ? __longlong_as_double(v) : fx_double(v, e); };
  auto exps = [&](const long long* p, int l) { return reinterpret_cast<const int*>(p + kRecExp + (l & 15))[r == 3 ? 1 : 0]; };
  double u[3] = {0.0, 0.0, 0.0};
  for (int i0 = 0; i0 < nk - 1; i0 += 8) {
    const bool live = i0 + q < nk - 1;
    const int k = k0 + i0 + q + (i0 + q >= kd ? 1 : 0);
    double d[4] = {0.0, 0.0, 0.0, 0.0};
    if (live) {
      for (int c = bptr[k]; c < bptr[k + 1]; ++c) {
        const int l = blist[c];
        const long long* p = rec + (size_t)(l >> 4) * kRecord;
        const int e = exps(p, l);
        const long long* v = p + kRecOff + 16 * off_index((l >> 2) & 3, l & 3) + 4 * r;
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] += value(v[j], j < 3 ? (short)e : e >> 16);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) u[j] += d[j];
    }
    transpose_quad<ADJ>(d, r);
    if (live) st4(A + 16ll * (ADJ ? btr[k] : k) + 4 * r, d[0], d[1], d[2], d[3]);
  }
  double d[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = bptr[k0 + kd] + q; i < bptr[k0 + kd + 1]; i += 8) {
    const int l = blist[i];
    const long long* p = rec + (size_t)(l >> 4) * kRecord;
    d[3] += value(p[kRecDiag + 4 * (l & 3) + r], exps(p, l) >> 16);
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    d[3] += __shfl_xor_sync(full, d[3], o);
#pragma unroll
    for (int j = 0; j < 3; ++j) u[j] += __shfl_xor_sync(full, u[j], o);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) d[j] = -u[j];
  transpose_quad<ADJ>(d, r);
  if (q == 0) st4(A + 16ll * (k0 + kd) + 4 * r, d[0], d[1], d[2], d[3]);
}

constexpr int kRowTerms = 192;  // list entries of a row kept in shared memory (96 on the Kuhn grid)
template <bool ADJ>
__global__ void __launch_bounds__(128, 8) k_gather_rows(int N, int row_blocks, const int* __restrict__ brow_ptr,
                                                     const int* __restrict__ diag, const int* __restrict__ btr,
                                                     const int* __restrict__ bptr, const int* __restrict__ blist,
                                                     const int* __restrict__ nptr, const int* __restrict__ nlist,
                                                     const long long* records, double* __restrict__ A,
                                                     double* __restrict__ R, const double* dbuf,
                                                     double* __restrict__ dMdu) {
  if ((int)blockIdx.x >= row_blocks) {
    const long long vectors = 2;  // R, then dM/du
    for (long long t = (blockIdx.x - row_blocks) * (long long)blockDim.x + threadIdx.x; t < vectors * 4ll * N;
         t += (long long)(gridDim.x - row_blocks) * blockDim.x) {
      const bool second = t >= 4ll * N;
      const long long i = second ? t - 4ll * N : t;
      const int n = (int)(i >> 2), q = (int)(i & 3);
      const int c0 = __ldg(nptr + n), c1 = __ldg(nptr + n + 1);
      const double* src = wait_for_elements(second ? dbuf : reinterpret_cast<const double*>(records));
      if (second && !dbuf) {  // no QoI: dM/du is cleared
        dMdu[i] = 0.0;
        continue;
      }
      const int stride = second ? 16 : kRecord;
      double acc = 0.0;
#pragma unroll 4
      for (int c = c0; c < c1; ++c) {
        const int v = __ldg(nlist + c);
        acc += src[(size_t)(v >> 2) * stride + 4 * (v & 3) + q];
      }
      (second ? dMdu : R)[i] = acc;
    }
    return;
  }
  const int lane = threadIdx.x & 31, q = lane >> 2, r = lane & 3;
  const unsigned full = 0xffffffffu;
  const long long* rec = wait_for_elements(records);
  constexpr int kNone = -32768;  // exponent of no term: every shift takes it to zero
  __shared__ int lists[4][kRowTerms];
  int* mine = lists[threadIdx.x >> 5];
  // T terms of a block from list entries w (those past `left` are none): the
  // accumulators go to the largest exponent once, then every term is added there
  auto add = [&](auto count, const int* w, int left, int extra, long long (&acc)[4], int& x0, int& x3) {
    constexpr int T = decltype(count)::value;
    int e0[T], e3[T], m0 = x0, m3 = x3;
    longlong4_32a v[T];
#pragma unroll
    for (int u = 0; u < T; ++u) {
      e0[u] = e3[u] = kNone;
      v[u] = longlong4_32a{0, 0, 0, 0};
      if (u < left) {
        const int l = w[u];
        const long long* p = rec + (size_t)(l >> 4) * kRecord;
        const int e = reinterpret_cast<const int*>(p + kRecExp + (l & 15))[r == 3 ? 1 : 0];
        v[u] = ld_row(p + kRecOff + 16 * off_index((l >> 2) & 3, l & 3) + 4 * r);
        e0[u] = (short)e + extra;
        e3[u] = (e >> 16) + extra;
      }
    }
#pragma unroll
    for (int u = 0; u < T; ++u) {
      m0 = max(m0, e0[u]);
      m3 = max(m3, e3[u]);
    }
    if (m0 > x0) {
      const int s0 = min(m0 - x0, 62);
      const long long h0 = (1ll << s0) >> 1;
      acc[0] = (acc[0] + h0) >> s0; acc[1] = (acc[1] + h0) >> s0; acc[2] = (acc[2] + h0) >> s0;
    }
    if (m3 > x3) {
      const int s3 = min(m3 - x3, 62);
      acc[3] = (acc[3] + ((1ll << s3) >> 1)) >> s3;
    }
#pragma unroll
    for (int u = 0; u < T; ++u) {
      const int d0 = min(m0 - e0[u] + extra, 62), d3 = min(m3 - e3[u] + extra, 62);
      const long long h0 = (1ll << d0) >> 1, h3 = (1ll << d3) >> 1;  // to round
      acc[0] += (v[u].x + h0) >> d0; acc[1] += (v[u].y + h0) >> d0; acc[2] += (v[u].z + h0) >> d0;
      acc[3] += (v[u].w + h3) >> d3;
    }
    x0 = m0;
    x3 = m3;
  };
  for (int n = blockIdx.x * 4 + (threadIdx.x >> 5); n < N; n += row_blocks * 4) {
    // the lists of the whole row before any record: its block pointers (one a
    // lane) and its terms (in shared memory) are contiguous
    const int k0 = __ldg(brow_ptr + n), nk = __ldg(brow_ptr + n + 1) - k0, nb = nk - 1, kd = __ldg(diag + n) - k0;
    const int bp = __ldg(bptr + k0 + min(lane, nk));
    const int t0 = __shfl_sync(full, bp, 0), t1 = nk < 32 ? __shfl_sync(full, bp, nk) : __ldg(bptr + k0 + nk);
    const bool ahead = t1 - t0 <= kRowTerms;
    const int* terms = ahead ? mine - t0 : blist;  // list entry c is terms[c]
    __syncwarp();
    if (ahead)
      for (int i = lane; i < t1 - t0; i += 32) mine[i] = __ldg(blist + t0 + i);
    __syncwarp();
    auto range = [&](int k, int& c0, int& c1) {  // of block k of the row; all lanes call it
      c0 = __shfl_sync(full, bp, k & 31);
      c1 = __shfl_sync(full, bp, (k + 1) & 31);
      if (k >= 31 && k < nk) {
        c0 = __ldg(bptr + k0 + k);
        c1 = __ldg(bptr + k0 + k + 1);
      }
    };
    RowSum row;
    for (int i0 = 0; i0 < nb; i0 += 8) {
      const bool live = i0 + q < nb;
      const int k = i0 + q + (i0 + q >= kd ? 1 : 0);
      int c, c1;
      range(k, c, c1);
      double d[4] = {0.0, 0.0, 0.0, 0.0};
      if (live) {
        const int extra = c1 - c > 1 ? 32 - __clz(c1 - c - 1) : 0;  // room for that many terms below 2^62
        long long acc[4] = {0, 0, 0, 0};
        int x0 = kNone, x3 = kNone;
        for (; c < c1; c += 4) {
          if (c1 - c > 2) add(std::integral_constant<int, 4>(), terms + c, c1 - c, extra, acc, x0, x3);
          else add(std::integral_constant<int, 2>(), terms + c, c1 - c, extra, acc, x0, x3);
        }
        row.add(acc, x0);
        d[0] = fx_double(acc[0], x0);
        d[1] = fx_double(acc[1], x0);
        d[2] = fx_double(acc[2], x0);
        d[3] = fx_double(acc[3], x3);
      }
      transpose_quad<ADJ>(d, r);
      if (live) st4(A + 16ll * (ADJ ? __ldg(btr + k0 + k) : k0 + k) + 4 * r, d[0], d[1], d[2], d[3]);
    }
    // column 3 of the diagonal block: the terms of block kd are the node's elements
    long long dacc = 0;
    int dx = kNone;
    {
      int c, c1;
      range(kd, c, c1);
      const int extra = c1 - c > 2 ? 31 - __clz(c1 - c - 1) : 0;  // terms below 2^61
#pragma unroll 2
      for (int i = c + q; i < c1; i += 8) {
        const int l = terms[i];
        const long long* p = rec + (size_t)(l >> 4) * kRecord;
        const int e = (reinterpret_cast<const int*>(p + kRecExp + (l & 15))[r == 3 ? 1 : 0] >> 16) + extra;
        const int top = max(dx, e), sa = min(top - dx, 62), sv = min(top - e + extra, 62);
        const long long v = p[kRecDiag + 4 * (l & 3) + r];
        dacc = ((dacc + ((1ll << sa) >> 1)) >> sa) + ((v + ((1ll << sv) >> 1)) >> sv);
        dx = top;
      }
    }
    // sums over the quads: exponents first, then the integers
    int rx = row.x, ex = dx;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      rx = max(rx, __shfl_xor_sync(full, rx, o));
      ex = max(ex, __shfl_xor_sync(full, ex, o));
    }
    // an element in FP64 is among the terms of the diagonal block, as of the others
    if (ex >= kFxFloat) {
      gather_row_fp64<ADJ>(k0, nk, kd, btr, bptr, blist, rec, A);
      continue;
    }
    dacc >>= fx_shift(ex - dx);
    row.raise(rx);
    // the row sums as 64 bits, shifted so far that eight of them cannot overflow
    long long t[3];
    int bits = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      t[k] = row.h[k] + (row.l[k] >> 32);
      bits = max(bits, 64 - __clzll(t[k] ^ (t[k] >> 63)));
    }
    bits = __reduce_max_sync(full, bits);
    const int sh = min(max(bits - 27, 0), 32);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      t[k] = sh == 32 ? t[k] : (t[k] << (32 - sh)) | (long long)((unsigned)row.l[k] >> sh);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      dacc += __shfl_xor_sync(full, dacc, o);
#pragma unroll
      for (int k = 0; k < 3; ++k) t[k] += __shfl_xor_sync(full, t[k], o);
    }
    double d[4];
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] = fx_double(-t[k], rx + sh);
    d[3] = fx_double(dacc, ex);
    transpose_quad<ADJ>(d, r);
    if (q == 0) st4(A + 16ll * (k0 + kd) + 4 * r, d[0], d[1], d[2], d[3]);
  }
}

int reduction_blocks(Mechanics& m, int n) {
  const int nb = std::min(grid_for(n, 256), 1024);
  if (m.red.n < 2 * (size_t)nb + 2) m.red.alloc(2 * nb + 2);
  return nb;
}

}  // namespace

void Mechanics::init() {
  const int E = disc->num_elems, N = disc->num_nodes;
  std::vector<double> m;
  for (const MaterialRow& r : mats_h) {
    double kappa = r.E / (3.0 * (1.0 - 2.0 * r.nu));
    double mu = r.E / (2.0 * (1.0 + r.nu));
    m.insert(m.end(), {kappa, mu, r.K, r.Y, r.c0, 1.0 / kappa, 0.5 * r.c0 / mu, 1.0 / (16.0 * kappa)});
  }
  static bool table_ready = false;
  if (!table_ready) {
    double t[80];
    for (int k = 0; k < 80; ++k) t[k] = 1.0 / (k + 1);
    GOAL_CUDA(cudaMemcpyToSymbol(c_inv_k, t, sizeof(t)));
    table_ready = true;
  }
  mats.upload(m.data(), m.size(), disc->stream);
  U.alloc(4ll * N);
  U.zero(disc->stream);
  st.sigma.alloc(9ll * E);
  st.sigma.zero(disc->stream);
  st.eqps.alloc(E);
  st.eqps.zero(disc->stream);
  st.eqps_old.alloc(E);
  st.eqps_old.zero(disc->stream);
  st.Fp.alloc(9ll * E);
  st.Fp_old.alloc(9ll * E);
  st.Cpinv.alloc(6ll * E);
  st.Apend.alloc(6ll * E);
  st.pend.alloc(E);
  st.pend.zero(disc->stream);
  k_fill_identity<<<grid_for(E, 256), 256, 0, disc->stream>>>(E, st.Fp.ptr);
  k_fill_identity<<<grid_for(E, 256), 256, 0, disc->stream>>>(E, st.Fp_old.ptr);
  GOAL_CHECK_LAUNCH();
  refresh_cpinv();
  qoi_elem.alloc(E);
  ticket.alloc(1);
  ticket.zero(disc->stream);
  results.alloc();
  GOAL_CUDA(cudaStreamSynchronize(disc->stream));  // the material rows above leave with this call
}

void Mechanics::refresh_cpinv() {
  const int E = disc->num_elems;
  k_cpinv<<<grid_for(E, 256), 256, 0, disc->stream>>>(E, st.Fp_old.ptr, st.Cpinv.ptr);
  GOAL_CHECK_LAUNCH();
}

void Mechanics::materialize_fp() {
  const int E = disc->num_elems;
  results.v->series = 0;
  k_materialize_fp<<<grid_for(E, 256), 256, 0, disc->stream>>>(E, st.Apend.ptr, st.pend.ptr, st.Fp_old.ptr, st.Fp.ptr,
                                                               &results.v->series);
  GOAL_CHECK_LAUNCH();
  GOAL_CUDA(cudaStreamSynchronize(disc->stream));
  GOAL_REQUIRE(!results.v->series, GOAL_ERR_RETURN_MAP, "J2: the exponential of the plastic increment did not converge");
}

void Mechanics::update_states() {
  const int E = disc->num_elems;
  materialize_fp();
  GOAL_CUDA(cudaMemcpyAsync(st.Fp_old.ptr, st.Fp.ptr, sizeof(double) * 9 * E, cudaMemcpyDeviceToDevice, disc->stream));
  GOAL_CUDA(cudaMemcpyAsync(st.eqps_old.ptr, st.eqps.ptr, sizeof(double) * E, cudaMemcpyDeviceToDevice, disc->stream));
  refresh_cpinv();
}

void SolInfo::init(Disc* d) {
  disc = d;
  R.alloc(4ll * d->num_nodes);
  dMdu.alloc(4ll * d->num_nodes);
  A.alloc(16ll * d->nnzb);
  R.zero(d->stream);
  dMdu.zero(d->stream);
  A.zero(d->stream);
}

void ks_prepass(Mechanics& m, double rho, double& max_vm, double& scale, cudaStream_t st) {
  const int E = m.disc->num_elems;
  const int nb = reduction_blocks(m, E);
  double* mx = m.red.ptr + 2 * nb;
  k_vm_max<<<nb, 256, 0, st>>>(m.st.sigma.ptr, E, m.red.ptr, m.ticket.ptr, mx, &m.results.v->max_vm);
  GOAL_CHECK_LAUNCH();
  k_ks_sum<<<nb, 256, 0, st>>>(m.st.sigma.ptr, m.disc->vol.ptr, E, rho, mx, m.red.ptr, m.ticket.ptr, &m.results.v->sum);
  GOAL_CHECK_LAUNCH();
  GOAL_CUDA(cudaStreamSynchronize(st));
  max_vm = m.results.v->max_vm;
  scale = m.results.v->sum;
}

namespace {
// Optional device timing of the two assembly phases (CUDA events on the
// assembly's stream, read after the stream synchronisation that ends every
// assembly). Off unless enabled.
struct PhaseTimer {
  bool on = false;
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  double elem_ms = 0.0, gather_ms = 0.0;
  long long count = 0;
} g_phase;
}  // namespace

void assembly_timing(bool enable) {
  if (enable && !g_phase.ev[0])
    for (auto& e : g_phase.ev) GOAL_CUDA(cudaEventCreate(&e));
  g_phase.on = enable;
  if (enable) {
    g_phase.elem_ms = g_phase.gather_ms = 0.0;
    g_phase.count = 0;
  }
}

void assembly_timing_read(double* ms, long long* count) {
  ms[0] = g_phase.elem_ms;
  ms[1] = g_phase.gather_ms;
  *count = g_phase.count;
}

namespace {
long long g_ebuf_limit = 0;  // bytes; 0 = a quarter of the device's memory
}

void set_element_buffer_limit(long long bytes) { g_ebuf_limit = bytes < 0 ? 0 : bytes; }

long long element_buffer_limit() {
  if (g_ebuf_limit > 0) return g_ebuf_limit;
  // a quarter of the device's memory, looked up once per device (the query is
  // too slow to repeat in every assembly)
  constexpr int kDevs = 64;
  static long long total[kDevs] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) return 8ll << 30;
  if (total[dev] == 0) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || total_b == 0) return 8ll << 30;
    total[dev] = (long long)total_b;
  }
  return total[dev] / 4;
}

double assemble(Mechanics& m, SolInfo* s, const Chain& c, const ErrorWeights* w, cudaStream_t st) {
  const Disc& d = *m.disc;
  ElemArgs a;
  std::memset(&a, 0, sizeof(a));
  a.d = d.view();
  a.mats = m.mats.ptr;
  a.U = m.U.ptr;
  a.Fp_old = m.st.Fp_old.ptr;
  a.eqps_old = m.st.eqps_old.ptr;
  a.Cpinv = m.st.Cpinv.ptr;
  a.sigma = m.st.sigma.ptr;
  a.Fp = m.st.Fp.ptr;
  a.eqps = m.st.eqps.ptr;
  a.Apend = m.st.Apend.ptr;
  a.pend = m.st.pend.ptr;
  a.failed = &m.results.v->return_map;
  a.stab = m.stabilization ? 1 : 0;
  a.save = c.save_states;
  a.fp_reset = m.fp_reset ? 1 : 0;
  a.overwrite = c.overwrite;
  a.qoi = c.qoi;
  a.rho = c.rho;
  a.qoi_elem = m.qoi_elem.ptr;
  if (c.mode != MODE_NONE || c.jacobian) {
    GOAL_REQUIRE(s != nullptr, GOAL_ERR_ARG, "assemble: SolInfo required for this chain");
    a.R = s->R.ptr;
    a.A = s->A.ptr;
    a.dMdu = s->dMdu.ptr;
  }
  if (c.error_chain) {
    GOAL_REQUIRE(w && w->Zd && w->Zc, GOAL_ERR_ARG, "error chain needs z weights");
    a.Zd = w->Zd;
    a.Zc = w->Zc;
  }
  double ks_max = 0.0, ks_scale = 1.0;
  if (c.qoi == QOI_KS_VM) {
    GOAL_REQUIRE(c.rho > 0.0, GOAL_ERR_ARG, "KS functional needs rho > 0");
    ks_prepass(m, c.rho, ks_max, ks_scale, st);
    GOAL_REQUIRE(ks_max > 0.0 && ks_scale > 0.0, GOAL_ERR_STATE, "KS functional: stored stresses are zero");
  }
  a.ks_max = ks_max;
  a.ks_scale = ks_scale;
  m.results.v->return_map = 0;
  const bool buf = !c.colored && (c.mode != MODE_NONE || c.jacobian);
  const bool scatter = c.mode != MODE_NONE;
  const int E = d.num_elems;
  int chunk = E;  // elements per pass of the two-phase assembly
  bool fix = false;
  if (buf) {
    a.estride = c.jacobian ? 272 : 16;
    const size_t per_elem = sizeof(double) * (a.estride + ((c.jacobian && c.qoi != QOI_NONE) ? 16 : 0));
    chunk = (int)std::max<long long>(1, std::min<long long>(E, element_buffer_limit() / per_elem));
    // Fixed point and diagonal blocks from row sums: Jacobian chains that overwrite,
    // in one pass, unless the mesh has so many flat elements that their second
    // evaluation, by whole warps, would cost more than it saves (384,000 elements,
    // us: FP64 throughout 997 neo-Hookean, 1,114 J2; fixed point with no flat
    // element 562 and 621, with 0.1% 625 and 695, with all of them 1,386 and 1,581;
    // one in 64 puts one into four of ten warps).
    fix = scatter && c.jacobian && c.overwrite && chunk == E && 64ll * d.flat_elems <= E;
    if (fix) {
      a.estride = kRecord;
      if (c.mode == MODE_ADJOINT) const_cast<Disc&>(d).block_transpose_map();
    }
    size_t need = (size_t)chunk * a.estride;
    if (m.ebuf.n < need) m.ebuf.alloc(need);
    a.ebuf = m.ebuf.ptr;
    if (c.jacobian && c.qoi != QOI_NONE) {
      if (m.dbuf.n < 16ull * chunk) m.dbuf.alloc(16ull * chunk);
      a.dbuf = m.dbuf.ptr;
    }
  }
  if (c.overwrite && c.jacobian && c.qoi == QOI_NONE && s && !fix) {
    // dMdu is not written by a chain without QoI: SolInfo::zero_all semantics (the fixed-point gather clears it)
    GOAL_CUDA(cudaMemsetAsync(s->dMdu.ptr, 0, sizeof(double) * s->dMdu.n, st));
  }
  const bool timed = g_phase.on;
  if (timed) GOAL_CUDA(cudaEventRecord(g_phase.ev[0], st));
  for (int e0 = 0; e0 < E; e0 += chunk) {
    const int e1 = buf ? std::min(E, e0 + chunk) : E;
    a.begin = e0;
    a.end = e1;
    a.ebase = e0;
    if (m.model == MODEL_J2) dispatch<MODEL_J2>(d, c, a, st, buf, fix);
    else dispatch<MODEL_NEOHOOKEAN>(d, c, a, st, buf, fix);
    if (timed && e0 == 0) GOAL_CUDA(cudaEventRecord(g_phase.ev[1], st));
    if (!buf) break;  // the coloured path covers every element itself
    if (fix) {
      const int rows = grid_for(d.num_nodes, 4, kSMs * 64);
      const bool dm = c.qoi != QOI_NONE;
      const int nodes = grid_for(8ll * d.num_nodes, 128, kSMs * 32);
      auto gather = c.mode == MODE_ADJOINT ? k_gather_rows<true> : k_gather_rows<false>;
      launch_gather(gather, rows + nodes, 128, st, d.num_nodes, rows, d.brow_ptr.ptr, d.diag.ptr, d.btr.ptr, d.bptr.ptr,
                    d.blist.ptr, d.nptr.ptr, d.nlist.ptr, reinterpret_cast<const long long*>(m.ebuf.ptr), s->A.ptr,
                    s->R.ptr, dm ? m.dbuf.ptr : nullptr, s->dMdu.ptr);
      break;
    }
    const int acc = (c.overwrite && e0 == 0) ? 0 : 1;
    const bool chunked = chunk < E;
    if (scatter) {
      launch_gather(k_gather_nodes, grid_for(4ll * d.num_nodes, 256), 256, st, d.num_nodes, d.nptr.ptr, d.nlist.ptr,
                    m.ebuf.ptr, a.estride, s->R.ptr, acc, e0, e1);
      if (c.jacobian) {
        const int noff = d.nnzb - d.num_nodes;
        const int* lists[2] = {d.offd.ptr, d.diag.ptr};
        const int counts[2] = {noff, d.num_nodes};
        for (int q = 0; q < 2; ++q) {
          if (counts[q] <= 0) continue;
          const int g = grid_for(4ll * counts[q], 256);
          if (chunked) {
            if (c.mode == MODE_ADJOINT)
              k_gather_blocks_chunk<true><<<g, 256, 0, st>>>(counts[q], lists[q], d.bptr.ptr, d.blist.ptr, m.ebuf.ptr,
                                                             a.estride, s->A.ptr, acc, e0, e1);
            else
              k_gather_blocks_chunk<false><<<g, 256, 0, st>>>(counts[q], lists[q], d.bptr.ptr, d.blist.ptr,
                                                              m.ebuf.ptr, a.estride, s->A.ptr, acc, e0, e1);
          } else if (c.mode == MODE_ADJOINT) {
            k_gather_blocks<true><<<g, 256, 0, st>>>(counts[q], lists[q], d.bptr.ptr, d.blist.ptr, m.ebuf.ptr,
                                                     a.estride, s->A.ptr, acc);
          } else {
            k_gather_blocks<false><<<g, 256, 0, st>>>(counts[q], lists[q], d.bptr.ptr, d.blist.ptr, m.ebuf.ptr,
                                                      a.estride, s->A.ptr, acc);
          }
          GOAL_CHECK_LAUNCH();
        }
      }
    }
    if (c.jacobian && c.qoi != QOI_NONE && s) {
      k_gather_nodes<<<grid_for(4ll * d.num_nodes, 256), 256, 0, st>>>(d.num_nodes, d.nptr.ptr, d.nlist.ptr,
                                                                          m.dbuf.ptr, 16, s->dMdu.ptr, acc, e0, e1);
      GOAL_CHECK_LAUNCH();
    }
  }
  if (timed) GOAL_CUDA(cudaEventRecord(g_phase.ev[2], st));
  if (c.qoi == QOI_AVG_DISP) {
    const int nb = reduction_blocks(m, E);
    k_sum<<<nb, 256, 0, st>>>(m.qoi_elem.ptr, E, m.red.ptr, m.ticket.ptr, &m.results.v->sum);
    GOAL_CHECK_LAUNCH();
  }
  GOAL_CUDA(cudaStreamSynchronize(st));
  double q = 0.0;
  if (c.qoi == QOI_AVG_DISP) q = m.results.v->sum;
  else if (c.qoi == QOI_KS_VM) q = ks_max + (1.0 / c.rho) * std::log(ks_scale);
  if (timed) {
    float e = 0.0f, g = 0.0f;
    GOAL_CUDA(cudaEventElapsedTime(&e, g_phase.ev[0], g_phase.ev[1]));
    GOAL_CUDA(cudaEventElapsedTime(&g, g_phase.ev[1], g_phase.ev[2]));
    g_phase.elem_ms += e;
    g_phase.gather_ms += g;
    g_phase.count += 1;
  }
  GOAL_REQUIRE(!m.results.v->return_map, GOAL_ERR_RETURN_MAP, "J2: return mapping failed");
  return q;
}

}  // namespace goal
