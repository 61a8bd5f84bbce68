// Stout link smearing and its force Jacobian on the device (FP64).
//
// Reference: Smear_APE::smear (src/lib/Smear/smear_APE.cpp:108-140),
// Projection_Stout_SU3::project / force_recursive / set_uw / set_fj
// (src/lib/Smear/projection_Stout_SU3.cpp:60-500), ForceSmear_APE::force_udiv /
// force_each / staple (src/lib/Smear/forceSmear_APE.cpp:95-260), driven by
// Director_Smear (src/lib/Smear/director_Smear.cpp) and
// AForce_F_Smeared_alt::mult_jacobian (src/lib_alt/Force/Fermion/
// aforce_F_Smeared_alt-tmpl.h:170-191).  In the reference these run on the
// host (the Accel build copies the links back for force_recursive); here each
// is one kernel over the 4*Nvol links, one thread per (site, mu).
//
// Links and forces use the lexical Field_G(Nvol, 4) layout
// ri + 2*(col + 3*row) + 18*(site + Nvol*mu).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/b200dwf.h"
#include "device_alloc.h"
#include "dwf_kernels.h"
#include "su3_lex.cuh"

namespace b200 {


// rho * sum_{nu != mu} (upper + lower) staples of U_mu(x)
__device__ __forceinline__ M3 staple_sum(const PlanarField& u, const LexHop& h, int x, int mu, double rho) {
  M3 c = zero3();
  const int um = h.up(mu);
#pragma unroll 1
  for (int k = 1; k < 4; ++k) {
    const int nu = (mu + k) & 3;
    const int un = h.up(nu), dn = h.dn(nu);
    // U_nu(x) U_mu(x+nu) U_nu(x+mu)^+
    mul3<false, true, true>(c, mul_nn(u.load(x, nu), u.load(x + un, mu)), u.load(x + um, nu));
    // U_nu(x-nu)^+ U_mu(x-nu) U_nu(x-nu+mu)
    mul3<false, false, true>(c, mul_dn(u.load(x + dn, nu), u.load(x + dn, mu)), u.load(x + dn + um, nu));
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) c.m[k] = rho * c.m[k];
  return c;
}

// ---------------------------------------------------------------------------
// exp(iQ) of a traceless Hermitian 3x3 matrix Q by the Cayley-Hamilton
// theorem, after C. Morningstar and M. Peardon, "Analytic smearing of SU(3)
// link variables in lattice QCD", Phys. Rev. D 69, 054501 (2004), sec. III:
//   exp(iQ) = f0 + f1 Q + f2 Q^2,
// the f_j being functions of the two invariants c0 = det Q = tr(Q^3)/3 and
// c1 = tr(Q^2)/2 only (through the eigenvalue parameters u and w).  The stout
// force needs their derivatives, B1 = sum_j (df_j/dc1) Q^j and
// B2 = sum_j (df_j/dc0) Q^j.  The closed forms are evaluated at |c0| (where
// they are best conditioned) and carried to c0 < 0 by the paper's symmetry
// f_j(-c0) = (-1)^j conj f_j(c0), whose derivative gives
// d f_j/dc1 (-c0) = (-1)^j conj(...) and d f_j/dc0 (-c0) = (-1)^(j+1) conj(...).
// ---------------------------------------------------------------------------

// (cos w - sin(w)/w) / w^2 = d/dw (sin(w)/w) / w, from w, sin w and cos w.
// For small w, where the closed form cancels, its Taylor series
//   sum_m (-1)^(m+1) (2m+2) w^(2m) / (2m+3)!
// is summed term by term (each term from the previous one).
__device__ double dsinc_w(double w, double sinw, double cosw) {
  if (w >= 0.5) return (cosw - sinw / w) / (w * w);
  const double w2 = w * w;
  double term = -1.0 / 3.0, sum = 0.0;
  for (int m = 1; m < 12; ++m) {
    sum += term;
    term *= -w2 * (2 * m + 2) / ((double)(2 * m) * (2 * m + 2) * (2 * m + 3));
  }
  return sum + term;
}

struct ExpCoef {
  Cx f[3];     // exp(iQ) = f0 + f1 Q + f2 Q^2
  Cx d1[3];    // d f_j / d c1
  Cx d0[3];    // d f_j / d c0
};

__device__ __forceinline__ Cx expi(double a) {
  Cx e;
  sincos(a, &e.i, &e.r);
  return e;
}
__device__ __forceinline__ Cx imul(double s, Cx a) { return cx(-s * a.i, s * a.r); }   // i s a

// kDeriv: also the derivatives (the force's B1, B2)
template <bool kDeriv>
__device__ ExpCoef expi_coef(double c0, double c1) {
  const bool flip = c0 < 0.0;
  const double a0 = fabs(c0);
  const double s3 = sqrt(c1 / 3.0);
  const double theta = acos(fmin(1.0, a0 / (2.0 * s3 * s3 * s3)));
  double st, ct, sw, cw;
  sincos(theta / 3.0, &st, &ct);
  const double u = s3 * ct;
  const double w = sqrt(c1) * st;
  const double uu = u * u, ww = w * w;
  sincos(w, &sw, &cw);
  const double ds = kDeriv ? dsinc_w(w, sw, cw) : 0.0;
  sw = (w == 0.0) ? 1.0 : sw / w;            // sin(w)/w
  const Cx m1 = expi(-u);                    // e^{-iu}
  const Cx p2 = conj(m1) * conj(m1);         // e^{2iu}
  const double den = 9.0 * uu - ww;
  ExpCoef r;
  // h_j / (9u^2 - w^2), paper eqs. (30)-(33)
  r.f[0] = (1.0 / den) * ((uu - ww) * p2 + m1 * cx(8.0 * uu * cw, 2.0 * u * (3.0 * uu + ww) * sw));
  r.f[1] = (1.0 / den) * ((2.0 * u) * p2 - m1 * cx(2.0 * u * cw, -(3.0 * uu - ww) * sw));
  r.f[2] = (1.0 / den) * (p2 - m1 * cx(cw, 3.0 * u * sw));
  if (kDeriv) {
    // the paper's r_j^(1), r_j^(2) (eqs. 58-60), written out per component
    Cx ra[3], rb[3];
    ra[0] = 2.0 * (cx(u, uu - ww) * p2) +
            2.0 * (m1 * cx(8.0 * u * cw + u * (3.0 * uu + ww) * sw,
                           -4.0 * uu * cw + (9.0 * uu + ww) * sw));
    ra[1] = 2.0 * (cx(1.0, 2.0 * u) * p2) +
            m1 * cx(-2.0 * cw + (3.0 * uu - ww) * sw, 2.0 * u * cw + 6.0 * u * sw);
    ra[2] = imul(2.0, p2) + m1 * cx(-3.0 * u * sw, cw - 3.0 * sw);
    rb[0] = -2.0 * p2 + m1 * cx(-8.0 * uu * sw, 2.0 * u * (cw + sw + 3.0 * uu * ds));
    rb[1] = m1 * cx(2.0 * u * sw, -(cw + sw - 3.0 * uu * ds));
    rb[2] = m1 * cx(sw, -3.0 * u * ds);
    const double inv = 1.0 / (2.0 * den * den);
    for (int j = 0; j < 3; ++j) {
      r.d1[j] = inv * ((2.0 * u) * ra[j] + (3.0 * uu - ww) * rb[j] - (30.0 * uu + 2.0 * ww) * r.f[j]);
      r.d0[j] = inv * (ra[j] - (3.0 * u) * rb[j] - (24.0 * u) * r.f[j]);
    }
  }
  if (flip) {
    for (int j = 0; j < 3; ++j) {
      const double sj = (j & 1) ? -1.0 : 1.0;
      r.f[j] = sj * conj(r.f[j]);
      if (kDeriv) {
        r.d1[j] = sj * conj(r.d1[j]);
        r.d0[j] = -sj * conj(r.d0[j]);
      }
    }
  }
  return r;
}

// a0 + a1 Q + a2 Q^2
__device__ __forceinline__ M3 qpoly(const Cx* a, const M3& Q, const M3& Q2) {
  M3 e;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const Cx id = (k % 4 == 0) ? a[0] : cx(0.0, 0.0);
    e.m[k] = id + a[1] * Q.m[k] + a[2] * Q2.m[k];
  }
  return e;
}

// tr(A B)
__device__ __forceinline__ Cx tr_mul(const M3& a, const M3& b) {
  Cx t = cx(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) t = t + a.m[3 * i + j] * b.m[3 * j + i];
  return t;
}

// The stout generator of one link: Q = -i TA(C U^+) (Hermitian, traceless),
// its square, and the invariants c0, c1.
struct StoutQ {
  M3 Q, Q2;
  double c0, c1;
};

__device__ __forceinline__ StoutQ stout_q(const M3& C, const M3& U) {
  StoutQ q;
  M3 a = mul_nd(C, U);
  at3(a);                                    // a = i Q
#pragma unroll
  for (int k = 0; k < 9; ++k) q.Q.m[k] = cx(a.m[k].i, -a.m[k].r);
  q.Q2 = mul_nn(q.Q, q.Q);
  q.c1 = 0.5 * (q.Q2.m[0].r + q.Q2.m[4].r + q.Q2.m[8].r);
  q.c0 = tr_mul(q.Q, q.Q2).r / 3.0;
  return q;
}

// The reference treats a link whose generator is negligible as unsmeared:
// exp(iQ) = 1 and no Lambda term in the force, when |iQ|^2 = tr(Q^2) = 2 c1
// is at most 1e-10 (Projection_Stout_SU3::force_recursive / project,
// src/lib/Smear/projection_Stout_SU3.cpp); the same cut keeps results equal
// on (near-)cold links.
__device__ __forceinline__ bool stout_negligible(const StoutQ& q) { return 2.0 * q.c1 <= 1.0e-10; }

struct StoutParams {
  PlanarField u;          // links of this level (input of the smearing step)
  PlanarField out;        // smeared links, planar (p null: not wanted)
  double* out_lex;        // smeared links, lexical (null: not wanted)
  PlanarField sig;        // force w.r.t. the smeared links in, w.r.t. u out
  const double* sig_in;   // the force arrives here in the lexical layout (null: in sig)
  double* sig_out;        // the finished force goes here in the lexical layout (null: to sig)
  PlanarField itheta;     // per-link i Theta (recursive -> force_each)
  double rho;
  LexGeom g;
};

// The kernels below run one thread per link, a block on the four directions
// (one a warp) of 32 consecutive sites, so that the directions find each
// other's links in L1 and L2, and read neighbours from planar copies
// (su3_lex.cuh).  They are bound by the FP64 pipe (12 products of 3x3
// matrices a link for the staples, 30 in force_each; 45 % busy) and, at the 8
// to 12 warps an SM that their registers leave, by the latency of the loads;
// at 4 resident blocks they spill and run 1.1-1.7x slower.  Two levels and the
// Jacobian at 24^3x48: 10.8 ms from lexical loads with 64-bit index divisions,
// 5.7 ms from the planar copies.

// U' = exp(iQ) U
__global__ void __launch_bounds__(128, 3) stout_smear_kernel(StoutParams p) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const int vol = (int)p.g.vol;
  const int x = blockIdx.x * 32 + lane;
  M3 o = zero3();
  if (x < vol) {
    const LexHop h(p.g, x);
    const M3 U = p.u.load(x, mu);
    const StoutQ q = stout_q(staple_sum(p.u, h, x, mu, p.rho), U);
    if (stout_negligible(q)) {
      o = U;
    } else {
      const ExpCoef k = expi_coef<false>(q.c0, q.c1);
      o = mul_nn(qpoly(k.f, q.Q, q.Q2), U);
    }
    if (p.out.p) p.out.store(x, mu, o);
  }
  if (p.out_lex) {
    const size_t base = (size_t)vol * mu;
    store3_warp(p.out_lex, base + blockIdx.x * 32, base + vol, buf[mu], lane, o);
  }
}

// One backward step of the stout chain for link (x, mu): with M = U Sigma'
//   Gamma  = tr(M B1) Q + tr(M B2) Q^2 + f1 M + f2 (Q M + M Q)
//   iLambda = TA(i Gamma),   iTheta = iLambda U   (kept for force_each)
//   Sigma  = Sigma' exp(iQ) + C^+ iLambda
// (paper eqs. 69-75); the staple derivative terms follow in force_each.
// Sigma' and Sigma are the thread's own link only, so sig is updated in place.
__global__ void __launch_bounds__(128, 2) stout_recursive_kernel(StoutParams p) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const int vol = (int)p.g.vol;
  const int x = blockIdx.x * 32 + lane;
  M3 Sp;
  if (p.sig_in) {
    const size_t base = (size_t)vol * mu;
    Sp = load3_warp(p.sig_in, base + blockIdx.x * 32, base + vol, buf[mu], lane);
  }
  if (x >= vol) return;
  if (!p.sig_in) Sp = p.sig.load(x, mu);
  const LexHop h(p.g, x);
  const M3 U = p.u.load(x, mu);
  const M3 C = staple_sum(p.u, h, x, mu, p.rho);
  const StoutQ q = stout_q(C, U);
  M3 e, il;
  if (stout_negligible(q)) {
    e = unit3();
    il = zero3();
  } else {
    const ExpCoef k = expi_coef<true>(q.c0, q.c1);
    e = qpoly(k.f, q.Q, q.Q2);
    const M3 M = mul_nn(U, Sp);
    const Cx g1 = tr_mul(M, qpoly(k.d1, q.Q, q.Q2));
    const Cx g0 = tr_mul(M, qpoly(k.d0, q.Q, q.Q2));
    M3 QM = mul_nn(q.Q, M);
    mul3<false, false, true>(QM, M, q.Q);
#pragma unroll
    for (int n = 0; n < 9; ++n) {
      Cx gam = g1 * q.Q.m[n];
      cmac(gam, g0, q.Q2.m[n]);
      cmac(gam, k.f[1], M.m[n]);
      cmac(gam, k.f[2], QM.m[n]);
      il.m[n] = imul(1.0, gam);
    }
    at3(il);
  }
  p.itheta.store(x, mu, mul_nn(il, U));
  M3 sig = mul_nn(Sp, e);
  mul3<true, false, true>(sig, C, il);
  p.sig.store(x, mu, sig);
}

// ForceSmear_APE::force_each summed over nu != mu, times rho, added to sig.
// Six products a plane and side, two of which share their outer factor:
//   above x:  V_nu(x+mu) [V_mu(x+nu)^+ iT_nu(x)^+ + iT_mu(x+nu)^+ V_nu(x)^+] + iT_nu(x+mu) V_mu(x+nu)^+ V_nu(x)^+
//   below:    V_nu(y+mu)^+ [iT_mu(y)^+ V_nu(y) + V_mu(y)^+ iT_nu(y)] + iT_nu(y+mu)^+ V_mu(y)^+ V_nu(y),  y = x - nu
__global__ void __launch_bounds__(128, 2) stout_force_each_kernel(StoutParams p) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const int vol = (int)p.g.vol;
  const int x = blockIdx.x * 32 + lane;
  const PlanarField& U = p.u;
  const PlanarField& T = p.itheta;
  M3 acc = zero3();
  if (x < vol) {
    const LexHop h(p.g, x);
    const int um = h.up(mu);
#pragma unroll 1
    for (int k = 1; k < 4; ++k) {
      const int nu = (mu + k) & 3;
      const int un = h.up(nu);
      {
        const M3 vm = U.load(x + un, mu), vn = U.load(x, nu);
        M3 s = mul_dd(vm, T.load(x, nu));
        mul3<true, true, true>(s, T.load(x + un, mu), vn);
        mul3<false, false, true>(acc, U.load(x + um, nu), s);
        mul3<false, true, true>(acc, mul_nd(T.load(x + um, nu), vm), vn);
      }
      {
        const int y = x + h.dn(nu);
        const M3 vm = U.load(y, mu), vn = U.load(y, nu);
        M3 s = mul_dn(T.load(y, mu), vn);
        mul3<true, false, true>(s, vm, T.load(y, nu));
        mul3<true, false, true>(acc, U.load(y + um, nu), s);
        mul3<false, false, true>(acc, mul_dd(T.load(y + um, nu), vm), vn);
      }
    }
    M3 out = p.sig.load(x, mu);
    add_to(out, acc, p.rho);
    acc = out;
    if (!p.sig_out) p.sig.store(x, mu, acc);
  }
  if (p.sig_out) {
    const size_t base = (size_t)vol * mu;
    store3_warp(p.sig_out, base + blockIdx.x * 32, base + vol, buf[mu], lane, acc);
  }
}

// planar -> lexical Field_G
__global__ void __launch_bounds__(128) planar_to_links_kernel(double* out, PlanarField in) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  M3 a = zero3();
  if (x < (int)in.vol) a = in.load(x, mu);
  const size_t base = (size_t)in.vol * mu;
  store3_warp(out, base + blockIdx.x * 32, base + in.vol, buf[mu], lane, a);
}

// AForce_F<ACCEL>::mult_generator (src/lib_alt_Accel/Force/Fermion/aforce_F.cpp:62-75):
// F_mu(x) <- -2 at(U_mu(x) F_mu(x))
__global__ void __launch_bounds__(128) mult_generator_kernel(double* f, const double* u, size_t nlink) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t first = blockIdx.x * (size_t)128 + warp * 32;
  const M3 a = load3_warp(u, first, nlink, buf[warp], lane);
  const M3 b = load3_warp(f, first, nlink, buf[warp], lane);
  M3 m = mul_nn(a, b);
  at3(m);
#pragma unroll
  for (int k = 0; k < 9; ++k) m.m[k] = -2.0 * m.m[k];
  store3_warp(f, first, nlink, buf[warp], lane, m);
}

}  // namespace b200

// ------------------------------------------------------------ smearing plan
using namespace b200;

// Levels 0 .. nsmear-1 are kept planar (what the next level and the Jacobian
// read), the top level in the lexical layout (what callers read).  Another
// level asked for by b200_smear_config gets a lexical copy then, refreshed by
// every later set_config, so the pointer handed out stays that level's.
struct b200_smear {
  LexGeom g;
  double rho;
  int nsmear;
  double2* block = nullptr;        // one allocation: the top level, then the arrays below
  double2* planar = nullptr;       // nsmear planar levels
  std::vector<double*> lex;        // lexical copies per level (top: in block)
  double2* itheta = nullptr;
  double2* sig = nullptr;
  std::mutex mu;                   // guards the lexical copies made on request
  int device = 0;                  // the device that the levels are on
  bool have_config = false;
};

namespace b200 {
void set_last_error(int code, const char* fmt, ...);
}

#define B200_SMEAR_CHECK(call)                                                      \
  do {                                                                              \
    cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess) {                                                        \
      set_last_error(B200_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));          \
      return B200_ECUDA;                                                            \
    }                                                                               \
  } while (0)

// Queues work on a stream of its own and waits for it, so that what is in
// progress on the caller's streams is not touched (the levels are complete when
// set_config returns).
template <class F>
static cudaError_t on_own_stream(F queue) {
  cudaStream_t st = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  e = queue(st);
  const cudaError_t es = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return e != cudaSuccess ? e : es;
}

static size_t nreal_cfg(const b200_smear* sm) { return 18 * 4 * sm->g.vol; }

extern "C" {

int b200_smear_create(b200_smear_t** out, const int lattice[4], double rho, int nsmear) {
  if (!out || !lattice || nsmear < 0 || nsmear > 16) {
    set_last_error(B200_EINVAL, "smear_create: invalid argument");
    return B200_EINVAL;
  }
  b200_smear* sm = new b200_smear();
  for (int mu = 0; mu < 4; ++mu) {
    if (lattice[mu] < 1) { delete sm; set_last_error(B200_EINVAL, "invalid lattice"); return B200_EINVAL; }
    sm->g.n[mu] = lattice[mu];
  }
  sm->g.vol = (size_t)lattice[0] * lattice[1] * lattice[2] * lattice[3];
  sm->rho = rho;
  sm->nsmear = nsmear;
  sm->lex.assign(nsmear + 1, nullptr);
  cudaGetDevice(&sm->device);
  const size_t n = nreal_cfg(sm) / 2;      // double2 of one field
  const size_t fields = nsmear > 0 ? nsmear + 3 : 1;
  if (sm->g.vol > 0x7fffffffu || device_malloc(&sm->block, fields * n * sizeof(double2)) != cudaSuccess) {
    sm->block = nullptr;
    b200_smear_destroy(sm);
    set_last_error(B200_ENOMEM, "smear_create: device allocation failed");
    return B200_ENOMEM;
  }
  sm->lex[nsmear] = reinterpret_cast<double*>(sm->block);
  if (nsmear > 0) {
    sm->itheta = sm->block + n;
    sm->sig = sm->block + 2 * n;
    sm->planar = sm->block + 3 * n;
  }
  *out = sm;
  return 0;
}

int b200_smear_destroy(b200_smear_t* sm) {
  if (!sm) return 0;
  for (int i = 0; i < sm->nsmear; ++i) cudaFree(sm->lex[i]);
  cudaFree(sm->block);
  gauge_scratch_trim();
  delete sm;
  return 0;
}

static PlanarField planar_level(const b200_smear* sm, int level) {
  return PlanarField{sm->planar + (size_t)level * 36 * sm->g.vol, (unsigned)sm->g.vol};
}

// The planar copy reads the caller's links 16 bytes at a time and from this
// device.  What it cannot read so (a view at an odd number of doubles, memory
// of another device, page-locked host memory) is copied first, as host links
// are.
static bool readable_in_place(const double* u) {
  if (reinterpret_cast<uintptr_t>(u) & 15u) return false;
  int dev = 0;
  cudaPointerAttributes a;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&a, u) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice && a.device == dev;
}

static unsigned link_grid(const b200_smear* sm) { return (unsigned)((sm->g.vol + 31) / 32); }

int b200_smear_set_config(b200_smear_t* sm, const double* u, int on_device, void* stream) {
  if (!sm || !u) { set_last_error(B200_EINVAL, "smear_set_config: invalid argument"); return B200_EINVAL; }
  cudaStream_t st = (cudaStream_t)stream;
  const size_t bytes = nreal_cfg(sm) * sizeof(double);
  std::lock_guard<std::mutex> lock(sm->mu);
  double* top = sm->lex[sm->nsmear];
  const double* thin = u;
  if (sm->nsmear == 0 || !on_device || !readable_in_place(u)) {
    // these links pass through the top level's buffer, which the last level
    // overwrites once the planar copy has been made
    B200_SMEAR_CHECK(cudaMemcpyAsync(top, u, bytes, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, st));
    thin = top;
  }
  if (sm->nsmear > 0) B200_SMEAR_CHECK(launch_links_to_planar(planar_level(sm, 0).p, thin, sm->g.vol, st));
  for (int i = 0; i < sm->nsmear; ++i) {
    StoutParams p{};
    p.u = planar_level(sm, i);
    if (i + 1 < sm->nsmear) p.out = planar_level(sm, i + 1);
    p.out_lex = sm->lex[i + 1];
    p.rho = sm->rho;
    p.g = sm->g;
    stout_smear_kernel<<<link_grid(sm), 128, 0, st>>>(p);
    B200_SMEAR_CHECK(cudaGetLastError());
  }
  if (sm->nsmear > 0 && sm->lex[0]) {
    planar_to_links_kernel<<<link_grid(sm), 128, 0, st>>>(sm->lex[0], planar_level(sm, 0));
    B200_SMEAR_CHECK(cudaGetLastError());
  }
  B200_SMEAR_CHECK(cudaStreamSynchronize(st));
  sm->have_config = true;
  return 0;
}

// The plan's device, whichever the calling thread has current, and a capture
// mode in which allocations do not disturb a capture in progress.
struct OnPlanDevice {
  int plan, current;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  explicit OnPlanDevice(const b200_smear* sm) : plan(sm->device), current(sm->device) {
    cudaGetDevice(&current);
    if (current != plan) cudaSetDevice(plan);
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  ~OnPlanDevice() {
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (current != plan) cudaSetDevice(current);
  }
};

// planar level -> lexical `out`
static cudaError_t level_to_lex(const b200_smear* sm, int level, double* out, cudaStream_t st) {
  planar_to_links_kernel<<<link_grid(sm), 128, 0, st>>>(out, planar_level(sm, level));
  return cudaGetLastError();
}

static int smear_fail(cudaError_t e, const char* what) {
  set_last_error(e == cudaErrorMemoryAllocation ? B200_ENOMEM : B200_ECUDA, "%s: %s", what, cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? B200_ENOMEM : B200_ECUDA;
}

// The lexical copy of a level below the top that stays with the plan.
static int make_lex(b200_smear* sm, int level) {
  OnPlanDevice on(sm);
  double* buf = nullptr;
  cudaError_t e = device_malloc(&buf, nreal_cfg(sm) * sizeof(double));
  if (e == cudaSuccess) e = on_own_stream([&](cudaStream_t st) { return level_to_lex(sm, level, buf, st); });
  if (e != cudaSuccess) {
    cudaFree(buf);
    return smear_fail(e, "smear_config");
  }
  sm->lex[level] = buf;
  return 0;
}

const double* b200_smear_config(b200_smear_t* sm, int level) {
  if (!sm || level < 0 || level > sm->nsmear || !sm->have_config) return nullptr;
  std::lock_guard<std::mutex> lock(sm->mu);
  if (!sm->lex[level] && make_lex(sm, level) != 0) return nullptr;
  return sm->lex[level];
}

// A level that has no lexical copy goes through one that is given back, or,
// where there is no room for it, is put in order on the host: the plan keeps no
// memory for this call, and later set_config calls do no more work after it.
static int planar_to_host(b200_smear* sm, int level, double* host_out) {
  OnPlanDevice on(sm);
  const size_t bytes = nreal_cfg(sm) * sizeof(double), vol = sm->g.vol;
  double* lex = nullptr;
  cudaError_t e = device_malloc(&lex, bytes);
  if (e == cudaSuccess) {
    e = on_own_stream([&](cudaStream_t st) {
      const cudaError_t ek = level_to_lex(sm, level, lex, st);
      return ek != cudaSuccess ? ek : cudaMemcpyAsync(host_out, lex, bytes, cudaMemcpyDeviceToHost, st);
    });
    cudaFree(lex);
    return e == cudaSuccess ? 0 : smear_fail(e, "smear_get_config");
  }
  if (e != cudaErrorMemoryAllocation) return smear_fail(e, "smear_get_config");
  double2* planar = new (std::nothrow) double2[36 * vol];
  if (!planar) return smear_fail(cudaErrorMemoryAllocation, "smear_get_config");
  e = on_own_stream([&](cudaStream_t st) {
    return cudaMemcpyAsync(planar, planar_level(sm, level).p, bytes, cudaMemcpyDeviceToHost, st);
  });
  if (e == cudaSuccess)
    for (size_t mu = 0; mu < 4; ++mu)
      for (size_t site = 0; site < vol; ++site)
        for (size_t k = 0; k < 9; ++k)
          memcpy(host_out + 18 * (site + vol * mu) + 2 * k, planar + (9 * mu + k) * vol + site, sizeof(double2));
  delete[] planar;
  return e == cudaSuccess ? 0 : smear_fail(e, "smear_get_config");
}

int b200_smear_get_config(b200_smear_t* sm, int level, double* host_out, void* stream) {
  if (!sm || !host_out || level < 0 || level > sm->nsmear || !sm->have_config) {
    set_last_error(B200_EINVAL, "smear_get_config: invalid level or no config");
    return B200_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lock(sm->mu);
  if (!sm->lex[level]) return planar_to_host(sm, level, host_out);
  B200_SMEAR_CHECK(cudaMemcpyAsync(host_out, sm->lex[level], nreal_cfg(sm) * sizeof(double), cudaMemcpyDeviceToHost, st));
  B200_SMEAR_CHECK(cudaStreamSynchronize(st));
  return 0;
}

int b200_smear_jacobian(b200_smear_t* sm, double* sigma, void* stream) {
  if (!sm || !sigma || !sm->have_config) {
    set_last_error(B200_EINVAL, "smear_jacobian: invalid argument or no config");
    return B200_EINVAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned vol = (unsigned)sm->g.vol;
  for (int i = sm->nsmear - 1; i >= 0; --i) {
    // Sigma_i = J_i^T Sigma_(i+1): recursion, then the staple derivatives
    StoutParams p{};
    p.u = planar_level(sm, i);
    p.sig = PlanarField{sm->sig, vol};
    p.itheta = PlanarField{sm->itheta, vol};
    if (i == sm->nsmear - 1) p.sig_in = sigma;
    if (i == 0) p.sig_out = sigma;
    p.rho = sm->rho;
    p.g = sm->g;
    stout_recursive_kernel<<<link_grid(sm), 128, 0, st>>>(p);
    B200_SMEAR_CHECK(cudaGetLastError());
    stout_force_each_kernel<<<link_grid(sm), 128, 0, st>>>(p);
    B200_SMEAR_CHECK(cudaGetLastError());
  }
  return 0;
}

int b200_force_mult_generator(const int lattice[4], double* force, const double* u, void* stream) {
  if (!lattice || !force || !u) { set_last_error(B200_EINVAL, "mult_generator: invalid argument"); return B200_EINVAL; }
  const size_t nlink = 4 * (size_t)lattice[0] * lattice[1] * lattice[2] * lattice[3];
  mult_generator_kernel<<<(int)((nlink + 127) / 128), 128, 0, (cudaStream_t)stream>>>(force, u, nlink);
  B200_SMEAR_CHECK(cudaGetLastError());
  return 0;
}

}  // extern "C"
