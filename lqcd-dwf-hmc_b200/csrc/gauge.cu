// Gauge-field side of the HMC step on the device (FP64): the Iwasaki /
// rectangle gauge force and action, the link update exp(alpha iP) U and the
// momentum update and kinetic energy.
//
// Reference (the corelib runs these on the host in every build):
//   Force_G_Rectangle::force_core  src/lib/Force/Gauge/force_G_Rectangle.cpp:84-220
//   Action_G_Rectangle::calcH      src/lib/Action/Gauge/action_G_Rectangle.cpp:97-200
//   Integrator_UpdateU::evolve     src/lib/HMC/integrator_UpdateU.cpp:79-86
//     -> mult_exp_Field_G (src/lib/Field/Imp/field_G_imp.cpp:496-522)
//     -> SU_N::mat_exp + Mat_SU_N::reunit_SU3 (src/lib/Tools/mat_SU_N.h:637-657,
//        src/lib/Tools/mat_SU_N.cpp:18-88)
//   Integrator_UpdateP::evolve     src/lib/HMC/integrator_UpdateP.cpp:44-66
//   HMC_General::calcH_P           src/lib/HMC/hmc_General.cpp:340-346
//
// One thread per link (site, mu) for the force and the update, one per site
// for the action; every staple and rectangle is formed from the links it
// touches (no shifted copies of the field are made).  The force reads the
// links from a planar copy, own links go through shared memory (su3_lex.cuh).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "../../include/b200dwf.h"
#include "device_alloc.h"
#include "dwf_kernels.h"
#include "su3_lex.cuh"

namespace b200 {

void set_last_error(int code, const char* fmt, ...);

namespace {

struct GaugeGeom {
  LexGeom g;
  __device__ M3 U(const double* u, size_t site, int mu) const { return load3(u, site + g.vol * mu); }
  __device__ size_t sh(size_t site, int mu, int d) const { return g.shift(site, mu, d); }
};

__device__ __forceinline__ void scale3(M3& a, double s) {
#pragma unroll
  for (int k = 0; k < 9; ++k) a.m[k] = s * a.m[k];
}

// Sum over nu != mu of the staples of U_mu(x) in the rectangle action:
// c_plaq (upper + lower plaquette staples) + c_rect (the six 2x1 rectangles
// through U_mu(x)), each a product S with U_mu(x) S^+ a closed loop at x.
// The eight products of a plane share their factors: with the 2x1 ends
//   A(y; a, b) = U_a(y) U_b(y+a) U_a(y+b)^+   (upper staple of U_b(y) along a)
//   B(y; a, b) = U_a(y-a)^+ U_b(y-a) U_a(y-a+b)   (lower staple)
// the sum is
//   U_nu(x) { [cp V + cr A(x+nu; nu,mu)] U_nu(x+mu)^+ + cr V A(x+mu; mu,nu)^+ } + cr B(x; mu,nu) V U_nu(x+mu)^+
// with V = U_mu(x+nu), and the mirror image below x: 22 products of 3x3
// matrices a plane instead of 28.
template <class F>
__device__ __forceinline__ M3 rect_staples(const F& U, const LexHop& h, int x, int mu, double cp, double cr) {
  M3 f = zero3();
  const int um = h.up(mu), dm = h.dn(mu), um2 = h.up2(mu);
#pragma unroll 1
  for (int k = 1; k < 4; ++k) {
    const int nu = (mu + k) & 3;
    const int un = h.up(nu), dn = h.dn(nu);
    {
      const M3 v = U.load(x + un, mu);
      const M3 t = mul_nd(v, U.load(x + um, nu));                       // V U_nu(x+mu)^+
      if (cr != 0.0) {
        const M3 a1 = mul_nd(mul_nn(U.load(x + un, nu), U.load(x + h.up2(nu), mu)), U.load(x + um + un, nu));
        M3 y = mul_nd(a1, U.load(x + um, nu));
        const M3 a2 = mul_nd(mul_nn(U.load(x + um, mu), U.load(x + um2, nu)), U.load(x + um + un, mu));
        mul3<false, true, true>(y, v, a2);
        scale3(y, cr);
        add_to(y, t, cp);
        mul3<false, false, true>(f, U.load(x, nu), y);
        M3 b = mul_nn(mul_dn(U.load(x + dm, mu), U.load(x + dm, nu)), U.load(x + dm + un, mu));
        scale3(b, cr);
        mul3<false, false, true>(f, b, t);
      } else {
        add_to(f, mul_nn(U.load(x, nu), t), cp);
      }
    }
    {
      const M3 v = U.load(x + dn, mu);
      const M3 t = mul_nn(v, U.load(x + dn + um, nu));                  // V U_nu(x-nu+mu)
      if (cr != 0.0) {
        const int dn2 = h.dn2(nu);
        const M3 b1 = mul_nn(mul_dn(U.load(x + dn2, nu), U.load(x + dn2, mu)), U.load(x + dn2 + um, nu));
        M3 y = mul_nn(b1, U.load(x + dn + um, nu));
        const M3 a2 = mul_nd(mul_nn(U.load(x + dn + um, mu), U.load(x + dn + um2, nu)), U.load(x + um, mu));
        mul3<false, false, true>(y, v, a2);
        scale3(y, cr);
        add_to(y, t, cp);
        mul3<true, false, true>(f, U.load(x + dn, nu), y);
        M3 z = mul_nn(mul_dd(U.load(x + dm, mu), U.load(x + dm + dn, nu)), U.load(x + dm + dn, mu));
        scale3(z, cr);
        mul3<false, false, true>(f, z, t);
      } else {
        add_to(f, mul_dn(U.load(x + dn, nu), t), cp);
      }
    }
  }
  return f;
}

// One thread per link, a block on 128 consecutive sites of one direction
// (blockIdx.y; four directions of 32 sites in one block, as in the stout
// kernels, ran 1.15x slower: their 66 loads crowd each other out of L1).  Bound by
// the latency of those loads at 8 warps an SM and by the FP64 pipe (66
// products of 3x3 matrices a link): the five or six matrices in flight need
// the registers of 2 resident blocks (at 3 they spill, 1.3x slower).  The
// whole molecular-dynamics step at 16^3x32 (this kernel, momentum and link
// update): 1096 us from lexical loads, 543 us from the planar copy.
template <class F>
__global__ void __launch_bounds__(128, 2) gauge_force_kernel(F u, double* force, LexGeom g, double beta, double cp,
                                                             double cr) {
  __shared__ double2 buf[4][kLinkBuf];
  const int mu = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int vol = (int)g.vol;
  const int x = blockIdx.x * 128 + threadIdx.x;
  M3 out = zero3();
  if (x < vol) {
    const LexHop h(g, x);
    const M3 f = rect_staples(u, h, x, mu, cp, cr);
    M3 w = mul_nd(u.load(x, mu), f);
    at3(w);
    add_to(out, w, -beta / 3.0);
  }
  const size_t base = (size_t)vol * mu;
  store3_warp(force, base + blockIdx.x * 128 + warp * 32, base + vol, buf[warp], lane, out);
}

// lexical Field_G -> planar copy
__global__ void __launch_bounds__(128) links_to_planar_kernel(PlanarField o, const double* u) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  const size_t base = (size_t)o.vol * mu;
  const M3 a = load3_warp(u, base + blockIdx.x * 32, base + o.vol, buf[mu], lane);
  if (x < (int)o.vol) o.store(x, mu, a);
}

__device__ __forceinline__ double retr_nd(const M3& a, const M3& b) {   // Re tr(a b^+)
  double t = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) t += a.m[k].r * b.m[k].r + a.m[k].i * b.m[k].i;
  return t;
}

// per-block partial sums of the plaquette and rectangle traces of calcH
__global__ void gauge_action_kernel(const double* u, LexGeom g, double* partial) {
  __shared__ double sp[256], sr[256];
  const size_t x = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  double pl = 0.0, re = 0.0;
  if (x < g.vol) {
    GaugeGeom G{g};
    for (int mu = 0; mu < 4; ++mu) {
      const M3 umu = G.U(u, x, mu);
      const size_t xpm = G.sh(x, mu, 1);
      for (int nu = mu + 1; nu < 4; ++nu) {
        const size_t xpn = G.sh(x, nu, 1);
        pl += retr_nd(umu, mul_nd(mul_nn(G.U(u, x, nu), G.U(u, xpn, mu)), G.U(u, xpm, nu)));
        const size_t xpmpn = G.sh(xpm, nu, 1);
        re += retr_nd(umu, mul_nd(mul_nd(mul_nn(mul_nn(G.U(u, x, nu), G.U(u, xpn, mu)), G.U(u, xpmpn, mu)),
                                         G.U(u, G.sh(xpm, mu, 1), nu)), G.U(u, xpm, mu)));
        re += retr_nd(umu, mul_nd(mul_nd(mul_nn(mul_nn(G.U(u, x, nu), G.U(u, xpn, nu)),
                                                G.U(u, G.sh(xpn, nu, 1), mu)), G.U(u, xpmpn, nu)),
                                  G.U(u, xpm, nu)));
      }
    }
  }
  sp[threadIdx.x] = pl;
  sr[threadIdx.x] = re;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) { sp[threadIdx.x] += sp[threadIdx.x + o]; sr[threadIdx.x] += sr[threadIdx.x + o]; }
    __syncthreads();
  }
  if (threadIdx.x == 0) { partial[2 * blockIdx.x] = sp[0]; partial[2 * blockIdx.x + 1] = sr[0]; }
}

// Back onto SU(3) after the link update, as Mat_SU_N::reunit_SU3 does
// (src/lib/Tools/mat_SU_N.cpp:18-88): Gram-Schmidt on the first two rows,
// then the third row completes a unit-determinant matrix.  With rows a, b:
//   a <- a / |a|;   b <- b - <a, b> a,  b <- b / |b|;   c = conj(a x b).
__device__ void reunit3(M3& m) {
  Cx* a = m.m;
  Cx* b = m.m + 3;
  Cx* c = m.m + 6;
  const double ia = 1.0 / sqrt(a[0].r * a[0].r + a[0].i * a[0].i + a[1].r * a[1].r + a[1].i * a[1].i +
                               a[2].r * a[2].r + a[2].i * a[2].i);
#pragma unroll
  for (int j = 0; j < 3; ++j) a[j] = ia * a[j];
  const Cx ab = conj(a[0]) * b[0] + conj(a[1]) * b[1] + conj(a[2]) * b[2];   // <a, b>
#pragma unroll
  for (int j = 0; j < 3; ++j) b[j] = b[j] - ab * a[j];
  const double ib = 1.0 / sqrt(b[0].r * b[0].r + b[0].i * b[0].i + b[1].r * b[1].r + b[1].i * b[1].i +
                               b[2].r * b[2].r + b[2].i * b[2].i);
#pragma unroll
  for (int j = 0; j < 3; ++j) b[j] = ib * b[j];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = (j + 1) % 3, l = (j + 2) % 3;
    c[j] = conj(a[k] * b[l] - a[l] * b[k]);
  }
}

// u <- reunit( (u + a iP (u + a/2 iP ( ... (u + a/n iP u) ...))) ), n = nprec
__global__ void __launch_bounds__(128) link_update_kernel(double* u, const double* ip, size_t nlink, double alpha,
                                                          int nprec) {
  __shared__ double2 buf[4][kLinkBuf];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t first = blockIdx.x * (size_t)128 + warp * 32;
  const M3 u0 = load3_warp(u, first, nlink, buf[warp], lane);
  const M3 iv = load3_warp(ip, first, nlink, buf[warp], lane);
  M3 t = u0;
  if (first + lane < nlink) {
    for (int k = 0; k < nprec; ++k) {
      const double f = alpha / (double)(nprec - k);
      const M3 p = mul_nn(iv, t);
      t = u0;
      add_to(t, p, f);
    }
    reunit3(t);
  }
  store3_warp(u, first, nlink, buf[warp], lane, t);
}

// y = a x + b y over link fields of n elements (b = 0: y = a x, y not read).
// HBM-bound: four independent 16-byte loads of each operand a thread keep
// enough bytes in flight (8-byte loads, one at a time, did not); T is double
// only for arrays that are not 16-byte aligned.
constexpr int kAxpyUnroll = 4;
__device__ __forceinline__ double axpby1(double a, double x, double b, double y) { return fma(a, x, b * y); }
__device__ __forceinline__ double2 axpby1(double a, double2 x, double b, double2 y) {
  return make_double2(fma(a, x.x, b * y.x), fma(a, x.y, b * y.y));
}
__device__ __forceinline__ double scale1(double a, double x) { return a * x; }
__device__ __forceinline__ double2 scale1(double a, double2 x) { return make_double2(a * x.x, a * x.y); }

template <typename T, bool kReadY>
__global__ void __launch_bounds__(256) axpby_links_kernel(T* y, const T* x, size_t n, double a, double b) {
  const size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += kAxpyUnroll * step) {
    T xv[kAxpyUnroll], yv[kAxpyUnroll];
#pragma unroll
    for (int k = 0; k < kAxpyUnroll; ++k) {
      const size_t j = i + k * step;
      if (j < n) {
        xv[k] = x[j];
        if (kReadY) yv[k] = y[j];
      }
    }
#pragma unroll
    for (int k = 0; k < kAxpyUnroll; ++k) {
      const size_t j = i + k * step;
      if (j < n) y[j] = kReadY ? axpby1(a, xv[k], b, yv[k]) : scale1(a, xv[k]);
    }
  }
}

template <typename T>
cudaError_t run_axpby_links(double* y, const double* x, size_t n, double a, double b, cudaStream_t st) {
  const size_t m = n * sizeof(double) / sizeof(T);           // n is a multiple of 18
  const size_t want = (m + 256 * kAxpyUnroll - 1) / (256 * kAxpyUnroll);
  const int nb = (int)(want < 148 * 8 ? want : 148 * 8);
  if (b == 0.0) axpby_links_kernel<T, false><<<nb, 256, 0, st>>>((T*)y, (const T*)x, m, a, b);
  else axpby_links_kernel<T, true><<<nb, 256, 0, st>>>((T*)y, (const T*)x, m, a, b);
  return cudaGetLastError();
}

cudaError_t launch_axpby_links(double* y, const double* x, size_t n, double a, double b, cudaStream_t st) {
  const bool wide = ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(x)) & 15u) == 0;
  return wide ? run_axpby_links<double2>(y, x, n, a, b, st) : run_axpby_links<double>(y, x, n, a, b, st);
}

// iP = i sum_a h_a lambda_a on every link (Langevin_Momentum::set_iP_SU3,
// src/lib/HMC/langevin_Momentum.cpp:150-210) from h = Field(8, Nvol, 4) of
// Gaussians, written into the Field_G layout entry by entry: the Gell-Mann
// matrices lambda_1..8 have at most two non-zero entries per position, and
// lambda_8's 1/sqrt(3) is passed in (s).  Diagonal: i (h_3 +- s h_8) and
// -2 i s h_8; off-diagonal (r, c) / (c, r): i h for the symmetric lambdas,
// +-h for the antisymmetric ones.
__global__ void momentum_from_gauss_kernel(const double* h, double* ip, size_t nlink, double s) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= nlink) return;
  double a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = h[8 * idx + k];
  double* o = ip + 18 * idx;
  const double d8 = __dmul_rn(s, a[7]);
  o[0] = 0.0;    o[1] = __dadd_rn(a[2], d8);               // (0,0)
  o[2] = a[1];   o[3] = a[0];                               // (0,1)
  o[4] = a[4];   o[5] = a[3];                               // (0,2)
  o[6] = -a[1];  o[7] = a[0];                               // (1,0)
  o[8] = 0.0;    o[9] = __dadd_rn(-a[2], d8);              // (1,1)
  o[10] = a[6];  o[11] = a[5];                              // (1,2)
  o[12] = -a[4]; o[13] = a[3];                              // (2,0)
  o[14] = -a[6]; o[15] = a[5];                              // (2,1)
  o[16] = 0.0;   o[17] = __dmul_rn(-2.0 * s, a[7]);        // (2,2)
}

__global__ void norm2_links_kernel(const double* x, size_t n, double* partial) {
  __shared__ double sh[256];
  double acc = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    acc = fma(x[i], x[i], acc);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

bool geom_ok(const int* L, LexGeom* g) {
  if (!L) return false;
  size_t v = 1;
  for (int mu = 0; mu < 4; ++mu) {
    if (L[mu] < 1) return false;
    g->n[mu] = L[mu];
    v *= (size_t)L[mu];
  }
  g->vol = v;
  return true;
}

int fail_code(int code, const char* msg) {
  set_last_error(code, "%s", msg);
  return code;
}

#define G_CHECK(call)                                                                  \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if (e_ != cudaSuccess) {                                                           \
      set_last_error(B200_ECUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,            \
                     cudaGetErrorString(e_));                                          \
      return B200_ECUDA;                                                               \
    }                                                                                  \
  } while (0)

// Scratch of the gauge force (a planar copy of the links): stream-ordered
// allocations from a pool of this library, one per device, so that calls on
// several streams and threads each have their own and a repeated call does
// not wait for the allocator.  At most kPoolKeep bytes stay with the pool
// between calls.  They go back to the device when a plan is destroyed, when
// b200_scratch_release asks for it and when an allocation of this library
// would fail without them.
constexpr int kMaxDevices = 64;
constexpr unsigned long long kPoolKeep = 2ull << 30;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};
bool g_pool_keeps[kMaxDevices] = {};      // the release threshold is kPoolKeep (else 0)

cudaError_t pool_keep(int dev, unsigned long long bytes) {
  g_pool_keeps[dev] = bytes != 0;
  return cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &bytes);
}

cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaMemPoolCreate(&g_pool[dev], &props) != cudaSuccess) {
      cudaGetLastError();
      g_pool[dev] = nullptr;
    }
  }
  if (g_pool[dev] && !g_pool_keeps[dev]) pool_keep(dev, kPoolKeep);
  return g_pool[dev];
}

}  // namespace

// What no call uses any more goes back at once; with the threshold at 0 (until
// the next gauge force) what a call still in flight frees goes back at the next
// synchronisation.
void gauge_scratch_trim() {
  // no stream is touched: safe while this thread captures one
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    for (int d = 0; d < kMaxDevices; ++d)
      if (g_pool[d]) {
        pool_keep(d, 0);
        cudaMemPoolTrimTo(g_pool[d], 0);
      }
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
}

cudaError_t device_malloc_bytes(void** p, size_t n) {
  const cudaError_t e = cudaMalloc(p, n);
  if (e != cudaErrorMemoryAllocation) return e;
  gauge_scratch_trim();
  const cudaError_t e2 = cudaMalloc(p, n);
  cudaGetLastError();      // the caller reports it; left set, the next launch would too
  return e2;
}

cudaError_t launch_links_to_planar(double2* out, const double* u, size_t vol, cudaStream_t st) {
  links_to_planar_kernel<<<(unsigned)((vol + 31) / 32), 128, 0, st>>>(PlanarField{out, (unsigned)vol}, u);
  return cudaGetLastError();
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_scratch_release(void) {
  gauge_scratch_trim();
  return 0;
}

int b200_gauge_force_rect(const int lattice[4], double beta, double c_plaq, double c_rect, double* force,
                          const double* u, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !force || !u) return fail_code(B200_EINVAL, "invalid argument");
  if (g.vol > 0x7fffffffu) return fail_code(B200_EINVAL, "lattice volume too large");
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid((unsigned)((g.vol + 127) / 128), 4);
  // The planar copy costs one pass over the links and makes the 66 link loads
  // of a thread whole lines.  Without room for it, and in a stream capture
  // (whose graph would own the copy and could be instantiated only once), the
  // links are read where they are, with the same arithmetic.
  double2* planar = nullptr;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
  cudaMemPool_t pool = capture == cudaStreamCaptureStatusNone ? scratch_pool() : nullptr;
  if (!pool || cudaMallocFromPoolAsync((void**)&planar, 4 * g.vol * 9 * sizeof(double2), pool, st) != cudaSuccess) {
    if (pool) cudaGetLastError();
    gauge_force_kernel<<<grid, 128, 0, st>>>(LexField{u, (unsigned)g.vol}, force, g, beta, c_plaq, c_rect);
    G_CHECK(cudaGetLastError());
    return 0;
  }
  cudaError_t e = launch_links_to_planar(planar, u, g.vol, st);
  if (e == cudaSuccess) {
    gauge_force_kernel<<<grid, 128, 0, st>>>(PlanarField{planar, (unsigned)g.vol}, force, g, beta, c_plaq, c_rect);
    e = cudaGetLastError();
  }
  const cudaError_t ef = cudaFreeAsync(planar, st);
  G_CHECK(e);
  G_CHECK(ef);
  return 0;
}

int b200_gauge_action_rect(const int lattice[4], double beta, double c_plaq, double c_rect, const double* u,
                           double* H, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !u || !H) return fail_code(B200_EINVAL, "invalid argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int nb = (int)((g.vol + 255) / 256);
  double* part = nullptr;
  G_CHECK(device_malloc(&part, sizeof(double) * 2 * nb));
  gauge_action_kernel<<<nb, 256, 0, st>>>(u, g, part);
  std::vector<double> h(2 * (size_t)nb);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), part, sizeof(double) * 2 * nb, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(part);
  G_CHECK(e);
  double plaqF = 0.0, rectF = 0.0;
  for (int b = 0; b < nb; ++b) { plaqF += h[2 * b]; rectF += h[2 * b + 1]; }
  const double V = (double)g.vol;
  *H = beta * (c_plaq * 6.0 * V - c_plaq * plaqF / 3.0 + c_rect * 12.0 * V - c_rect * rectF / 3.0);
  return 0;
}

int b200_link_update(const int lattice[4], double alpha, const double* ip, double* u, int nprec, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !ip || !u || nprec < 1) return fail_code(B200_EINVAL, "invalid argument");
  const size_t n = 4 * g.vol;
  link_update_kernel<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(u, ip, n, alpha, nprec);
  G_CHECK(cudaGetLastError());
  return 0;
}

int b200_momentum_update(const int lattice[4], double eps, const double* force, double* ip, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !force || !ip) return fail_code(B200_EINVAL, "invalid argument");
  const size_t n = 18 * 4 * g.vol;
  G_CHECK(launch_axpby_links(ip, force, n, eps, 1.0, (cudaStream_t)stream));
  return 0;
}

int b200_momentum_energy(const int lattice[4], const double* ip, double* H, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !ip || !H) return fail_code(B200_EINVAL, "invalid argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int nb = 592;
  double* part = nullptr;
  G_CHECK(device_malloc(&part, sizeof(double) * nb));
  norm2_links_kernel<<<nb, 256, 0, st>>>(ip, 18 * 4 * g.vol, part);
  std::vector<double> h(nb);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), part, sizeof(double) * nb, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(part);
  G_CHECK(e);
  double s = 0.0;
  for (int b = 0; b < nb; ++b) s += h[b];
  *H = 0.5 * s;
  return 0;
}

int b200_links_axpby(const int lattice[4], double a, const double* x, double b, double* y, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !x || !y) return fail_code(B200_EINVAL, "invalid argument");
  G_CHECK(launch_axpby_links(y, x, 18 * 4 * g.vol, a, b, (cudaStream_t)stream));
  return 0;
}

int b200_momentum_from_gauss(const int lattice[4], const double* h, double* ip, void* stream) {
  LexGeom g;
  if (!geom_ok(lattice, &g) || !h || !ip) return fail_code(B200_EINVAL, "invalid argument");
  const size_t n = 4 * g.vol;
  momentum_from_gauss_kernel<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      h, ip, n, 1.0 / std::sqrt(3.0));
  G_CHECK(cudaGetLastError());
  return 0;
}

}  // extern "C"
