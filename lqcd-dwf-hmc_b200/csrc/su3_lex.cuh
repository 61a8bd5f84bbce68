// Small SU(3) / lexical-lattice helpers shared by the link-field kernels
// (stout smearing, gauge force and action, link update): complex numbers,
// 3x3 complex matrices in the reference Field_G layout
// ri + 2*(col + 3*row) + 18*(site + Nvol*mu), and periodic lexical shifts.
#pragma once

#include <cuda_runtime.h>

namespace b200 {

struct Cx {
  double r, i;
};
__device__ __forceinline__ Cx cx(double r, double i) { return Cx{r, i}; }
__device__ __forceinline__ Cx operator+(Cx a, Cx b) { return cx(a.r + b.r, a.i + b.i); }
__device__ __forceinline__ Cx operator-(Cx a, Cx b) { return cx(a.r - b.r, a.i - b.i); }
__device__ __forceinline__ Cx operator*(Cx a, Cx b) { return cx(a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r); }
__device__ __forceinline__ Cx operator*(double s, Cx a) { return cx(s * a.r, s * a.i); }

struct M3 {
  Cx m[9];   // row-major
};

__device__ __forceinline__ M3 load3(const double* base, size_t idx) {
  M3 a;
  const double2* p = reinterpret_cast<const double2*>(base + 18 * idx);
#pragma unroll
  for (int k = 0; k < 9; ++k) { double2 v = p[k]; a.m[k] = cx(v.x, v.y); }
  return a;
}
__device__ __forceinline__ void store3(double* base, size_t idx, const M3& a) {
  double2* p = reinterpret_cast<double2*>(base + 18 * idx);
#pragma unroll
  for (int k = 0; k < 9; ++k) p[k] = make_double2(a.m[k].r, a.m[k].i);
}
__device__ __forceinline__ M3 zero3() {
  M3 a;
#pragma unroll
  for (int k = 0; k < 9; ++k) a.m[k] = cx(0, 0);
  return a;
}
__device__ __forceinline__ M3 unit3() {
  M3 a = zero3();
  a.m[0] = a.m[4] = a.m[8] = cx(1, 0);
  return a;
}
__device__ __forceinline__ Cx conj(Cx a) { return cx(a.r, -a.i); }
// s += a b as four chained multiply-adds (a product formed first and added
// afterwards costs two more instructions: the FP64 pipe bounds these kernels)
__device__ __forceinline__ void cmac(Cx& s, Cx a, Cx b) {
  s.r = fma(a.r, b.r, s.r); s.r = fma(-a.i, b.i, s.r);
  s.i = fma(a.r, b.i, s.i); s.i = fma(a.i, b.r, s.i);
}
// c (+)= op(A) op(B), op the adjoint where its flag is set
template <bool kDagA, bool kDagB, bool kAcc>
__device__ __forceinline__ void mul3(M3& c, const M3& a, const M3& b) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Cx s = kAcc ? c.m[3 * i + j] : cx(0, 0);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const Cx x = kDagA ? conj(a.m[3 * k + i]) : a.m[3 * i + k];
        const Cx y = kDagB ? conj(b.m[3 * j + k]) : b.m[3 * k + j];
        cmac(s, x, y);
      }
      c.m[3 * i + j] = s;
    }
}
// A B, A B^+, A^+ B, A^+ B^+
__device__ __forceinline__ M3 mul_nn(const M3& a, const M3& b) { M3 c; mul3<false, false, false>(c, a, b); return c; }
__device__ __forceinline__ M3 mul_nd(const M3& a, const M3& b) { M3 c; mul3<false, true, false>(c, a, b); return c; }
__device__ __forceinline__ M3 mul_dn(const M3& a, const M3& b) { M3 c; mul3<true, false, false>(c, a, b); return c; }
__device__ __forceinline__ M3 mul_dd(const M3& a, const M3& b) { M3 c; mul3<true, true, false>(c, a, b); return c; }
__device__ __forceinline__ void add_to(M3& a, const M3& b, double s = 1.0) {
#pragma unroll
  for (int k = 0; k < 9; ++k) { a.m[k].r = fma(s, b.m[k].r, a.m[k].r); a.m[k].i = fma(s, b.m[k].i, a.m[k].i); }
}
// traceless anti-Hermitian part (Mat_SU_N::at, src/lib/Tools/mat_SU_N.h:375-398)
__device__ __forceinline__ void at3(M3& a) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i + 1; j < 3; ++j) {
      const double re = a.m[3 * i + j].r - a.m[3 * j + i].r;
      const double im = a.m[3 * i + j].i + a.m[3 * j + i].i;
      a.m[3 * i + j] = cx(0.5 * re, 0.5 * im);
      a.m[3 * j + i] = cx(-0.5 * re, 0.5 * im);
    }
  const double tr = (a.m[0].i + a.m[4].i + a.m[8].i) / 3.0;
  a.m[0] = cx(0.0, a.m[0].i - tr);
  a.m[4] = cx(0.0, a.m[4].i - tr);
  a.m[8] = cx(0.0, a.m[8].i - tr);
}
__device__ __forceinline__ double norm2_3(const M3& a) {
  double t = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) t += a.m[k].r * a.m[k].r + a.m[k].i * a.m[k].i;
  return t;
}

struct LexGeom {
  int n[4];
  size_t vol;
  __device__ size_t shift(size_t site, int mu, int dir) const {   // site + dir*mu (periodic)
    int c[4];
    size_t s = site;
    c[0] = (int)(s % n[0]); s /= n[0];
    c[1] = (int)(s % n[1]); s /= n[1];
    c[2] = (int)(s % n[2]); s /= n[2];
    c[3] = (int)s;
    c[mu] = (c[mu] + dir + n[mu]) % n[mu];
    return c[0] + (size_t)n[0] * (c[1] + (size_t)n[1] * (c[2] + (size_t)n[2] * c[3]));
  }
};

// ---------------------------------------------------------------- planar link fields
// Working copies of link fields with entry k of all links of one direction
// contiguous: double2 p[(9 mu + k) vol + site].  A warp's load of one entry
// for 32 consecutive sites (shifted or not) is then four full 128-byte lines;
// from the lexical layout, whose links are 144 bytes apart, every 16-byte
// load of a warp touches 32 lines, and that lookup rate, not the arithmetic,
// bounded the staple kernels.
struct PlanarField {
  double2* p;
  unsigned vol;
  __device__ __forceinline__ M3 load(int site, int mu) const {
    M3 a;
    const double2* q = p + (size_t)(9 * mu) * vol + site;
#pragma unroll
    for (int k = 0; k < 9; ++k) { const double2 v = q[(size_t)k * vol]; a.m[k] = cx(v.x, v.y); }
    return a;
  }
  __device__ __forceinline__ void store(int site, int mu, const M3& a) const {
    double2* q = p + (size_t)(9 * mu) * vol + site;
#pragma unroll
    for (int k = 0; k < 9; ++k) q[(size_t)k * vol] = make_double2(a.m[k].r, a.m[k].i);
  }
};

// The same loads from the lexical layout, where no planar copy can be had.
struct LexField {
  const double* u;
  unsigned vol;
  __device__ __forceinline__ M3 load(int site, int mu) const { return load3(u, site + (size_t)vol * mu); }
};

// Offsets from a site to its neighbours (periodic); shifts along different
// directions add.
struct LexHop {
  int n[4];
  int c[4];
  int st[4];
  __device__ __forceinline__ LexHop(const LexGeom& g, int site) {
    int s = site, stride = 1;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
      n[mu] = g.n[mu];
      st[mu] = stride;
      const int q = s / n[mu];
      c[mu] = s - q * n[mu];
      s = q;
      stride *= n[mu];
    }
  }
  __device__ __forceinline__ void pick(int mu, int* cc, int* nn, int* ss) const {
    *cc = mu == 0 ? c[0] : mu == 1 ? c[1] : mu == 2 ? c[2] : c[3];
    *nn = mu == 0 ? n[0] : mu == 1 ? n[1] : mu == 2 ? n[2] : n[3];
    *ss = mu == 0 ? st[0] : mu == 1 ? st[1] : mu == 2 ? st[2] : st[3];
  }
  __device__ __forceinline__ int up(int mu) const {
    int a, b, s;
    pick(mu, &a, &b, &s);
    return (a + 1 == b) ? -(b - 1) * s : s;
  }
  __device__ __forceinline__ int dn(int mu) const {
    int a, b, s;
    pick(mu, &a, &b, &s);
    return (a == 0) ? (b - 1) * s : -s;
  }
  __device__ __forceinline__ int up2(int mu) const {
    int a, b, s;
    pick(mu, &a, &b, &s);
    int d = a + 1 == b ? 0 : a + 1;
    d = d + 1 == b ? 0 : d + 1;
    return (d - a) * s;
  }
  __device__ __forceinline__ int dn2(int mu) const {
    int a, b, s;
    pick(mu, &a, &b, &s);
    int d = a == 0 ? b - 1 : a - 1;
    d = d == 0 ? b - 1 : d - 1;
    return (d - a) * s;
  }
};

// A warp's own links (up to 32 consecutive ones of a lexical field) through
// a 4,608-byte shared-memory buffer: the global side moves whole lines, the
// shared side (144-byte stride) is free of bank conflicts.  first: the
// warp's first link, nlink: the field's number of links; lanes past the end
// read zeros and write nothing.
__device__ __forceinline__ M3 load3_warp(const double* base, size_t first, size_t nlink, double2* buf, int lane) {
  const double2* g = reinterpret_cast<const double2*>(base) + 9 * first;
  const int np = first < nlink ? 9 * (int)(nlink - first < 32 ? nlink - first : 32) : 0;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int i = lane + 32 * k;
    buf[i] = i < np ? g[i] : make_double2(0.0, 0.0);
  }
  __syncwarp();
  M3 a;
#pragma unroll
  for (int k = 0; k < 9; ++k) { const double2 v = buf[9 * lane + k]; a.m[k] = cx(v.x, v.y); }
  return a;
}
__device__ __forceinline__ void store3_warp(double* base, size_t first, size_t nlink, double2* buf, int lane,
                                            const M3& a) {
  double2* g = reinterpret_cast<double2*>(base) + 9 * first;
  const int np = first < nlink ? 9 * (int)(nlink - first < 32 ? nlink - first : 32) : 0;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 9; ++k) buf[9 * lane + k] = make_double2(a.m[k].r, a.m[k].i);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int i = lane + 32 * k;
    if (i < np) g[i] = buf[i];
  }
}
constexpr int kLinkBuf = 288;      // double2 per warp

// lexical Field_G links -> planar copy (gauge.cu)
cudaError_t launch_links_to_planar(double2* out, const double* u, size_t vol, cudaStream_t st);
// gives up the scratch that the gauge force keeps between calls (gauge.cu)
void gauge_scratch_trim();

}  // namespace b200
