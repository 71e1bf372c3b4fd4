// adjoint.cu -- reverse-mode derivatives of the Wilson action and of the Wilson flow (SU(2)).
//
// Conventions (those of the reference): the algebra element (a, b, c) of adjointsu2
// (adjointfield.hh:12-51) is X = i(a s_x + b s_y + c s_z) (s = Pauli matrices) and exp_gauge.cc
// computes exp(X); in the (a, b) storage of an SU(2) element, X itself is {a: i c, b: b + i a}.
// get_deriv(S)_k = -ReTr(i s_k S) (adjointfield.hh:53-56).  Derivatives are left derivatives:
// grad O(x, mu)_k = d/dw O(exp(i w s_k) U_mu(x)) at w = 0; with them the derivative of
// get_S_G_hmc is gaugemonomial::derivative (flat-gaugemonomial.hh:105-131).
//
// Force field g(x, mu) = get_deriv(U_mu(x) K_mu(x)) (K = staple sum, get_staples.hh:26-80).
// Its vector-Jacobian product for a cotangent field mu is
//   VJP(x, nu) = get_deriv( U_nu(x) * sum_staples D ),
// where for a staple A B C of the link (A, B, C links or their daggers) the decorated sum is
//   D = A B C M_l + [A] B C + A [B] C + A B [C],   M = i mu.s = {a: i mu_c, b: mu_b + i mu_a},
//   [X] = +M_X X when X is a link traversed forwards, -X M_X when traversed backwards,
// M_l being the cotangent of the link itself.  (Derivation: mu.g = -sum ReTr(M U K); each
// staple term is a plaquette with M inserted at the front of one of its links.)
//
// One RK3 flow step (flat-gradient_flow.hh:17-50): Z_0 = a_0 g(W_0), W_1 = exp(b_0 Z_0) W_0,
// Z_1 = Z_0 + a_1 g(W_1), W_2 = exp(b_1 Z_1) W_1, Z_2 = Z_1 + a_2 g(W_2), W_3 = exp(b_2 Z_2) W_2.
// Reverse through W' = exp(x) W, x = b Z: the cotangent of W is R(x)^T lam' and that of Z is
// b J(x)^T lam', with R the rotation of the adjoint action of exp(x) and J the
// left-trivialised differential of exp (for su(2): ad_x v = -2 x cross v, theta = 2|x|,
// J = 1 + (1 - cos th)/th^2 ad + (th - sin th)/th^3 ad^2).
#include <sys/mman.h>
#include <unistd.h>

#include <cerrno>
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

#include "site_ops.cuh"
#include "su2b.h"
#include "su2b_ctx.h"

using namespace su2b;

namespace {

// an algebra element i (x s_x + y s_y + z s_z): {Im b, Re b, Im a} of the (a, b) storage
template <class T> struct V3 {
  T x, y, z;
};
template <class T> __device__ __forceinline__ V3<T> operator+(const V3<T> &a, const V3<T> &b) {
  return V3<T>{a.x + b.x, a.y + b.y, a.z + b.z};
}
template <class T> __device__ __forceinline__ V3<T> operator-(const V3<T> &a, const V3<T> &b) {
  return V3<T>{a.x - b.x, a.y - b.y, a.z - b.z};
}
template <class T> __device__ __forceinline__ V3<T> cross(const V3<T> &a, const V3<T> &b) {
  return V3<T>{fm(a.y, b.z, -a.z * b.y), fm(a.z, b.x, -a.x * b.z), fm(a.x, b.y, -a.y * b.x)};
}
// The rotation v -> d^+ v d / |d|^2 of d = (d0, e): v + d0 w + e x w with w = f x v,
// f = 2 e / |d|^2 (any w for a zero link, the plaquettes that it is in are zero).  FP32: the fast
// quotient (2 ulp) and a Newton step.  FP64, where a division is a branch: 2 / n = 4 - 2 n up to
// (1 - n)^2, below rounding for links that are unitary to 2^-27; a field uploaded unnormalised has
// others, for which `far` asks for the site once more with EXACT.
template <class T> struct Rot {
  T d0;
  V3<T> e, f;
};
template <class T> __device__ __forceinline__ Rot<T> rot_by(const Su2<T> &d, T w) {
  return Rot<T>{d.ar, V3<T>{d.bi, d.br, d.ai}, V3<T>{w * d.bi, w * d.br, w * d.ai}};
}
template <bool EXACT>
__device__ __forceinline__ Rot<double> rot_of(const Su2<double> &d, bool &far) {
  const double n = fm(d.ar, d.ar, fm(d.ai, d.ai, fm(d.br, d.br, d.bi * d.bi)));
  if constexpr (EXACT) return rot_by(d, n > 1e-300 ? 2.0 / n : 0.0);
  far |= !(fabs(n - 1.0) < 0x1p-27);
  return rot_by(d, fm(-2.0, n, 4.0));
}
template <bool EXACT>
__device__ __forceinline__ Rot<float> rot_of(const Su2<float> &d, bool &) {
  const float n = fm(d.ar, d.ar, fm(d.ai, d.ai, fm(d.br, d.br, d.bi * d.bi)));
  const float m = fmaxf(n, 1e-37f), r = __fdividef(1.0f, m);
  const float y = fm(r, fm(-m, r, 1.0f), r);
  return rot_by(d, y + y);
}
// d^+ v d (inverse: d v d^+) over |d|^2
template <class T>
__device__ __forceinline__ V3<T> rotate(const Rot<T> &r, const V3<T> &v, bool inverse) {
  const T s = inverse ? T(-1) : T(1);
  const V3<T> w = cross(r.f, v), u = cross(r.e, w);
  return V3<T>{fm(s * r.d0, w.x, v.x + u.x), fm(s * r.d0, w.y, v.y + u.y),
               fm(s * r.d0, w.z, v.z + u.z)};
}

// What pass 1 leaves for pass 2, component by component (each a field of V reals): the
// 3 ND (ND - 1) reals a site sends to its forward neighbours, then the 3 ND of its own links.  Two
// spare link buffers hold 4 ND components each, the staging buffer (4 ND doubles) the others.
template <class T, int ND> struct Sent {
  T *a, *b, *c;
  __device__ __forceinline__ T *at(int k, size_t V) const {
    return k < 4 * ND ? a + k * V : k < 8 * ND ? b + (k - 4 * ND) * V : c + (k - 8 * ND) * V;
  }
};

// VJP of the force field, lam(x,nu) (+)= coef * VJP(x,nu), in two passes.  For the plaquette
// P = A B C^+ D^+ with A = U_mu(x), B = U_nu(x+mu), C = U_mu(x+nu), D = U_nu(x), cotangents
// m_A .. m_D, n_B = A m_B A^+, n_C = D m_C D^+, N = m_A + n_B - n_C - m_D and P = (p0, p), the
// decorated sums of its four links reduce to
//   A: v - w + 2 p x n_B        D: -(v + w + 2 p x n_C)
//   B: A^+ (v - w) A            C: -D^+ (v + w) D            v = p0 N, w = p x N,
// (vec(P N) = v - w, vec(N P) = v + w).  Pass 1, one thread per site: every plaquette once, its
// four results into `sent`; pass 2 adds a link's own sum and what the backward neighbours sent.
// 930 FMAs and 16 links per site in d = 4 and 384 B (FP32) of intermediate values, where one
// thread per link forming all staples with a cotangent in each of their four places took 5,000
// FMAs and 76 links.  Memory bounds both passes: at 24^4 FP32, cold, 33 us and 38 us with the
// reverse of a link update in the second, against 109 us and 27 us for that update by itself.
// An FP64 site whose own links are far from unit norm is done again with exact rotations, after
// the loads and stores of the first time.  With the division's branch in each rotation, between
// the loads, 20 steps at 24^4 took 10.8 ms instead of 10.45 (10.25 without any other than unit
// links), mixed 7.3 instead of 7.0 (6.9).
template <bool EXACT, class T, int ND>
__device__ __forceinline__ bool vjp_site(const Geom &g, const LinkT<T> *U, const T *mu,
                                         const Sent<T, ND> &sent, int p, int cb) {
  const int q = 1 - p;
  const Site s = site_from_eo(g, p, cb);
  const size_t V = (size_t)g.V, NL = V * ND, self = (size_t)p * g.Vh + cb;
  auto M = [&](size_t l) {
    return V3<T>{ld_real(mu + l), ld_real(mu + NL + l), ld_real(mu + 2 * NL + l)};
  };
  bool far = false;
  Su2<T> u[ND];
  V3<T> S[ND];
#pragma unroll
  for (int d = 0; d < ND; d++) u[d] = ld_link(U + d * V + self), S[d] = V3<T>{0, 0, 0};
#pragma unroll
  for (int d = 0; d < ND - 1; d++)
#pragma unroll
    for (int e = d + 1; e < ND; e++) {
      const size_t lb = e * V + eo_of(g, s.lex + fwd(g, s, d), q);
      const size_t lc = d * V + eo_of(g, s.lex + fwd(g, s, e), q);
      const Su2<T> P = mul(mul(u[d], ld_link(U + lb)), dag(mul(u[e], ld_link(U + lc))));
      const V3<T> pv{P.bi, P.br, P.ai};
      const Rot<T> ra = rot_of<EXACT>(u[d], far), rd = rot_of<EXACT>(u[e], far);
      const V3<T> nb = rotate(ra, M(lb), true), nc = rotate(rd, M(lc), true);
      const V3<T> N = (M(d * V + self) + nb) - (nc + M(e * V + self));
      const V3<T> v{P.ar * N.x, P.ar * N.y, P.ar * N.z}, x = cross(pv, N);
      const V3<T> lo = v - x, hi = v + x;
      const V3<T> xb = cross(pv, nb), xc = cross(pv, nc);
      S[d] = S[d] + (lo + (xb + xb));
      S[e] = S[e] - (hi + (xc + xc));
      // to U_e(x + d) and U_d(x + e): components [direction of the step][link]
      const V3<T> to_b = rotate(ra, lo, false), to_c = rotate(rd, hi, false);
      const int kb = 3 * ((ND - 1) * d + (e - 1)), kc = 3 * ((ND - 1) * e + d);
      sent.at(kb, V)[self] = to_b.x;
      sent.at(kb + 1, V)[self] = to_b.y;
      sent.at(kb + 2, V)[self] = to_b.z;
      sent.at(kc, V)[self] = -to_c.x;
      sent.at(kc + 1, V)[self] = -to_c.y;
      sent.at(kc + 2, V)[self] = -to_c.z;
    }
#pragma unroll
  for (int d = 0; d < ND; d++) {
    const int k = 3 * ND * (ND - 1) + 3 * d;
    sent.at(k, V)[self] = S[d].x;
    sent.at(k + 1, V)[self] = S[d].y;
    sent.at(k + 2, V)[self] = S[d].z;
  }
  return far;
}
template <class T, int ND, int NT>
__global__ void __launch_bounds__(NT, sizeof(T) == 4 ? 5 : 3)
  k_force_vjp(Geom g, const LinkT<T> *U, const T *mu, Sent<T, ND> sent) {
  const int w = threadIdx.x >> 5, p = w & 1;
  int cb = blockIdx.x * (NT / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  pdl_start<(sizeof(T) == 4 ? 5 : 3)>(cb);
  if (cb >= g.Vh) return;
  const bool far = vjp_site<false>(g, U, mu, sent, p, cb);
  if (sizeof(T) == 8 && far) {
    asm volatile("" : "+r"(cb));  // loads of its own, so that none is kept for it
    vjp_site<sizeof(T) == 8>(g, U, mu, sent, p, cb);
  }
}

// Horner steps k = K .. 0 of sum_k (-1)^k t2^k / (2k + j)!, j = 1, 2, 3
template <int k> struct SeriesJ {
  static __device__ __forceinline__ void run(double t2, double &s1, double &c1, double &c2) {
    constexpr double sg = (k & 1) ? -1.0 : 1.0;
    s1 = fma(s1, t2, sg / detail::fact(2 * k + 1));
    c1 = fma(c1, t2, sg / detail::fact(2 * k + 2));
    c2 = fma(c2, t2, sg / detail::fact(2 * k + 3));
    SeriesJ<k - 1>::run(t2, s1, c1, c2);
  }
};
template <> struct SeriesJ<-1> {
  static __device__ __forceinline__ void run(double, double &, double &, double &) {}
};

// reverse of W' = exp(b Z) W for link l with cotangent (l0, l1, l2):
// lam <- R(bZ)^T lam ; mu (+)= b J(bZ)^T lam
template <class T>
__device__ __forceinline__ void exp_adjoint_link(size_t l, size_t NL, const T *__restrict__ Z, T b,
                                                 double l0, double l1, double l2,
                                                 T *__restrict__ lam, T *__restrict__ mu,
                                                 int accumulate) {
  const double x0 = (double)b * Z[l], x1 = (double)b * Z[NL + l], x2 = (double)b * Z[2 * NL + l];
  const double t2 = 4.0 * (x0 * x0 + x1 * x1 + x2 * x2);  // th^2, th = 2 |x|
  // ad v = -2 x cross v ; ad^2 v = 4 (x (x.v) - |x|^2 v)
  auto ad = [&](double v0, double v1, double v2, double &r0, double &r1, double &r2) {
    r0 = -2.0 * (x1 * v2 - x2 * v1);
    r1 = -2.0 * (x2 * v0 - x0 * v2);
    r2 = -2.0 * (x0 * v1 - x1 * v0);
  };
  double c1, c2, s1, s2;  // J = 1 + c1 ad + c2 ad^2 ; R = exp(ad) = 1 + s1 ad + s2 ad^2
  if (t2 <= 0.25) {
    // sin(th)/th, (1 - cos th)/th^2, (th - sin th)/th^3 as their series in th^2 (the first
    // omitted terms are below 1e-16): every flow step in practice, and no cancellation.  A
    // quarter of the FP64 work of the square root, sincospi and five divisions below
    s1 = c1 = c2 = 0.;
    SeriesJ<6>::run(t2, s1, c1, c2);
    s2 = c1;
  } else {
    const double th = sqrt(t2);
    double sn, cs;
    sincospi(th * M_1_PI_D, &sn, &cs);
    c1 = (1.0 - cs) / (th * th);
    c2 = (th - sn) / (th * th * th);
    s1 = sn / th;
    s2 = (1.0 - cs) / (th * th);
  }
  // transposes: ad^T = -ad (skew), (ad^2)^T = ad^2
  double a0, a1, a2v, b0, b1, b2;
  ad(l0, l1, l2, a0, a1, a2v);
  ad(a0, a1, a2v, b0, b1, b2);
  const double r0 = l0 - s1 * a0 + s2 * b0, r1 = l1 - s1 * a1 + s2 * b1,
               r2 = l2 - s1 * a2v + s2 * b2;
  const double j0 = (double)b * (l0 - c1 * a0 + c2 * b0),
               j1 = (double)b * (l1 - c1 * a1 + c2 * b1),
               j2 = (double)b * (l2 - c1 * a2v + c2 * b2);
  lam[l] = (T)r0;
  lam[NL + l] = (T)r1;
  lam[2 * NL + l] = (T)r2;
  if (accumulate) {
    mu[l] += (T)j0;
    mu[NL + l] += (T)j1;
    mu[2 * NL + l] += (T)j2;
  } else {
    mu[l] = (T)j0;
    mu[NL + l] = (T)j1;
    mu[2 * NL + l] = (T)j2;
  }
}
template <class T>
__global__ void k_exp_adjoint(size_t NL, const T *__restrict__ Z, T b, T *__restrict__ lam,
                              T *__restrict__ mu) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x)
    exp_adjoint_link(l, NL, Z, b, (double)lam[l], (double)lam[NL + l], (double)lam[2 * NL + l], lam,
                     mu, 0);
}

// Pass 2 of the VJP, then (EXP) the reverse of the link update before the stage in the same
// pass over the cotangent: lam is read and written once instead of twice
template <class T, int ND, int NT, bool EXP>
__global__ void __launch_bounds__(NT, 7)
  k_force_vjp_gather(Geom g, Sent<T, ND> sent, T *__restrict__ lam, T coef,
                     int acc_lam, const T *Z, T b, T *__restrict__ mu, int acc_mu) {
  const int w = threadIdx.x >> 5, p = w & 1, q = 1 - p;
  int cb = blockIdx.x * (NT / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  pdl_start<7>(cb);
  if (cb >= g.Vh) return;
  const Site s = site_from_eo(g, p, cb);
  const size_t V = (size_t)g.V, NL = V * ND, self = (size_t)p * g.Vh + cb;
  T S[3 * ND];
#pragma unroll
  for (int k = 0; k < 3 * ND; k++) S[k] = sent.at(3 * ND * (ND - 1) + k, V)[self];
#pragma unroll
  for (int d = 0; d < ND; d++) {
    const size_t z = eo_of(g, s.lex + bwd(g, s, d), q);
#pragma unroll
    for (int m = 0; m < ND; m++) {
      if (m == d) continue;
      const int k = 3 * ((ND - 1) * d + (m < d ? m : m - 1));
#pragma unroll
      for (int i = 0; i < 3; i++) S[3 * m + i] += sent.at(k + i, V)[z];
    }
  }
  const T c2 = T(2) * coef;
#pragma unroll
  for (int m = 0; m < ND; m++) {
    const size_t l = m * V + self;
    T v[3];
#pragma unroll
    for (int i = 0; i < 3; i++)
      v[i] = acc_lam ? fm(c2, S[3 * m + i], lam[i * NL + l]) : c2 * S[3 * m + i];
    if (EXP) {
      exp_adjoint_link(l, NL, Z, b, (double)v[0], (double)v[1], (double)v[2], lam, mu, acc_mu);
    } else {
#pragma unroll
      for (int i = 0; i < 3; i++) lam[i * NL + l] = v[i];
    }
  }
}

// The two passes.  spare: two link buffers and the staging buffer of the context, none of which
// holds anything between calls; they carry what pass 1 sends to pass 2.  With Z pass 2 also takes
// the reverse of exp(b Z) (lam, and mu accumulated).
template <class T, int ND> Sent<T, ND> sent_in(void *const (&spare)[3]) {
  return Sent<T, ND>{(T *)spare[0], (T *)spare[1], (T *)spare[2]};
}
template <class T>
cudaError_t force_vjp_send(const Geom &g, const void *U, const T *mu, void *const (&spare)[3],
                           cudaStream_t s) {
  constexpr int NT = 128;
  const int grid = (g.Vh + NT / 2 - 1) / (NT / 2);
  const LinkT<T> *u = (const LinkT<T> *)U;
#define SU2B_SEND(ND)                                                                      \
  launch_force(k_force_vjp<T, ND, NT>, dim3(grid), NT, s, true, 0, g, u, mu, sent_in<T, ND>(spare))
  return g.nd == 2 ? SU2B_SEND(2) : g.nd == 3 ? SU2B_SEND(3) : SU2B_SEND(4);
#undef SU2B_SEND
}
template <class T>
cudaError_t force_vjp_gather(const Geom &g, T *lam, double coef, int acc, void *const (&spare)[3],
                             const T *Z, double b, T *mu, int acc_mu, cudaStream_t s) {
  constexpr int NT = 128;
  const int grid = (g.Vh + NT / 2 - 1) / (NT / 2);
#define SU2B_GATHER(ND, EXP)                                                               \
  launch_force(k_force_vjp_gather<T, ND, NT, EXP>, dim3(grid), NT, s, true, 0, g,           \
               sent_in<T, ND>(spare), lam, (T)coef, acc, Z, (T)b, mu, acc_mu)
  switch (g.nd) {
    case 2: return Z ? SU2B_GATHER(2, true) : SU2B_GATHER(2, false);
    case 3: return Z ? SU2B_GATHER(3, true) : SU2B_GATHER(3, false);
    default: return Z ? SU2B_GATHER(4, true) : SU2B_GATHER(4, false);
  }
#undef SU2B_GATHER
}
template <class T>
cudaError_t exp_adjoint(const Geom &g, const T *Z, double b, T *lam, T *mu, cudaStream_t s) {
  const size_t NL = (size_t)g.V * g.nd;
  const int grid = (int)std::min<size_t>((NL + 255) / 256, 148 * 32);
  k_exp_adjoint<T><<<grid, 256, 0, s>>>(NL, Z, (T)b, lam, mu);
  return cudaGetLastError();
}

// Scratch of one adjoint computation, carved from the context's arena.  The arena stays
// allocated between calls (allocating and freeing the 2.2 GB of a gradient of 20 steps at 24^4
// takes 2.4 ms), until the context ends, a call asks for checkpoints and needs less than half of
// it, or another allocation of the process finds no memory.
struct Scratch {
  char *base = nullptr;
  size_t off = 0, cap = 0;
  void *get(size_t bytes) {
    const size_t b = (bytes + 255) & ~(size_t)255;
    if (off + b > cap) return nullptr;
    void *q = base + off;
    off += b;
    return q;
  }
};
int arena(su2b_ctx *ctx, size_t bytes, Scratch *sc, bool shrink, size_t limit) {
  if (ctx->arena_bytes < bytes || (shrink && ctx->arena_bytes / 2 > bytes)) {
    const cudaError_t e = su2b_arena_reserve(ctx, bytes, limit);
    if (e != cudaSuccess)
      return su2b_fail(ctx, SU2B_ERR_NOMEM, "flow adjoint scratch (%zu bytes): %s", bytes,
                       cudaGetErrorString(e));
  }
  sc->base = (char *)ctx->arena;
  sc->off = 0;
  sc->cap = ctx->arena_bytes;
  return SU2B_OK;
}
// a call's claim on the arena, held until the device is done with it
struct ArenaUse {
  su2b_ctx *ctx;
  explicit ArenaUse(su2b_ctx *c) : ctx(c) { su2b_arena_busy(ctx, true); }
  ~ArenaUse() {
    cudaStreamSynchronize(ctx->stream);
    su2b_arena_busy(ctx, false);
  }
};

// Maps the pages of a host buffer that is about to be written, while the device still works on
// what goes there: the 8,000 pages of a fresh 32 MB array (a gradient at 24^4) otherwise fault
// one by one inside the copy (a call of 20 steps there: 13.5 ms, 10.1 ms with this and without
// the wait for the objective in its middle).  The contents stay; where the kernel or the mapping does not take
// the advice, the copy faults them in as before.
void populate(void *p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t a = (uintptr_t)p / page * page, e = ((uintptr_t)p + bytes + page - 1) / page * page;
  const int saved = errno;
  (void)madvise((void *)a, e - a, MADV_POPULATE_WRITE);
  errno = saved;
#endif
}

struct FlowCoef {
  double a[3], b[3];
};
FlowCoef flow_coef(const su2b_ctx *ctx, double eps) {
  // flat-gradient_flow.hh:20-47 via gaugemonomial::derivative's fac*beta/Nc
  const double zfac[3] = {(-17.0) / (36.0), (8.0) / (9.0), (-3.0) / (4.0)};
  const double expfac[3] = {-36.0 / 4. / 17.0, 1., -1.};
  const int Nc = 2;
  FlowCoef c;
  for (int f = 0; f < 3; f++) {
    const double fac = 2. * Nc * zfac[f] / ctx->beta;
    c.a[f] = fac * ctx->beta / (double)Nc;
    c.b[f] = -eps * expfac[f];
  }
  return c;
}

// the reverse of the flow's steps: lam, the cotangent of the field that the last step ended with,
// becomes that of the field it began with
template <class T> struct Reverse {
  su2b_ctx *ctx;
  T *lam, *mu;
  void *const spare[3];
  // The VJP's second pass waits for the next link update's reverse, which takes it along (or
  // for the end); nothing in between touches the cotangent or the spare buffers.
  bool sent = false;
  double sent_a = 0.;
  int vjp(const void *W, double a) {
    SU2B_LAUNCH(SU2B_K_FORCE, force_vjp_send<T>(ctx->g, W, mu, spare, ctx->stream));
    sent = true;
    sent_a = a;
    return SU2B_OK;
  }
  int gather(const T *Z, double bz, int acc_mu) {
    SU2B_LAUNCH(SU2B_K_FORCE, force_vjp_gather<T>(ctx->g, lam, sent_a, 1, spare, Z, bz, mu, acc_mu,
                                                  ctx->stream));
    sent = false;
    return SU2B_OK;
  }
  // one step with the fields W and the accumulators Z of its stages; the last stage's update
  // starts the step's mu
  int step(const void *const (&W)[3], T *const (&Z)[3], const FlowCoef &c) {
    if (sent)
      SU2B_CKS(gather(Z[2], c.b[2], 0));
    else
      SU2B_LAUNCH(SU2B_K_OTHER, exp_adjoint<T>(ctx->g, Z[2], c.b[2], lam, mu, ctx->stream));
    SU2B_CKS(vjp(W[2], c.a[2]));
    SU2B_CKS(gather(Z[1], c.b[1], 1));
    SU2B_CKS(vjp(W[1], c.a[1]));
    SU2B_CKS(gather(Z[0], c.b[0], 1));
    return vjp(W[0], c.a[0]);
  }
  int end() { return sent ? gather(nullptr, 0., 0) : SU2B_OK; }
};

// objective t^2 E_p(t), E_p = d(d-1)/2 - P/(V Nc) (flat-gradient_flow.hh:151), P in h_red[40]
void read_objective(const su2b_ctx *ctx, double t, double *objective) {
  const double d = ctx->g.nd, VNc = (double)ctx->V * ctx->Nc();
  if (objective) *objective = t * t * (d * (d - 1) / 2.0 - ctx->h_red[40] / VNc);
}
int get_gradient(su2b_ctx *ctx, const void *lam, double t, double *objective, double *grad_host) {
  populate(grad_host, sizeof(double) * 3 * ctx->NL);
  SU2B_CKS(su2b_adj_download(ctx, lam, grad_host));
  read_objective(ctx, t, objective);
  return SU2B_OK;
}

// The arena for a tape: the arenas of all contexts hold at most 8 GB with it, and it takes at
// most a quarter of what is free.
bool tape_arena(su2b_ctx *ctx, size_t bytes, Scratch *sc) {
  constexpr size_t LIMIT = (size_t)8 << 30;
  if (bytes > ctx->arena_bytes) {
    size_t free = 0, total = 0;
    if (bytes > LIMIT || cudaMemGetInfo(&free, &total) != cudaSuccess) return false;
    if (bytes - ctx->arena_bytes > free / 4) return false;
  }
  if (arena(ctx, bytes, sc, false, LIMIT) == SU2B_OK) return true;
  ctx->err.clear();
  return false;
}

// the gradient with every stage's field W[3 st + f] and accumulator Z[3 st + f] kept
template <class T>
int flow_adjoint_tape(su2b_ctx *ctx, double eps, int n, Scratch *sc, double *objective,
                      double *grad_host) {
  const size_t lb = ctx->link_bytes() * ctx->NL, ab = ctx->adj_bytes() * ctx->NL;
  std::vector<void *> W(3 * n + 1);
  std::vector<T *> Z(3 * n);
  for (void *&w : W) w = sc->get(lb);
  for (T *&z : Z) z = (T *)sc->get(ab);
  T *const lam = (T *)sc->get(ab), *const mu = (T *)sc->get(ab);
  const FlowCoef c = flow_coef(ctx, eps);
  SU2B_CK(cudaMemcpyAsync(W[0], ctx->U, lb, cudaMemcpyDeviceToDevice, ctx->stream));
  for (int st = 0; st < n; st++) {
    for (int f = 0; f < 3; f++) {
      const int k = 3 * st + f;
      SU2B_CKS(su2b_q_force(ctx, W[k], Z[k], f ? Z[k - 1] : nullptr, c.a[f], 1.0,
                            FM_UPDATE | (f ? FM_EXTRA : 0), nullptr, nullptr, W[k + 1], c.b[f]));
    }
    if (!ctx->link64) SU2B_CKS(su2b_q_restore(ctx, W[3 * st + 3]));
  }
  SU2B_CKS(su2b_q_plaq(ctx, W[3 * n], ctx->h_red + 40));
  const double t = n * eps, VNc = (double)ctx->V * ctx->Nc();
  // d O / d V_T (left derivative) = t^2/(V Nc) g(V_T)
  SU2B_CKS(su2b_q_force(ctx, W[3 * n], lam, nullptr, t * t / VNc, 1.0, 0, nullptr, nullptr));
  Reverse<T> rev{ctx, lam, mu, {ctx->U_old, ctx->U2, ctx->stage}};
  for (int st = n - 1; st >= 0; st--) {
    const void *const w[3] = {W[3 * st], W[3 * st + 1], W[3 * st + 2]};
    T *const z[3] = {Z[3 * st], Z[3 * st + 1], Z[3 * st + 2]};
    SU2B_CKS(rev.step(w, z, c));
  }
  SU2B_CKS(rev.end());
  return get_gradient(ctx, lam, t, objective, grad_host);
}

template <class T>
int flow_adjoint_t(su2b_ctx *ctx, double eps, int n, int every, double *objective,
                   double *grad_host) {
  cudaStream_t s = ctx->stream;
  const size_t NL = ctx->NL, lb = ctx->link_bytes() * NL, ab = ctx->adj_bytes() * NL;
  const size_t lb_a = (lb + 255) & ~(size_t)255, ab_a = (ab + 255) & ~(size_t)255;
  Scratch sc;
  // Every stage's field and Z kept from the forward pass where there is room for them and the
  // caller asked for no checkpoints: the reverse pass then runs no force again.  20 steps at
  // 24^4, mixed precision: 7.0 ms and 2.2 GB against 9.85 ms and 0.3 GB.
  const size_t tape = (size_t)n * 3 * (lb_a + ab_a) + lb_a + 2 * ab_a;
  const ArenaUse use(ctx);
  if (grad_host && every <= 0 && tape_arena(ctx, tape, &sc))
    return flow_adjoint_tape<T>(ctx, eps, n, &sc, objective, grad_host);
  const bool asked = every > 0;
  if (!asked) every = std::max(1, (int)std::lround(std::sqrt((double)n)));
  const int nseg = (n + every - 1) / every;
  SU2B_CKS(arena(ctx, (nseg + every + 3) * lb_a + 5 * ab_a, &sc, asked, 0));
  std::vector<void *> ck(nseg), seg(every);
  for (int i = 0; i < nseg; i++) ck[i] = sc.get(lb);
  for (int i = 0; i < every; i++) seg[i] = sc.get(lb);
  void *W1 = sc.get(lb), *W2 = sc.get(lb), *cur = sc.get(lb);
  T *Zs[3], *lam, *mu;
  for (int f = 0; f < 3; f++) Zs[f] = (T *)sc.get(ab);
  lam = (T *)sc.get(ab);
  mu = (T *)sc.get(ab);
  const FlowCoef c = flow_coef(ctx, eps);
  Reverse<T> rev{ctx, lam, mu, {ctx->U_old, ctx->U2, ctx->stage}};
  // Z = a g(W) (+ Z with FM_HAS_IN, + Z0 with FM_EXTRA: the stages' Z are kept without copies, a
  // gradient of 20 steps at 24^4 9.85 ms against 10.13); with Wn, also Wn = exp(b Z) W from the
  // same kernel
  auto force = [&](const void *W, T *Z, double a, int mode, void *Wn = nullptr, double b = 0.0,
                   const T *Z0 = nullptr) {
    return su2b_q_force(ctx, W, Z, Z0, a, 1.0, Wn ? (mode | FM_UPDATE) : mode, nullptr, nullptr,
                        Wn, b);
  };
  // forward with checkpoints every `every` steps; the field alternates between cur and W1
  // (W1 is free until the backward pass), so every stage is fused with its link update
  SU2B_CK(cudaMemcpyAsync(cur, ctx->U, lb, cudaMemcpyDeviceToDevice, s));
  void *fa = cur, *fb = W1;
  for (int st = 0; st < n; st++) {
    if (st % every == 0)
      SU2B_CK(cudaMemcpyAsync(ck[st / every], fa, lb, cudaMemcpyDeviceToDevice, s));
    SU2B_CKS(su2b_q_flow_step_to(ctx, fa, fb, eps));
    std::swap(fa, fb);
  }
  cur = fa;
  SU2B_CKS(su2b_q_plaq(ctx, cur, ctx->h_red + 40));
  const double t = n * eps, VNc = (double)ctx->V * ctx->Nc();
  if (!grad_host) {
    SU2B_CK(cudaStreamSynchronize(s));
    read_objective(ctx, t, objective);
    return SU2B_OK;
  }
  // d O / d V_T (left derivative) = t^2/(V Nc) g(V_T)
  SU2B_CKS(force(cur, lam, t * t / VNc, 0));
  for (int sg = nseg - 1; sg >= 0; sg--) {
    const int s0 = sg * every, s1 = std::min(n, s0 + every);
    SU2B_CK(cudaMemcpyAsync(seg[0], ck[sg], lb, cudaMemcpyDeviceToDevice, s));
    for (int j = 1; j < s1 - s0; j++) {  // seg[j-1] -> seg[j] through W2, seg[j-1] kept
      SU2B_CKS(force(seg[j - 1], Zs[0], c.a[0], 0, seg[j], c.b[0]));
      SU2B_CKS(force(seg[j], Zs[0], c.a[1], FM_HAS_IN, W2, c.b[1]));
      SU2B_CKS(force(W2, Zs[0], c.a[2], FM_HAS_IN, seg[j], c.b[2]));
      if (!ctx->link64) SU2B_CKS(su2b_q_restore(ctx, seg[j]));
    }
    for (int j = s1 - s0 - 1; j >= 0; j--) {
      const void *W0 = seg[j];
      // stages of this step, each fused with its link update
      SU2B_CKS(force(W0, Zs[0], c.a[0], 0, W1, c.b[0]));
      SU2B_CKS(force(W1, Zs[1], c.a[1], FM_EXTRA, W2, c.b[1], Zs[0]));
      SU2B_CKS(force(W2, Zs[2], c.a[2], FM_EXTRA, nullptr, 0.0, Zs[1]));
      const void *const W[3] = {W0, W1, W2};
      SU2B_CKS(rev.step(W, Zs, c));
    }
  }
  SU2B_CKS(rev.end());
  return get_gradient(ctx, lam, t, objective, grad_host);
}

}  // namespace

extern "C" int su2b_action_backward(su2b_ctx *ctx, double grad_out, double *S, double *dS_host) {
  if (!ctx) return SU2B_ERR_INVALID;
  ctx->begin_call();
  SU2B_CK(cudaSetDevice(ctx->device));
  if (S) {
    SU2B_CKS(su2b_q_plaq(ctx, ctx->U, ctx->h_red + 40));
    SU2B_CK(cudaStreamSynchronize(ctx->stream));
    *S = -ctx->beta * ctx->h_red[42] / ctx->Nc();
  }
  if (!dS_host) return SU2B_OK;
  SU2B_CKS(su2b_q_force(ctx, ctx->U, ctx->Z, nullptr, grad_out * ctx->beta / ctx->Nc(), 1.0, 0,
                        nullptr, nullptr));
  return su2b_adj_download(ctx, ctx->Z, dS_host);
}

extern "C" int su2b_force_vjp(su2b_ctx *ctx, const double *mu_host, double *out_host) {
  if (!ctx) return SU2B_ERR_INVALID;
  ctx->begin_call();
  SU2B_CK(cudaSetDevice(ctx->device));
  SU2B_NEED(mu_host && out_host, "NULL buffer");
  if (ctx->group != SU2B_GROUP_SU2)
    return su2b_fail(ctx, SU2B_ERR_UNSUPPORTED, "the force VJP is provided for SU(2)");
  SU2B_CKS(su2b_adj_upload(ctx, mu_host, ctx->P));
  void *const spare[3] = {ctx->U_old, ctx->U2, ctx->stage};
  auto vjp = [&](auto zero) -> int {
    using T = decltype(zero);
    SU2B_LAUNCH(SU2B_K_FORCE, force_vjp_send<T>(ctx->g, ctx->U, (const T *)ctx->P, spare,
                                                ctx->stream));
    SU2B_LAUNCH(SU2B_K_FORCE, force_vjp_gather<T>(ctx->g, (T *)ctx->Z, 1.0, 0, spare, (const T *)nullptr,
                                                  0.0, (T *)nullptr, 0, ctx->stream));
    return SU2B_OK;
  };
  SU2B_CKS(ctx->link64 ? vjp(0.0) : vjp(0.0f));
  return su2b_adj_download(ctx, ctx->Z, out_host);
}

extern "C" int su2b_flow_adjoint(su2b_ctx *ctx, double eps, int n_steps, int checkpoint_every,
                                 double *objective, double *grad_host) {
  if (!ctx) return SU2B_ERR_INVALID;
  ctx->begin_call();
  SU2B_CK(cudaSetDevice(ctx->device));
  SU2B_NEED(n_steps >= 1 && eps > 0, "n_steps >= 1 and eps > 0 required");
  if (ctx->group != SU2B_GROUP_SU2)
    return su2b_fail(ctx, SU2B_ERR_UNSUPPORTED, "the flow adjoint is provided for SU(2)");
  SU2B_NEED(ctx->xi == 1.0, "the flow adjoint needs the isotropic action (xi = 1)");
  const int rc = ctx->link64 ? flow_adjoint_t<double>(ctx, eps, n_steps, checkpoint_every,
                                                      objective, grad_host)
                             : flow_adjoint_t<float>(ctx, eps, n_steps, checkpoint_every,
                                                     objective, grad_host);
  if (rc == SU2B_OK) SU2B_CK(cudaStreamSynchronize(ctx->stream));
  return rc;
}
