// clover.cu -- clover-leaf energy density and topological charge
// (flat-energy_density.hh:57-164), FP64 arithmetic whatever the link storage.
//
// Per site and plane mu<nu the four leaves
//   U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+            (the plaquette)
//   U_nu(x) U_mu(x-mu+nu)^+ U_nu(x-mu)^+ U_mu(x-mu)
//   U_mu(x-mu)^+ U_nu(x-mu-nu)^+ U_mu(x-mu-nu) U_nu(x-nu)
//   U_nu(x-nu)^+ U_mu(x-nu) U_nu(x+mu-nu) U_mu(x)^+
// are summed (cloverdef) or only the first is used, G = traceless_antiherm(leaf sum),
// E += ReTr(G G), and for d = 4 Q += eps_{i1 i2 i3 i4} ReTr(G_{i1 i2} G_{i3 i4}) over the
// terms with i1<i2, i3<i4; for U(1) in d = 2, Q += -Im G_01.  Per-block partials
// {sum E (all planes), sum E (planes mu >= 1), sum Q}.
#include <type_traits>
#include "su2b_internal.h"

namespace su2b {
namespace {

template <class T> using LinkT = typename LinkOf<T>::type;

template <class T>
__device__ __forceinline__ Su2<double> L(const Geom &g, const LinkT<T> *U, int mu, int lex,
                                         int p) {
  return to64(ld_link(U + (size_t)mu * g.V + eo_of(g, lex, p)));
}

// The antihermitian traceless part (su2.hh:83-85, a -> i Im a, b unchanged) of the leaf sum of
// one plane.  An antihermitian part changes sign under ^+, so leaves 1 and 4^+ share U_mu(x)
// on the left, leaves 2 and 3^+ share U_mu(x-mu) on the right, and each pair is closed by one
// product whose real component is never formed:
//   U_mu(x) [U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+ - U_nu(x+mu-nu)^+ U_mu(x-nu)^+ U_nu(x-nu)]
//   [U_nu(x) U_mu(x-mu+nu)^+ U_nu(x-mu)^+ - U_nu(x-nu)^+ U_mu(x-mu-nu)^+ U_nu(x-mu-nu)] U_mu(x-mu)
// ten products per plane instead of twelve.
template <class T, int MU, int NU>
__device__ __forceinline__ Su2<double> clover_plane(const Geom &g, const LinkT<T> *U,
                                                    const Site &s, int p, int cloverdef) {
  const int fm = fwd(g, s, MU), bm = bwd(g, s, MU), fn = fwd(g, s, NU), bn = bwd(g, s, NU);
  const int x = s.lex, q = 1 - p;
  const Su2<double> unu = L<T>(g, U, NU, x, p);
  Su2<double> a = mul(L<T>(g, U, NU, x + fm, q), dag(mul(unu, L<T>(g, U, MU, x + fn, q))));
  if (cloverdef)
    a = add(a, scale(-1.0, mul(dag(mul(L<T>(g, U, MU, x + bn, q), L<T>(g, U, NU, x + fm + bn, p))),
                               L<T>(g, U, NU, x + bn, q))));
  Su2<double> r = mul(L<T>(g, U, MU, x, p), a);
  if (cloverdef) {
    const Su2<double> b = mul(unu, dag(mul(L<T>(g, U, NU, x + bm, q),
                                           L<T>(g, U, MU, x + bm + fn, p))));
    const Su2<double> c = mul(dag(mul(L<T>(g, U, MU, x + bm + bn, p), L<T>(g, U, NU, x + bn, q))),
                              L<T>(g, U, NU, x + bm + bn, p));
    r = add(r, mul(add(b, scale(-1.0, c)), L<T>(g, U, MU, x + bm, q)));
  }
  r.ar = 0.0;
  return r;
}

// planes third of three: a complementary pair in d = 4, one plane in d = 3
template <class T, int ND>
__device__ __forceinline__ void clover_third(const Geom &g, const LinkT<T> *__restrict__ U,
                                             const Site &s, int p, int cloverdef, int third,
                                             double (&v)[3]) {
  auto plane = [&](auto mu, auto nu) {
    const Su2<double> G =
      clover_plane<T, decltype(mu)::value, decltype(nu)::value>(g, U, s, p, cloverdef);
    const double t = retr_mul(G, G);
    v[0] += t;
    if (decltype(mu)::value >= 1) v[1] += t;
    return G;
  };
  using std::integral_constant;
  constexpr integral_constant<int, 0> d0{};
  constexpr integral_constant<int, 1> d1{};
  constexpr integral_constant<int, ND >= 3 ? 2 : 1> d2{};
  constexpr integral_constant<int, ND == 4 ? 3 : 1> d3{};
  if constexpr (ND == 2) {
    plane(d0, d1);
  } else if constexpr (ND == 3) {
    if (third == 0)
      plane(d0, d1);
    else if (third == 1)
      plane(d0, d2);
    else
      plane(d1, d2);
  } else {
    // eps_{i1 i2 i3 i4} over i1<i2, i3<i4 (tensors.hh): every pair of planes twice, the
    // middle one with a minus sign
    if (third == 0)
      v[2] += 2. * retr_mul(plane(d0, d1), plane(d2, d3));
    else if (third == 1)
      v[2] -= 2. * retr_mul(plane(d0, d2), plane(d1, d3));
    else
      v[2] += 2. * retr_mul(plane(d0, d3), plane(d1, d2));
  }
}

// One thread per site, blocks stay and take band after band: bound by the reads of 72 links a
// site through L1.  Four blocks per SM (128 registers, no spills; a call at 32^4 takes 133 us,
// with three 150, with five and spills 147; the twelve-product form 149).  In d = 4 a pair of
// complementary planes (01,23), (02,13), (03,12) gives one term of the charge, so a third of a
// site keeps two plane sums alive instead of six; three warps per site instead of one thread
// were slower from 16^4 on (they share no link reads: 174 us at 32^4).
constexpr int CLOVER_BLOCKS = 4;
template <class T, int ND, int NT>
__global__ void __launch_bounds__(NT, CLOVER_BLOCKS)
  k_clover_su2(Geom g, const LinkT<T> *__restrict__ U, int cloverdef, double *part, Finish fin) {
  __shared__ double shk[3 * (NT / 32)];
  double v[3] = {0., 0., 0.};  // E of all planes, E of the planes mu >= 1, Q
  // the sites cb0 .. cb0 + ncb - 1 of each parity (all of them but in a time slab)
  for (int c = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); 32 * (c >> 1) < g.ncb;
       c += gridDim.x * (NT / 32)) {  // band c/2 of 32 sites, parity c%2
    const int b = 32 * (c >> 1) + (threadIdx.x & 31), p = c & 1;
    if (b >= g.ncb) continue;
    const Site s = site_from_eo(g, p, g.cb0 + b);
#pragma unroll
    for (int third = 0; third < (ND == 2 ? 1 : 3); third++)
      clover_third<T, ND>(g, U, s, p, cloverdef, third, v);
  }
  finish_sums<NT, 3>(v, part, fin, shk);
}

template <int ND, int NT>
__global__ void __launch_bounds__(NT)
  k_clover_u1(Geom g, const double *__restrict__ U, int cloverdef, double *part, Finish fin) {
  __shared__ double shk[3 * (NT / 32)];
  const int p = blockIdx.x & 1;
  const int cb = (blockIdx.x >> 1) * NT + threadIdx.x;
  double e_all = 0., e_ss = 0., q = 0.;
  if (cb < g.Vh) {
    const Site s = site_from_eo(g, p, cb);
    double G[ND][ND];
    auto A = [&](int mu, int lex, int par) { return U[(size_t)mu * g.V + eo_of(g, lex, par)]; };
#pragma unroll
    for (int mu = 0; mu < ND - 1; mu++)
#pragma unroll
      for (int nu = mu + 1; nu < ND; nu++) {
        const int fm = fwd(g, s, mu), bm = bwd(g, s, mu), fn = fwd(g, s, nu),
                  bn = bwd(g, s, nu);
        const int x = s.lex, q_ = 1 - p;
        double im = sin_pi_scaled(((A(mu, x, p) + A(nu, x + fm, q_)) + (-A(mu, x + fn, q_))) +
                        (-A(nu, x, p)));
        if (cloverdef) {
          im += sin_pi_scaled(((A(nu, x, p) + (-A(mu, x + bm + fn, p))) + (-A(nu, x + bm, q_))) +
                    A(mu, x + bm, q_));
          im += sin_pi_scaled((((-A(mu, x + bm, q_)) + (-A(nu, x + bm + bn, p))) + A(mu, x + bm + bn, p)) +
                    A(nu, x + bn, q_));
          im += sin_pi_scaled((((-A(nu, x + bn, q_)) + A(mu, x + bn, q_)) + A(nu, x + fm + bn, p)) +
                    (-A(mu, x, p)));
        }
        G[mu][nu] = im;  // G = i*im (u1.hh:201-203)
        const double t = -im * im;
        e_all += t;
        if (mu >= 1) e_ss += t;
      }
    if (ND == 4) {
      q += -(G[0][1] * G[2][3]);
      q -= -(G[0][2] * G[1][3]);
      q += -(G[0][3] * G[1][2]);
      q += -(G[1][2] * G[0][3]);
      q -= -(G[1][3] * G[0][2]);
      q += -(G[2][3] * G[0][1]);
    }
    if (ND == 2) q += -G[0][1];
  }
  double v[3] = {e_all, e_ss, q};
  finish_sums<NT, 3>(v, part, fin, shk);
}

}  // namespace

template <class T>
cudaError_t clover_partials(const Geom &g, const void *U, int group, int cloverdef,
                            double *part, int *nblocks, cudaStream_t s, Finish fin) {
  if (group == 0) {
    const LinkT<T> *u = (const LinkT<T> *)U;
    constexpr int NT = 128;
    const dim3 grid(min((g.ncb + NT / 2 - 1) / (NT / 2), 148 * CLOVER_BLOCKS));
    *nblocks = grid.x;
    switch (g.nd) {
      case 2: k_clover_su2<T, 2, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
      case 3: k_clover_su2<T, 3, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
      default: k_clover_su2<T, 4, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
    }
  } else {
    constexpr int NT = 128;
    const dim3 grid(2 * ((g.Vh + NT - 1) / NT));
    *nblocks = grid.x;
    const double *u = (const double *)U;
    switch (g.nd) {
      case 2: k_clover_u1<2, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
      case 3: k_clover_u1<3, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
      default: k_clover_u1<4, NT><<<grid, NT, 0, s>>>(g, u, cloverdef, part, fin); break;
    }
  }
  return cudaGetLastError();
}

template cudaError_t clover_partials<double>(const Geom &, const void *, int, int, double *,
                                             int *, cudaStream_t, Finish);
template cudaError_t clover_partials<float>(const Geom &, const void *, int, int, double *, int *,
                                            cudaStream_t, Finish);

}  // namespace su2b
