// gauge.cu -- gauge-field kernels of libsu2b: layout conversion, plaquette reductions, the
// fused staple/force/momentum kernel, link update, reunitarisation, Philox momenta, the
// deterministic final reduction and the HMC accept/reject.
//
// Roofline per link (FP64 / FP32 storage), algorithmic bytes:
//   force+momentum  read U 32/16, read+write P 48/24            = 80 / 40 B
//   link update     read P 24/12, read+write U 64/32            = 88 / 44 B
//   plaquette       read U once                                 = 32 / 16 B
#include "site_ops.cuh"

namespace su2b {

namespace {

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// ------------------------------------------------------------------------------------
// layout conversion between the reference's host order and the even/odd device layout
// SU(2) links go through shared memory, both sides coalesced: a block takes a tile of
// 64 consecutive reference sites (32 half-indices h in both parities).  The device side is
// read (or written) as 32 consecutive links per direction and parity -- the site of
// half-index h and parity p is 2h or 2h+1, whichever has parity p -- and the host side as
// the tile's 64 nd consecutive 32-byte records.
constexpr int CONV_TILE = 64;  // sites per block; 64 nd <= 256 threads
__device__ __forceinline__ int tile_lex(const Geom &g, int h, int p) {
  const Site s = site_from_lex(g, 2 * h);
  return 2 * h + (s.p != p);
}
template <class T>
__global__ void __launch_bounds__(256)
  k_links_to_host_tiled(Geom g, const LinkT<T> *__restrict__ U, double *aos) {
  __shared__ Link64 tile[CONV_TILE * 4];
  const int lex0 = blockIdx.x * CONV_TILE, t = threadIdx.x;
  const int nl = CONV_TILE * g.nd;
  if (t < nl) {
    const int mu = t / CONV_TILE, r = t % CONV_TILE, p = r / 32;
    const int h = lex0 / 2 + (r % 32);
    if (h < g.Vh) {
      const int lex = tile_lex(g, h, p);
      const Su2<double> u = to64(ld_link(U + (size_t)mu * g.V + (size_t)p * g.Vh + h));
      tile[(lex - lex0) * g.nd + mu] = Link64{u.ar, u.ai, u.br, u.bi};
    }
  }
  __syncthreads();
  const long i = (long)lex0 * g.nd + t;
  if (t < nl && i < (long)g.V * g.nd) {
    const Link64 v = tile[t];
    st_link((Link64 *)aos + i, Su2<double>{v.ar, v.ai, v.br, v.bi});
  }
}
template <class T>
__global__ void __launch_bounds__(256)
  k_links_from_host_tiled(Geom g, const double *__restrict__ aos, LinkT<T> *U) {
  __shared__ Link64 tile[CONV_TILE * 4];
  const int lex0 = blockIdx.x * CONV_TILE, t = threadIdx.x;
  const int nl = CONV_TILE * g.nd;
  const long i = (long)lex0 * g.nd + t;
  if (t < nl && i < (long)g.V * g.nd) tile[t] = ((const Link64 *)aos)[i];
  __syncthreads();
  if (t < nl) {
    const int mu = t / CONV_TILE, r = t % CONV_TILE, p = r / 32;
    const int h = lex0 / 2 + (r % 32);
    if (h < g.Vh) {
      const int lex = tile_lex(g, h, p);
      const Link64 v = tile[(lex - lex0) * g.nd + mu];
      st_link(U + (size_t)mu * g.V + (size_t)p * g.Vh + h,
              from64<T>(Su2<double>{v.ar, v.ai, v.br, v.bi}));
    }
  }
}

// U(1) angles and adjoint fields: na reals per link, SoA on the device
template <class T>
__global__ void k_adj_from_host(Geom g, const double *__restrict__ aos, T *P, int na) {
  const long n = (long)g.V * g.nd;
  const size_t NL = (size_t)g.V * g.nd;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    const int lex = (int)(i / g.nd), mu = (int)(i - (long)lex * g.nd);
    const Site s = site_from_lex(g, lex);
    const size_t l = (size_t)mu * g.V + eo_of(g, lex, s.p);
    for (int k = 0; k < na; k++) P[k * NL + l] = (T)aos[na * i + k];
  }
}
template <class T>
__global__ void k_adj_to_host(Geom g, const T *__restrict__ P, double *aos, int na) {
  const long n = (long)g.V * g.nd;
  const size_t NL = (size_t)g.V * g.nd;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    const int lex = (int)(i / g.nd), mu = (int)(i - (long)lex * g.nd);
    const Site s = site_from_lex(g, lex);
    const size_t l = (size_t)mu * g.V + eo_of(g, lex, s.p);
    for (int k = 0; k < na; k++) aos[na * i + k] = (double)P[k * NL + l];
  }
}
__global__ void k_spinor_from_host(Geom g, const double2 *__restrict__ aos, double2 *psi) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.V; i += gridDim.x * blockDim.x) {
    const Site s = site_from_lex(g, i);
    psi[eo_of(g, i, s.p)] = aos[i];
  }
}
__global__ void k_spinor_to_host(Geom g, const double2 *__restrict__ psi, double2 *aos) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.V; i += gridDim.x * blockDim.x) {
    const Site s = site_from_lex(g, i);
    aos[i] = psi[eo_of(g, i, s.p)];
  }
}

// ------------------------------------------------------------------------------------
// plaquettes: per site, sum over planes mu<nu of ReTr U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
// (flat-gauge_energy.hpp:31-94), FP64 products.  Partials {full, spatial, xi-weighted}.
// Resident blocks of 256 threads: four with FP32 links (64 registers), three with FP64 links
// (80 registers, no spills; the plaquette call 67 against 71 us at 32^4 with two).  The
// plaquette kernel's blocks stay and take band after band of 32 sites of one parity, so there
// is one wave of them to finish: 55 us at 32^4, 27 us at 24^4 (35 with a block per band and the
// sum in a second launch).
template <class T, int NT> constexpr int plaq_min_blocks() {
  return sizeof(T) == 8 ? 768 / NT : 1024 / NT;
}

template <class T, int ND, int NT>
__device__ __forceinline__ void plaq_bands(const Geom &g, const LinkT<T> *__restrict__ U,
                                           double xi, int first, double (&v)[3]) {
  for (int c = first; 32 * (c >> 1) < g.ncb;
       c += gridDim.x * (NT / 32)) {  // band c/2 of 32 sites, parity c%2
    const int b = 32 * (c >> 1) + (threadIdx.x & 31);
    if (b < g.ncb) plaq_site<T, ND>(g, U, c & 1, g.cb0 + b, xi, v[0], v[1], v[2]);
  }
}
template <class T, int ND, int NT>
__global__ void __launch_bounds__(NT, plaq_min_blocks<T, NT>())
  k_plaq_su2(Geom g, const LinkT<T> *__restrict__ U, double xi, double *part, Finish fin) {
  __shared__ double shk[3 * (NT / 32)];
  double v[3] = {0., 0., 0.};
  plaq_bands<T, ND, NT>(g, U, xi, blockIdx.x * (NT / 32) + (threadIdx.x >> 5), v);
  finish_sums<NT, 3>(v, part, fin, shk);
}

// The start of a trajectory in one pass over the sites: the Philox momenta of the site's
// links (as k_momenta) with their |P|^2, and the site's plaquettes (as k_plaq_su2) for H_old.
// Per block: {sum |P|^2, plaquettes, spatial plaquettes, xi-weighted plaquettes}.
// Without PLAQ only the momenta and |P|^2 (the start plaquettes are known from the previous
// trajectory); the partial layout stays the same, so the kinetic sums are identical.
template <class T, int ND, int NT, bool PLAQ = true>
__global__ void __launch_bounds__(NT, plaq_min_blocks<T, NT>())
  k_momenta_plaq_su2(Geom g, const LinkT<T> *__restrict__ U, T *__restrict__ P,
                     const TrajParams *__restrict__ tp, double xi, double *part) {
  __shared__ double shk[4 * (NT / 32)];
  const int w = threadIdx.x >> 5, p = w & 1;
  const int cb = g.cb0 + blockIdx.x * (NT / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  pdl_trigger();
  double k2 = 0., full = 0., spat = 0., wsum = 0.;
  if (cb < g.cb0 + g.ncb) {
    const uint64_t seed = tp->seed;
    const uint32_t traj = tp->traj;
    const Site s = site_from_eo(g, p, cb);
    const size_t NL = (size_t)g.V * ND;
#pragma unroll
    for (int mu = 0; mu < ND; mu++) {
      const uint32_t lref = (uint32_t)(s.lex + g.lex0) * (uint32_t)ND + (uint32_t)mu;
      const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
      T n0, n1, n2;
      momentum_normals<T>(lref, traj, seed, 3, n0, n1, n2);
      P[l] = n0;
      P[NL + l] = n1;
      P[2 * NL + l] = n2;
      k2 += (double)n0 * n0 + (double)n1 * n1 + (double)n2 * n2;
    }
    if (PLAQ) plaq_site<T, ND>(g, U, p, cb, xi, full, spat, wsum);
  }
  const int b = blockIdx.x;
  double v[4] = {k2, full, spat, wsum};
  block_sums<NT, 4>(v, shk);
  if (threadIdx.x == 0) {
    part[4 * b] = v[0];
    part[4 * b + 1] = v[1];
    part[4 * b + 2] = v[2];
    part[4 * b + 3] = v[3];
  }
}

template <int ND, int NT>
__global__ void __launch_bounds__(NT)
  k_plaq_u1(Geom g, const double *__restrict__ U, double xi, double *part, Finish fin) {
  __shared__ double shk[3 * (NT / 32)];
  const int w = threadIdx.x >> 5, p = w & 1;
  const int cb = blockIdx.x * (NT / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  double full = 0., spat = 0., wsum = 0.;
  if (cb < g.Vh) {
    const Site s = site_from_eo(g, p, cb);
    double u[ND];
#pragma unroll
    for (int mu = 0; mu < ND; mu++) u[mu] = U[(size_t)mu * g.V + p * g.Vh + cb];
#pragma unroll
    for (int mu = 0; mu < ND - 1; mu++) {
      const int lpm = s.lex + fwd(g, s, mu);
#pragma unroll
      for (int nu = mu + 1; nu < ND; nu++) {
        const int lpn = s.lex + fwd(g, s, nu);
        const double A = U[(size_t)nu * g.V + eo_of(g, lpm, 1 - p)];
        const double B = U[(size_t)mu * g.V + eo_of(g, lpn, 1 - p)];
        const double tr = cospi((((u[mu] + A) + (-B)) + (-u[nu])) * M_1_PI_D);
        full += tr;
        if (mu >= 1) spat += tr;
        wsum += (((mu == 0) ^ (nu == 0)) ? 1.0 / xi : xi) * tr;
      }
    }
  }
  double v[3] = {full, spat, wsum};
  finish_sums<NT, 3>(v, part, fin, shk);
}

// out[k] = sum over b of part[b*ncomp + k], one block, in an order fixed by n: thread t sums
// the entries t + i NT into four accumulators (i mod 4), so four loads are in flight at a
// time, then adds them pairwise and the block reduces in a fixed tree
template <int NT>
__device__ __forceinline__ void reduce_into(const double *__restrict__ part, int n, int ncomp,
                                            double *out, double *sh) {
  for (int k = 0; k < ncomp; k++) {
    double a0 = 0., a1 = 0., a2 = 0., a3 = 0.;
    int b = threadIdx.x;
    for (; b + 3 * NT < n; b += 4 * NT) {
      a0 += part[(size_t)b * ncomp + k];
      a1 += part[(size_t)(b + NT) * ncomp + k];
      a2 += part[(size_t)(b + 2 * NT) * ncomp + k];
      a3 += part[(size_t)(b + 3 * NT) * ncomp + k];
    }
    for (; b < n; b += NT) a0 += part[(size_t)b * ncomp + k];
    const double r = block_sum<NT>((a0 + a1) + (a2 + a3), sh);
    if (threadIdx.x == 0) out[k] = r;
  }
}
template <int NT>
__global__ void __launch_bounds__(NT)
  k_reduce_final(const double *__restrict__ part, int n, int ncomp, double *out) {
  __shared__ double sh[NT / 32];
  reduce_into<NT>(part, n, ncomp, out, sh);
}

// fused staple/force/momentum(/link update) kernel: one thread per site, force_site body
template <class T, int ND, int NT, int MINB, bool ANISO>
__global__ void __launch_bounds__(NT, MINB)
  k_force_su2(Geom g, const LinkT<T> *U, T *__restrict__ P,
              const T *extra, T f, T scale_, int mode, T wt, T ws,
              double *kin_part, LinkT<T> *__restrict__ Uout, T dt_upd) {
  __shared__ double sh[NT / 32];
  // warps alternate between the parities of one band of NT/2 sites per parity, so the
  // +-z / +-y neighbours of a site are mostly the own links of another warp of the block
  const int w = threadIdx.x >> 5;
  const int p = w & 1;
  int cb = g.cb0 + blockIdx.x * (NT / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  pdl_start<MINB>(cb);
  double k2 = 0.;
  if (cb < g.cb0 + g.ncb)
    k2 = force_site_impl<T, ND, ANISO>(g, U, P, extra, f, scale_, mode, wt, ws, Uout, dt_upd, p,
                                       cb);
  if (mode & FM_KINETIC) {
    const double r = block_sum<NT>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.x] = r;
  }
}


// the fused force step with one thread per link (force_link_impl): warp mu of block b takes
// the links in direction mu of 32 sites of parity b & 1, so a block holds all d links of its
// sites; for lattices too small to fill the GPU one thread per site
template <class T, int ND, int MINB>
__global__ void __launch_bounds__(32 * ND, MINB)
  k_force_su2_link(Geom g, const LinkT<T> *U, T *__restrict__ P,
                   const T *extra, T f, T scale_, int mode, T wt, T ws,
                   double *kin_part, LinkT<T> *__restrict__ Uout, T dt_upd) {
  constexpr int NT = 32 * ND;
  __shared__ double sh[NT / 32];
  const int mu = threadIdx.x >> 5, p = blockIdx.x & 1;
  int cb = g.cb0 + (blockIdx.x >> 1) * 32 + (threadIdx.x & 31);
  pdl_start<MINB>(cb);
  double k2 = 0.;
  // the direction is a compile-time constant in each warp's body (static site indexing)
#define SU2B_LINK_BODY(M)                                                                     \
  k2 = force_link_impl<T, ND, (M < ND ? M : 0)>(g, U, P, extra, f, scale_, mode, Uout, dt_upd, \
                                                 p, cb)
  if (cb < g.cb0 + g.ncb) {
    switch (mu) {
      case 0: SU2B_LINK_BODY(0); break;
      case 1: SU2B_LINK_BODY(1); break;
      case 2: SU2B_LINK_BODY(2); break;
      default: SU2B_LINK_BODY(3); break;
    }
  }
#undef SU2B_LINK_BODY
  if (mode & FM_KINETIC) {
    const double r = block_sum<NT>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.x] = r;
  }
}

// The fused force step of a d = 4 lattice that leaves most of the GPU idle: three threads per
// link, one for each plane it lies in.  Warp mu + 4 j of a block takes the j-th plane of the
// links mu of 32 sites; the staple sums meet in shared memory and warps 0..3 finish the links.
// What a launch of so few threads takes is one thread's chain of loads and products: two
// staples long here, six with one thread per link.  8^4, ten steps: FP64 49.5 us a trajectory
// (one thread per link 55.3), FP32 44.4 us (48.4); 12^4, where the SMs are full: 99 us (75).
template <class T>
__global__ void __launch_bounds__(384, 1)
  k_force_su2_planes(Geom g, const LinkT<T> *U, T *__restrict__ P,
                     const T *extra, T f, T scale_, int mode, T wt, T ws,
                     double *kin_part, LinkT<T> *__restrict__ Uout, T dt_upd) {
  __shared__ double sh[12];
  __shared__ LinkT<T> xs[2][4][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, mu = w & 3, j = w >> 2;
  const int p = blockIdx.x & 1, cb = g.cb0 + (blockIdx.x >> 1) * 32 + lane;
  const bool on = cb < g.cb0 + g.ncb;  // lanes past the end compute the last site, write nothing
  const int c = on ? cb : g.cb0 + g.ncb - 1;
  Site s = site_from_eo(g, p, c);
  pdl_start<1>(s.lex);
  const size_t V = (size_t)g.V, l = mu * V + eo_of(g, s.lex, p);
  if (j == 0 && (mode & FM_HAS_IN)) prefetch_momenta(P, l, 4 * V);
  Su2<T> K;
  switch (w) {  // direction and plane are compile-time constants in each warp's body
    case 0: K = staple_pair<T, 0, 1>(g, U, s, p); break;
    case 1: K = staple_pair<T, 1, 0>(g, U, s, p); break;
    case 2: K = staple_pair<T, 2, 0>(g, U, s, p); break;
    case 3: K = staple_pair<T, 3, 0>(g, U, s, p); break;
    case 4: K = staple_pair<T, 0, 2>(g, U, s, p); break;
    case 5: K = staple_pair<T, 1, 2>(g, U, s, p); break;
    case 6: K = staple_pair<T, 2, 1>(g, U, s, p); break;
    case 7: K = staple_pair<T, 3, 1>(g, U, s, p); break;
    case 8: K = staple_pair<T, 0, 3>(g, U, s, p); break;
    case 9: K = staple_pair<T, 1, 3>(g, U, s, p); break;
    case 10: K = staple_pair<T, 2, 3>(g, U, s, p); break;
    default: K = staple_pair<T, 3, 2>(g, U, s, p); break;
  }
  if (j > 0) xs[j - 1][mu][lane] = as_link(K);
  Su2<T> u;
  if (j == 0) u = ld_link(U + l);
  __syncthreads();
  double k2 = 0.;
  if (j == 0 && on) {
    K = add(add(K, from_link(xs[0][mu][lane])), from_link(xs[1][mu][lane]));
    k2 = finish_link<T>(u, K, l, 4 * V, P, extra, f, scale_, mode, Uout, dt_upd);
  }
  if (mode & FM_KINETIC) {
    const double r = block_sum<384>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.x] = r;
  }
}

template <int ND, int NT>
__global__ void __launch_bounds__(NT)
  k_force_u1(Geom g, const double *__restrict__ U, double *__restrict__ P,
             const double *__restrict__ extra, double f, double scale_, int mode, int aniso,
             double wt, double ws, double *kin_part) {
  __shared__ double sh[NT / 32];
  const int mu = blockIdx.y >> 1, p = blockIdx.y & 1;
  const int cb = blockIdx.x * NT + threadIdx.x;
  double k2 = 0.;
  if (cb < g.Vh) {
    const Site s = site_from_eo(g, p, cb);
    const int lpm = s.lex + fwd_rt(g, s, mu);  // mu from the block index
    double Kr = 0., Ki = 0.;
#pragma unroll
    for (int nu = 0; nu < ND; nu++) {
      if (nu == mu) continue;
      const int lpn = s.lex + fwd(g, s, nu);
      const double A = U[(size_t)nu * g.V + eo_of(g, lpm, 1 - p)];
      const double B = U[(size_t)mu * g.V + eo_of(g, lpn, 1 - p)];
      const double D = U[(size_t)nu * g.V + eo_of(g, s.lex, p)];
      double sn, cs;
      sincospi(((A + (-B)) + (-D)) * M_1_PI_D, &sn, &cs);
      const double w = aniso ? ((nu == 0 || mu == 0) ? wt : ws) : 1.0;
      Kr += w * cs;
      Ki += w * sn;
    }
#pragma unroll
    for (int nu = 0; nu < ND; nu++) {
      if (nu == mu) continue;
      const int b = bwd(g, s, nu);
      const double A = U[(size_t)nu * g.V + eo_of(g, lpm + b, p)];
      const double B = U[(size_t)mu * g.V + eo_of(g, s.lex + b, 1 - p)];
      const double D = U[(size_t)nu * g.V + eo_of(g, s.lex + b, 1 - p)];
      double sn, cs;
      sincospi((((-A) + (-B)) + D) * M_1_PI_D, &sn, &cs);
      const double w = aniso ? ((nu == 0 || mu == 0) ? wt : ws) : 1.0;
      Kr += w * cs;
      Ki += w * sn;
    }
    const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
    double su, cu;
    sincospi(U[l] * M_1_PI_D, &su, &cu);
    double d = f * (cu * Ki + su * Kr);  // Im(e^{i theta} K), adjointfield.hh:79-81
    if (mode & FM_EXTRA) d += extra[l];
    const double pn = (mode & FM_HAS_IN) ? P[l] + scale_ * d : scale_ * d;
    P[l] = pn;
    k2 = pn * pn;
  }
  if (mode & FM_KINETIC) {
    const double r = block_sum<NT>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.y * gridDim.x + blockIdx.x] = r;
  }
}

// ------------------------------------------------------------------------------------
// U <- exp(dt P) U (update_gauge.hh:8-16)
template <class T>
__global__ void k_update_su2(size_t NL, LinkT<T> *__restrict__ U, const T *__restrict__ P,
                             T dt) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x) {
    const Su2<T> e = exp_alg(dt * P[l], dt * P[NL + l], dt * P[2 * NL + l]);
    st_link(U + l, mul(e, ld_link_rw(U + l)));
  }
}
__global__ void k_update_u1(size_t NL, double *__restrict__ U, const double *__restrict__ P,
                            double dt) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x)
    U[l] = dt * P[l] + U[l];
}
// The rounding of the low-precision integrators, round(x dn) / dn with an IEEE multiply and
// divide in FP64 (std::round and a division: adjointfield.hh:28-31, su2.hh:29-33).
__device__ __forceinline__ double round_dn(double x, double dn) {
  return __ddiv_rn(round(__dmul_rn(x, dn)), dn);
}
// round_and_update_gauge (update_gauge.hh:20-26): U = exp(dt P) round(U)
template <class T>
__global__ void k_update_su2_round(size_t NL, LinkT<T> *__restrict__ U, const T *__restrict__ P,
                                   T dt, double dn) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x) {
    const Su2<T> u = ld_link_rw(U + l);
    const Su2<double> r{round_dn((double)u.ar, dn), round_dn((double)u.ai, dn),
                        round_dn((double)u.br, dn), round_dn((double)u.bi, dn)};
    const Su2<T> e = exp_alg(dt * P[l], dt * P[NL + l], dt * P[2 * NL + l]);
    st_link(U + l, mul(e, from64<T>(r)));
  }
}
// U(1): the angle as _u1::round writes it (u1.hh:31-33), round(a) * dn / dn
__global__ void k_update_u1_round(size_t NL, double *__restrict__ U,
                                  const double *__restrict__ P, double dt, double dn) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x)
    U[l] = dt * P[l] + __ddiv_rn(__dmul_rn(round(U[l]), dn), dn);
}
// round_and_update_momenta (update_momenta.hh:36-58): P -= dt * round(D), multiply and
// subtract rounded separately as there
template <class T>
__global__ void k_adj_round_axpy(size_t n, T *__restrict__ P, const T *__restrict__ D,
                                 double dt, double dn) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    P[i] = (T)__dsub_rn((double)P[i], __dmul_rn(dt, round_dn((double)D[i], dn)));
}

// restoreSU in FP64 (gaugeconfig.hh:115-120)
template <class T> __global__ void k_restore(size_t NL, LinkT<T> *__restrict__ U) {
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < NL;
       l += (size_t)gridDim.x * blockDim.x)
    st_link(U + l, from64<T>(restore_su(to64(ld_link_rw(U + l)))));
}

// ------------------------------------------------------------------------------------
// ------------------------------------------------------------------------------------
// momenta: standard normal per component from Philox(seed; {ref link, draw, traj, MOM})
template <class T, int NT>
__global__ void __launch_bounds__(NT)
  k_momenta(Geom g, T *__restrict__ P, int na, const TrajParams *__restrict__ tp,
            double *kin_part) {
  __shared__ double sh[NT / 32];
  const uint64_t seed = tp->seed;
  const uint32_t traj = tp->traj;
  const int mu = blockIdx.y >> 1, p = blockIdx.y & 1;
  const int cb = blockIdx.x * NT + threadIdx.x;
  double k2 = 0.;
  if (cb < g.Vh) {
    const Site s = site_from_eo(g, p, cb);
    const uint32_t lref = (uint32_t)s.lex * (uint32_t)g.nd + (uint32_t)mu;
    const size_t NL = (size_t)g.V * g.nd;
    const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
    T n0, n1, n2;
    momentum_normals<T>(lref, traj, seed, na, n0, n1, n2);
    P[l] = n0;
    k2 = (double)n0 * n0;
    if (na == 3) {
      P[NL + l] = n1;
      P[2 * NL + l] = n2;
      k2 += (double)n1 * n1 + (double)n2 * n2;
    }
  }
  const double rr = block_sum<NT>(k2, sh);
  if (threadIdx.x == 0) kin_part[blockIdx.y * gridDim.x + blockIdx.x] = rr;
}

template <class T, int NT>
__global__ void __launch_bounds__(NT)
  k_kinetic(Geom g, const T *__restrict__ P, int na, double *part) {
  __shared__ double sh[NT / 32];
  const int mu = blockIdx.y >> 1, p = blockIdx.y & 1;
  const int cb = blockIdx.x * NT + threadIdx.x;
  double k2 = 0.;
  if (cb < g.Vh) {
    const size_t NL = (size_t)g.V * g.nd;
    const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
    for (int k = 0; k < na; k++) {
      const double v = (double)P[k * NL + l];
      k2 += v * v;
    }
  }
  const double rr = block_sum<NT>(k2, sh);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = rr;
}

template <class T> __global__ void k_negate(size_t n, T *P) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    P[i] = -P[i];
}

// ------------------------------------------------------------------------------------
// accept/reject (md_update.hh:45-60), one thread
__device__ __forceinline__ void accept_body(const double *red, const TrajParams *__restrict__ tp,
                                            TrajDev *out) {
  const TrajParams in = *tp;
  TrajDev t;
  t.H_old[0] = 0.5 * red[0];
  t.H_old[1] = -in.beta * red[3] / in.Nc;
  t.H_old[2] = red[8];
  t.H_new[0] = 0.5 * red[4];
  t.H_new[1] = -in.beta * red[7] / in.Nc;
  t.H_new[2] = red[9];
  double dH = 0.;
  dH += t.H_new[0] - t.H_old[0];
  dH += t.H_new[1] - t.H_old[1];
  dH += t.H_new[2] - t.H_old[2];
  t.dH = dH;
  t.accepted = 1;
  t.u = -1.0;
  if (in.accept_reject && dH > 0) {
    double u = in.u_host;
    if (u < 0.0) {
      uint32_t r[4];
      philox(0u, 0u, in.traj, TAG_ACCEPT, in.seed, r);
      u = u01_53(r[0], r[1]) - 0x1p-53;
    }
    t.u = u;
    if (u > exp(-dH)) t.accepted = 0;
  }
  t.pad = 0;
  *out = t;
}
__global__ void k_accept(const double *__restrict__ red, const TrajParams *__restrict__ tp,
                         TrajDev *out) {
  accept_body(red, tp, out);
}
// The end of a fused trajectory in one launch: the plaquettes of the final field (as
// k_plaq_su2), the closing sums and the accept step.  Each block also adds its share of the
// start partials (momenta pass, 4 components, none when ns = 0) and of the final kinetic
// partials; the block that finishes last adds the blocks up into red[0..3], red[4] (skipped when
// nk = 0) and red[5..7], in an order fixed by the grids, and writes red[0..9] and the result to
// the pinned host copies as well.  A separate reduction launch, two copies and a memset that it
// replaces took 13 us of the 70 us of a trajectory of ten steps at 8^4; with all the earlier
// partials left to the last block a mixed trajectory at 32^4 takes 805 to 820 us instead of 785
// to 790.
// cached_start: the momenta pass summed no plaquettes (its components 1..3 are zero); the
// start field is the previous trajectory's result, whose plaquette sums are still in red[]:
// red[5..7] if that trajectory was accepted (out->accepted), else red[1..3].  They are taken
// before the end plaquettes overwrite red[5..7].
template <class T, int ND, int NT>
__global__ void __launch_bounds__(NT, plaq_min_blocks<T, NT>())
  k_plaq_accept_su2(Geom g, const LinkT<T> *U, double xi, double *part,
                    TrajTail e) {
  constexpr int NC = 8;  // start |P|^2 and three plaquette sums, end |P|^2, three plaquette sums
  __shared__ double shk[NC * (NT / 32)];
  int band = blockIdx.x * (NT / 32) + (threadIdx.x >> 5);
  pdl_wait(band);
  double v[3] = {0., 0., 0.}, a[NC];
  plaq_bands<T, ND, NT>(g, U, xi, band, v);
#pragma unroll
  for (int k = 0; k < NC; k++) a[k] = k < 5 ? 0. : v[k - 5];
  // every block also takes its share of the earlier launches' partials (16,384 of the force
  // launch at 32^4), so the last one adds only the blocks of this launch
  const int first = blockIdx.x * NT + threadIdx.x, stride = gridDim.x * NT;
  for (int b = first; b < e.ns; b += stride)
#pragma unroll
    for (int k = 0; k < 4; k++) a[k] += e.ps[(size_t)b * 4 + k];
  for (int b = first; b < e.nk; b += stride) a[4] += e.pk[b];
  if (!leave_sums<NT, NC>(a, part, e.ticket, shk)) return;
#pragma unroll
  for (int k = 0; k < NC; k++) a[k] = 0.;
#pragma unroll 2
  for (int b = threadIdx.x; b < (int)gridDim.x; b += NT)
#pragma unroll
    for (int k = 0; k < NC; k++) a[k] += __ldcg(part + (size_t)b * NC + k);
  block_sums<NT, NC>(a, shk);
  if (threadIdx.x == 0) {
    double *red = e.red;
    if (e.cached_start) {
      const bool prev_accepted = e.out->accepted != 0;
#pragma unroll
      for (int k = 1; k < 4; k++) red[k] = prev_accepted ? red[4 + k] : red[k];
      red[0] = a[0];
    } else if (e.ns > 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) red[k] = a[k];
    }
    if (e.nk > 0) red[4] = a[4];
#pragma unroll
    for (int k = 5; k < 8; k++) red[k] = a[k];
    red[8] = red[9] = 0.;  // no fermion action
    accept_body(red, e.tp, e.out);
    *e.h_out = *e.out;
#pragma unroll
    for (int k = 0; k < 10; k++) e.h_red[k] = red[k];
  }
}

template <class T>
__global__ void k_cond_restore(size_t n, T *__restrict__ U, const T *__restrict__ U_old,
                               const TrajDev *__restrict__ flag) {
  if (flag->accepted) return;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    U[i] = U_old[i];
}

constexpr int NT_RED = 256;

inline int flat_grid(size_t n, int nt) {
  const size_t b = (n + nt - 1) / nt;
  return (int)(b < 148u * 32u ? (b > 0 ? b : 1) : 148u * 32u);
}

}  // namespace

// =====================================================================================
// launchers
// =====================================================================================

template <class T>
cudaError_t links_from_host(const Geom &g, const double *aos, void *U, int group,
                            cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd;
  if (group == 0)
    k_links_from_host_tiled<T><<<cdiv(g.V, CONV_TILE), 256, 0, s>>>(g, aos, (LinkT<T> *)U);
  else
    k_adj_from_host<double><<<flat_grid(n, 256), 256, 0, s>>>(g, aos, (double *)U, 1);
  return cudaGetLastError();
}
template <class T>
cudaError_t links_to_host(const Geom &g, const void *U, double *aos, int group,
                          cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd;
  if (group == 0)
    k_links_to_host_tiled<T><<<cdiv(g.V, CONV_TILE), 256, 0, s>>>(g, (const LinkT<T> *)U, aos);
  else
    k_adj_to_host<double><<<flat_grid(n, 256), 256, 0, s>>>(g, (const double *)U, aos, 1);
  return cudaGetLastError();
}
template <class T>
cudaError_t adj_from_host(const Geom &g, const double *aos, T *P, int group, cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd;
  k_adj_from_host<T><<<flat_grid(n, 256), 256, 0, s>>>(g, aos, P, group == 0 ? 3 : 1);
  return cudaGetLastError();
}
template <class T>
cudaError_t adj_to_host(const Geom &g, const T *P, double *aos, int group, cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd;
  k_adj_to_host<T><<<flat_grid(n, 256), 256, 0, s>>>(g, P, aos, group == 0 ? 3 : 1);
  return cudaGetLastError();
}
cudaError_t spinor_from_host(const Geom &g, const double *aos, double2 *psi, cudaStream_t s) {
  k_spinor_from_host<<<flat_grid(g.V, 256), 256, 0, s>>>(g, (const double2 *)aos, psi);
  return cudaGetLastError();
}
cudaError_t spinor_to_host(const Geom &g, const double2 *psi, double *aos, cudaStream_t s) {
  k_spinor_to_host<<<flat_grid(g.V, 256), 256, 0, s>>>(g, psi, (double2 *)aos);
  return cudaGetLastError();
}

template <class T>
cudaError_t plaq_partials(const Geom &g, const void *U, int group, double xi, double *part,
                          int *nblocks, cudaStream_t s, Finish fin) {
  constexpr int NT = 256;
  const dim3 grid(group == 0 ? min(cdiv(g.ncb, NT / 2), 148 * plaq_min_blocks<T, NT>())
                             : cdiv(g.Vh, NT / 2));
  *nblocks = grid.x;
  if (group == 0) {
    const LinkT<T> *u = (const LinkT<T> *)U;
    switch (g.nd) {
      case 2: k_plaq_su2<T, 2, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
      case 3: k_plaq_su2<T, 3, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
      default: k_plaq_su2<T, 4, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
    }
  } else {
    const double *u = (const double *)U;
    switch (g.nd) {
      case 2: k_plaq_u1<2, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
      case 3: k_plaq_u1<3, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
      default: k_plaq_u1<4, NT><<<grid, NT, 0, s>>>(g, u, xi, part, fin); break;
    }
  }
  return cudaGetLastError();
}

cudaError_t reduce_final(const double *part, int nblocks, int ncomp, double *out,
                         cudaStream_t s) {
  k_reduce_final<1024><<<1, 1024, 0, s>>>(part, nblocks, ncomp, out);
  return cudaGetLastError();
}

// the force step with two threads per site (d = 4): warps (4k, 4k+1) are the two halves of 32
// sites of one parity, warps (4k+2, 4k+3) of the 32 sites of the other parity beside them
template <class T, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
  k_force_su2_split(Geom g, const LinkT<T> *U, T *__restrict__ P,
                    const T *extra, T f, T scale_, int mode, T wt, T ws,
                    double *kin_part, LinkT<T> *__restrict__ Uout, T dt_upd) {
  __shared__ double sh[NT / 32];
  const int w = threadIdx.x >> 5;
  const int half = w & 1, p = (w >> 1) & 1;
  int cb = g.cb0 + blockIdx.x * (NT / 4) + (w >> 2) * 32 + (threadIdx.x & 31);
  pdl_start<MINB>(cb);
  double k2 = 0.;
  if (cb < g.cb0 + g.ncb)
    k2 = half == 0 ? force_half_impl<T, 0, false>(g, U, P, extra, f, scale_, mode, wt, ws, Uout,
                                                  dt_upd, p, cb)
                   : force_half_impl<T, 1, false>(g, U, P, extra, f, scale_, mode, wt, ws, Uout,
                                                  dt_upd, p, cb);
  if (mode & FM_KINETIC) {
    const double r = block_sum<NT>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.x] = r;
  }
}

// the split force step with the cross-plane products formed once per site and swapped
// between the two warps of a site pair through shared memory (force_half_x); isotropic d = 4.
// Every thread reaches its pair barrier: threads past the lattice end run on a clamped site.
template <class T, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
  k_force_su2_xsplit(Geom g, const LinkT<T> *U, T *__restrict__ P,
                     const T *extra, T f, T scale_, int mode, T wt, T ws,
                     double *kin_part, LinkT<T> *__restrict__ Uout, T dt_upd) {
  static_assert(NT == 128, "two warp pairs per block, hardware barriers 1 and 2");
  __shared__ double sh[NT / 32];
  __shared__ LinkT<T> xs[2][NT];
  const int w = threadIdx.x >> 5;
  const int half = w & 1, p = (w >> 1) & 1;
  int cb = g.cb0 + blockIdx.x * (NT / 4) + (w >> 2) * 32 + (threadIdx.x & 31);
  pdl_start<MINB>(cb);
  const bool valid = cb < g.cb0 + g.ncb;
  const int cbc = valid ? cb : g.cb0 + g.ncb - 1;
  const int bar_id = 1 + (w >> 1);
  const double k2 =
    half == 0 ? force_half_x<T, 0>(g, U, P, extra, f, scale_, mode, Uout, dt_upd, p, cbc, valid,
                                   xs, bar_id)
              : force_half_x<T, 1>(g, U, P, extra, f, scale_, mode, Uout, dt_upd, p, cbc, valid,
                                   xs, bar_id);
  if (mode & FM_KINETIC) {
    const double r = block_sum<NT>(k2, sh);
    if (threadIdx.x == 0) kin_part[blockIdx.x] = r;
  }
}

// Three threads per link or (256, 3) for shape 5.  Up to about 160 blocks of 32 sites the three
// threads are the fastest of all shapes (10 x 8 x 8 x 12 FP64 59.6 us a trajectory of ten steps,
// one thread per link 60.4; 10^4, 314 blocks: 79 against 64), and (256, 3) is not, which on
// larger lattices ties with (128, 6).  The line is drawn in the sites of a time slice, not in
// all sites, so that a slab takes the shape that the whole lattice takes, bit for bit; long
// lattices that it admits are left to the tuner, which times the other shapes as well.
bool force_planes_apply(const Geom &g) {
  return g.nd == 4 && (long)g.L[1] * g.L[2] * g.L[3] <= 1024;
}

template <class T>
cudaError_t force_update(const Geom &g, const void *U, int group, T *P, const T *extra, double f,
                         double scale, double xi, int mode, double *kin_part, int *nblocks,
                         void *Uout, double dt_upd, cudaStream_t s, int variant, bool pdl) {
  constexpr int NT = 128;
  const int aniso = xi != 1.0;
  if (group == 0) {
    const LinkT<T> *u = (const LinkT<T> *)U;
    const T wt = (T)(1.0 / xi), ws = (T)xi;
    LinkT<T> *uo = (LinkT<T> *)Uout;
    int nb = 0;
    const int v = (variant >= 0 && variant < FORCE_VARIANTS) ? variant : 1;
#define SU2B_FORCE_ARGS g, u, P, extra, (T)f, (T)scale, mode, wt, ws, kin_part, uo, (T)dt_upd
#define SU2B_FORCE_LAUNCH(NTV, MB, AN)                                                       \
  do {                                                                                     \
    const dim3 grid(cdiv(g.ncb, NTV / 2));                                                  \
    nb = grid.x;                                                                           \
    cudaError_t e_;                                                                        \
    switch (g.nd) {                                                                        \
      case 2:                                                                              \
        e_ = launch_force(k_force_su2<T, 2, NTV, MB, AN>, grid, NTV, s, pdl, 0,             \
                          SU2B_FORCE_ARGS);                                                \
        break;                                                                             \
      case 3:                                                                              \
        e_ = launch_force(k_force_su2<T, 3, NTV, MB, AN>, grid, NTV, s, pdl, 0,             \
                          SU2B_FORCE_ARGS);                                                \
        break;                                                                             \
      default:                                                                             \
        e_ = launch_force(k_force_su2<T, 4, NTV, MB, AN>, grid, NTV, s, pdl, 0,             \
                          SU2B_FORCE_ARGS);                                                \
        break;                                                                             \
    }                                                                                      \
    if (e_ != cudaSuccess) return e_;                                                      \
  } while (0)
#define SU2B_FORCE_SPLIT(NTV, MB)                                                            \
  do {                                                                                     \
    if (g.nd != 4) {                                                                       \
      SU2B_FORCE_LAUNCH(128, 8, false);                                                    \
      break;                                                                               \
    }                                                                                      \
    const dim3 grid(cdiv(g.ncb, NTV / 4));                                                  \
    nb = grid.x;                                                                           \
    const cudaError_t e_ =                                                                 \
      launch_force(k_force_su2_split<T, NTV, MB>, grid, NTV, s, pdl, 0, SU2B_FORCE_ARGS);     \
    if (e_ != cudaSuccess) return e_;                                                      \
  } while (0)
#define SU2B_FORCE_LINK(MB)                                                                  \
  do {                                                                                     \
    const dim3 grid(2 * cdiv(g.ncb, 32));                                                   \
    nb = grid.x;                                                                           \
    cudaError_t e_;                                                                        \
    switch (g.nd) {                                                                        \
      case 2:                                                                              \
        e_ = launch_force(k_force_su2_link<T, 2, MB>, grid, 64, s, pdl, 0, SU2B_FORCE_ARGS);  \
        break;                                                                             \
      case 3:                                                                              \
        e_ = launch_force(k_force_su2_link<T, 3, MB>, grid, 96, s, pdl, 0, SU2B_FORCE_ARGS);  \
        break;                                                                             \
      default:                                                                             \
        e_ = launch_force(k_force_su2_link<T, 4, MB>, grid, 128, s, pdl, 0, SU2B_FORCE_ARGS); \
        break;                                                                             \
    }                                                                                      \
    if (e_ != cudaSuccess) return e_;                                                      \
  } while (0)
#define SU2B_FORCE_XSPLIT(NTV, MB)                                                           \
  do {                                                                                     \
    if (g.nd != 4) {                                                                       \
      SU2B_FORCE_LAUNCH(128, 8, false);                                                    \
      break;                                                                               \
    }                                                                                      \
    const dim3 grid(cdiv(g.ncb, NTV / 4));                                                  \
    nb = grid.x;                                                                           \
    const cudaError_t e_ =                                                                 \
      launch_force(k_force_su2_xsplit<T, NTV, MB>, grid, NTV, s, pdl, 0, SU2B_FORCE_ARGS);    \
    if (e_ != cudaSuccess) return e_;                                                      \
  } while (0)
    // the anisotropic action (rare) runs one launch shape; the tuned shapes are isotropic and
    // carry no code for the plane weights
    if (aniso) {
      SU2B_FORCE_LAUNCH(128, 6, true);
    } else {
      switch (v) {
        case 0: SU2B_FORCE_LAUNCH(256, 4, false); break;
        case 1: SU2B_FORCE_LAUNCH(128, 8, false); break;
        case 2: SU2B_FORCE_LAUNCH(128, 4, false); break;
        case 3: SU2B_FORCE_LAUNCH(128, 6, false); break;
        case 4: SU2B_FORCE_LAUNCH(256, 2, false); break;
        case 5:
          if (force_planes_apply(g)) {
            const dim3 grid(2 * cdiv(g.ncb, 32));
            nb = grid.x;
            const cudaError_t e_ =
              launch_force(k_force_su2_planes<T>, grid, 384, s, pdl, 0, SU2B_FORCE_ARGS);
            if (e_ != cudaSuccess) return e_;
          } else {
            SU2B_FORCE_LAUNCH(256, 3, false);
          }
          break;
        case 6: SU2B_FORCE_SPLIT(128, 8); break;
        case 8: SU2B_FORCE_XSPLIT(128, 8); break;
        case 9: SU2B_FORCE_LINK(6); break;
        case 10: SU2B_FORCE_SPLIT(128, 5); break;
        case 11: SU2B_FORCE_LINK(6); break;  // site pairs: the standard-layout stand-in
        default: SU2B_FORCE_LAUNCH(64, 16, false); break;
      }
    }
#undef SU2B_FORCE_LAUNCH
#undef SU2B_FORCE_SPLIT
#undef SU2B_FORCE_XSPLIT
#undef SU2B_FORCE_LINK
#undef SU2B_FORCE_ARGS
    if (nblocks) *nblocks = nb;
  } else {
    if (sizeof(T) != 8) return cudaErrorNotSupported;
    const dim3 grid(cdiv(g.Vh, NT), 2 * g.nd);
    if (nblocks) *nblocks = grid.x * grid.y;
    const double *u = (const double *)U;
    double *PP = (double *)P;
    const double *ex = (const double *)extra;
    switch (g.nd) {
      case 2:
        k_force_u1<2, NT><<<grid, NT, 0, s>>>(g, u, PP, ex, f, scale, mode, aniso, 1.0 / xi, xi,
                                              kin_part);
        break;
      case 3:
        k_force_u1<3, NT><<<grid, NT, 0, s>>>(g, u, PP, ex, f, scale, mode, aniso, 1.0 / xi, xi,
                                              kin_part);
        break;
      default:
        k_force_u1<4, NT><<<grid, NT, 0, s>>>(g, u, PP, ex, f, scale, mode, aniso, 1.0 / xi, xi,
                                              kin_part);
        break;
    }
  }
  return cudaGetLastError();
}

template <class T>
cudaError_t link_update(const Geom &g, void *U, int group, const T *P, double dt,
                        cudaStream_t s, double round_dn) {
  const size_t NL = (size_t)g.V * g.nd;
  if (group == 0) {
    if (round_dn > 0.)
      k_update_su2_round<T><<<flat_grid(NL, 256), 256, 0, s>>>(NL, (LinkT<T> *)U, P, (T)dt,
                                                               round_dn);
    else
      k_update_su2<T><<<flat_grid(NL, 256), 256, 0, s>>>(NL, (LinkT<T> *)U, P, (T)dt);
  } else {
    if (sizeof(T) != 8) return cudaErrorNotSupported;
    if (round_dn > 0.)
      k_update_u1_round<<<flat_grid(NL, 256), 256, 0, s>>>(NL, (double *)U, (const double *)P,
                                                           dt, round_dn);
    else
      k_update_u1<<<flat_grid(NL, 256), 256, 0, s>>>(NL, (double *)U, (const double *)P, dt);
  }
  return cudaGetLastError();
}

template <class T>
cudaError_t adj_round_axpy(const Geom &g, T *P, const T *D, int group, double dt, double dn,
                           cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd * (group == 0 ? 3 : 1);
  k_adj_round_axpy<T><<<flat_grid(n, 256), 256, 0, s>>>(n, P, D, dt, dn);
  return cudaGetLastError();
}

template <class T> cudaError_t restore_links(const Geom &g, void *U, int group, cudaStream_t s) {
  if (group != 0) return cudaSuccess;  // u1.hh:178-179
  const size_t NL = (size_t)g.V * g.nd;
  k_restore<T><<<flat_grid(NL, 256), 256, 0, s>>>(NL, (LinkT<T> *)U);
  return cudaGetLastError();
}

template <class T>
cudaError_t momenta_philox(const Geom &g, T *P, int group, const TrajParams *tp,
                           double *kin_part, int *nblocks, cudaStream_t s) {
  constexpr int NT = NT_RED;
  const dim3 grid(cdiv(g.Vh, NT), 2 * g.nd);
  *nblocks = grid.x * grid.y;
  k_momenta<T, NT><<<grid, NT, 0, s>>>(g, P, group == 0 ? 3 : 1, tp, kin_part);
  return cudaGetLastError();
}

template <class T>
cudaError_t momenta_plaq(const Geom &g, const void *U, T *P, const TrajParams *tp, double xi,
                         double *part, int *nblocks, cudaStream_t s, bool plaq) {
  constexpr int NT = 256;
  const dim3 grid(cdiv(g.ncb, NT / 2));
  *nblocks = grid.x;
  const LinkT<T> *u = (const LinkT<T> *)U;
#define SU2B_MP(ND)                                                                          \
  (plaq ? (k_momenta_plaq_su2<T, ND, NT, true><<<grid, NT, 0, s>>>(g, u, P, tp, xi, part), 0) \
        : (k_momenta_plaq_su2<T, ND, NT, false><<<grid, NT, 0, s>>>(g, u, P, tp, xi, part), 0))
  switch (g.nd) {
    case 2: SU2B_MP(2); break;
    case 3: SU2B_MP(3); break;
    default: SU2B_MP(4); break;
  }
#undef SU2B_MP
  return cudaGetLastError();
}

template <class T>
cudaError_t kinetic_partials(const Geom &g, const T *P, int group, double *part, int *nblocks,
                             cudaStream_t s) {
  constexpr int NT = NT_RED;
  const dim3 grid(cdiv(g.Vh, NT), 2 * g.nd);
  *nblocks = grid.x * grid.y;
  k_kinetic<T, NT><<<grid, NT, 0, s>>>(g, P, group == 0 ? 3 : 1, part);
  return cudaGetLastError();
}

template <class T> cudaError_t negate_adj(const Geom &g, T *P, int group, cudaStream_t s) {
  const size_t n = (size_t)g.V * g.nd * (group == 0 ? 3 : 1);
  k_negate<T><<<flat_grid(n, 256), 256, 0, s>>>(n, P);
  return cudaGetLastError();
}

cudaError_t accept_step(const double *red, const TrajParams *tp, TrajDev *out, cudaStream_t s) {
  k_accept<<<1, 1, 0, s>>>(red, tp, out);
  return cudaGetLastError();
}
template <class T>
cudaError_t plaq_accept(const Geom &g, const void *U, double xi, double *part,
                        const TrajTail &e, bool pdl, cudaStream_t s) {
  constexpr int NT = 256;
  const dim3 grid(min(cdiv(g.ncb, NT / 2), 148 * plaq_min_blocks<T, NT>()));
  const LinkT<T> *u = (const LinkT<T> *)U;
  switch (g.nd) {
    case 2: return launch_force(k_plaq_accept_su2<T, 2, NT>, grid, NT, s, pdl, 0, g, u, xi, part, e);
    case 3: return launch_force(k_plaq_accept_su2<T, 3, NT>, grid, NT, s, pdl, 0, g, u, xi, part, e);
    default: return launch_force(k_plaq_accept_su2<T, 4, NT>, grid, NT, s, pdl, 0, g, u, xi, part, e);
  }
}

template <class T>
cudaError_t cond_restore(const Geom &g, void *U, const void *U_old, int group,
                         const TrajDev *flag, cudaStream_t s) {
  const size_t NL = (size_t)g.V * g.nd;
  if (group == 0) {
    // copy as 16-byte words
    const size_t n = NL * sizeof(LinkT<T>) / sizeof(float4);
    k_cond_restore<float4><<<flat_grid(n, 256), 256, 0, s>>>(n, (float4 *)U,
                                                             (const float4 *)U_old, flag);
  } else {
    k_cond_restore<double><<<flat_grid(NL, 256), 256, 0, s>>>(NL, (double *)U,
                                                              (const double *)U_old, flag);
  }
  return cudaGetLastError();
}

#define INST(T)                                                                              \
  template cudaError_t links_from_host<T>(const Geom &, const double *, void *, int,         \
                                          cudaStream_t);                                      \
  template cudaError_t links_to_host<T>(const Geom &, const void *, double *, int,           \
                                        cudaStream_t);                                        \
  template cudaError_t adj_from_host<T>(const Geom &, const double *, T *, int, cudaStream_t); \
  template cudaError_t adj_to_host<T>(const Geom &, const T *, double *, int, cudaStream_t);   \
  template cudaError_t plaq_partials<T>(const Geom &, const void *, int, double, double *,   \
                                        int *, cudaStream_t, Finish);                                 \
  template cudaError_t force_update<T>(const Geom &, const void *, int, T *, const T *,      \
                                       double, double, double, int, double *, int *, void *,  \
                                       double, cudaStream_t, int, bool);                      \
  template cudaError_t link_update<T>(const Geom &, void *, int, const T *, double,          \
                                      cudaStream_t, double);                                  \
  template cudaError_t adj_round_axpy<T>(const Geom &, T *, const T *, int, double, double,  \
                                         cudaStream_t);                                       \
  template cudaError_t restore_links<T>(const Geom &, void *, int, cudaStream_t);            \
  template cudaError_t plaq_accept<T>(const Geom &, const void *, double, double *,          \
                                      const TrajTail &, bool, cudaStream_t);                 \
  template cudaError_t momenta_philox<T>(const Geom &, T *, int, const TrajParams *,         \
                                         double *, int *, cudaStream_t);                      \
  template cudaError_t momenta_plaq<T>(const Geom &, const void *, T *, const TrajParams *,  \
                                       double, double *, int *, cudaStream_t, bool);          \
  template cudaError_t kinetic_partials<T>(const Geom &, const T *, int, double *, int *,    \
                                           cudaStream_t);                                     \
  template cudaError_t negate_adj<T>(const Geom &, T *, int, cudaStream_t);                  \
  template cudaError_t cond_restore<T>(const Geom &, void *, const void *, int,              \
                                       const TrajDev *, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace su2b
