// metropolis.cu -- checkerboard Metropolis pass (flat-sweep.hh:64-164 update rule).
//
// One launch updates every link (x, mu) with parity(x) = p for one direction mu.  Such links
// share no staple: the staple of U_mu(x) contains U_mu(x +- nu) (opposite parity) and links
// of other directions only, so all of them update independently and in any order.  A sweep
// is 2*nd launches.  Per link: staples once (get_staples.hh:26-80), then N_hit proposals
// U -> U R with R = random_element(delta) (random_element.hh:9-34), dS = beta/Nc (ReTr(U K) -
// ReTr(U R K)), accept with min(1, exp(-dS)), restoreSU after each accepted hit.
//   FP64 links: all arithmetic in FP64.
//   FP32 links (mixed precision): the staple sum, the proposal R and the product U R in FP32;
//   the action change dS (the traces of the FP32 values, in FP64), the accept test and the
//   reunitarisation in FP64.
// In both, the accept test u < exp(-dS) goes through accept_fp64, which takes the FP64
// test's decisions (FP32 exp with a guard band, FP64 exp inside the band).  Random numbers:
// one Philox4x32-10 draw per hit, counter {reference link index, hit, sweep, TAG_METRO}:
// 32-bit uniforms for alpha, u, theta and the accept test, the same stream in both
// precisions.
#include <climits>

#include "site_ops.cuh"

namespace su2b {
namespace {

// The FP64 accept test u < exp(-dS) (dS >= 0), decided by FP32 exp where that is safe.  The
// FP32 value differs from the FP64 one by at most the rounding of dS to float (|dS| 2^-24
// relative to the result) plus expf's error (2 ulp); outside a guard band of twice that
// bound the FP32 comparison gives the FP64 decision, inside it (and where expf underflows)
// the test is taken in FP64.  The decisions are those of the FP64 test.
__device__ __forceinline__ bool accept_fp64(double u, double dS) {
  const float ef = expf(-(float)dS);
  if (!(ef > 1e-30f)) return u < exp(-dS);
  const double band = (double)ef * (2.0 * (double)dS * 0x1p-24 + 8.0 * 0x1p-24);
  if (u < (double)ef - band) return true;
  if (u >= (double)ef + band) return false;
  return u < exp(-dS);
}

// restoreSU in FP64 of a product of two unit elements: |u|^2 = 1 + e with e at the rounding of the
// storage precision, and two Newton steps from 1 for its inverse square root leave 1e-20 for
// e up to 2^-16, where a square root and a division cost forty FP64 instructions and the
// longest latency of a hit.  Anything further from 1 (a field uploaded unnormalised) takes those.
__device__ __forceinline__ Su2<double> restore_near(const Su2<double> &u) {
  const double n = fma(u.ar, u.ar, fma(u.ai, u.ai, fma(u.br, u.br, u.bi * u.bi)));
  if (!(fabs(n - 1.0) < 0x1p-16)) return restore_su(u);
  const double y = fma(-0.5, n, 1.5), ir = y * fma(-0.5 * n, y * y, 1.5);
  return Su2<double>{u.ar * ir, u.ai * ir, u.br * ir, u.bi * ir};
}

// random_element (random_element.hh:9-34) of hit n, in the storage precision, and the hit's
// accept uniform
__device__ __forceinline__ Su2<double> proposal(uint32_t lref, int n, uint32_t sweep, uint64_t seed,
                                                double delta, double &accept) {
  uint32_t r[4];
  philox(lref, (uint32_t)n, sweep, TAG_METRO, seed, r);
  double sa, ca, st, ct;
  sincospi(2.0 * delta * u01_32(r[0]), &sa, &ca);
  const double uu = 2.0 * u01_32(r[1]) - 1.0;
  sincospi(2.0 * u01_32(r[2]), &st, &ct);
  const double rr = sqrt(1.0 - uu * uu);
  accept = u01_32(r[3]);
  return Su2<double>{ca, sa * uu, sa * rr * st, sa * rr * ct};
}
__device__ __forceinline__ Su2<float> proposal(uint32_t lref, int n, uint32_t sweep, uint64_t seed,
                                               float delta, double &accept) {
  uint32_t r[4];
  philox(lref, (uint32_t)n, sweep, TAG_METRO, seed, r);
  float sa, ca, st, ct;
  // x 2^-32 rounded once to FP32 (a power of two: as the FP64 uniform rounded); the conversions
  // through FP64 run at a quarter of the rate (32^4 mixed 446 us a sweep instead of 434)
  auto u01 = [](uint32_t x) { return __uint2float_rn(x) * 0x1p-32f; };
  sincospif(2.0f * delta * u01(r[0]), &sa, &ca);
  const float uu = fmaf(2.0f, u01(r[1]), -1.0f);
  sincospif(2.0f * u01(r[2]), &st, &ct);
  const float rr = sqrtf(fmaxf(0.0f, fmaf(-uu, uu, 1.0f)));
  accept = u01_32(r[3]);
  return Su2<float>{ca, sa * uu, sa * rr * st, sa * rr * ct};
}

// the staple sum of U_mu(x) (get_staples.hh:26-80) in the storage precision.  Plain loads: with
// programmatic launches the read-only cache may hold lines from before the previous pass.
template <class T, int ND>
__device__ __forceinline__ Su2<T> staple_sum(const Geom &g, const LinkT<T> *U, const Site &s, int mu,
                                             T wt, T ws) {
  const int p = s.p;
  const int lpm = s.lex + fwd_rt(g, s, mu);  // mu is known at run time only
  Su2<T> K = zero_su2<T>();
#pragma unroll
  for (int nu = 0; nu < ND; nu++) {
    if (nu == mu) continue;
    const int lpn = s.lex + fwd(g, s, nu);
    const Su2<T> A = ld_link_rw(U + (size_t)nu * g.V + eo_of(g, lpm, 1 - p));
    const Su2<T> B = ld_link_rw(U + (size_t)mu * g.V + eo_of(g, lpn, 1 - p));
    const Su2<T> D = ld_link_rw(U + (size_t)nu * g.V + eo_of(g, s.lex, p));
    K = mul_acc(K, scale((nu == 0 || mu == 0) ? wt : ws, mul(A, dag(B))), dag(D));
  }
#pragma unroll
  for (int nu = 0; nu < ND; nu++) {
    if (nu == mu) continue;
    const int b = bwd(g, s, nu);
    const Su2<T> A = ld_link_rw(U + (size_t)nu * g.V + eo_of(g, lpm + b, p));
    const Su2<T> B = ld_link_rw(U + (size_t)mu * g.V + eo_of(g, s.lex + b, 1 - p));
    const Su2<T> D = ld_link_rw(U + (size_t)nu * g.V + eo_of(g, s.lex + b, 1 - p));
    K = mul_acc(K, scale((nu == 0 || mu == 0) ? wt : ws, mul(dag(A), dag(B))), D);
  }
  return K;
}
// hit n: U -> U R with the accept test on dS = beta/Nc (ReTr(U K) - ReTr(U R K))
template <class T>
__device__ __forceinline__ unsigned metro_hit(Su2<T> &u, double &tr_u, const Su2<double> &K64,
                                              const Su2<T> &R, double accept, double beta_nc) {
  const Su2<T> uR = mul(u, R);
  const double dS = beta_nc * (tr_u - retr_mul(to64(uR), K64));
  const Su2<T> v = from64<T>(restore_near(to64(uR)));
  const double tr_v = retr_mul(to64(v), K64);
  if (!(dS < 0 || accept_fp64(accept, dS))) return 0;
  u = v;
  tr_u = tr_v;
  return 1;
}

// a block's accepted hits (one thread of each block); a memset before each sweep and a copy after
// it: 44 us a sweep at 100^2 instead of 41, 70 instead of 64 at 48x40x36
__device__ __forceinline__ void leave_count(const MetroCounts &c, unsigned acc, int mu) {
  if (acc) {
    atomicAdd(c.total, (unsigned long long)acc);
    if (mu == 0) atomicAdd(c.total + 1, (unsigned long long)acc);
  }
  if (!c.out) return;
  __threadfence();
  if (atomicInc(c.ticket, gridDim.x - 1) != gridDim.x - 1) return;
  __threadfence();
  c.out[0] = atomicExch(c.total, 0ull);
  c.out[1] = atomicExch(c.total + 1, 0ull);
}

template <class T, int ND, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
  k_metro_su2(Geom g, LinkT<T> *__restrict__ U, int mu, int p, double beta_nc, double delta,
              int N_hit, uint64_t seed, uint32_t sweep, MetroCounts counts, T wt, T ws) {
  __shared__ unsigned int sh_acc;
  if (threadIdx.x == 0) sh_acc = 0;
  // as pdl_start: the next pass's blocks enter early behind the last wave of several, not
  // beside a single one (a sweep at 16^4 FP64 106 us against 115 us)
  if (gridDim.x > 148u * MINB) pdl_trigger();
  // the sites cb0 .. cb0 + ncb - 1 of parity p (all of them but in a time slab)
  const int cb = g.cb0 + blockIdx.x * NT + threadIdx.x;
  const bool on = cb < g.cb0 + g.ncb;
  const Site s = site_from_eo(g, p, on ? cb : g.cb0);
  const uint32_t lref = (uint32_t)(s.lex + g.lex0) * (uint32_t)g.nd + (uint32_t)mu;
  double ua;
  Su2<T> R = proposal(lref, 0, sweep, seed, (T)delta, ua);
  pdl_wait();  // the previous pass's links
  __syncthreads();
  unsigned int acc = 0;
  if (on) {
    const Su2<T> K = staple_sum<T, ND>(g, U, s, mu, wt, ws);
    const Su2<double> K64 = to64(K);
    const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
    Su2<T> u = ld_link_rw(U + l);
    double tr_u = retr_mul(to64(u), K64);
    for (int n = 0; n < N_hit; n++) {
      const Su2<T> Rn = R;
      const double un = ua;
      if (n + 1 < N_hit) R = proposal(lref, n + 1, sweep, seed, (T)delta, ua);
      acc += metro_hit(u, tr_u, K64, Rn, un, beta_nc);
    }
    st_link(U + l, u);
  }
  if (acc) atomicAdd(&sh_acc, acc);
  __syncthreads();
  if (threadIdx.x == 0) leave_count(counts, sh_acc, mu);
}

// The same for passes of few links, which the chain of a link's hits bounds: a block of eight
// warps takes 32 links; all warps draw proposals (they depend on nothing but the hit) into
// shared memory, sixteen hits at a time and the first ones while the previous pass still runs,
// and warp 0 applies them.  At 100^2, ten hits: 47 us per sweep, 57 us with
// one thread per link (65 us before the chain of a hit lost its square root and division and the
// passes their launch gaps).
constexpr int WIDE_HITS = 16;
// chunks of N hits and the hits of chunk c < chunks, in the range of int for every N
__host__ __device__ constexpr int wide_chunks(int N) {
  return N / WIDE_HITS + (N % WIDE_HITS != 0);
}
__host__ __device__ constexpr int wide_hits(int c, int N) {
  return N - c * WIDE_HITS < WIDE_HITS ? N - c * WIDE_HITS : WIDE_HITS;
}
static_assert(wide_chunks(0) == 0 && wide_chunks(16) == 1 && wide_chunks(17) == 2 &&
              wide_hits(0, 16) == 16 && wide_hits(1, 17) == 1, "chunks of sixteen hits");
static_assert(wide_chunks(INT_MAX) == INT_MAX / WIDE_HITS + 1 &&
              wide_hits(wide_chunks(INT_MAX) - 1, INT_MAX) == INT_MAX % WIDE_HITS,
              "the last chunk of the most hits, whose successor's first hit is no int");
template <class T, int ND>
__global__ void __launch_bounds__(256, 2)
  k_metro_su2_wide(Geom g, LinkT<T> *__restrict__ U, int mu, int p, double beta_nc, double delta,
                   int N_hit, uint64_t seed, uint32_t sweep, MetroCounts counts, T wt,
                   T ws) {
  __shared__ LinkT<T> prop[2][WIDE_HITS][32];
  __shared__ double acc_u[2][WIDE_HITS][32];
  pdl_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int cb = g.cb0 + blockIdx.x * 32 + lane;
  const bool on = cb < g.cb0 + g.ncb;
  const Site s = site_from_eo(g, p, on ? cb : g.cb0);
  const uint32_t lref = (uint32_t)(s.lex + g.lex0) * (uint32_t)g.nd + (uint32_t)mu;
  const int chunks = wide_chunks(N_hit);
  auto draw = [&](int chunk, int first, int step) {
    if (chunk >= chunks) return;
    const int n = wide_hits(chunk, N_hit);
    for (int i = first; i < n; i += step)
      prop[chunk & 1][i][lane] = as_link(proposal(lref, chunk * WIDE_HITS + i, sweep, seed, (T)delta,
                                                  acc_u[chunk & 1][i][lane]));
  };
  draw(0, w, 8);
  pdl_wait();  // the previous pass's links
  const size_t l = (size_t)mu * g.V + s.p * (size_t)g.Vh + (s.lex >> 1);
  Su2<T> u;
  Su2<double> K64;
  double tr_u = 0.;
  if (w == 0) {
    u = ld_link_rw(U + l);
    K64 = to64(staple_sum<T, ND>(g, U, s, mu, wt, ws));
    tr_u = retr_mul(to64(u), K64);
  }
  unsigned acc = 0;
  for (int c = 0; c < chunks; c++) {
    __syncthreads();
    if (w == 0) {
      const int n = wide_hits(c, N_hit);
      for (int i = 0; i < n; i++)
        acc += metro_hit(u, tr_u, K64, from_link(prop[c & 1][i][lane]), acc_u[c & 1][i][lane],
                         beta_nc);
    } else {
      draw(c + 1, w - 1, 7);
    }
  }
  if (w) return;
  if (on)
    st_link(U + l, u);
  else
    acc = 0;
  acc = __reduce_add_sync(0xffffffffu, acc);
  if (lane == 0) leave_count(counts, acc, mu);
}

template <int ND, int NT>
__global__ void __launch_bounds__(NT)
  k_metro_u1(Geom g, double *__restrict__ U, int mu, int p, double beta, double delta,
             int N_hit, uint64_t seed, uint32_t sweep, MetroCounts counts, double wt,
             double ws) {
  __shared__ unsigned int sh_acc;
  if (threadIdx.x == 0) sh_acc = 0;
  __syncthreads();
  const int cb = blockIdx.x * NT + threadIdx.x;
  unsigned int acc = 0;
  if (cb < g.Vh) {
    const Site s = site_from_eo(g, p, cb);
    const int lpm = s.lex + fwd_rt(g, s, mu);  // mu is known at run time only
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
      const double w = (nu == 0 || mu == 0) ? wt : ws;
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
      const double w = (nu == 0 || mu == 0) ? wt : ws;
      Kr += w * cs;
      Ki += w * sn;
    }
    const size_t l = (size_t)mu * g.V + (size_t)p * g.Vh + cb;
    double u = U[l];
    const uint32_t lref = (uint32_t)s.lex * (uint32_t)g.nd + (uint32_t)mu;
    for (int n = 0; n < N_hit; n++) {
      uint32_t r[4];
      philox(lref, (uint32_t)n, sweep, TAG_METRO, seed, r);
      const double th = M_PI * delta * (2.0 * u01_32(r[0]) - 1.0);
      double s0, c0, s1, c1;
      sincospi(u * M_1_PI_D, &s0, &c0);
      sincospi((u + th) * M_1_PI_D, &s1, &c1);
      const double dS = beta * ((c0 * Kr - s0 * Ki) - (c1 * Kr - s1 * Ki));
      bool a = dS < 0;
      if (!a) a = u01_32(r[1]) < exp(-dS);
      if (a) {
        u = u + th;
        acc++;
      }
    }
    U[l] = u;
  }
  if (acc) atomicAdd(&sh_acc, acc);
  __syncthreads();
  if (threadIdx.x == 0) leave_count(counts, sh_acc, mu);
}

}  // namespace

template <class T>
cudaError_t metropolis_pass(const Geom &g, void *U, int group, int mu, int parity, double beta,
                            double xi, double delta, int N_hit, uint64_t seed, uint32_t sweep,
                            const MetroCounts &counts, cudaStream_t s) {
  constexpr int NT = 128, MINB = 8;
  // anisotropic weights of get_staples (get_staples.hh:58-79): 1/xi for planes with
  // direction 0, xi otherwise; both 1 (exactly) for the isotropic action
  const double wt = xi == 1.0 ? 1.0 : 1.0 / xi, ws = xi;
  const int grid = ((group == 0 ? g.ncb : g.Vh) + NT - 1) / NT;
  if (group == 0) {
    LinkT<T> *u = (LinkT<T> *)U;
    const double bn = beta / 2.0;
    // up to two blocks of 32 links per SM the chain of a link's hits bounds a pass (10^4, eight
    // hits: 73 us per sweep against 95 us); at 12^4, 10,368 links, the eight warps of a block
    // cost more than they hide (109 us against 103 us)
    const bool wide = g.ncb <= 2 * 148 * 32;
#define SU2B_METRO(ND)                                                                     \
  (wide ? launch_force(k_metro_su2_wide<T, ND>, dim3((g.ncb + 31) / 32), 256, s, true, 0, g, u, mu, \
                       parity, bn, delta, N_hit, seed, sweep, counts, (T)wt, (T)ws)        \
        : launch_force(k_metro_su2<T, ND, NT, MINB>, dim3(grid), NT, s, true, 0, g, u, mu, parity, bn, \
                       delta, N_hit, seed, sweep, counts, (T)wt, (T)ws))
    switch (g.nd) {
      case 2: return SU2B_METRO(2);
      case 3: return SU2B_METRO(3);
      default: return SU2B_METRO(4);
    }
#undef SU2B_METRO
  }
  double *u = (double *)U;
  switch (g.nd) {
    case 2:
      k_metro_u1<2, NT><<<grid, NT, 0, s>>>(g, u, mu, parity, beta, delta, N_hit, seed, sweep,
                                            counts, wt, ws);
      break;
    case 3:
      k_metro_u1<3, NT><<<grid, NT, 0, s>>>(g, u, mu, parity, beta, delta, N_hit, seed, sweep,
                                            counts, wt, ws);
      break;
    default:
      k_metro_u1<4, NT><<<grid, NT, 0, s>>>(g, u, mu, parity, beta, delta, N_hit, seed, sweep,
                                            counts, wt, ws);
      break;
  }
  return cudaGetLastError();
}

template cudaError_t metropolis_pass<double>(const Geom &, void *, int, int, int, double, double,
                                             double, int, uint64_t, uint32_t,
                                             const MetroCounts &, cudaStream_t);
template cudaError_t metropolis_pass<float>(const Geom &, void *, int, int, int, double, double,
                                            double, int, uint64_t, uint32_t,
                                            const MetroCounts &, cudaStream_t);

}  // namespace su2b
