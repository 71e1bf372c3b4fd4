// cg_tile.cu -- the CG on D D^+ and the BiCGStab on D for two-dimensional lattices, the whole
// solve in one launch with the lattice held in registers and shared memory.
//
// A block owns a tile of the lattice, a thread K of its sites: p, x, r, t = D^+ p and b live in
// registers for the whole solve.  A phase needs two things from the other blocks, the vector's
// values beside the tile and the sum of the blocks' partials; the rest of its time is FP64
// latency (a division, two tree sums, a stencil: about 1,000 cycles).  Two forms:
//   k_cg_cluster, up to 16,384 sites: the blocks are one thread-block cluster and push both into
//     each other's shared memory.  1,800 cycles a phase at 64^2: 0.76 ms a solve of 414
//     iterations, where k_cg_persistent (staggered.cu: a grid barrier a phase) takes 3.56 ms.
//   k_cg_tile, up to about 150,000 sites: blocks over the whole GPU.  Both travel as 16-byte
//     packets {64 bits of data, epoch} in global memory that the receiver polls until the epoch
//     of the phase arrives: the data come with their own arrival flag, so no barrier, no memory
//     fence and no second read follow, and the stencil runs while the partials travel.  An L2
//     round trip or two bound it: 4,300 cycles a phase at 256^2, 1.96 ms for 443 iterations
//     against 4.40 ms.
//
// The iteration, the convergence tests and the true-residual restart are those of cg64
// (solve.cu, CG.hpp:36-94), with <p, A p> = |D^+ p|^2 and D^+ p carried by linearity:
//   A: publish t;  alpha = rr / |t|^2;  x += alpha p;  r -= alpha D t
//   B: publish r;  beta = |r|^2 / rr;  p = r + beta p;  t = D^+ r + beta t
// The BiCGStab on D runs on the same tiles in three phases an iteration (bi_run), mass 0.05 to
// 1e-12: 2.8 ms for 717 iterations at 64^2 where k_bicgstab_persistent takes 9.4 ms for 723,
// 7.3 ms at 256^2 against 11.9 ms.
// Every block adds the partials in the same order, so all take the same decisions.  Every wait
// is bounded: one that gives up tells the host, and all blocks return, those that the missing
// data were meant for when their own waits run out, a second later at most.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "solver.h"
#include "su2b_internal.h"

namespace su2b {
namespace {

constexpr int MAX_THREADS = 512;
constexpr int MAX_BLOCKS = 160;  // partials a warp polls: 5 per lane
constexpr int BI_SUMS = 5;  // sums of one phase at most: the BiCGStab's (the CG: 1)
// When a wait gives up, after about a second: k_cg_tile counts its polls, an L2 round trip each;
// k_cg_cluster's try_wait suspends the thread for a time of the hardware's choosing (TRY_NS is a
// hint), so there the clock is read.
constexpr long POLL_LIMIT = 1L << 21, CYCLE_LIMIT = 2000000000L;
constexpr unsigned TRY_NS = 1000000;

__device__ __forceinline__ void put_packet(ulonglong2 *p, double v, unsigned long long epoch) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}"
               ::"l"(p), "l"(__double_as_longlong(v)), "l"(epoch)
               : "memory");
}
// one poll of a packet where `want` is set: its data into v and want cleared if the epoch is there
__device__ __forceinline__ void poll_issue(const ulonglong2 *p, int want, unsigned long long &a,
                                           unsigned long long &e) {
  asm volatile("{\n\t.reg .pred w;\n\t.reg .b128 q;\n\tsetp.ne.s32 w, %3, 0;\n\tmov.b128 q, {%0, %1};\n\t"
               "@w ld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "+l"(a), "+l"(e)
               : "l"(p), "r"(want)
               : "memory");
}

struct CgTileArgs {
  Geom g;
  CgTilePlan tp;
  const double2 *ph;
  double m;
  const double2 *b;
  double2 *x;
  ulonglong2 *halo;  // [2][V][2] packets: a boundary site's value by epoch parity
  ulonglong2 *sums;  // [2][BI_SUMS][MAX_BLOCKS], alternating from phase to phase with sums
  unsigned long long epoch;  // last epoch used by earlier solves
  CgTileResult *out;
  int *err;
  double tol;
  long max_iter;
  long limit;  // POLL_LIMIT or CYCLE_LIMIT; a test sets 0, and every wait of a cluster runs out
};

// m v + sgn hop(v) at a site of slice t: the arithmetic of hop_site64 (staggered.cu) in d = 2.
// uf: the phases of the site's links, ub: of the links behind it; f / b: the neighbours' values
__device__ __forceinline__ double2 hop2(double m, double sgn, double2 v, const double2 (&uf)[2],
                                        const double2 (&ub)[2], double2 tf, double2 tb, double2 xf,
                                        double2 xb, int t) {
  double ar = 0, ai = 0;
  auto dir = [&](double eta, double2 u, double2 w, double2 fp, double2 fm) {
    const double tr = (u.x * fp.x - u.y * fp.y) - (w.x * fm.x + w.y * fm.y);
    const double ti = (u.x * fp.y + u.y * fp.x) - (w.x * fm.y - w.y * fm.x);
    ar += eta * tr;
    ai += eta * ti;
  };
  dir(0.5, uf[0], ub[0], tf, tb);
  dir((t & 1) ? -0.5 : 0.5, uf[1], ub[1], xf, xb);
  return make_double2(m * v.x + sgn * ar, m * v.y + sgn * ai);
}

// The solve on any tiling.  phase<N sums, hop>(v, sgn, out, part, total): out = m v + sgn hop(v)
// where hop is set, and the lattice's sums of part[0..N-1] into total; false: give up.
template <int N> using Sums = std::integral_constant<int, N>;
using Hop = std::true_type;
using NoHop = std::false_type;
struct CgEnd {
  double rn, ex;
  long iters, restarts;
  int done;
};
template <int K, class Phase>
__device__ __forceinline__ bool cg_run(const bool (&on)[K], double2 (&x)[K], const double2 (&b)[K],
                                       double tol, long max_iter, Phase &&phase_n, CgEnd &end) {
  auto phase = [&](const double2 (&v)[K], double sgn, double2 (&out)[K], bool sum, double part,
                   double &total) {
    return sum ? phase_n(Sums<1>(), Hop(), v, sgn, out, &part, &total)
               : phase_n(Sums<0>(), Hop(), v, sgn, out, &part, &total);
  };
  double2 r[K], p[K], t[K], w[K], aw[K];
  auto norm = [&](const double2 (&v)[K]) {
    double s = 0.;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (on[k]) s += v[k].x * v[k].x + v[k].y * v[k].y;
    return s;
  };

  const double near = tol * tol * (1. + 1e-12);  // |r|^2 above it: |r| > tol
  double total = 0., rr = 0., rn = 0., ex = 0.;
  long iters = 0, restarts = 0;
  int done = 0;
#pragma unroll
  for (int k = 0; k < K; k++) w[k] = aw[k] = r[k] = p[k] = t[k] = make_double2(0., 0.);
  for (bool start = true;; start = false) {
    // the true residual b - D D^+ x
    if (!phase(x, -1., w, false, 0., total)) return false;
    if (!phase(w, 1., aw, false, 0., total)) return false;
#pragma unroll
    for (int k = 0; k < K; k++) w[k] = make_double2(b[k].x - aw[k].x, b[k].y - aw[k].y);
    // its norm and D^+ of it (the first t if a CG starts from it)
    if (!phase(w, -1., aw, true, norm(w), total)) return false;
    ex = sqrt(total);
    if (!start) {
      // converged: restart from x while the iterated residual is below the true one
      if (!(rn < ex && iters < max_iter)) break;
      restarts++;
    }
    rr = total;
    rn = ex;
    if (!(rn > tol)) {
      done = 1;
      break;
    }
    done = 0;
#pragma unroll
    for (int k = 0; k < K; k++) p[k] = r[k] = w[k], t[k] = aw[k];
    while (!done) {
      if (!phase(t, 1., aw, true, norm(t), total)) return false;
      const double alpha = rr / total;
#pragma unroll
      for (int k = 0; k < K; k++) {
        x[k].x += alpha * p[k].x, x[k].y += alpha * p[k].y;
        r[k].x -= alpha * aw[k].x, r[k].y -= alpha * aw[k].y;
      }
      if (!phase(r, -1., w, true, norm(r), total)) return false;
      const double beta = total / rr;
      rr = total;
      iters++;
      // |r| itself (a square root's latency) only where it is near the tolerance or wanted
      if (!(total > near) || iters >= max_iter) {
        rn = sqrt(total);
        if (rn != rn) done = 3;
        else if (!(rn > tol)) done = 1;
        else if (iters >= max_iter) done = 2;
        if (done) break;
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        p[k] = make_double2(r[k].x + beta * p[k].x, r[k].y + beta * p[k].y);
        t[k] = make_double2(w[k].x + beta * t[k].x, w[k].y + beta * t[k].y);
      }
    }
    if (done != 1) break;
  }
  end = CgEnd{rn, ex, iters, restarts, done};
  return true;
}

// BiCGStab on D (BiCGStab.hpp:36-106, the iteration of bicgstab64 in solve.cu), three phases each:
//   A: publish p;  v = D p;  <r0, v> = <D^+ r0, p>, which needs no v;  |r|^2 of the last iteration
//   B: publish s = r - alpha v;  t = D s;  <r0, s>
//   C: sums alone: <t, s>, |t|^2, <r0, t>;  omega;  x += alpha p + omega s;  r = s - omega t;
//      <r0, r> = <r0, s> - omega <r0, t>;  beta;  p = r + beta p - beta omega v
// D p and D s are applied directly, not carried by recurrences.  A step's |r|^2 arrives with the
// next step's phase A, which is where it is looked at.
template <int K, class Phase>
__device__ __forceinline__ bool bi_run(const bool (&on)[K], double2 (&x)[K], const double2 (&b)[K],
                                       double tol, long max_iter, Phase &&phase, CgEnd &end) {
  double2 r[K], p[K], v[K], t[K], r0[K], w0[K];
  // <a, c> over the thread's sites
  auto dot = [&](const double2 (&a)[K], const double2 (&c)[K], double *re, double *im) {
    double sr = 0., si = 0.;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (on[k]) {
        sr += a[k].x * c[k].x + a[k].y * c[k].y;
        if (im) si += a[k].x * c[k].y - a[k].y * c[k].x;
      }
    *re = sr;
    if (im) *im = si;
  };
  double part[BI_SUMS], sum[BI_SUMS];
  double rn = 0., ex = 0.;
  long iters = 0, restarts = 0;
  int done = 0;
#pragma unroll
  for (int k = 0; k < K; k++) r[k] = p[k] = v[k] = t[k] = r0[k] = w0[k] = make_double2(0., 0.);
  for (bool start = true;; start = false) {
    // the true residual b - D x, its norm and D^+ of it
    if (!phase(Sums<0>(), Hop(), x, 1., v, part, sum)) return false;
#pragma unroll
    for (int k = 0; k < K; k++) r0[k] = make_double2(b[k].x - v[k].x, b[k].y - v[k].y);
    dot(r0, r0, part, nullptr);
    if (!phase(Sums<1>(), Hop(), r0, -1., w0, part, sum)) return false;
    ex = sqrt(sum[0]);
    if (!start) {
      if (!(rn < ex && iters < max_iter)) break;
      restarts++;
    }
    rn = ex;
    if (!(rn > tol)) {
      done = 1;
      break;
    }
    done = 0;
    double2 rho = make_double2(sum[0], 0.);
#pragma unroll
    for (int k = 0; k < K; k++) r[k] = p[k] = r0[k];
    for (bool first = true;; first = false) {
      dot(w0, p, part, part + 1);
      dot(r, r, part + 2, nullptr);
      if (!phase(Sums<3>(), Hop(), p, 1., v, part, sum)) return false;
      if (!first) {
        rn = sqrt(sum[2]);
        if (rn != rn) done = 3;
        else if (!(rn > tol)) done = 1;
        else if (iters >= max_iter) done = 2;
        if (done) break;
      }
      const double2 alpha = cdivs(rho, make_double2(sum[0], sum[1]));
#pragma unroll
      for (int k = 0; k < K; k++) {
        const double2 av = cm(alpha, v[k]);
        r[k] = make_double2(r[k].x - av.x, r[k].y - av.y);
      }
      dot(r0, r, part, part + 1);
      if (!phase(Sums<2>(), Hop(), r, 1., t, part, sum)) return false;
      const double2 r0s = make_double2(sum[0], sum[1]);
      dot(t, r, part, part + 1);
      dot(t, t, part + 2, nullptr);
      dot(r0, t, part + 3, part + 4);
      if (!phase(Sums<5>(), NoHop(), r, 1., t, part, sum)) return false;
      const double2 omega = make_double2(sum[0] / sum[2], sum[1] / sum[2]);
      const double2 ot = cm(omega, make_double2(sum[3], sum[4]));
      const double2 next = make_double2(r0s.x - ot.x, r0s.y - ot.y);
      const double2 beta = cm(cdivs(next, rho), cdivs(alpha, omega));
      const double2 bo = cm(beta, omega);
      rho = next;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const double2 ap = cm(alpha, p[k]), os = cm(omega, r[k]), wt = cm(omega, t[k]);
        x[k] = make_double2(x[k].x + os.x + ap.x, x[k].y + os.y + ap.y);
        r[k] = make_double2(r[k].x - wt.x, r[k].y - wt.y);
        const double2 bp = cm(beta, p[k]), bv = cm(bo, v[k]);
        p[k] = make_double2(r[k].x + bp.x - bv.x, r[k].y + bp.y - bv.y);
      }
      iters++;
    }
    if (done != 1) break;
  }
  end = CgEnd{rn, ex, iters, restarts, done};
  return true;
}

__device__ __forceinline__ void write_result(CgTileResult *out, const CgEnd &e,
                                             unsigned long long epoch) {
  out->rn = e.rn;
  out->true_residual = e.done == 1 ? e.ex : 0.;
  out->iters = e.iters;
  out->restarts = e.restarts;
  out->done = e.done;
  out->epoch = epoch;
}

template <int K, bool BI>
__global__ void __launch_bounds__(MAX_THREADS, 1) k_cg_tile(CgTileArgs a) {
  constexpr int NSM = BI ? BI_SUMS : 1;
  __shared__ double2 tile[K * MAX_THREADS];
  __shared__ double shw[NSM][MAX_THREADS / 32];
  __shared__ double sh_sum[NSM];
  __shared__ int sh_bad;
  const CgTilePlan tp = a.tp;
  const int Lt = a.g.L[0], Lx = a.g.L[1], V = a.g.V, Vh = a.g.Vh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = (blockDim.x + 31) >> 5;
  const int bt = blockIdx.x / tp.gx, bx = blockIdx.x - bt * tp.gx;
  const int t0 = bt * tp.ht, x0 = bx * tp.hx;
  const int rows = min(tp.ht, Lt - t0), cols = min(tp.hx, Lx - x0);
  const int c = tid % tp.hx, r0 = tid / tp.hx;  // threads past the tile have r0 >= rp
  if (tid == 0) sh_bad = 0;

  bool on[K];
  double2 uf[K][2], ub[K][2];  // e^{i th} of the site's links and of the links behind it
  double2 x[K], b[K];
  const int xc = x0 + c;
  const int xf = xc + 1 == Lx ? 0 : xc + 1, xb = xc == 0 ? Lx - 1 : xc - 1;
  auto eo = [&](int tt, int xx) { return ((tt + xx) & 1) * Vh + ((tt * Lx + xx) >> 1); };
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int row = r0 + k * tp.rp, tt = t0 + row;
    on[k] = r0 < tp.rp && row < rows && c < cols;
    const int tc = on[k] ? tt : t0, xx = on[k] ? xc : x0;
    const int s = eo(tc, xx);
    uf[k][0] = a.ph[s], uf[k][1] = a.ph[V + s];
    ub[k][0] = a.ph[eo(tc == 0 ? Lt - 1 : tc - 1, xx)];
    ub[k][1] = a.ph[V + eo(tc, xx == 0 ? Lx - 1 : xx - 1)];
    x[k] = a.x[s], b[k] = a.b[s];
  }
  unsigned long long ep = a.epoch;
  unsigned nsum = 0;

  // waits for N packets at once (their loads are in flight together); want: which of them
  auto wait = [&](auto n, const ulonglong2 *const *q, unsigned want, double *v) {
    constexpr int N = decltype(n)::value;
    long spins = 0;
    while (want) {
      unsigned long long d[N], e[N];
#pragma unroll
      for (int j = 0; j < N; j++) d[j] = e[j] = 0, poll_issue(q[j], want >> j & 1, d[j], e[j]);
#pragma unroll
      for (int j = 0; j < N; j++)
        if ((want >> j & 1) && e[j] == ep) v[j] = __longlong_as_double((long long)d[j]), want &= ~(1u << j);
      spins++;
      if (spins > a.limit || ((spins & 255) == 0 && *(volatile int *)a.err)) {
        atomicExch(a.err, 1);
        *(volatile int *)&a.out->failed = 1;
        sh_bad = 1;
        return;
      }
    }
  };
  // One phase: v to the neighbours, out = m v + sgn hop(v); the sums of part[] over the lattice
  // (out's stencil runs meanwhile), each by a warp of its own.  false: a wait gave up.
  auto phase = [&](auto ns, auto hop, const double2 (&v)[K], double sgn, double2 (&out)[K],
                   const double *part, double *total) -> bool {
    constexpr int NS = decltype(ns)::value;
    constexpr bool HOP = decltype(hop)::value;
    ep++;
    ulonglong2 *const hb = a.halo + (size_t)(ep & 1) * 2 * V;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int row = r0 + k * tp.rp;
      if (!HOP || !on[k]) continue;
      tile[row * tp.hx + c] = v[k];
      if ((tp.gt > 1 && (row == 0 || row == rows - 1)) || (tp.gx > 1 && (c == 0 || c == cols - 1))) {
        ulonglong2 *q = hb + 2 * ((t0 + row) * Lx + xc);
        put_packet(q, v[k].x, ep);
        put_packet(q + 1, v[k].y, ep);
      }
    }
#pragma unroll
    for (int j = 0; j < NS; j++) {
      double s = part[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) shw[j][warp] = s;
    }
    __syncthreads();
    if (NS) nsum++;
    ulonglong2 *const sb = a.sums + (size_t)(nsum & 1) * BI_SUMS * MAX_BLOCKS;
    for (int j = warp; j < NS; j += nw) {
      double s = lane < nw ? shw[j][lane] : 0.;
#pragma unroll
      for (int o = MAX_THREADS / 64; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) put_packet(sb + j * MAX_BLOCKS + blockIdx.x, s, ep);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (!HOP || !on[k]) continue;
      const int row = r0 + k * tp.rp, tt = t0 + row;
      // forward and backward in t, then in x: inside the tile (or around the lattice in it)
      // from shared memory, else from its packets
      const int tf = tt + 1 == Lt ? 0 : tt + 1, tb = tt == 0 ? Lt - 1 : tt - 1;
      const bool rem[4] = {row + 1 == rows && tp.gt > 1, row == 0 && tp.gt > 1,
                           c + 1 == cols && tp.gx > 1, c == 0 && tp.gx > 1};
      const int src[4] = {(row + 1 < rows ? row + 1 : 0) * tp.hx + c,
                          (row > 0 ? row - 1 : rows - 1) * tp.hx + c,
                          row * tp.hx + (c + 1 < cols ? c + 1 : 0),
                          row * tp.hx + (c > 0 ? c - 1 : cols - 1)};
      const ulonglong2 *q[8];
      double w[8];
      unsigned want = 0;
      const int far[4] = {tf * Lx + xc, tb * Lx + xc, tt * Lx + xf, tt * Lx + xb};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        q[2 * j] = hb + 2 * far[j], q[2 * j + 1] = q[2 * j] + 1;
        const double2 in = tile[src[j]];
        w[2 * j] = in.x, w[2 * j + 1] = in.y;
        if (rem[j]) want |= 3u << (2 * j);
      }
      wait(std::integral_constant<int, 8>(), q, want, w);
      const double2 vtf = make_double2(w[0], w[1]), vtb = make_double2(w[2], w[3]),
                    vxf = make_double2(w[4], w[5]), vxb = make_double2(w[6], w[7]);
      out[k] = hop2(a.m, sgn, v[k], uf[k], ub[k], vtf, vtb, vxf, vxb, tt);
    }
    for (int i = warp; i < NS; i += nw) {
      constexpr int N = MAX_BLOCKS / 32;
      const ulonglong2 *src[N];
      double q[N], s = 0.;
      unsigned want = 0;
#pragma unroll
      for (int j = 0; j < N; j++) {
        q[j] = 0.;
        src[j] = sb + i * MAX_BLOCKS + lane + 32 * j;
        if (lane + 32 * j < (int)gridDim.x) want |= 1u << j;
      }
      wait(std::integral_constant<int, N>(), src, want, q);
#pragma unroll
      for (int j = 0; j < N; j++) s += q[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) sh_sum[i] = s;
    }
    __syncthreads();  // the sums are in; the tile may be rewritten
#pragma unroll
    for (int j = 0; j < NS; j++) total[j] = sh_sum[j];
    return sh_bad == 0;
  };
  CgEnd end;
  const bool good = BI ? bi_run<K>(on, x, b, a.tol, a.max_iter, phase, end)
                       : cg_run<K>(on, x, b, a.tol, a.max_iter, phase, end);
  if (!good) return;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (on[k]) a.x[eo(t0 + r0 + k * tp.rp, xc)] = x[k];
  if (blockIdx.x == 0 && tid == 0) write_result(a.out, end, ep);
}

// The same on one thread-block cluster (up to 16 blocks, 16,384 sites).  Each block pushes its
// rim into its neighbours' shared memory and its partial into every block's, with st.async: the
// stores count on a barrier (mbarrier) of the receiving block, whose wait is the only one of a
// phase besides the block's own.  (The cluster's barrier instruction took 1,000 to 1,400 of the
// 2,600 cycles of a phase at 64^2; partials by warp instead of by block, 128 stores into each
// barrier, as much.)  Every phase carries the sum, so no block is two phases ahead of another
// and two buffers alternate.
constexpr int MAX_CLUSTER = 16;
constexpr int MAX_RIM = 320;  // rim values of a tile, 2 (ht + hx)
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ double2 lds(uint32_t a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
template <int K, bool BI> struct ClusterBuf {
  static constexpr int NSM = BI ? BI_SUMS : 1;
  double2 tile[K * MAX_THREADS];
  double2 rim[MAX_RIM];        // t forward, t backward, x forward, x backward
  double thr[NSM][MAX_THREADS];   // the threads' partials
  double part[NSM][MAX_CLUSTER];  // the blocks' partials
  unsigned long long bar;
};
template <int K, bool BI>
__global__ void __launch_bounds__(MAX_THREADS, 1) k_cg_cluster(CgTileArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Buf = ClusterBuf<K, BI>;
  Buf *const B = (Buf *)smem;
  constexpr uint32_t STEP = sizeof(Buf);
  __shared__ unsigned sh_bad;  // the phase in which a wait gave up
  const CgTilePlan tp = a.tp;
  const int Lt = a.g.L[0], Lx = a.g.L[1], V = a.g.V, Vh = a.g.Vh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int nb = gridDim.x;  // one cluster
  const int bt = blockIdx.x / tp.gx, bx = blockIdx.x - bt * tp.gx;
  const int t0 = bt * tp.ht, x0 = bx * tp.hx;
  const int rows = max(0, min(tp.ht, Lt - t0)), cols = min(tp.hx, Lx - x0);
  const int c = tid % tp.hx, r0 = tid / tp.hx, xc = x0 + c;
  auto saddr = [](const void *q) { return (uint32_t)__cvta_generic_to_shared(q); };
  if (tid == 0) {
    sh_bad = ~0u;
#pragma unroll
    for (int k = 0; k < 2; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&B[k].bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 2 * Buf::NSM * MAX_CLUSTER; i += blockDim.x)
    B[i / (Buf::NSM * MAX_CLUSTER)].part[0][i % (Buf::NSM * MAX_CLUSTER)] = 0.;
  const uint32_t my_bar = saddr(&B[0].bar);
  // this block's slot in the partials of block `lane`, and that block's barrier
  const int peer = lane < nb ? lane : 0;
  const uint32_t mine = cluster_addr(saddr(&B[0].part[0][blockIdx.x]), peer);
  const uint32_t peer_bar = cluster_addr(my_bar, peer);
  // bytes of a phase besides the sums
  const int rims =
    rows > 0 ? 16 * ((tp.gt > 1 ? 2 * cols : 0) + (tp.gx > 1 ? 2 * rows : 0)) : 0;

  bool on[K];
  double2 uf[K][2], ub[K][2], x[K], b[K];
  uint32_t own[K], src[K][4];         // the site's value and its neighbours' in buffer 0
  uint32_t dst[K][2], dbar[K][2];     // where the value goes: along t, along x (0: nowhere)
  uint32_t dst2[K], dbar2[K];         // a tile one row or column wide sends to both sides
  auto eo = [&](int tt, int xx) { return ((tt + xx) & 1) * Vh + ((tt * Lx + xx) >> 1); };
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int row = r0 + k * tp.rp;
    on[k] = r0 < tp.rp && row < rows && c < cols;
    const int rr = on[k] ? row : 0, cc = on[k] ? c : 0;
    const int tt = on[k] ? t0 + row : 0, xx = on[k] ? xc : 0;
    const int s = eo(tt, xx);
    uf[k][0] = a.ph[s], uf[k][1] = a.ph[V + s];
    ub[k][0] = a.ph[eo(tt == 0 ? Lt - 1 : tt - 1, xx)];
    ub[k][1] = a.ph[V + eo(tt, xx == 0 ? Lx - 1 : xx - 1)];
    x[k] = a.x[s], b[k] = a.b[s];
    const double2 *const T = B[0].tile, *const Q = B[0].rim;
    const int hx = tp.hx, ht = tp.ht;
    own[k] = saddr(T + rr * hx + cc);
    src[k][0] = saddr(rr + 1 < rows ? T + (rr + 1) * hx + cc : tp.gt > 1 ? Q + cc : T + cc);
    src[k][1] = saddr(rr > 0 ? T + (rr - 1) * hx + cc
                      : tp.gt > 1 ? Q + hx + cc : T + max(rows - 1, 0) * hx + cc);
    src[k][2] = saddr(cc + 1 < cols ? T + rr * hx + cc + 1 : tp.gx > 1 ? Q + 2 * hx + rr : T + rr * hx);
    src[k][3] = saddr(cc > 0 ? T + rr * hx + cc - 1
                      : tp.gx > 1 ? Q + 2 * hx + ht + rr : T + rr * hx + max(cols - 1, 0));
    // the block behind in t takes the first row as its forward rim, the block ahead the last one
    // as its backward rim; the same in x
    const int back = (bt == 0 ? tp.gt - 1 : bt - 1) * tp.gx + bx;
    const int ahead = (bt + 1 == tp.gt ? 0 : bt + 1) * tp.gx + bx;
    const int left = bt * tp.gx + (bx == 0 ? tp.gx - 1 : bx - 1);
    const int right = bt * tp.gx + (bx + 1 == tp.gx ? 0 : bx + 1);
    dst[k][0] = dst[k][1] = dst2[k] = 0;
    dbar[k][0] = dbar[k][1] = dbar2[k] = 0;
    auto send = [&](uint32_t &d, uint32_t &db, int rank, int slot) {
      d = cluster_addr(saddr(Q + slot), rank);
      db = cluster_addr(my_bar, rank);
    };
    if (on[k] && tp.gt > 1) {
      if (row == 0) send(dst[k][0], dbar[k][0], back, c);
      if (row == rows - 1) {
        if (row == 0) send(dst2[k], dbar2[k], ahead, hx + c);
        else send(dst[k][0], dbar[k][0], ahead, hx + c);
      }
    }
    if (on[k] && tp.gx > 1) {
      if (c == 0) send(dst[k][1], dbar[k][1], left, 2 * hx + row);
      if (c == cols - 1) send(dst[k][1], dbar[k][1], right, 2 * hx + ht + row);
    }
  }
  cluster_sync();  // every block runs and its barriers are set before anything is sent to it
  unsigned n = 0;
  auto phase = [&](auto ns, auto hop, const double2 (&v)[K], double sgn, double2 (&out)[K],
                   const double *pt, double *total) -> bool {
    constexpr int NS = decltype(ns)::value > 1 ? decltype(ns)::value : 1;
    constexpr bool HOP = decltype(hop)::value;
    const uint32_t off = (n & 1) * STEP, parity = (n >> 1) & 1;
    Buf &C = B[n & 1];
    n++;
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(my_bar + off),
                   "r"(NS * nb * 8 + (HOP ? rims : 0))
                   : "memory");
#pragma unroll
    for (int j = 0; j < NS; j++) C.thr[j][tid] = decltype(ns)::value ? pt[j] : 0.;
#pragma unroll
    for (int k = 0; k < (HOP ? K : 0); k++) {
      auto push = [&](uint32_t d, uint32_t db) {
        if (d)
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(d + off),
                       "d"(v[k].x), "d"(v[k].y), "r"(db + off)
                       : "memory");
      };
      if (on[k])
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(own[k] + off), "d"(v[k].x), "d"(v[k].y)
                     : "memory");
      push(dst[k][0], dbar[k][0]);
      push(dst[k][1], dbar[k][1]);
      push(dst2[k], dbar2[k]);
    }
    __syncthreads();
    if (*(volatile unsigned *)&sh_bad < n) return false;  // in the last phase: the same for all
    for (int i = warp; i < NS; i += nw) {  // a warp for each sum
      double q[MAX_THREADS / 32];
#pragma unroll
      for (int j = 0; j < MAX_THREADS / 32; j++) q[j] = j < nw ? C.thr[i][lane + 32 * j] : 0.;
#pragma unroll
      for (int o = MAX_THREADS / 64; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; j++) q[j] += q[j + o];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q[0] += __shfl_xor_sync(0xffffffffu, q[0], o);
      if (lane < nb)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(mine + off + (uint32_t)(i * 8 * MAX_CLUSTER)),
                     "d"(q[0]), "r"(peer_bar + off)
                     : "memory");
    }
    // A warp waits as one.  One that gives up joins the barrier at which the block's other warps
    // next meet, in their next phase or after their last one, and so tells them all.
    for (long long since = 0;;) {
      uint32_t ok = 0;
      asm volatile("{\n\t.reg .pred q;\n\t"
                   "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2, %3;\n\t"
                   "selp.u32 %0, 1, 0, q;\n\t}"
                   : "=r"(ok)
                   : "r"(my_bar + off), "r"(parity), "r"(TRY_NS)
                   : "memory");
      if (__all_sync(0xffffffffu, ok) && a.limit > 0) break;
      const long long now = clock64();
      if (since == 0) since = now;
      if (__any_sync(0xffffffffu, now - since >= a.limit)) {
        *(volatile int *)&a.out->failed = 1;
        *(volatile unsigned *)&sh_bad = n;
        __syncthreads();
        return false;
      }
    }
    double2 w[K][4];
#pragma unroll
    for (int k = 0; k < (HOP ? K : 0); k++)
#pragma unroll
      for (int j = 0; j < 4; j++) w[k][j] = lds(src[k][j] + off);
    // every thread adds the blocks' partials in the same order
    const uint32_t pa = saddr(&B[0].part[0][0]) + off;
#pragma unroll
    for (int i = 0; i < NS; i++) {
      double2 q[MAX_CLUSTER / 2];
#pragma unroll
      for (int j = 0; j < MAX_CLUSTER / 2; j++) q[j] = lds(pa + 8 * MAX_CLUSTER * i + 16 * j);
#pragma unroll
      for (int o = MAX_CLUSTER / 4; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; j++) q[j].x += q[j + o].x, q[j].y += q[j + o].y;
      total[i] = q[0].x + q[0].y;
    }
#pragma unroll
    for (int k = 0; k < (HOP ? K : 0); k++)
      out[k] = hop2(a.m, sgn, v[k], uf[k], ub[k], w[k][0], w[k][1], w[k][2], w[k][3],
                    t0 + r0 + k * tp.rp);
    return true;
  };
  CgEnd end;
  bool good = BI ? bi_run<K>(on, x, b, a.tol, a.max_iter, phase, end)
                 : cg_run<K>(on, x, b, a.tol, a.max_iter, phase, end);
  if (good) {
    __syncthreads();
    good = *(volatile unsigned *)&sh_bad > n;
  }
  if (good) {
#pragma unroll
    for (int k = 0; k < K; k++)
      if (on[k]) a.x[eo(t0 + r0 + k * tp.rp, xc)] = x[k];
    if (blockIdx.x == 0 && tid == 0) write_result(a.out, end, a.epoch);
  } else {
    // what was sent to a block that no longer waits for it is still to arrive: a millisecond
    for (const long long since = clock64(); clock64() - since < 2000000;) {
    }
  }
  cluster_sync();  // no block leaves while another may send to it
}

template <int K> int tile_blocks(int *slots) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (slots[dev] == 0) {
    int coop = 0, sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_tile<K, false>, MAX_THREADS, 0);
    slots[dev] = 1 + (coop && per_sm >= 1 ? sms : 0);
  }
  return slots[dev] - 1;
}

// the tiling of at most `most` blocks of K-site threads with the least time per phase: the
// sites of a block cost its SM FP64 issue, its rim packets, its blocks the sum
double plan(const Geom &g, int K, int most, int max_rim, CgTilePlan *best) {
  const int Lt = g.L[0], Lx = g.L[1];
  double cost = 1e30;
  for (int hx = 2; hx <= std::min(Lx, MAX_THREADS); hx += 2)
    for (int rp = 1; rp * hx <= MAX_THREADS; rp++) {
      const int ht = K * rp, gt = (Lt + ht - 1) / ht, gx = (Lx + hx - 1) / hx;
      if ((long)gt * gx > most || (rp > 1 && K * (rp - 1) >= Lt)) continue;
      if (gt * gx > 1 && 2 * (hx + ht) > max_rim) continue;
      const double c = K * rp * hx + 2. * ((gt > 1 ? hx : 0) + (gx > 1 ? ht : 0)) + 0.5 * gt * gx;
      if (c < cost) cost = c, *best = CgTilePlan{K, ht, hx, gt, gx, rp, 0};
    }
  return cost;
}

// a launch of one cluster of `size` blocks; attr holds its launch attribute
inline cudaLaunchConfig_t cluster_config(int size, int nt, size_t smem, cudaStream_t s, cudaLaunchAttribute *attr) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = size;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}
template <int K, bool BI> bool set_cluster_attributes() {
  if (cudaFuncSetAttribute(k_cg_cluster<K, BI>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess &&
      cudaFuncSetAttribute(k_cg_cluster<K, BI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(2 * sizeof(ClusterBuf<K, BI>))) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}
template <int K, bool BI> bool cluster_fits(int size, const CgTilePlan &q) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config(size, (q.rp * q.hx + 31) / 32 * 32,
                                                 2 * sizeof(ClusterBuf<K, BI>), nullptr, &attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_cg_cluster<K, BI>, &cfg) == cudaSuccess && n >= 1)
    return true;
  cudaGetLastError();
  return false;
}
template <int K> bool plan_cluster(const Geom &g, CgTilePlan *p) {
  if (!set_cluster_attributes<K, false>()) return false;
  double best = 1e30;
  for (int size = 1; size <= MAX_CLUSTER; size *= 2) {
    CgTilePlan q{};
    // a second block costs the cluster's barrier, as much as 200 sites
    const double c = plan(g, K, size, MAX_RIM, &q) + (size > 1 ? 200. : 0.);
    if (!q.K || c >= best) continue;
    if (!cluster_fits<K, false>(size, q)) continue;
    best = c;
    *p = q;
    p->cluster = size;
  }
  return best < 1e30;
}

}  // namespace

CgTilePlan cg_tile_plan(const Geom &g) {
  CgTilePlan p{};
  if (g.nd != 2) return p;
  if (plan_cluster<1>(g, &p) || plan_cluster<2>(g, &p)) return p;
  static int slots[2][64];
  plan(g, 1, std::min(tile_blocks<1>(slots[0]), MAX_BLOCKS), 1 << 30, &p);
  if (!p.K) plan(g, 2, std::min(tile_blocks<2>(slots[1]), MAX_BLOCKS), 1 << 30, &p);
  return p;
}
// whether the BiCGStab runs on a plan made for the CG
bool cg_tile_bicgstab(const CgTilePlan &p) {
  if (!p.K) return false;
  if (p.cluster)
    return p.K == 1 ? set_cluster_attributes<1, true>() && cluster_fits<1, true>(p.cluster, p)
                    : set_cluster_attributes<2, true>() && cluster_fits<2, true>(p.cluster, p);
  int per_sm = 0;
  const cudaError_t e =
    p.K == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_tile<1, true>, MAX_THREADS, 0)
             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_tile<2, true>, MAX_THREADS, 0);
  cudaGetLastError();
  return e == cudaSuccess && per_sm >= 1;
}
size_t cg_tile_bytes(const Geom &g) {
  return sizeof(ulonglong2) * ((size_t)4 * g.V + 2 * BI_SUMS * MAX_BLOCKS + 1);
}

cudaError_t cg_tile(const Geom &g, const CgTilePlan &tp, bool bicgstab, const double2 *ph,
                    double m, const double2 *b, double2 *x, double tol, long max_iter, void *work,
                    unsigned long long epoch, CgTileResult *out, cudaStream_t s, long limit) {
  CgTileArgs a{};
  a.g = g, a.tp = tp, a.ph = ph, a.m = m, a.b = b, a.x = x, a.tol = tol, a.max_iter = max_iter;
  a.halo = (ulonglong2 *)work;
  a.sums = a.halo + (size_t)4 * g.V;
  a.err = (int *)(a.sums + 2 * BI_SUMS * MAX_BLOCKS);
  a.epoch = epoch, a.out = out;
  a.limit = limit >= 0 ? limit : tp.cluster ? CYCLE_LIMIT : POLL_LIMIT;
  const int nt = (tp.rp * tp.hx + 31) / 32 * 32;
  if (tp.cluster) {
    const auto kern = bicgstab ? (tp.K == 1 ? k_cg_cluster<1, true> : k_cg_cluster<2, true>)
                               : (tp.K == 1 ? k_cg_cluster<1, false> : k_cg_cluster<2, false>);
    const size_t buf = bicgstab ? (tp.K == 1 ? sizeof(ClusterBuf<1, true>) : sizeof(ClusterBuf<2, true>))
                                : (tp.K == 1 ? sizeof(ClusterBuf<1, false>) : sizeof(ClusterBuf<2, false>));
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config(tp.cluster, nt, 2 * buf, s, &attr);
    return cudaLaunchKernelEx(&cfg, kern, a);
  }
  cudaError_t e = cudaMemsetAsync(a.err, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  void *args[] = {&a};
  const auto kern = bicgstab ? (tp.K == 1 ? k_cg_tile<1, true> : k_cg_tile<2, true>)
                             : (tp.K == 1 ? k_cg_tile<1, false> : k_cg_tile<2, false>);
  e = cudaLaunchCooperativeKernel((const void *)kern, dim3(tp.gt * tp.gx), dim3(nt), args, 0, s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs free: the other forms
    cudaGetLastError();
    return cudaErrorNotSupported;
  }
  return e;
}

}  // namespace su2b
