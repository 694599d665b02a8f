// afl_poisson_brick.cu -- brick-resident FP64 CG: the whole solve in one
// cooperative launch with every CG vector on chip.
//
// The direction d lives in shared memory (the brick, its side ring, and the
// cell above each column); the residual r in registers, one column of up to
// 32 cells per thread; q = A d and the pressure p in tensor memory (in
// registers too when a thread has at most 8 cells).  Per iteration only the
// faces cross L2, as tagged packets of q, and one grid-wide sum of four
// doubles.  The ring keeps the neighbours' r and d: it applies the owners'
// updates to them, bit for bit, so q is all it needs.
//
// What bounds it (128^3: 128 CTAs of 32 x 16 x 32 cells, cycles at 1.9 GHz of
// one 16.6 k cycle iteration, stamped per CTA): the stencil 7.8 k (five
// shared-memory reads of 8 bytes per cell alone take 5.1 k), the CTA's partial
// sums 0.7-1.2 k, the wait for the neighbours' packets and the slowest CTA's
// sum 3.6 k (one hop between the dies is 0.95 k), the scalars and the ring 1.6 k,
// the update 2.2 k.  On small grids only the hops are left: 3 us an iteration
// whatever the size.
//
// Per iteration, CUDA events over 200-iteration solves, this kernel against the
// column-resident one (afl_poisson_resident.cu: q through L2, faces after a
// fence, all threads of a CTA behind each step of the sum):
//   128^3 17.3 -> 8.9 us, 90 x 133 x 77 14.4 -> 5.3 us, 64^3 7.8 -> 3.2 us,
//   36 x 52 x 36 7.6 -> 3.1 us.
// What mattered, in this order: q and p in tensor memory and r in registers (no
// vector in L2); all packet loads of a thread in flight at once (one after the
// other: +3 us at 128^3); no vector spilled (the shared-memory carve-out leaves no
// L1 for local memory: +4 us; the instances of 32 planes still spill 108 bytes of
// addresses and scalars a thread, 180 in the queue); packets polled before the sum
// (+0.8 us after it).
// Tried and slower: polling the neighbours' sum slots before asking for their
// packets, and pushing the partial sums into a mailbox per reader (+2 us: the
// extra words crowd the lines being waited for).
//
// Built with -fmad=false; the FMAs of the solve are written out (__fma_rn).
#include <algorithm>
#include <numeric>
#include <type_traits>

#include "afl_brick.cuh"

namespace afl {
namespace {

struct BrickCgArgs {
  Dims g;
  int nbx, nby, nbz, cz, czp;
  double *p;
  const double *b;
  Packet *inbox;
  int parity;  // packets between an inbox's two parities
  int max_iters;
  double rel_tol;
  SolveReport *report;
};

// r = b - A p at one interior cell from global memory (src/fluid.rs:455-458),
// 0 elsewhere: the pressure is written only at the end of the solve, after
// every CTA has passed the first sum.
__device__ __forceinline__ double brick_residual(const Dims &g, const double *p, const double *b,
                                                 int c, int i, int j, int k) {
  if (!interior(g, i, j, k)) return 0.0;
  double diag = 0.0, nb = 0.0;
  if (i > 1) { diag += 1.0; nb += p[c - 1]; }
  if (i + 2 < g.nx) { diag += 1.0; nb += p[c + 1]; }
  if (j > 1) { diag += 1.0; nb += p[c - g.nx]; }
  if (j + 2 < g.ny) { diag += 1.0; nb += p[c + g.nx]; }
  if (k > 1) { diag += 1.0; nb += p[c - g.nxy]; }
  if (k + 2 < g.nz) { diag += 1.0; nb += p[c + g.nxy]; }
  return b[c] - (diag * p[c] - nb);
}

// solve_poisson_conjugate_gradient (src/fluid.rs:445-493) with the relative
// tolerance extension.  One grid-wide sum per iteration carries d.q, r.q, q.q
// and the r.r of the current residual: alpha = delta/(d.q) takes the true
// delta = r.r; the next r.r is formed as delta - 2 alpha r.q + alpha^2 q.q for
// beta (src/fluid.rs:482); the stopping tests after an update (:479, relative
// tolerance) read the true r.r, which arrives with the next iteration's sum,
// and run there before any further update.
//
// Wall cells take no part in the stencil: A d is 0 there and interior cells
// skip them, so r stays b, d = s_k b with s_0 = 1, s_{k+1} = 1 + beta_k s_k, and
// p gains b times the sum of alpha_k s_k.  Their r.r joins the sums as one
// number, and p gets its gain at the end (b is 0 there after a divergence; a
// caller's own right-hand side may not be).
template <int BX, int CZ, typename Sums>
__device__ __forceinline__ void cg_brick_f64_body(const BrickCgArgs &a, const Sums &bs,
                                                  double *D, double *red, double *keep, unsigned tm) {
  using S = BrickShape<BX>;
  constexpr bool TM = CZ > 8;             // q and p in tensor memory, else in registers
  constexpr int NCH = CZ / 4;             // chunks of 4 planes
  constexpr int NI = (CZ + S::kLanes - 1) / S::kLanes;  // side ring cells per thread
  constexpr int SXY = S::SXY;
  constexpr int RSTEP = S::kLanes * S::kSide;  // ring cells the CTA covers at once
  const Dims &g = a.g;
  const int t = threadIdx.x;
  const int cz = a.cz;
  const BrickCells<S> cl(g, a.nbx, a.nby, cz, t, bs.block());
  const BrickFaces<S, Sums::kQueued> fc(g, cl, a.nbx, a.nby, a.nbz, a.czp, t);
  // z of the brick's plane m is k0 + m; chunks whose four planes all have both
  // z neighbours take the plain path of the operator
  const int k0 = cl.z0, k_lo = 2 - k0, k_hi = min(g.nz - 3 - k0, cl.nzb - 1);
  // shared memory: d (plane cz of a column: the cell above it), then per
  // thread r and d of the cell below and r of the cell above, then r of the
  // side ring, RSTEP apart, then the staged x faces, XSTEP per plane
  constexpr int XSTEP = 2 * S::BY;
  double *const Dc = D + (t / S::BX + 1) * S::SX + t % S::BX + 1;
  double *const Z = D + (CZ + 1) * SXY + t;
  double *const RS = D + (CZ + 1) * SXY + 3 * kBT + t;
  double *const X = D + (CZ + 1) * SXY + 3 * kBT + NI * RSTEP;
  int *const I = reinterpret_cast<int *>(X + CZ * XSTEP) + t;
  constexpr int kYdst = 0, kZlo = kBT, kZhi = 2 * kBT, kXdst = 3 * kBT, kSide = 4 * kBT,
                kSideD = 5 * kBT;
  double r[CZ];
  double qreg[TM ? 1 : CZ], preg[TM ? 1 : CZ];
  unsigned tag = 1;

  // ---- r = b - A p, d = r, on the brick and its ring --------------------------
  for (int s = t; s < (CZ + 1) * SXY; s += kBT) D[s] = 0.0;
  for (int s = t; s < brick_inbox_packets(S::kSide, a.czp); s += kBT) {
    a.inbox[fc.own + s] = Packet{0, 0};
    a.inbox[fc.own + a.parity + s] = Packet{0, 0};
  }
  __syncthreads();
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    unsigned pw[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = 4 * ch + e;
      double rv = 0.0, pv = 0.0;
      if (cl.in_ij && m < cl.nzb) {
        const int c = cl.c0 + m * g.nxy;
        rv = brick_residual(g, a.p, a.b, c, cl.i, cl.j, cl.z0 + m);
        pv = a.p[c];
        const double bc = a.b[c];
        const bool in = interior(g, cl.i, cl.j, cl.z0 + m);
        acc[0] += in ? rv * rv : bc * bc;
        acc[1] += bc * bc;
        acc[2] += in ? 0.0 : bc * bc;
        Dc[m * SXY] = rv;
      }
      r[m] = rv;
      if constexpr (TM) put_double(pw, e, pv);
      else preg[m] = pv;
    }
    if constexpr (TM) brick_tm_st8(tm + 16u * ch + 8u, pw);
  }
  {
    double lo = 0.0, hi = 0.0;
    if (fc.zlo_dst >= 0) lo = brick_residual(g, a.p, a.b, cl.c0 - g.nxy, cl.i, cl.j, cl.z0 - 1);
    if (fc.zhi_dst >= 0) hi = brick_residual(g, a.p, a.b, cl.c0 + cz * g.nxy, cl.i, cl.j, cl.z0 + cz);
    Z[0] = lo;
    Z[kBT] = lo;
    Z[2 * kBT] = hi;
    Dc[cz * SXY] = hi;
    for (int n = 0; n * S::kLanes < fc.side_lim; ++n) {
      const int k = k0 + t / S::kSide + n * S::kLanes;
      const double rv =
          brick_residual(g, a.p, a.b, (k * g.ny + fc.sj) * g.nx + fc.si, fc.si, fc.sj, k);
      RS[n * RSTEP] = rv;
      D[fc.side_d + n * S::kLanes * SXY] = rv;
    }
  }
  if constexpr (TM) brick_tm_wait_st();
  brick_partials(acc, red);
  brick_publish<true>(bs, tag, red);
  double tot[4];
  if (!brick_gather(bs, tag, tot, red + 4 * kBW, true)) return;
  __threadfence();  // the neighbours' inboxes are cleared before packets go there
  ++tag;
  // scalars that an iteration does not need stay in shared memory: keep[0..2]
  // = r.r at the start, b.b, the squared tolerance; of the wall cells keep[3..5]
  // = r.r, s_k, the sum of alpha_k s_k
  double delta = tot[0];
  {
    double tol2 = -1.0;
    if (a.rel_tol > 0.0) {
      const double tl = a.rel_tol * sqrt(tot[1]);
      tol2 = tl * tl;
    }
    if (t == 0) {
      keep[0] = delta;
      keep[1] = tot[1];
      keep[2] = tol2;
      keep[3] = tot[2];
      keep[4] = 1.0;
      keep[5] = 0.0;
    }
  }
  __syncthreads();
  double last = delta;
  int it = 0, converged = 0;
  if (!(delta > 1e-24) || (keep[2] >= 0.0 && delta <= keep[2])) {  // src/fluid.rs:462
    converged = isfinite(delta) ? 1 : 0;
  } else {
    // What a thread needs of its faces once per iteration waits in shared memory:
    // the registers hold r.
    I[kYdst] = fc.ydst;
    I[kZlo] = fc.zlo_dst;
    I[kZhi] = fc.zhi_dst;
    I[kXdst] = fc.xdst;
    I[kSideD] = fc.side_d;
    // side_lim, and whether the own and the side column are interior
    I[kSide] = max(fc.side_lim, 0) | (cl.column_interior(g) ? 256 : 0) |
               (fc.si >= 1 && fc.si <= g.nx - 2 && fc.sj >= 1 && fc.sj <= g.ny - 2 ? 512 : 0);
    const double dg2 = double(cl.diag2(g));  // the diagonal with both z neighbours
    double rr = 0.0;  // this thread's part of r.r; thread 0 of CTA 0 adds the walls'
    for (;;) {
      Packet *const box = a.inbox + ((it & 1) ? a.parity : 0);
      // ---- q = A d (src/fluid.rs:465), the faces' q, the four dot products ----
      acc[0] = acc[1] = acc[2] = 0.0;
      acc[3] = rr;
      {
        // Off the interior columns q comes out as garbage instead of 0; it is
        // kept out of the sums here and out of the updates by a zero alpha.
        double below = Z[kBT], mid = Dc[0];
        const int ydst = I[kYdst];
        const int xstage = t % S::BX == 0           ? t / S::BX
                           : t % S::BX == S::BX - 1 ? S::BY + t / S::BX
                                                    : -1;
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          if (4 * ch >= cz) break;
          unsigned qw[8];
          double qv[4];
          auto cell = [&](int e, double dg) {
            const int m = 4 * ch + e;
            const double above = Dc[(m + 1) * SXY];
            double nb = Dc[m * SXY - 1];
            nb += Dc[m * SXY + 1];
            nb += Dc[m * SXY - S::SX];
            nb += Dc[m * SXY + S::SX];
            nb += below;
            nb += above;
            const double q = __fma_rn(dg, mid, -nb);
            below = mid;
            mid = above;
            return q;
          };
          auto sums = [&](int e, double d, double q) {
            acc[0] = __fma_rn(d, q, acc[0]);
            acc[1] = __fma_rn(r[4 * ch + e], q, acc[1]);
            acc[2] = __fma_rn(q, q, acc[2]);
            qv[e] = q;
          };
          if (4 * ch >= k_lo && 4 * ch + 3 <= k_hi) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const double d = mid;
              sums(e, d, cell(e, dg2));
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int m = 4 * ch + e, k = k0 + m;
              const double d = mid;
              const double q = cell(e, k == 1 || k == g.nz - 2 ? dg2 - 1.0 : dg2);
              sums(e, d, k >= 1 && k <= g.nz - 2 && m < cz ? q : 0.0);
            }
          }
          if (xstage >= 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) X[(4 * ch + e) * XSTEP + xstage] = qv[e];
          }
          if (ydst >= 0) {
            if (!Sums::kQueued || 4 * ch + 4 <= cl.nzb) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                st_packet(box + S::y_at(ydst, 4 * ch + e, 4 * ch + 4), qv[e], tag);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (const int at = S::y_at(ydst, 4 * ch + e, cl.nzb); at >= 0)
                  st_packet(box + at, qv[e], tag);
            }
          }
          if (ch == 0) {
            const int zlo = I[kZlo];
            if (zlo >= 0) st_packet(box + zlo, qv[0], tag);
          }
          if (4 * ch + 4 >= cz) {
            const int zhi = I[kZhi];
            const int e = (cz - 1) & 3;
            const double qt = e == 0 ? qv[0] : e == 1 ? qv[1] : e == 2 ? qv[2] : qv[3];
            if (zhi >= 0) st_packet(box + zhi, qt, tag);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if constexpr (TM) put_double(qw, e, qv[e]);
            else qreg[4 * ch + e] = qv[e];
          }
          if constexpr (TM) brick_tm_st8(tm + 16u * ch, qw);
        }
        if constexpr (TM) brick_tm_wait_st();
        if (!(I[kSide] & 256)) acc[0] = acc[1] = acc[2] = 0.0;
      }
      brick_partials(acc, red);
      if (const int xdst = I[kXdst]; xdst >= 0) {
#pragma unroll
        for (int n = 0; n < CZ / S::kXLanes || n == 0; ++n)
          if (const int at = S::template x_at<Sums::kQueued>(xdst, t, n, cz, cl.nzb); at >= 0)
            st_packet(box + at, X[t + n * kBT], tag);
      }
      brick_publish<false>(bs, tag, red);
      // ---- the ring's q, the neighbours' packets, then the grid-wide sum --------
      double q_lo, q_hi, q_side[NI], sum[4];
      bool ok = true;
      {
        const Packet *const own = box + bs.block() * brick_inbox_packets(S::kSide, a.czp) + t;
        RawPacket lo, hi, side[NI];
        const int side_lim = I[kSide] & 255;
        const bool zlo = I[kZlo] >= 0, zhi = I[kZhi] >= 0;
        BoundedWait w;
        for (;;) {
          lo.ld(zlo, own + S::kSide * a.czp, tag);
          hi.ld(zhi, own + S::kSide * a.czp + kBT, tag);
#pragma unroll
          for (int n = 0; n < NI; ++n) side[n].ld(S::side_on(n, side_lim), own + n * RSTEP, tag);
          bool got = lo.has(tag) & hi.has(tag);
#pragma unroll
          for (int n = 0; n < NI; ++n) got &= side[n].has(tag);
          if (got) break;
          if (!w.again(bs.abort_flag, bs.timeout_ns)) {
            ok = false;
            break;
          }
        }
        q_lo = lo.value();
        q_hi = hi.value();
#pragma unroll
        for (int n = 0; n < NI; ++n) q_side[n] = side[n].value();
      }
      if (!brick_gather(bs, tag, sum, red + 4 * kBW, ok)) return;
      ++tag;
      if (it > 0) {  // the tests after the previous update (src/fluid.rs:478-481)
        last = sum[3];
        if (!isfinite(last)) break;
        if (last < 1e-20) { converged = 1; break; }
        const double tol2 = keep[2];
        if (tol2 >= 0.0 && last <= tol2) { converged = 1; break; }
        delta = last;
      }
      if (it >= a.max_iters) break;
      if (fabs(sum[0]) < 1e-28) break;  // src/fluid.rs:469
      // alpha = delta / d.q and beta = (delta - 2 alpha r.q + alpha^2 q.q) / delta, the
      // latter over d.q too: the two divisions do not wait for one another
      const double inv = 1.0 / sum[0];
      const double alpha = delta / sum[0];
      const double beta = __fma_rn(__fma_rn(alpha, sum[2], -2.0 * sum[1]), inv, 1.0);
      // ---- p += alpha d, r -= alpha q, d = r + beta d (src/fluid.rs:472-485) -----
      // the ring first, with the owners' expressions on the owners' operands
      const int side = I[kSide];
      const double a_col = side & 256 ? -alpha : -0.0, a_side = side & 512 ? -alpha : -0.0;
      double dh;
      {
        const double rl = __fma_rn(a_col, q_lo, Z[0]);
        Z[0] = rl;
        Z[kBT] = __fma_rn(beta, Z[kBT], rl);
        const double rh = __fma_rn(a_col, q_hi, Z[2 * kBT]);
        Z[2 * kBT] = rh;
        dh = __fma_rn(beta, Dc[cz * SXY], rh);
        double *const DS = D + I[kSideD];
        const int side_lim = side & 255;
#pragma unroll
        for (int n = 0; n < NI; ++n)
          if (n * S::kLanes < side_lim) {
            const double rv = __fma_rn(a_side, q_side[n], RS[n * RSTEP]);
            RS[n * RSTEP] = rv;
            double &ds = DS[n * S::kLanes * SXY];
            ds = __fma_rn(beta, ds, rv);
          }
      }
      rr = 0.0;
      if (t == 0) {
        keep[5] += alpha * keep[4];
        keep[4] = 1.0 + beta * keep[4];
        if (bs.block() == 0) rr = keep[3];
      }
      auto update = [&](int m, double q, double &p) {
        const double dv = Dc[m * SXY];
        p = __fma_rn(alpha, dv, p);
        const double rv = __fma_rn(a_col, q, r[m]);
        r[m] = rv;
        Dc[m * SXY] = __fma_rn(beta, dv, rv);
        rr = __fma_rn(rv, rv, rr);
      };
      if constexpr (TM) {
        unsigned w[2][16];
        brick_tm_ld16(tm, w[0]);
        brick_tm_wait_ld(w[0]);
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          if (4 * ch >= cz) break;
          if (ch + 1 < NCH) brick_tm_ld16(tm + 16u * (ch + 1), w[(ch + 1) & 1]);
          unsigned pw[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            double pv = get_double(w[ch & 1], 8 + 2 * e);
            update(4 * ch + e, get_double(w[ch & 1], 2 * e), pv);
            put_double(pw, e, pv);
          }
          brick_tm_st8(tm + 16u * ch + 8u, pw);
          if (ch + 1 < NCH) brick_tm_wait_ld(w[(ch + 1) & 1]);
        }
        brick_tm_wait_st();
      } else {
#pragma unroll
        for (int m = 0; m < CZ; ++m) {
          if (m >= cz) break;
          update(m, qreg[m], preg[m]);
        }
      }
      Dc[cz * SXY] = dh;  // past the update of the column's padding planes
      __syncthreads();
      ++it;
    }
  }
  // ---- the pressure back to global memory ----------------------------------------
  int t2;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t2));  // kept apart: no register across the loop
  const BrickCells<S> cw(g, a.nbx, a.nby, cz, t2, bs.block());
  __syncthreads();
  const bool wall = it > 0 && keep[3] != 0.0;  // without a step 0 * inf would be added
  const double gain = keep[5];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    if (4 * ch >= cz) break;
    unsigned cur[16];
    if constexpr (TM) {
      brick_tm_ld16(tm + 16u * ch, cur);
      brick_tm_wait_ld(cur);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = 4 * ch + e;
      double pv;
      if constexpr (TM) pv = get_double(cur, 8 + 2 * e);
      else pv = preg[m];
      if (cw.in_ij && m < cw.nzb) {
        const int c = cw.c0 + m * g.nxy;
        if (wall && !interior(g, cw.i, cw.j, cw.z0 + m)) pv += gain * a.b[c];
        a.p[c] = pv;
      }
    }
  }
  if (bs.block() == 0 && t2 == 0 && a.report) {
    SolveReport rep;
    rep.iterations = it;
    rep.refinements = 0;
    rep.converged = converged;
    rep.status = isfinite(last) ? 0 : 4;
    rep.initial_residual = sqrt(keep[0]);
    rep.final_residual = sqrt(last);
    rep.rhs_norm = sqrt(keep[1]);
    *a.report = rep;
  }
}

template <int BX, int CZ>
__global__ void __launch_bounds__(kBT, 1)
    k_cg_brick_f64(const __grid_constant__ BrickCgArgs a, const __grid_constant__ BrickSums bs) {
  extern __shared__ double Dsm[];
  __shared__ double red[2 * 4 * kBW], keep[6];
  __shared__ unsigned tm_base;
  constexpr bool TM = CZ > 8;
  constexpr int COLS = 16 * CZ;  // 4 warps share a quarter of the lanes: 4*CZ columns each
  if constexpr (TM) {
    const int warp = threadIdx.x >> 5;
    if (warp == 0) brick_tm_alloc<COLS>(&tm_base);
    brick_tm_sync_threads();
    cg_brick_f64_body<BX, CZ>(a, bs, Dsm, red, keep,
                              tm_base + ((32u * unsigned(warp & 3)) << 16) +
                                  unsigned(4 * CZ) * unsigned(warp >> 2));
    brick_tm_sync_threads();  // every TMEM access of the CTA is complete
    if (warp == 0) brick_tm_dealloc<COLS>(tm_base);
  } else {
    cg_brick_f64_body<BX, CZ>(a, bs, Dsm, red, keep, 0u);
  }
}

// Several systems, each CTA its list of them.
template <int CZ>
__global__ void __launch_bounds__(kBT, 1)
    k_cg_brick_queue_f64(const __grid_constant__ BrickQueue<BrickCgArgs> q) {
  extern __shared__ double Dsm[];
  __shared__ double red[2 * 4 * kBW], keep[6];
  __shared__ unsigned tm_base;
  __shared__ BrickCgArgs a;
  __shared__ QueuedSums bs;
  constexpr bool TM = CZ > 8;
  constexpr int COLS = 16 * CZ;
  const int warp = threadIdx.x >> 5;
  unsigned tm = 0;
  if constexpr (TM) {
    if (warp == 0) brick_tm_alloc<COLS>(&tm_base);
    brick_tm_sync_threads();
    tm = tm_base + ((32u * unsigned(warp & 3)) << 16) + unsigned(4 * CZ) * unsigned(warp >> 2);
  }
  run_queue(q, a, bs, [&] { cg_brick_f64_body<kQueueBX, CZ>(a, bs, Dsm, red, keep, tm); });
  if constexpr (TM) {
    brick_tm_sync_threads();
    if (warp == 0) brick_tm_dealloc<COLS>(tm_base);
  }
}

using BrickFn = void (*)(BrickCgArgs, BrickSums);

template <int BX>
BrickFn brick_fn(int cz) {
  if (cz <= 4) return &k_cg_brick_f64<BX, 4>;
  if (cz <= 8) return &k_cg_brick_f64<BX, 8>;
  if constexpr (BX < 64) {
    if (cz > 16) return &k_cg_brick_f64<BX, 32>;
  }
  return &k_cg_brick_f64<BX, 16>;
}

}  // namespace

bool plan_brick(const Dims &g, BrickPlan *plan) {
  int dev = 0, sms = 0, smem = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return plan_brick_on(g, sms, smem, plan);
}

namespace {
// scratch: the abort flag and the sums' slots (zeroed before a launch), the
// inboxes (which clear themselves)
size_t slot_bytes(const BrickPlan &p) { return sizeof(Packet) * 8 * static_cast<size_t>(p.ctas()); }
}  // namespace

size_t brick_scratch_bytes(const BrickPlan &plan) {
  return kBrickHeader + slot_bytes(plan) + plan.inbox_bytes;
}

int launch_cg_brick(const BrickSolve &s, const BrickPlan &plan, cudaStream_t st) {
  BrickFn fn = plan.bx == 32   ? brick_fn<32>(plan.cz)
               : plan.bx == 16 ? brick_fn<16>(plan.cz)
                               : brick_fn<64>(plan.cz);
  const int blocks = plan.ctas();
  cudaError_t err =
      cudaFuncSetAttribute(reinterpret_cast<const void *>(fn),
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(plan.smem_bytes));
  if (err != cudaSuccess) return -static_cast<int>(err);
  cudaMemsetAsync(s.scratch, 0, kBrickHeader + slot_bytes(plan), st);
  auto *base = static_cast<unsigned char *>(s.scratch);
  auto *slots = base + kBrickHeader, *inbox = slots + slot_bytes(plan);
  BrickCgArgs a{s.g, plan.nbx, plan.nby, plan.nbz, plan.cz, (plan.cz + 3) / 4 * 4, s.p, s.b,
                reinterpret_cast<Packet *>(inbox),
                static_cast<int>(plan.inbox_bytes / (2 * sizeof(Packet))), s.max_iters, s.rel_tol,
                s.report};
  BrickSums bs{reinterpret_cast<Packet *>(slots), blocks, reinterpret_cast<int *>(base),
               s.timeout_ns};
  void *params[] = {&a, &bs};
  err = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fn), dim3(blocks), dim3(kBT),
                                    params, plan.smem_bytes, st);
  return err == cudaSuccess ? blocks : -static_cast<int>(err);
}

// Planes per CTA: the fewest of 4, 8, 16, 32 at which all systems run side by side, else up
// to 32 and several systems per CTA.  Largest first, each where it can start earliest.
// A solve is taken to need 3.5 iterations per cell of its longest side (32^3 115, 48^3 165).
//
// Against the streaming solve, which takes every system at once at 6.6 ps a cell and
// iteration (FP64 13) and not less than 4 us an iteration.  ms per step, streaming -> this:
// the 48 plumes 16.2 -> 11.4 (FP64 31.4 -> 11.9), one 32^3 1.6 -> 0.44, one 128^3 5.2 -> 2.4,
// 140 of 16^3 1.6 -> 0.9, 9 of 96^3 13.2 -> 11.0; several per CTA on bricks that the grids
// leave half empty lose in f32: 40 of 40^3 3.8 -> 4.5 (FP64 5.2 -> 4.5), 300 of 16^3
// 2.0 -> 2.2 (2.5 -> 2.2).
bool plan_brick_queue(const std::vector<Dims> &g, int max_iters, bool f64, BrickQueuePlan *q) {
  using S = BrickShape<kQueueBX>;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  sms = std::min(sms, 160);
  const int count = static_cast<int>(g.size());
  for (q->cz_class = 4;; q->cz_class *= 2) {
    q->plan.clear();
    q->total = 0;
    int most = 0;
    for (const Dims &d : g) {
      BrickPlan p{};
      p.bx = S::BX;
      p.nbx = (d.nx + S::BX - 1) / S::BX;
      p.nby = (d.ny + S::BY - 1) / S::BY;
      const int layers = (d.nz + q->cz_class - 1) / q->cz_class;
      p.cz = (d.nz + layers - 1) / layers;
      p.nbz = (d.nz + p.cz - 1) / p.cz;
      if (static_cast<long long>(p.nbx) * p.nby * p.nbz > sms) most = sms + 1;
      else q->total += p.ctas(), most = std::max(most, p.ctas());
      q->plan.push_back(p);
    }
    if (most <= sms && q->total <= sms) break;
    if (q->cz_class == kBrickMaxPlanes) {
      if (most > sms) return false;
      break;
    }
  }
  std::vector<int> order(count);
  std::iota(order.begin(), order.end(), 0);
  int most_planes = 0;
  for (const BrickPlan &p : q->plan) most_planes = std::max(most_planes, p.cz);
  q->cz_class = brick_cz_class(most_planes);
  auto iterations = [&](int m) {
    return std::min(double(max_iters), 3.5 * std::max(g[m].nx, std::max(g[m].ny, g[m].nz)));
  };
  auto cost = [&](int m) { return iterations(m) * 0.2 * (12 + q->plan[m].cz); };  // us
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return cost(a) * q->plan[a].ctas() > cost(b) * q->plan[b].ctas();
  });
  std::vector<double> free(sms, 0.0);
  std::vector<std::vector<int>> lists(sms);
  q->begin.assign(count, 0);
  q->ctas = 0;
  for (int m : order) {
    const int n = q->plan[m].ctas();
    double best = 0.0;
    for (int b = 0; b + n <= sms; ++b) {
      const double at = *std::max_element(free.begin() + b, free.begin() + b + n);
      if (b > 0 && at >= best) continue;
      best = at;
      q->begin[m] = b;
    }
    for (int c = q->begin[m]; c < q->begin[m] + n; ++c) {
      free[c] = best + cost(m);
      lists[c].push_back(m);
    }
    q->ctas = std::max(q->ctas, q->begin[m] + n);
  }
  double cells = 0.0, longest = 0.0;
  for (int m = 0; m < count; ++m) {
    cells += iterations(m) * g[m].n;
    longest = std::max(longest, iterations(m));
  }
  const double streaming = cells * (f64 ? 13e-6 : 6.6e-6) + longest * 4.0;
  if (*std::max_element(free.begin(), free.end()) > streaming) return false;
  q->first.assign(1, 0);
  q->list.clear();
  for (int c = 0; c < q->ctas; ++c) {
    q->list.insert(q->list.end(), lists[c].begin(), lists[c].end());
    q->first.push_back(static_cast<int>(q->list.size()));
  }
  return true;
}

cudaError_t setup_brick_queue(const std::vector<BrickSolve> &s, const BrickQueuePlan &plan,
                              void *scratch, int *abort_flag, unsigned long long timeout_ns) {
  return write_queue<BrickCgArgs, Packet>(plan, scratch, abort_flag, timeout_ns,
                                          [&](size_t m, BrickCgArgs &a) {
                                            a.g = s[m].g;
                                            a.p = s[m].p;
                                            a.b = s[m].b;
                                            a.max_iters = s[m].max_iters;
                                            a.rel_tol = s[m].rel_tol;
                                            a.report = s[m].report;
                                          });
}

size_t brick_queue_scratch_bytes(const BrickQueuePlan &plan, bool f64) {
  return f64 ? QueueLayout(plan, sizeof(BrickJob<BrickCgArgs>), sizeof(Packet)).bytes
             : mixed_queue_scratch_bytes(plan);
}

int launch_cg_brick_queue(const BrickQueuePlan &q, bool f64, void *scratch, cudaStream_t st) {
  if (!f64) return launch_cg_brick_queue_mixed(q, scratch, st);
  const auto fn = q.cz_class == 4    ? &k_cg_brick_queue_f64<4>
                  : q.cz_class == 8  ? &k_cg_brick_queue_f64<8>
                  : q.cz_class == 16 ? &k_cg_brick_queue_f64<16>
                                     : &k_cg_brick_queue_f64<32>;
  return launch_queue<BrickCgArgs, Packet>(fn, brick_smem<kQueueBX>(q.cz_class), q, scratch, st);
}

}  // namespace afl
