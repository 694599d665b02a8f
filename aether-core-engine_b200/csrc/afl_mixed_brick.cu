// afl_mixed_brick.cu -- brick-resident mixed CG: f64 iterative refinement around
// an f32 CG whose vectors never leave the SM (solve_poisson_conjugate_gradient,
// src/fluid.rs:445-493, on the correction).
//
// The FP64 kernel's scheme (afl_poisson_brick.cu) on f32 vectors: the direction
// d in shared memory, the residual r and q = A d in registers, the correction e
// in shared memory too (in registers when a thread has at most 8 cells), faces as
// tagged words of q, and one grid-wide sum of four doubles per inner iteration
// (d.q, r.q, q.q, r.r, every product and sum in f64).
//
// What bounds it: as the FP64 kernel, the stencil and the hops; the words are half
// as wide, and the conversions to f64 for the sums (three per cell) take the place
// of the second half.  Per inner iteration, CUDA events over 200-iteration solves,
// against the column-resident kernel (two grid-wide sums):
//   128^3 13.7 -> 7.4 us, 96 x 96 x 97 11.0 -> 4.7, 64^3 7.7 -> 2.8.
// e is in shared memory because there is room; keeping it in tensor memory, with
// constant zeros stored to start it, raised an illegal instruction.
//
// Built with -fmad=false; the FMAs are written out.
#include "afl_brick.cuh"

namespace afl {
namespace {

struct BrickMixedArgs {
  Dims g;
  int nbx, nby, nbz, cz, czp;
  double *p;
  const double *b;
  unsigned long long *inbox;
  int parity;  // words between an inbox's two parities
  int max_total, max_inner, max_refine;
  double inner_rel_tol, rel_tol;
  SolveReport *report;
};

// b - A p in f64 at an interior cell, 0 elsewhere.  The pressure is read through
// L2: other CTAs write it between refinement passes.
__device__ __forceinline__ double mixed_residual(const Dims &g, const double *p, const double *b,
                                                 int c, int i, int j, int k) {
  if (!interior(g, i, j, k)) return 0.0;
  double diag = 0.0, nb = 0.0;
  if (i > 1) { diag += 1.0; nb += __ldcg(p + c - 1); }
  if (i + 2 < g.nx) { diag += 1.0; nb += __ldcg(p + c + 1); }
  if (j > 1) { diag += 1.0; nb += __ldcg(p + c - g.nx); }
  if (j + 2 < g.ny) { diag += 1.0; nb += __ldcg(p + c + g.nx); }
  if (k > 1) { diag += 1.0; nb += __ldcg(p + c - g.nxy); }
  if (k + 2 < g.nz) { diag += 1.0; nb += __ldcg(p + c + g.nxy); }
  return b[c] - (diag * __ldcg(p + c) - nb);
}

template <int BX, int CZ, typename Sums>
__device__ __forceinline__ void cg_brick_mixed_body(const BrickMixedArgs &a, const Sums &bs,
                                                    float *D, double *red, double *keep) {
  using S = BrickShape<BX>;
  constexpr bool SM = CZ > 8;             // e in shared memory, else in registers
  constexpr int NCH = CZ / 4;             // chunks of 4 planes
  constexpr int NI = (CZ + S::kLanes - 1) / S::kLanes;  // side ring cells per thread
  constexpr int SXY = S::SXY;
  constexpr int RSTEP = S::kLanes * S::kSide;
  const Dims &g = a.g;
  const int t = threadIdx.x;
  const int cz = a.cz;
  const BrickCells<S> cl(g, a.nbx, a.nby, cz, t, bs.block());
  const BrickFaces<S, Sums::kQueued> fc(g, cl, a.nbx, a.nby, a.nbz, a.czp, t);
  const int k0 = cl.z0, k_lo = 2 - k0, k_hi = min(g.nz - 3 - k0, cl.nzb - 1);
  const bool col_in = cl.column_interior(g);
  const bool side_in = fc.si >= 1 && fc.si <= g.nx - 2 && fc.sj >= 1 && fc.sj <= g.ny - 2;
  // shared memory as in the FP64 kernel: d, then r and d of the cell below and r of
  // the cell above each column, then r of the side ring, then the staged x faces,
  // then e
  constexpr int XSTEP = 2 * S::BY;
  float *const Dc = D + (t / S::BX + 1) * S::SX + t % S::BX + 1;
  float *const Z = D + (CZ + 1) * SXY + t;
  float *const RS = D + (CZ + 1) * SXY + 3 * kBT + t;
  float *const X = D + (CZ + 1) * SXY + 3 * kBT + NI * RSTEP;
  float *const E = X + CZ * XSTEP + t;  // e of the column, kBT per plane
  float *const DS = D + fc.side_d;
  const int xstage = t % S::BX == 0           ? t / S::BX
                     : t % S::BX == S::BX - 1 ? S::BY + t / S::BX
                                              : -1;
  float r[CZ], q[CZ];
  float ereg[SM ? 1 : CZ];
  unsigned tag = 1;

  for (int s = t; s < (CZ + 1) * SXY; s += kBT) D[s] = 0.0f;
  for (int s = t; s < brick_inbox_packets(S::kSide, a.czp); s += kBT) {
    a.inbox[fc.own + s] = 0;
    a.inbox[fc.own + a.parity + s] = 0;
  }
  __syncthreads();

  // r = b - A p in f64, rounded once to f32, on the brick and its ring; d = r,
  // e = 0.  Sums: the f64 r.r, b.b, the rounded r.r and its wall cells' part.  A
  // wall cell takes no part in the stencil: its r stays b, so its part of r.r is
  // one number and its correction b times the sum of alpha_k s_k, as in the FP64
  // kernel.
  double acc[4];
  auto outer_residual = [&] {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 4 * ch + e;
        float rf = 0.0f;
        if (cl.in_ij && m < cl.nzb) {
          const int c = cl.c0 + m * g.nxy;
          const double bc = a.b[c];
          const bool in = interior(g, cl.i, cl.j, k0 + m);
          const double rv = in ? mixed_residual(g, a.p, a.b, c, cl.i, cl.j, k0 + m) : bc;
          rf = float(rv);
          acc[0] += rv * rv;
          acc[1] += bc * bc;
          acc[2] += double(rf) * double(rf);
          if (!in) {
            acc[3] += double(rf) * double(rf);
            rf = 0.0f;
          }
        }
        r[m] = rf;
        if (m < cz) Dc[m * SXY] = rf;
        if constexpr (SM) E[m * kBT] = 0.0f;
        else ereg[m] = 0.0f;
      }
    }
    float lo = 0.0f, hi = 0.0f;
    if (fc.zlo_dst >= 0)
      lo = float(mixed_residual(g, a.p, a.b, cl.c0 - g.nxy, cl.i, cl.j, k0 - 1));
    if (fc.zhi_dst >= 0)
      hi = float(mixed_residual(g, a.p, a.b, cl.c0 + cz * g.nxy, cl.i, cl.j, k0 + cz));
    Z[0] = Z[kBT] = lo;
    Z[2 * kBT] = hi;
    Dc[cz * SXY] = hi;
    for (int n = 0; n * S::kLanes < fc.side_lim; ++n) {
      const int k = k0 + t / S::kSide + n * S::kLanes;
      const float rv =
          float(mixed_residual(g, a.p, a.b, (k * g.ny + fc.sj) * g.nx + fc.si, fc.si, fc.sj, k));
      RS[n * RSTEP] = rv;
      DS[n * S::kLanes * SXY] = rv;
    }
  };

  outer_residual();
  brick_partials(acc, red);
  brick_publish<true>(bs, tag, red);
  double tot[4];
  if (!brick_gather(bs, tag, tot, red + 4 * kBW, true)) return;
  __threadfence();  // the neighbours' inboxes are cleared before words go there
  ++tag;
  // scalars that an iteration does not need: keep[0..2] = r.r at the start, b.b,
  // the squared tolerance; of the wall cells keep[3..5] = r.r, s_k, the sum of
  // alpha_k s_k
  double rr = tot[0];
  if (t == 0) {
    double tol2 = -1.0;
    if (a.rel_tol > 0.0) {
      const double tl = a.rel_tol * sqrt(tot[1]);
      tol2 = tl * tl;
    }
    keep[0] = rr;
    keep[1] = tot[1];
    keep[2] = tol2;
    keep[3] = tot[3];
  }
  __syncthreads();
  int total = 0, passes = 0, converged = 0;
  unsigned exchange = 0;  // numbers the inner iterations over all passes
  if (!(rr > 1e-24) || (keep[2] >= 0.0 && rr <= keep[2])) converged = isfinite(rr) ? 1 : 0;

  while (!converged && passes < a.max_refine && total < a.max_total && isfinite(rr)) {
    const double tol2 = keep[2];
    double inner_rel = a.inner_rel_tol;
    if (tol2 >= 0.0) inner_rel = fmax(inner_rel, 0.5 * sqrt(tol2 / rr));
    double delta = tot[2];
    const double inner_tol2 = inner_rel * inner_rel * delta;
    const float dg2 = float(cl.diag2(g));
    if (t == 0) {
      keep[4] = 1.0;
      keep[5] = 0.0;
    }
    int it = 0;
    for (;;) {
      auto *const box = a.inbox + ((exchange & 1u) ? a.parity : 0);
      ++exchange;
      // ---- q = A d, the faces' q, the four products ---------------------------------
      // Off the interior columns q comes out as garbage instead of 0; it is kept
      // out of the sums here and out of the updates by a zero alpha.
      acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
      {
        float below = Z[kBT], mid = Dc[0];
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          if (4 * ch >= cz) break;
          auto cell = [&](int e, float dg, bool in) {
            const int m = 4 * ch + e;
            const float above = Dc[(m + 1) * SXY];
            float nb = Dc[m * SXY - 1];
            nb += Dc[m * SXY + 1];
            nb += Dc[m * SXY - S::SX];
            nb += Dc[m * SXY + S::SX];
            nb += below;
            nb += above;
            const float qv = in ? __fmaf_rn(dg, mid, -nb) : 0.0f;
            const double dd = double(mid), qd = double(qv), rd = double(r[m]);
            acc[0] = __fma_rn(dd, qd, acc[0]);
            acc[1] = __fma_rn(rd, qd, acc[1]);
            acc[2] = __fma_rn(qd, qd, acc[2]);
            acc[3] = __fma_rn(rd, rd, acc[3]);
            q[m] = qv;
            below = mid;
            mid = above;
          };
          if (4 * ch >= k_lo && 4 * ch + 3 <= k_hi) {
#pragma unroll
            for (int e = 0; e < 4; ++e) cell(e, dg2, true);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int m = 4 * ch + e, k = k0 + m;
              cell(e, k == 1 || k == g.nz - 2 ? dg2 - 1.0f : dg2,
                   k >= 1 && k <= g.nz - 2 && m < cz);
            }
          }
          if (xstage >= 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) X[(4 * ch + e) * XSTEP + xstage] = q[4 * ch + e];
          }
          if (fc.ydst >= 0) {
            if (!Sums::kQueued || 4 * ch + 4 <= cl.nzb) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                st_packet(box + S::y_at(fc.ydst, 4 * ch + e, 4 * ch + 4), q[4 * ch + e], tag);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (const int at = S::y_at(fc.ydst, 4 * ch + e, cl.nzb); at >= 0)
                  st_packet(box + at, q[4 * ch + e], tag);
            }
          }
          if (ch == 0 && fc.zlo_dst >= 0) st_packet(box + fc.zlo_dst, q[0], tag);
          if (4 * ch + 4 >= cz && fc.zhi_dst >= 0) {
            const int e = (cz - 1) & 3;
            const float qt = e == 0   ? q[4 * ch]
                             : e == 1 ? q[4 * ch + 1]
                             : e == 2 ? q[4 * ch + 2]
                                      : q[4 * ch + 3];
            st_packet(box + fc.zhi_dst, qt, tag);
          }
        }
        if (!col_in) acc[0] = acc[1] = acc[2] = 0.0;
        if (bs.block() == 0 && t == 0) acc[3] += keep[3];
      }
      brick_partials(acc, red);
      if (fc.xdst >= 0) {
#pragma unroll
        for (int n = 0; n < CZ / S::kXLanes || n == 0; ++n)
          if (const int at = S::template x_at<Sums::kQueued>(fc.xdst, t, n, cz, cl.nzb); at >= 0)
            st_packet(box + at, X[t + n * kBT], tag);
      }
      brick_publish<false>(bs, tag, red);
      // ---- the ring's q, then the grid-wide sum ----------------------------------------
      RawWord lo, hi, side[NI];
      bool ok = true;
      {
        const auto *const own = box + fc.own + t;
        BoundedWait w;
        for (;;) {
          lo.ld(fc.zlo_dst >= 0, own + S::kSide * a.czp, tag);
          hi.ld(fc.zhi_dst >= 0, own + S::kSide * a.czp + kBT, tag);
#pragma unroll
          for (int n = 0; n < NI; ++n)
            side[n].ld(S::side_on(n, fc.side_lim), own + n * RSTEP, tag);
          bool got = lo.has(tag) & hi.has(tag);
#pragma unroll
          for (int n = 0; n < NI; ++n) got &= side[n].has(tag);
          if (got) break;
          if (!w.again(bs.abort_flag, bs.timeout_ns)) {
            ok = false;
            break;
          }
        }
      }
      double sum[4];
      if (!brick_gather(bs, tag, sum, red + 4 * kBW, ok)) return;
      ++tag;
      if (it > 0) {  // the tests after the previous update, on its true r.r
        const double dn = sum[3];
        if (!isfinite(dn) || dn <= inner_tol2 || dn < 1e-30) break;
        delta = dn;
      }
      if (it >= a.max_inner || total >= a.max_total) break;
      if (!(fabs(sum[0]) >= 1e-30)) break;
      const double inv = 1.0 / sum[0];
      const double alpha = delta / sum[0];
      const float bf = float(__fma_rn(__fma_rn(alpha, sum[2], -2.0 * sum[1]), inv, 1.0));
      const float af = float(alpha);
      if (t == 0) {
        keep[5] += double(af) * keep[4];
        keep[4] = 1.0 + double(bf) * keep[4];
      }
      // ---- e += alpha d, r -= alpha q, d = r + beta d, on the ring first -----------------
      const float a_col = col_in ? -af : -0.0f, a_side = side_in ? -af : -0.0f;
      const float rl = __fmaf_rn(a_col, lo.value(), Z[0]);
      Z[0] = rl;
      Z[kBT] = __fmaf_rn(bf, Z[kBT], rl);
      const float rh = __fmaf_rn(a_col, hi.value(), Z[2 * kBT]);
      Z[2 * kBT] = rh;
      const float dh = __fmaf_rn(bf, Dc[cz * SXY], rh);
#pragma unroll
      for (int n = 0; n < NI; ++n)
        if (n * S::kLanes < fc.side_lim) {
          const float rv = __fmaf_rn(a_side, side[n].value(), RS[n * RSTEP]);
          RS[n * RSTEP] = rv;
          float &ds = DS[n * S::kLanes * SXY];
          ds = __fmaf_rn(bf, ds, rv);
        }
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        if (4 * ch >= cz) break;
        float dv[4], ev[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // all loads before the stores
          const int m = 4 * ch + e;
          dv[e] = Dc[m * SXY];
          if constexpr (SM) ev[e] = E[m * kBT];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int m = 4 * ch + e;
          if constexpr (SM) E[m * kBT] = __fmaf_rn(af, dv[e], ev[e]);
          else ereg[m] = __fmaf_rn(af, dv[e], ereg[m]);
          const float rv = __fmaf_rn(a_col, q[m], r[m]);
          r[m] = rv;
          Dc[m * SXY] = __fmaf_rn(bf, dv[e], rv);
        }
      }
      Dc[cz * SXY] = dh;  // past the update of the column's padding planes
      __syncthreads();
      ++it;
      ++total;
    }
    // ---- p += e in f64, then the true residual again -----------------------------------
    const bool wall = keep[3] != 0.0;
    const double gain = keep[5];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      if (4 * ch >= cz) break;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 4 * ch + e;
        if (cl.in_ij && m < cl.nzb) {
          const int c = cl.c0 + m * g.nxy;
          float ec = SM ? E[m * kBT] : ereg[SM ? 0 : m];
          if (wall && !interior(g, cl.i, cl.j, k0 + m)) ec = float(a.b[c] * gain);
          a.p[c] = __ldcg(a.p + c) + double(ec);
        }
      }
    }
    // every CTA's pressure is written before any reads it: a sum of nothing
    // that releases the writes
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    brick_partials(acc, red);
    brick_publish<true>(bs, tag, red);
    if (!brick_gather(bs, tag, tot, red + 4 * kBW, true)) return;
    __threadfence();
    ++tag;
    outer_residual();
    brick_partials(acc, red);
    // what it read of the neighbours' pressure comes before the next pass's writes
    brick_publish<true>(bs, tag, red);
    if (!brick_gather(bs, tag, tot, red + 4 * kBW, true)) return;
    __threadfence();
    ++tag;
    rr = tot[0];
    ++passes;
    if (rr < 1e-20 || (keep[2] >= 0.0 && rr <= keep[2])) converged = 1;
  }
  if (bs.block() == 0 && t == 0 && a.report) {
    SolveReport rep;
    rep.iterations = total;
    rep.refinements = passes;
    rep.converged = converged;
    rep.status = isfinite(rr) ? 0 : 4;
    rep.initial_residual = sqrt(keep[0]);
    rep.final_residual = sqrt(rr);
    rep.rhs_norm = sqrt(keep[1]);
    *a.report = rep;
  }
}

template <int BX, int CZ>
__global__ void __launch_bounds__(kBT, 1)
    k_cg_brick_mixed(const __grid_constant__ BrickMixedArgs a,
                     const __grid_constant__ BrickSums bs) {
  extern __shared__ float Fsm[];
  __shared__ double red[2 * 4 * kBW], keep[6];
  cg_brick_mixed_body<BX, CZ>(a, bs, Fsm, red, keep);
}

template <int CZ>
__global__ void __launch_bounds__(kBT, 1)
    k_cg_brick_queue_mixed(const __grid_constant__ BrickQueue<BrickMixedArgs> q) {
  extern __shared__ float Fsm[];
  __shared__ double red[2 * 4 * kBW], keep[6];
  __shared__ BrickMixedArgs a;
  __shared__ QueuedSums bs;
  run_queue(q, a, bs, [&] { cg_brick_mixed_body<kQueueBX, CZ>(a, bs, Fsm, red, keep); });
}

using BrickMixedFn = void (*)(BrickMixedArgs, BrickSums);

template <int BX>
BrickMixedFn mixed_fn(int cz) {
  if (cz <= 4) return &k_cg_brick_mixed<BX, 4>;
  if (cz <= 8) return &k_cg_brick_mixed<BX, 8>;
  if constexpr (BX < 64) {
    if (cz > 16) return &k_cg_brick_mixed<BX, 32>;
  }
  return &k_cg_brick_mixed<BX, 16>;
}

template <int BX>
size_t mixed_smem(int cz) {
  using S = BrickShape<BX>;
  const int c = cz <= 4 ? 4 : cz <= 8 ? 8 : cz <= 16 ? 16 : 32;
  const int rows = (c + S::kLanes - 1) / S::kLanes;
  return sizeof(float) * (static_cast<size_t>(c + 1) * S::SXY + 3 * kBT +
                          rows * S::kLanes * S::kSide + c * 2 * S::BY +
                          (c > 8 ? c * kBT : 0));
}

}  // namespace

int launch_cg_brick_mixed(const BrickMixedSolve &s, const BrickPlan &plan, cudaStream_t st) {
  BrickMixedFn fn = plan.bx == 32   ? mixed_fn<32>(plan.cz)
                    : plan.bx == 16 ? mixed_fn<16>(plan.cz)
                                    : mixed_fn<64>(plan.cz);
  const size_t smem = plan.bx == 32   ? mixed_smem<32>(plan.cz)
                      : plan.bx == 16 ? mixed_smem<16>(plan.cz)
                                      : mixed_smem<64>(plan.cz);
  const int blocks = plan.ctas();
  cudaError_t err =
      cudaFuncSetAttribute(reinterpret_cast<const void *>(fn),
                           cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return -static_cast<int>(err);
  const size_t slots = sizeof(Packet) * 8 * static_cast<size_t>(blocks);
  cudaMemsetAsync(s.scratch, 0, kBrickHeader + slots, st);
  auto *base = static_cast<unsigned char *>(s.scratch);
  BrickMixedArgs a{s.g, plan.nbx, plan.nby, plan.nbz, plan.cz, (plan.cz + 3) / 4 * 4, s.p, s.b,
                   reinterpret_cast<unsigned long long *>(base + kBrickHeader + slots),
                   static_cast<int>(plan.inbox_bytes / (2 * sizeof(Packet))), s.max_total,
                   s.max_inner, s.max_refine, s.inner_rel_tol, s.rel_tol, s.report};
  BrickSums bs{reinterpret_cast<Packet *>(base + kBrickHeader), blocks,
               reinterpret_cast<int *>(base), s.timeout_ns};
  void *params[] = {&a, &bs};
  err = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fn), dim3(blocks), dim3(kBT),
                                    params, smem, st);
  return err == cudaSuccess ? blocks : -static_cast<int>(err);
}

cudaError_t setup_brick_queue(const std::vector<BrickMixedSolve> &s, const BrickQueuePlan &plan,
                              void *scratch, int *abort_flag, unsigned long long timeout_ns) {
  return write_queue<BrickMixedArgs, unsigned long long>(
      plan, scratch, abort_flag, timeout_ns, [&](size_t m, BrickMixedArgs &a) {
        a.g = s[m].g;
        a.p = s[m].p;
        a.b = s[m].b;
        a.max_total = s[m].max_total;
        a.max_inner = s[m].max_inner;
        a.max_refine = s[m].max_refine;
        a.inner_rel_tol = s[m].inner_rel_tol;
        a.rel_tol = s[m].rel_tol;
        a.report = s[m].report;
      });
}

size_t mixed_queue_scratch_bytes(const BrickQueuePlan &plan) {
  return QueueLayout(plan, sizeof(BrickJob<BrickMixedArgs>), sizeof(unsigned long long)).bytes;
}

int launch_cg_brick_queue_mixed(const BrickQueuePlan &q, void *scratch, cudaStream_t st) {
  const auto fn = q.cz_class == 4    ? &k_cg_brick_queue_mixed<4>
                  : q.cz_class == 8  ? &k_cg_brick_queue_mixed<8>
                  : q.cz_class == 16 ? &k_cg_brick_queue_mixed<16>
                                     : &k_cg_brick_queue_mixed<32>;
  return launch_queue<BrickMixedArgs, unsigned long long>(fn, mixed_smem<kQueueBX>(q.cz_class), q,
                                                          scratch, st);
}

}  // namespace afl
