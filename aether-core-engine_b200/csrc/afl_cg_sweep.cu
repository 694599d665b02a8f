// afl_cg_sweep.cu -- streaming CG at one sweep over memory per iteration, for
// grids that do not fit on chip (FP64, and the f32 inner CG of the mixed form).
//
// A sweep applies iteration k's update and forms iteration k+1's products in one
// pass: from (r, d) of iteration k and its alpha, beta it computes
//   r' = r - alpha A d,  d' = r' + beta d,  q' = A d'
// and the sums d'.q', r'.q', q'.q', r'.r', so an iteration reads r and d and
// writes r' and d' once (16 + 16 bytes FP64) and has one grid-wide sum.  A CTA
// owns an x-y tile and marches along z: d of a plane is staged in shared memory
// with a two-cell halo and r with a one-cell halo (one TMA box each, two planes
// ahead), d' is computed on the tile and its one-cell ring into shared memory, and
// q' follows one plane behind.  The ring's d' are the neighbours' own expressions
// on the same operands, so all CTAs agree bit for bit.
//
// The solution takes alpha d every second sweep, for two iterations at once: the
// older direction is still in the buffer that this sweep overwrites.
//
// Sweeps alternate their z direction, so each starts on planes still in L2.
//
// What bounds it (256^3 FP64, 153 us an iteration): 41 bytes of DRAM traffic per
// cell would take 104 us at the measured copy rate; the rest is the chain of a
// plane step (box, stencil, barrier, stencil) with 16 warps per SM and 128 of 148
// SMs (tiles of 128 x 16 in 4 chunks of z).  The two-pass kernel moves 60 bytes in
// 207 us.  Mixed: 87 us against 107.
// What mattered: TMA boxes instead of cp.async per thread (235 -> 173 us), four
// cells per thread and no branches around cells (173 -> 153; the loop's overhead per
// step was 3 of 4 instructions).
//
// Built with -fmad=false; the FMAs of the solve are written out.
#include <cuda.h>

#include <algorithm>

#include "afl_brick.cuh"
#include "afl_cg_stream_body.cuh"
#include "afl_sweep_plan.h"

namespace afl {
namespace {

constexpr int kSY = kSweepRows;
constexpr int kAhead = 2;   // planes staged ahead of the one being computed
static_assert(kAhead == 2, "a unit starts with groups -1 and 0; a barrier takes one at a time");
constexpr int kDSlots = 3 + kAhead, kRSlots = 1 + kAhead, kNSlots = 3;

// NC cells per thread, 32 apart in x: tiles of 32 * NC x 16 cells.
template <typename T, int NC>
struct SweepShape {
  static constexpr int BX = 32 * NC;
  static constexpr int XH = 16 / int(sizeof(T));       // staged x halo: boxes start on 16 bytes
  static constexpr int RW = BX + 2 * XH;               // staged row
  // slots of a staged d and r plane, 128-byte aligned as the boxes need
  static constexpr int A = 128 / int(sizeof(T));
  static constexpr int DP = (RW * (kSY + 4) + A - 1) / A * A;
  static constexpr int RP = (RW * (kSY + 2) + A - 1) / A * A;
  static constexpr int NW = BX + 2, NP = NW * (kSY + 2);  // d' plane with its ring
  static constexpr int kRing = 2 * BX + 2 * kSY;
  static constexpr unsigned kDBytes = RW * (kSY + 4) * sizeof(T);
  static constexpr unsigned kRBytes = RW * (kSY + 2) * sizeof(T);
  static constexpr size_t kBytes =
      128 + sizeof(T) * (size_t(kDSlots) * DP + size_t(kRSlots) * RP + size_t(kNSlots) * NP);
};

// ---- TMA boxes and the barriers they complete on ------------------------------------
__device__ __forceinline__ void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_done(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ void tma_box(unsigned dst, const CUtensorMap *map, int x, int y, int z,
                                        unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
// Orders generic-proxy writes to global memory before the TMA reads of a later
// sweep (by the writers after their writes, by the issuer before its reads).
__device__ __forceinline__ void proxy_fence() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// The boxes of a sweep's inputs: r by parity, d by parity, and r[1] with d's halo
// (the first sweep starts d = r).
struct SweepMaps {
  CUtensorMap r[2], d[2], d_first;
};

template <typename T>
struct SweepVecs {
  T *r[2], *d[2];  // by sweep parity
  T *x;            // the solution
};

__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// A CTA's shared memory and the state of its barriers across sweeps.
template <typename T, int NC>
struct SweepSmem {
  using S = SweepShape<T, NC>;
  T *ds, *rs, *ns;
  unsigned ds_at, rs_at, bars;  // shared addresses; kRSlots barriers of 8 bytes
  unsigned parity;              // bit b: parity of barrier b's next completion
  __device__ __forceinline__ SweepSmem(unsigned char *raw, unsigned long long *bar) {
    const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(raw));
    ds = reinterpret_cast<T *>(raw + ((128u - (at & 127u)) & 127u));
    rs = ds + kDSlots * S::DP;
    ns = rs + kRSlots * S::RP;
    ds_at = static_cast<unsigned>(__cvta_generic_to_shared(ds));
    rs_at = static_cast<unsigned>(__cvta_generic_to_shared(rs));
    bars = static_cast<unsigned>(__cvta_generic_to_shared(bar));
    parity = 0;
    if (threadIdx.x == 0) {
      for (int b = 0; b < kRSlots; ++b) mbar_init(bars + 8u * b);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      proxy_fence();
    }
    __syncthreads();
  }
};

// One sweep over this CTA's units: (r, d) behind the maps -> (rout, dout); acc
// gains the four sums.  xup: the solution takes a_old * (old dout) + alpha * d.
// False when a box never arrived.
template <typename T, int NC>
__device__ __forceinline__ bool sweep(const Dims &g, const SweepPlan &pl, const CUtensorMap *rmap,
                                      const CUtensorMap *dmap, T *rout, T *dout, T *x, T alpha,
                                      T beta, T a_old, bool xup, bool up,
                                      SweepSmem<T, NC> &sm, const BrickSums &bs,
                                      double (&acc)[4]) {
  using S = SweepShape<T, NC>;
  const int t = threadIdx.x, lane = t & 31, row = t >> 5;
  const int per_chunk = pl.tiles_x * pl.tiles_y;
  for (int unit = blockIdx.x; unit < pl.units(); unit += gridDim.x) {
    const int ch = unit / per_chunk, tile = unit - ch * per_chunk;
    const int ty = tile / pl.tiles_x, tx = tile - ty * pl.tiles_x;
    const int x0 = tx * S::BX, y0 = ty * kSY;
    const int z0 = ch * pl.depth, cnt = min(pl.depth, g.nz - z0);
    const int base = up ? z0 : z0 + cnt - 1, dir = up ? 1 : -1;
    const int j = y0 + row;
    // Plane p of the march is z = base + dir * p.  d of plane p sits in slot
    // (p + 2) % kDSlots, r in slot (p + 1) % kRSlots.  Step s needs d of planes
    // s-1 .. s+1 and r of plane s; group s brings what it still lacks, on barrier
    // (s + 1) % kRSlots.
    auto box_d = [&](int p, unsigned bar) {
      tma_box(sm.ds_at + unsigned((p + 2) % kDSlots) * unsigned(S::DP * sizeof(T)), dmap,
              x0 - S::XH, y0 - 2, base + dir * p, bar);
    };
    auto group = [&](int s) {
      if (s > cnt) return;
      const unsigned bar = sm.bars + 8u * unsigned((s + 1) % kRSlots);
      mbar_expect(bar, (s == -1 ? 3 : 1) * S::kDBytes + S::kRBytes);
      if (s == -1) {
        box_d(-2, bar);
        box_d(-1, bar);
      }
      box_d(s + 1, bar);
      tma_box(sm.rs_at + unsigned((s + 1) % kRSlots) * unsigned(S::RP * sizeof(T)), rmap,
              x0 - S::XH, y0 - 1, base + dir * s, bar);
    };
    __syncthreads();  // the previous unit (or sweep) is done with the buffers
    if (t == 0) {
      group(-1);
      group(0);
    }

    // the ring cell of this thread (threads below kRing)
    int ri = 0, rj = 0;
    const bool ring = t < S::kRing;
    if (t < 2 * S::BX) {
      ri = t % S::BX;
      rj = t < S::BX ? -1 : kSY;
    } else {
      rj = (t - 2 * S::BX) % kSY;
      ri = t - 2 * S::BX < kSY ? -1 : S::BX;
    }
    // per column: whether it is interior and in the grid, and the diagonal of its
    // cells with both z neighbours
    auto diag2 = [&](int i, int jj) {
      return T(int(i > 1) + int(i + 2 < g.nx) + int(jj > 1) + int(jj + 2 < g.ny) + 2);
    };
    auto inside = [&](int i, int jj) {
      return i >= 1 && i <= g.nx - 2 && jj >= 1 && jj <= g.ny - 2;
    };
    bool in[NC], live[NC];
    T dg2[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int i = x0 + lane + 32 * c;
      in[c] = inside(i, j);
      live[c] = i < g.nx && j < g.ny;
      dg2[c] = diag2(i, j);
    }
    const bool ring_in = ring && inside(x0 + ri, y0 + rj);
    const T ring_dg2 = diag2(x0 + ri, y0 + rj);
    const int o_own = (row + 2) * S::RW + lane + S::XH, o_ring = (rj + 2) * S::RW + ri + S::XH;
    const int n_own = (row + 1) * S::NW + lane + 1, n_ring = (rj + 1) * S::NW + ri + 1;
    T dprev[NC], dmid[NC], rmid[NC];  // own d' of planes s-2 and s-1, own r' of s-1
#pragma unroll
    for (int c = 0; c < NC; ++c) dprev[c] = dmid[c] = rmid[c] = T(0);
    // slots of planes s-1, s, s+1 (d), s (r, and its barrier), s and s-1 (d')
    const T *dm = sm.ds, *d0 = dm + S::DP, *dp = d0 + S::DP;
    const T *const d_end = sm.ds + kDSlots * S::DP;
    T *nw = sm.ns, *np = sm.ns + (kNSlots - 1) * S::NP;
    int rslot = 0;
    int at = ((base - dir) * g.ny + j) * g.nx + x0 + lane;  // own cell of plane s
    const int at_step = dir * g.nxy;
    const T na = -alpha;
    bool q_in = false;  // plane s-1 is interior
    T q_edge = T(0);    // ... and has one z neighbour only

    // (r', d') of a cell; nothing is branched around: staged cells outside the grid
    // are 0, and what a wall cell computes is dropped
    auto update = [&](int o, bool ok, T dg, T mid, const T *r0, T &rv, T &dv) {
      T nb = d0[o - 1];
      nb += d0[o + 1];
      nb += d0[o - S::RW];
      nb += d0[o + S::RW];
      nb += dm[o];
      nb += dp[o];
      const T q = fma_t(dg, mid, -nb);
      const T r_ = fma_t(na, q, r0[o]);
      const T d_ = fma_t(beta, mid, r_);
      rv = ok ? r_ : T(0);
      dv = ok ? d_ : T(0);
    };

    for (int s = -1; s <= cnt; ++s) {
      if (t == 0) group(s + kAhead);  // into slots last read in step s-1
      const int k = base + dir * s;
      const bool own = s >= 0 && s < cnt;
      // the solution's own plane, used at the end of the step
      T xv[NC], od[NC];
      if (xup && own) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          xv[c] = live[c] ? x[at + 32 * c] : T(0);
          od[c] = live[c] ? dout[at + 32 * c] : T(0);
        }
      }
      {
        // this CTA's own copies: nobody else holds them up, and they must have landed
        // before the CTA may leave, so the limit is not the caller's
        const unsigned bar = sm.bars + 8u * unsigned(rslot);
        const unsigned want = (sm.parity >> rslot) & 1u;
        unsigned spins = 0;
        unsigned long long t_start = 0;
        while (!mbar_done(bar, want)) {
          if ((spins++ & 255u) == 0u) {
            const unsigned long long now = global_ns();
            if (spins == 1u) t_start = now;
            if (now - t_start > 2000000000ull) {
              atomicCAS(bs.abort_flag, 0, 1);
              return false;
            }
          }
        }
        sm.parity ^= 1u << rslot;
      }
      const bool kin = k >= 1 && k <= g.nz - 2;
      const T edge = k == 1 || k == g.nz - 2 ? T(1) : T(0);
      const T *const r0 = sm.rs + rslot * S::RP - S::RW;  // rows one less into the halo than d's
      T rnew[NC], dnew[NC], mid[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        mid[c] = d0[o_own + 32 * c];
        update(o_own + 32 * c, in[c] && kin, dg2[c] - edge, mid[c], r0, rnew[c], dnew[c]);
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) nw[n_own + 32 * c] = dnew[c];
      if (ring) {
        T rv, dv;
        update(o_ring, ring_in && kin, ring_dg2 - edge, d0[o_ring], r0, rv, dv);
        nw[n_ring] = dv;
      }
      __syncthreads();  // d' of plane s is complete; step s is done with its planes
      // q' of plane s-1: its d' neighbours in the plane from shared memory, along z
      // from registers (0 in the first steps)
      if (s >= 1) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const T *const n0 = np + n_own + 32 * c;
          T nb = n0[-1];
          nb += n0[1];
          nb += n0[-S::NW];
          nb += n0[S::NW];
          nb += dprev[c];
          nb += dnew[c];
          const T q_ = fma_t(dg2[c] - q_edge, dmid[c], -nb);
          const T q = in[c] && q_in ? q_ : T(0);
          const double qd = double(q), dd = double(dmid[c]), rd = double(rmid[c]);
          acc[0] = __fma_rn(dd, qd, acc[0]);
          acc[1] = __fma_rn(rd, qd, acc[1]);
          acc[2] = __fma_rn(qd, qd, acc[2]);
          acc[3] = __fma_rn(rd, rd, acc[3]);
        }
      }
      if (own) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          if (live[c]) {
            rout[at + 32 * c] = rnew[c];
            dout[at + 32 * c] = dnew[c];
            if (xup) x[at + 32 * c] = fma_t(alpha, mid[c], fma_t(a_old, od[c], xv[c]));
          }
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        dprev[c] = dmid[c];
        dmid[c] = dnew[c];
        rmid[c] = rnew[c];
      }
      q_in = kin;
      q_edge = edge;
      at += at_step;
      dm = d0;
      d0 = dp;
      dp = dp + S::DP == d_end ? sm.ds : dp + S::DP;
      rslot = rslot == kRSlots - 1 ? 0 : rslot + 1;
      np = nw;
      nw = nw + S::NP == sm.ns + kNSlots * S::NP ? sm.ns : nw + S::NP;
    }
  }
  proxy_fence();  // the next sweep reads these writes through TMA
  return true;
}

// The grid-wide total of acc, ordering every CTA's writes before it ahead of the
// reads after it.  The polls cover 4 * kBT / 4 = 512 CTAs.
__device__ __forceinline__ bool sweep_total(const BrickSums &bs, unsigned tag, double (&v)[4],
                                            double *red) {
  brick_partials(v, red);
  brick_publish<true>(bs, tag, red);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Packet *const slot = bs.of(tag) + threadIdx.x;
  const int mine = bs.nblocks * 4 - static_cast<int>(threadIdx.x);
  double *const red2 = red + 4 * kBW;
  RawPacket p[4];
  bool ok = true;
  BoundedWait w;
  for (;;) {
    bool got = true;
#pragma unroll
    for (int n = 0; n < 4; ++n) p[n].ld(mine > n * kBT, slot + n * kBT, tag);
#pragma unroll
    for (int n = 0; n < 4; ++n) got &= p[n].has(tag);
    if (got) break;
    if (!w.again(bs.abort_flag, bs.timeout_ns)) {
      ok = false;
      break;
    }
    __nanosleep(100);  // leaves the issue slots to the SM's other CTA
  }
  __threadfence();
  proxy_fence();
  double x = (p[0].value() + p[1].value()) + (p[2].value() + p[3].value());
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  x += __shfl_xor_sync(0xffffffffu, x, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 16);
  if (lane < 4) red2[warp * 4 + lane] = x;
  const bool all = __syncthreads_and(ok ? 1 : 0) != 0;
  const double y = brick_cta_sum(red2);
#pragma unroll
  for (int a = 0; a < 4; ++a) v[a] = __shfl_sync(0xffffffffu, y, a);
  return all;
}

// ------------------------------------------------------------------ FP64 ----
struct SweepCgArgs {
  SweepMaps maps;
  Dims g;
  SweepPlan plan;
  SweepVecs<double> v;
  const double *b;
  int max_iters;
  double rel_tol;
  SolveReport *report;
};

// Residual of the caller's pressure, wall cells 0 (afl_poisson_brick.cu explains
// how they are carried): sums r.r with them, b.b, their own part.
template <int NC>
__global__ void __launch_bounds__(kBT, NC == 4 ? 1 : 2)
    k_cg_sweep_f64(const __grid_constant__ SweepCgArgs a, const __grid_constant__ BrickSums bs) {
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  __shared__ double red[2 * 4 * kBW];
  __shared__ unsigned long long bar[kRSlots];
  SweepSmem<double, NC> sm(sweep_smem, bar);
  const Dims &g = a.g;
  double *const p = a.v.x;
  const int t0 = blockIdx.x * kBT + threadIdx.x, stride = gridDim.x * kBT;
  unsigned tag = 1;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = t0; c < g.n; c += stride) {
    const Run ru = decode_run<1>(g, c);
    Vec<double, 1> ap;
    lap_p_run<1>(g, ru, p, ap);
    const double bc = a.b[c];
    const bool in = interior(g, ru.i0, ru.j, ru.k);
    const double rv = bc - ap.v[0];
    a.v.r[1][c] = in ? rv : 0.0;
    acc[0] += rv * rv;
    acc[1] += bc * bc;
    acc[2] += in ? 0.0 : bc * bc;
  }
  proxy_fence();
  if (!sweep_total(bs, tag++, acc, red)) return;
  const double delta0 = acc[0], bb = acc[1], walls = acc[2];
  double tol2 = -1.0;
  if (a.rel_tol > 0.0) {
    const double tl = a.rel_tol * sqrt(bb);
    tol2 = tl * tl;
  }
  double delta = delta0, last = delta0;
  int it = 0, converged = 0;
  double s_k = 1.0, gain = 0.0;  // the walls' direction and correction, in units of b
  if (!(delta > 1e-24) || (tol2 >= 0.0 && delta <= tol2)) {  // src/fluid.rs:462
    converged = isfinite(delta) ? 1 : 0;
  } else {
    double alpha = 0.0, beta = 0.0, a_old = 0.0;
    for (;; ++it) {
      // sweep `it`: state it, in the arrays of parity it & 1, from state it - 1
      // (the first one starts d = r)
      const int o = it & 1;
      acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
      if (!sweep<double, NC>(g, a.plan, &a.maps.r[o ^ 1],
                             it == 0 ? &a.maps.d_first : &a.maps.d[o ^ 1], a.v.r[o], a.v.d[o], p,
                             alpha, beta, a_old, it > 0 && o == 0, o == 0, sm, bs, acc))
        return;
      if (blockIdx.x == 0 && threadIdx.x == 0) acc[3] += walls;
      if (!sweep_total(bs, tag++, acc, red)) return;
      if (it > 0) {  // the tests after the previous update (src/fluid.rs:478-481)
        last = acc[3];
        if (!isfinite(last)) break;
        if (last < 1e-20) { converged = 1; break; }
        if (tol2 >= 0.0 && last <= tol2) { converged = 1; break; }
        delta = last;
      }
      if (it >= a.max_iters) break;
      if (fabs(acc[0]) < 1e-28) break;  // src/fluid.rs:469
      a_old = alpha;
      alpha = delta / acc[0];
      beta = __fma_rn(__fma_rn(alpha, acc[2], -2.0 * acc[1]), 1.0 / acc[0], 1.0);
      gain += alpha * s_k;
      s_k = 1.0 + beta * s_k;
    }
    // an odd sweep left its alpha d for the next one
    if (it & 1) {
      const double *const d = a.v.d[0];
      for (int c = t0; c < g.n; c += stride) p[c] = __fma_rn(alpha, d[c], p[c]);
    }
  }
  if (it > 0 && walls != 0.0) {  // without a step 0 * inf would be added
    for (int c = t0; c < g.n; c += stride) {
      const Run ru = decode_run<1>(g, c);
      if (!interior(g, ru.i0, ru.j, ru.k)) p[c] += gain * a.b[c];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.report) {
    SolveReport rep;
    rep.iterations = it;
    rep.refinements = 0;
    rep.converged = converged;
    rep.status = isfinite(last) ? 0 : 4;
    rep.initial_residual = sqrt(delta0);
    rep.final_residual = sqrt(last);
    rep.rhs_norm = sqrt(bb);
    *a.report = rep;
  }
}

// ----------------------------------------------------------------- mixed ----
struct SweepMixedArgs {
  SweepMaps maps;
  Dims g;
  SweepPlan plan;
  SweepVecs<float> v;  // x: the f32 correction e
  double *p;
  const double *b;
  int max_inner, max_total, max_refine;
  double inner_rel_tol, rel_tol;
  SolveReport *report;
};

template <int NC>
__global__ void __launch_bounds__(kBT, 2)
    k_cg_sweep_mixed(const __grid_constant__ SweepMixedArgs a,
                     const __grid_constant__ BrickSums bs) {
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  __shared__ double red[2 * 4 * kBW];
  __shared__ unsigned long long bar[kRSlots];
  SweepSmem<float, NC> sm(sweep_smem, bar);
  const Dims &g = a.g;
  const int t0 = blockIdx.x * kBT + threadIdx.x, stride = gridDim.x * kBT;
  unsigned tag = 1;
  double acc[4];
  // r = b - A p in f64, rounded once to f32; e = 0.  Sums: the f64 r.r, b.b, the
  // rounded r.r and its wall cells' part.
  auto outer_residual = [&] {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    for (int c = t0; c < g.n; c += stride) {
      const Run ru = decode_run<1>(g, c);
      Vec<double, 1> ap;
      lap_p_run<1>(g, ru, a.p, ap);
      const double bc = a.b[c], rv = bc - ap.v[0];
      const float rf = float(rv);
      const bool in = interior(g, ru.i0, ru.j, ru.k);
      a.v.r[1][c] = in ? rf : 0.0f;
      a.v.x[c] = 0.0f;
      acc[0] += rv * rv;
      acc[1] += bc * bc;
      acc[2] += double(rf) * double(rf);
      acc[3] += in ? 0.0 : double(rf) * double(rf);
    }
    proxy_fence();
  };
  outer_residual();
  if (!sweep_total(bs, tag++, acc, red)) return;
  double rr = acc[0];
  const double rr0 = rr, bb = acc[1], walls = acc[3];
  double tol2 = -1.0;
  if (a.rel_tol > 0.0) {
    const double tl = a.rel_tol * sqrt(bb);
    tol2 = tl * tl;
  }
  int total = 0, passes = 0, converged = 0;
  if (!(rr > 1e-24) || (tol2 >= 0.0 && rr <= tol2)) converged = isfinite(rr) ? 1 : 0;
  while (!converged && passes < a.max_refine && total < a.max_total && isfinite(rr)) {
    double inner_rel = a.inner_rel_tol;
    if (tol2 >= 0.0) inner_rel = fmax(inner_rel, 0.5 * sqrt(tol2 / rr));
    double delta = acc[2];
    const double inner_tol2 = inner_rel * inner_rel * delta;
    double s_k = 1.0, gain = 0.0;
    float alpha = 0.0f, beta = 0.0f, a_old = 0.0f;
    int it = 0;
    for (;; ++it, ++total) {
      const int o = it & 1;
      acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
      if (!sweep<float, NC>(g, a.plan, &a.maps.r[o ^ 1],
                            it == 0 ? &a.maps.d_first : &a.maps.d[o ^ 1], a.v.r[o], a.v.d[o],
                            a.v.x, alpha, beta, a_old, it > 0 && o == 0, o == 0, sm, bs, acc))
        return;
      if (blockIdx.x == 0 && threadIdx.x == 0) acc[3] += walls;
      if (!sweep_total(bs, tag++, acc, red)) return;
      if (it > 0) {
        const double dn = acc[3];
        if (!isfinite(dn) || dn <= inner_tol2 || dn < 1e-30) break;
        delta = dn;
      }
      if (it >= a.max_inner || total >= a.max_total) break;
      if (!(fabs(acc[0]) >= 1e-30)) break;
      a_old = alpha;
      const double al = delta / acc[0];
      alpha = float(al);
      beta = float(__fma_rn(__fma_rn(al, acc[2], -2.0 * acc[1]), 1.0 / acc[0], 1.0));
      gain += double(alpha) * s_k;
      s_k = 1.0 + double(beta) * s_k;
    }
    // p += e in f64 (an odd sweep left its alpha d for the next one)
    for (int c = t0; c < g.n; c += stride) {
      float e = a.v.x[c];
      if (it & 1) e = __fmaf_rn(alpha, a.v.d[0][c], e);
      if (walls != 0.0) {
        const Run ru = decode_run<1>(g, c);
        if (!interior(g, ru.i0, ru.j, ru.k)) e = float(a.b[c] * gain);
      }
      a.p[c] = a.p[c] + double(e);
    }
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    if (!sweep_total(bs, tag++, acc, red)) return;
    outer_residual();
    if (!sweep_total(bs, tag++, acc, red)) return;
    rr = acc[0];
    ++passes;
    if (rr < 1e-20 || (tol2 >= 0.0 && rr <= tol2)) converged = 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.report) {
    SolveReport rep;
    rep.iterations = total;
    rep.refinements = passes;
    rep.converged = converged;
    rep.status = isfinite(rr) ? 0 : 4;
    rep.initial_residual = sqrt(rr0);
    rep.final_residual = sqrt(rr);
    rep.rhs_norm = sqrt(bb);
    *a.report = rep;
  }
}

// CTAs that are co-resident, at most what a sum's polls cover.
template <typename T, int NC>
int sweep_ctas(const void *fn) {
  const int smem = static_cast<int>(SweepShape<T, NC>::kBytes);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return 0;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBT, smem);
  return std::min(sms * per_sm, kBT);
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                 const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) !=
          cudaSuccess ||
      found != cudaDriverEntryPointSuccess)
    return nullptr;
  return reinterpret_cast<EncodeTiled>(fn);
}

template <typename T, int NC>
bool encode(EncodeTiled fn, CUtensorMap *map, const Dims &g, T *base, int rows) {
  using S = SweepShape<T, NC>;
  const cuuint64_t dims[3] = {cuuint64_t(g.nx), cuuint64_t(g.ny), cuuint64_t(g.nz)};
  const cuuint64_t strides[2] = {cuuint64_t(g.nx) * sizeof(T), cuuint64_t(g.nxy) * sizeof(T)};
  const cuuint32_t box[3] = {cuuint32_t(S::RW), cuuint32_t(rows), 1}, unit[3] = {1, 1, 1};
  return fn(map, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
            3, base, dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 0 when the sweep does not pay, or there are no tensor maps for it (the caller keeps the
// two-pass kernel).
template <typename T, int NC, typename Args>
int launch_sweep(const void *fn, Args a, const PersistentState &ps, cudaStream_t st) {
  int ctas = sweep_ctas<T, NC>(fn);
  // the sums' slots take the place of the streaming kernels' partials
  ctas = std::min(ctas, static_cast<int>(12 * sizeof(double) * size_t(ps.max_blocks) /
                                         (8 * sizeof(Packet))));
  if (ctas < 1) return 0;
  a.plan = sweep_plan(a.g, NC, ctas);
  if (!sweep_pays(a.g, a.plan, NC, ctas, sizeof(T) == 8)) return 0;
  const EncodeTiled enc = encode_tiled();
  bool ok = enc != nullptr;
  for (int q = 0; q < 2 && ok; ++q)
    ok = encode<T, NC>(enc, &a.maps.r[q], a.g, a.v.r[q], kSY + 2) &&
         encode<T, NC>(enc, &a.maps.d[q], a.g, a.v.d[q], kSY + 4);
  ok = ok && encode<T, NC>(enc, &a.maps.d_first, a.g, a.v.r[1], kSY + 4);
  if (!ok) {
    cudaGetLastError();
    return 0;
  }
  const int blocks = std::min(ctas, a.plan.units());
  cudaMemsetAsync(ps.abort_flag, 0, sizeof(int), st);
  cudaMemsetAsync(ps.partials, 0, sizeof(Packet) * 8 * static_cast<size_t>(blocks), st);
  BrickSums bs{reinterpret_cast<Packet *>(ps.partials), blocks, ps.abort_flag, ps.timeout_ns};
  void *params[] = {&a, &bs};
  const cudaError_t err = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kBT), params,
                                                      SweepShape<T, NC>::kBytes, st);
  return err == cudaSuccess ? blocks : -static_cast<int>(err);
}

}  // namespace

bool sweep_fits(const Dims &g, bool f64) {
  int dev = 0, l2 = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
  return sweep_fits(g, f64, static_cast<size_t>(l2));
}

int launch_cg_sweep_f64(const CgArgs &a, const PersistentState &ps, cudaStream_t st) {
  SweepCgArgs s{{}, a.g, {}, {{a.r, a.q}, {a.d0, a.d1}, a.p}, a.b, a.max_iters, a.rel_tol,
                a.report};
  if (sweep_wide(a.g))
    return launch_sweep<double, 4>(reinterpret_cast<const void *>(&k_cg_sweep_f64<4>), s, ps, st);
  return launch_sweep<double, 1>(reinterpret_cast<const void *>(&k_cg_sweep_f64<1>), s, ps, st);
}

int launch_cg_sweep_mixed(const MixedCgArgs &a, const PersistentState &ps, cudaStream_t st) {
  SweepMixedArgs s{{},           a.g,          {},
                   {{a.r, a.q}, {a.d0, a.d1}, a.e},
                   a.p,          a.b,          a.max_inner,
                   a.max_total,  a.max_refine, a.inner_rel_tol,
                   a.rel_tol,    a.report};
  return launch_sweep<float, 4>(reinterpret_cast<const void *>(&k_cg_sweep_mixed<4>), s, ps, st);
}

}  // namespace afl
