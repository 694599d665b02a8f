// afl_sor_brick.cu -- brick-resident red-black SOR (solve_poisson_gauss_seidel,
// src/fluid.rs:397-442), FP64 and the mixed form's f32 correction: all sweeps in
// one cooperative launch with the solved quantity in shared memory and the
// right-hand side in registers.
//
// A half-sweep updates the cells of one colour in place (each reads only the
// other colour), sends the face cells it changed to the neighbours as tagged
// packets, and takes the neighbours' packets of that colour into its ring.  CTAs
// wait only for their neighbours; there is no grid-wide barrier.  The FP64 update
// is the reference's expression with its neighbour order, so a sweep equals the
// reference's bit for bit.
//
// What bounds it (128^3 FP64, cycles of one 11.1 k cycle half-sweep, stamped per
// CTA): the update 8 k (six shared-memory reads and one write of 8 bytes per
// updated cell take 3.6 k, 14 FP64 operations 1.8 k, the sends of the face warps
// the rest), the wait for the slowest neighbour 1.9 k, the barrier 0.7 k.
// Per half-sweep, CUDA events over 80 sweeps, against the streaming sweep (two
// L2 passes and a grid barrier each):
//   FP64 128^3 13.2 -> 5.9 us, 96 x 96 x 97 9.0 -> 3.9, 64^3 7.3 -> 2.3;
//   mixed 128^3 12.4 -> 4.0 us, 64^3 6.8 -> 1.8.
// What mattered: the right-hand side in registers (b re-read from L2 every
// half-sweep kept the FP64 column tiles behind the streaming sweep), and the
// quotient by an exact Newton step (a wall lane's 0/d took its whole warp through
// the division's slow path: 7.8 us).
//
// Built with -fmad=false.
#include "afl_brick.cuh"

namespace afl {
namespace {

template <typename T>
struct BrickSorArgs {
  Dims g;
  int nbx, nby, nbz, cz, czp;
  double *p;
  const double *b;
  typename PacketOf<T>::Mem *inbox;
  int *abort_flag;
  unsigned long long timeout_ns;
  int sweeps;
  double omega;
  SolveReport *report;
};

// x / d for d = 3 .. 6, correctly rounded, with rd = 1/d rounded to nearest:
// one Newton correction of x * rd by the exact remainder gives the rounded
// quotient when the reciprocal is correctly rounded and nothing over- or
// underflows (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  div_unsafe: x outside a safe exponent range
// (zeros, subnormals, infinities, NaN), where the division itself is due unless
// x is 0.
__device__ __forceinline__ double div_small(double x, double d, double rd) {
  const double q = x * rd;
  return __fma_rn(__fma_rn(-d, q, x), rd, q);
}
__device__ __forceinline__ bool div_unsafe(double x) {
  return (static_cast<unsigned>(__double2hiint(x)) & 0x7fffffffu) - 0x08000000u > 0x6ff00000u;
}
__device__ __forceinline__ float div_small(float x, float d, float rd) {
  const float q = x * rd;
  return __fmaf_rn(__fmaf_rn(-d, q, x), rd, q);
}
__device__ __forceinline__ bool div_unsafe(float x) {
  return (__float_as_uint(x) & 0x7fffffffu) - 0x10000000u > 0x5f000000u;
}

// Right-hand side of one cell's sweep: b (FP64), or the f64 residual b - A p
// rounded once (mixed).
template <typename T>
__device__ __forceinline__ T sor_rhs(const Dims &g, const double *p, const double *b, int c, int i,
                                     int j, int k) {
  if constexpr (sizeof(T) == 8) {
    return b[c];
  } else {
    double diag = 0.0, nb = 0.0;
    if (i > 1) { diag += 1.0; nb += p[c - 1]; }
    if (i + 2 < g.nx) { diag += 1.0; nb += p[c + 1]; }
    if (j > 1) { diag += 1.0; nb += p[c - g.nx]; }
    if (j + 2 < g.ny) { diag += 1.0; nb += p[c + g.nx]; }
    if (k > 1) { diag += 1.0; nb += p[c - g.nxy]; }
    if (k + 2 < g.nz) { diag += 1.0; nb += p[c + g.nxy]; }
    return float(b[c] - (diag * p[c] - nb));
  }
}

template <typename T, int BX, int CZ>
__global__ void __launch_bounds__(kBT, 1) k_sor_brick(const __grid_constant__ BrickSorArgs<T> a) {
  using S = BrickShape<BX>;
  using Raw = typename PacketOf<T>::Raw;
  constexpr int NI = (CZ + S::kLanes - 1) / S::kLanes;  // side ring cells per thread
  constexpr int SXY = S::SXY, H = CZ / 2, U = H < 4 ? H : 4;
  constexpr int RSTEP = S::kLanes * S::kSide;
  extern __shared__ __align__(16) unsigned char smem[];
  T *const P = reinterpret_cast<T *>(smem);  // plane cz of a column: the cell above it
  const Dims &g = a.g;
  const int t = threadIdx.x;
  const int cz = a.cz;
  const BrickCells<S> cl(g, a.nbx, a.nby, cz, t, static_cast<int>(blockIdx.x));
  const BrickFaces<S> fc(g, cl, a.nbx, a.nby, a.nbz, a.czp, t);
  T *const Pc = P + (t / S::BX + 1) * S::SX + t % S::BX + 1;
  T *const Z = P + (CZ + 1) * SXY + t;  // the cell below the column
  const int k0 = cl.z0, k_lo = 2 - k0, k_hi = min(g.nz - 3 - k0, cl.nzb - 1);
  const bool col_in = cl.column_interior(g);
  // A face carries values only between two interior cells: a wall cell reads
  // none, and the handshake below needs an answer at every position sent to.
  const int side_s = t % S::kSide;
  const int oi = fc.si + (side_s < S::BY ? 1 : side_s < 2 * S::BY ? -1 : 0);
  const int oj = fc.sj + (side_s < 2 * S::BY ? 0 : side_s < 2 * S::BY + S::BX ? 1 : -1);
  const bool side_in = min(fc.si, oi) >= 1 && max(fc.si, oi) <= g.nx - 2 &&
                       min(fc.sj, oj) >= 1 && max(fc.sj, oj) <= g.ny - 2;
  const int ii = t % S::BX, jj = t / S::BX;
  const bool xsend = fc.xcol >= 0 && (ii == 0 ? cl.i >= 2 : cl.i <= g.nx - 3);
  const bool ysend = fc.ydst >= 0 && (jj == 0 ? cl.j >= 2 : cl.j <= g.ny - 3);
  const bool zlo = fc.zlo_dst >= 0 && col_in && k0 >= 2 && k0 <= g.nz - 2;
  const bool zhi = fc.zhi_dst >= 0 && col_in && k0 + cz >= 2 && k0 + cz <= g.nz - 2;
  const int side_par = (fc.si + fc.sj + k0 + t / S::kSide) & 1;
  const int par = (cl.i + cl.j + k0) & 1;  // colour of plane 0's cell

  // The solved quantity on the brick and its ring: the pressure, or a zero
  // correction; wall cells (which no cell reads) stay 0.  The thread's cell s of
  // colour c is plane 2s + (c ^ par).
  T rhs[2][H];
  for (int s = t; s < (CZ + 1) * SXY; s += kBT) P[s] = T(0);
  *Z = T(0);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int s = 0; s < H; ++s) {
      const int m = 2 * s + (c ^ par), k = k0 + m;
      rhs[c][s] = T(0);
      if (col_in && m < cl.nzb && k >= 1 && k <= g.nz - 2) {
        const int at = cl.c0 + m * g.nxy;
        rhs[c][s] = sor_rhs<T>(g, a.p, a.b, at, cl.i, cl.j, k);
        if constexpr (sizeof(T) == 8) Pc[m * SXY] = a.p[at];
      }
    }
  if constexpr (sizeof(T) == 8) {
    if (zlo) *Z = a.p[cl.c0 - g.nxy];
    if (zhi) Pc[cz * SXY] = a.p[cl.c0 + cz * g.nxy];
    for (int n = 0; side_in && n * S::kLanes < fc.side_lim; ++n) {
      const int k = k0 + t / S::kSide + n * S::kLanes;
      if (k >= 1 && k <= g.nz - 2)
        P[fc.side_d + n * S::kLanes * SXY] = a.p[(k * g.ny + fc.sj) * g.nx + fc.si];
    }
  }
  // What was read of the neighbours' pressure stays ordered before their writes of it at
  // the end: they have had a packet of this CTA's by then, and the fence there is the
  // other half.
  __threadfence();
  __syncthreads();

  const T omega = T(a.omega), keep = T(1) - omega;
  const int d2 = cl.diag2(g);
  const T dg2 = T(d2), dg1 = T(d2 - 1), rd2 = T(1) / dg2, rd1 = T(1) / dg1;
  auto *const box = a.inbox;
  // ring cells of either colour that this thread takes in: bit n side cell n, bits
  // NI and NI + 1 the cells below and above its column
  unsigned ring_on[2] = {0, 0};
  for (int n = 0; n < NI; ++n) {
    const int k = k0 + t / S::kSide + n * S::kLanes;
    if (side_in && n * S::kLanes < fc.side_lim && k >= 1 && k <= g.nz - 2)
      ring_on[(side_par + n * S::kLanes) & 1] |= 1u << n;
  }
  if (zlo) ring_on[par ^ 1] |= 1u << NI;
  if (zhi) ring_on[(par + cz) & 1] |= 2u << NI;
  unsigned tag = 1;
  for (int sweep = 0; sweep < a.sweeps; ++sweep) {
#pragma unroll
    for (int c = 0; c < 2; ++c, ++tag) {
      const int o = c ^ par;
      T *const Po = Pc + o * SXY;
      auto *const xd = box + fc.xcol + o * S::kSide, *const yd = box + fc.ydst + o * S::kSide;
      // U cells at a time, all loads before the first store, which would order them
#pragma unroll
      for (int s0 = 0; s0 < H; s0 += U) {
        if (2 * s0 >= cz) break;
        T v[U];
        unsigned in = col_in ? (1u << U) - 1u : 0u;  // bit u: cell u is updated
        T dg[U], rd[U];
        const bool plain = 2 * s0 >= k_lo && 2 * (s0 + U) - 1 <= k_hi;  // for all threads
#pragma unroll
        for (int u = 0; u < U; ++u) {
          dg[u] = dg2;
          rd[u] = rd2;
        }
        if (!plain) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int m = 2 * (s0 + u) + o, k = k0 + m;
            if (k == 1 || k == g.nz - 2) {
              dg[u] = dg1;
              rd[u] = rd1;
            }
            if (k < 1 || k > g.nz - 2 || m >= cz) in &= ~(1u << u);
          }
        }
        bool odd = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int s = s0 + u;
          const T *const x = Po + 2 * s * SXY;
          T nb = x[-1];
          nb += x[1];
          nb += x[-S::SX];
          nb += x[S::SX];
          nb += s == 0 && o == 0 ? *Z : x[-SXY];
          nb += x[SXY];
          v[u] = rhs[c][s] + nb;
        }
        T target[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          target[u] = div_small(v[u], dg[u], rd[u]);
          odd |= div_unsafe(v[u]);
        }
        if (odd && in) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (div_unsafe(v[u]) && v[u] != T(0)) target[u] = v[u] / dg[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = keep * Po[2 * (s0 + u) * SXY] + omega * target[u];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (in >> u & 1u) Po[2 * (s0 + u) * SXY] = v[u];
        if (xsend) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (in >> u & 1u) st_packet(xd + 2 * (s0 + u) * S::kSide, v[u], tag);
        }
        if (ysend) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (in >> u & 1u) st_packet(yd + 2 * (s0 + u) * S::kSide, v[u], tag);
        }
        if (zlo && s0 == 0 && o == 0 && (in & 1u)) st_packet(box + fc.zlo_dst, v[0], tag);
        if (zhi && 2 * (s0 + U) >= cz) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (2 * (s0 + u) + o == cz - 1 && (in >> u & 1u)) st_packet(box + fc.zhi_dst, v[u], tag);
        }
      }
      // The ring cells of this colour.  Nobody reads them in this half-sweep; a
      // packet's slot is free again once the neighbour has had this CTA's answer
      // at the same face position, one half-sweep later.
      const auto *const own = box + fc.own + t;
      const unsigned on = ring_on[c];
      Raw lo, hi, side[NI];
      int ok = 1;
      BoundedWait w;
      for (;;) {
        lo.ld(on >> NI & 1u, own + S::kSide * a.czp, tag);
        hi.ld(on >> NI & 2u, own + S::kSide * a.czp + kBT, tag);
#pragma unroll
        for (int n = 0; n < NI; ++n) side[n].ld(on >> n & 1u, own + n * RSTEP, tag);
        bool got = lo.has(tag) & hi.has(tag);
#pragma unroll
        for (int n = 0; n < NI; ++n) got &= side[n].has(tag);
        if (got) break;
        if (!w.again(a.abort_flag, a.timeout_ns)) {
          ok = 0;
          break;
        }
      }
      if (on >> NI & 1u) *Z = lo.value();
      if (on >> NI & 2u) Pc[cz * SXY] = hi.value();
#pragma unroll
      for (int n = 0; n < NI; ++n)
        if (on >> n & 1u) P[fc.side_d + n * S::kLanes * SXY] = side[n].value();
      if (!__syncthreads_and(ok)) return;
    }
  }
  __threadfence();
  __syncthreads();
#pragma unroll
  for (int m = 0; m < CZ; ++m) {
    const int k = k0 + m;
    if (m >= cl.nzb || !col_in || k < 1 || k > g.nz - 2) continue;
    double &p = a.p[cl.c0 + m * g.nxy];
    if constexpr (sizeof(T) == 8) p = Pc[m * SXY];
    else p = p + double(Pc[m * SXY]);
  }
  if (blockIdx.x == 0 && t == 0 && a.report) {
    SolveReport rep{};
    rep.iterations = a.sweeps;
    rep.refinements = sizeof(T) == 8 ? 0 : 1;
    *a.report = rep;
  }
}

template <typename T, int BX>
const void *sor_fn(int cz) {
  if (cz <= 4) return reinterpret_cast<const void *>(&k_sor_brick<T, BX, 4>);
  if (cz <= 8) return reinterpret_cast<const void *>(&k_sor_brick<T, BX, 8>);
  if constexpr (BX < 64) {
    if (cz > 16) return reinterpret_cast<const void *>(&k_sor_brick<T, BX, 32>);
  }
  return reinterpret_cast<const void *>(&k_sor_brick<T, BX, 16>);
}

template <typename T, int BX>
size_t sor_smem(int cz) {
  using S = BrickShape<BX>;
  const int c = cz <= 4 ? 4 : cz <= 8 ? 8 : cz <= 16 ? 16 : 32;
  return sizeof(T) * (static_cast<size_t>(c + 1) * S::SXY + kBT);
}

template <typename T>
int launch(const BrickSor &s, const BrickPlan &plan, cudaStream_t st) {
  const void *fn = plan.bx == 32   ? sor_fn<T, 32>(plan.cz)
                   : plan.bx == 16 ? sor_fn<T, 16>(plan.cz)
                                   : sor_fn<T, 64>(plan.cz);
  const size_t smem = plan.bx == 32   ? sor_smem<T, 32>(plan.cz)
                      : plan.bx == 16 ? sor_smem<T, 16>(plan.cz)
                                      : sor_smem<T, 64>(plan.cz);
  cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
  if (err != cudaSuccess) return -static_cast<int>(err);
  using Mem = typename PacketOf<T>::Mem;
  // one inbox per CTA; packets start without a tag
  const size_t inbox = plan.inbox_bytes / (2 * sizeof(Packet)) * sizeof(Mem);
  cudaMemsetAsync(s.scratch, 0, kBrickHeader + inbox, st);
  auto *base = static_cast<unsigned char *>(s.scratch);
  BrickSorArgs<T> a{s.g, plan.nbx, plan.nby, plan.nbz, plan.cz, (plan.cz + 3) / 4 * 4, s.p, s.b,
                    reinterpret_cast<Mem *>(base + kBrickHeader), reinterpret_cast<int *>(base),
                    s.timeout_ns, s.sweeps, s.omega, s.report};
  void *params[] = {&a};
  err = cudaLaunchCooperativeKernel(fn, dim3(plan.ctas()), dim3(kBT), params, smem, st);
  return err == cudaSuccess ? plan.ctas() : -static_cast<int>(err);
}

}  // namespace

int launch_sor_brick(const BrickSor &s, const BrickPlan &plan, bool f64, cudaStream_t st) {
  return f64 ? launch<double>(s, plan, st) : launch<float>(s, plan, st);
}

}  // namespace afl
