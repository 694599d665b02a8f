// afl_brick.cuh -- the pieces shared by the brick-resident Poisson kernels
// (afl_poisson_brick.cu): where a CTA's cells sit, the tagged packets that
// carry face values between neighbouring CTAs, the tagged grid-wide sums, and
// tensor memory as per-thread storage.
//
// A CTA of 512 threads owns a brick of BX x BY x cz cells (BX * BY = 512):
// one thread per (x, y) column, marching up the brick's cz planes.  Splitting
// z as well as x and y keeps the faces small (a 32 x 16 x 32 brick has 4096
// neighbour cells where a 16 x 8 column over 128 planes has 6144) and lets a
// small grid spread over all SMs with few planes per thread.
//
// No fence, no counter and no acquire is on an iteration's path: every word
// that crosses CTAs carries the number of the exchange in its upper half and
// half of a double in its lower half (aligned 64-bit stores are single-copy
// atomic), so seeing the tag is seeing the data.
#pragma once

#include "afl_launch.h"

namespace afl {
namespace {

constexpr int kBT = 512;        // threads per CTA
constexpr int kBW = kBT / 32;   // warps per CTA

// ---- tagged words ------------------------------------------------------------
struct alignas(16) Packet {
  unsigned long long lo, hi;  // tag << 32 | half of the double
};

__device__ __forceinline__ void st_packet(Packet *p, double v, unsigned tag) {
  unsigned long long a, b;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(__double2loint(v)), "r"(tag));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "r"(__double2hiint(v)), "r"(tag));
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b)
               : "memory");
}

// A packet on the way in; loading and checking are apart, so that several loads
// are in flight at once (a packet that is not wanted reads as a tagged 0).
struct RawPacket {
  unsigned long long a, b;
  __device__ __forceinline__ void ld(bool on, const Packet *p, unsigned tag) {
    a = b = static_cast<unsigned long long>(tag) << 32;
    asm volatile(
        "{\n.reg .pred on;\nsetp.ne.s32 on, %3, 0;\n"
        "@on ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n}"
        : "+l"(a), "+l"(b)
        : "l"(p), "r"(static_cast<int>(on))
        : "memory");
  }
  __device__ __forceinline__ bool has(unsigned tag) const {
    return (static_cast<unsigned>(a >> 32) == tag) & (static_cast<unsigned>(b >> 32) == tag);
  }
  __device__ __forceinline__ double value() const {
    return __hiloint2double(static_cast<int>(b & 0xffffffffull),
                            static_cast<int>(a & 0xffffffffull));
  }
};

// The f32 form: one word.
__device__ __forceinline__ void st_packet(unsigned long long *p, float v, unsigned tag) {
  unsigned long long a;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(__float_as_uint(v)), "r"(tag));
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
struct RawWord {
  unsigned long long a;
  __device__ __forceinline__ void ld(bool on, const unsigned long long *p, unsigned tag) {
    a = static_cast<unsigned long long>(tag) << 32;
    asm volatile(
        "{\n.reg .pred on;\nsetp.ne.s32 on, %2, 0;\n"
        "@on ld.relaxed.gpu.global.u64 %0, [%1];\n}"
        : "+l"(a)
        : "l"(p), "r"(static_cast<int>(on))
        : "memory");
  }
  __device__ __forceinline__ bool has(unsigned tag) const {
    return static_cast<unsigned>(a >> 32) == tag;
  }
  __device__ __forceinline__ float value() const {
    return __uint_as_float(static_cast<unsigned>(a & 0xffffffffull));
  }
};
// The packet of a value type: its word(s) in memory, and one on the way in.
template <typename T>
struct PacketOf;
template <>
struct PacketOf<double> {
  using Mem = Packet;
  using Raw = RawPacket;
};
template <>
struct PacketOf<float> {
  using Mem = unsigned long long;
  using Raw = RawWord;
};

// Bookkeeping of a bounded wait: call once per failed poll; false = give up
// (another CTA aborted, or the limit ran out; a limit of 0 gives up at the
// first failed poll).
struct BoundedWait {
  unsigned spins = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool again(int *abort_flag, unsigned long long limit_ns) {
    if ((spins++ & 255u) == 0u) {
      const unsigned long long now = global_ns();
      if (spins == 1u) t0 = now;
      if (ld_relaxed_i32(abort_flag) != 0) return false;
      if (limit_ns == 0 || now - t0 > limit_ns) {
        atomicCAS(abort_flag, 0, 1);
        return false;
      }
    }
    return true;
  }
};

// ---- grid-wide sums of four doubles ---------------------------------------------
// CTA b's partials of sum number `tag` are four packets at
// slots[(tag & 1) * nblocks + b][4].  A CTA publishes sum k+1 only after it has
// read all of sum k, and k+2 only after every CTA published k+1, so the two
// halves never mix.  Slots start at 0, tags at 1.
struct BrickSums {
  static constexpr bool kQueued = false;
  Packet *slots;
  int nblocks;
  int *abort_flag;
  unsigned long long timeout_ns;
  __device__ __forceinline__ Packet *of(unsigned tag) const {
    return slots + static_cast<size_t>(tag & 1u) * 4 * nblocks;
  }
  __device__ __forceinline__ int block() const { return static_cast<int>(blockIdx.x); }
};
// ... of one system of several in a launch (afl_launch.h, BrickQueue): this CTA is
// block vblock of it.
struct QueuedSums : BrickSums {
  static constexpr bool kQueued = true;
  int vblock;
  __device__ __forceinline__ int block() const { return vblock; }
};

// First half of publishing a sum: warp sums of v (a butterfly that halves the
// values per lane first: 6 double shuffles instead of 20) into `red` (4 * kBW
// doubles).  Ends with a CTA barrier.
__device__ __forceinline__ void brick_partials(const double (&v)[4], double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool h16 = lane & 16, h8 = lane & 8;
  double k0 = h16 ? v[2] : v[0], k1 = h16 ? v[3] : v[1];
  const double s0 = h16 ? v[0] : v[2], s1 = h16 ? v[1] : v[3];
  k0 += __shfl_xor_sync(0xffffffffu, s0, 16);
  k1 += __shfl_xor_sync(0xffffffffu, s1, 16);
  double x = h8 ? k1 : k0;
  x += __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  if ((lane & 7) == 0) red[warp * 4 + (lane >> 3)] = x;  // lane >> 3 = value held
  __syncthreads();
}

// The CTA's partial of value lane & 3 in every thread, from `red`.
__device__ __forceinline__ double brick_cta_sum(const double *red) {
  const int lane = threadIdx.x & 31;
  double y = red[lane] + red[lane + 32];
  y += __shfl_xor_sync(0xffffffffu, y, 4);
  y += __shfl_xor_sync(0xffffffffu, y, 8);
  y += __shfl_xor_sync(0xffffffffu, y, 16);
  return y;
}

// Second half: warp 0 publishes the CTA's partials as sum number `tag`.
// RELEASE: also releases the CTA's writes before the barrier.
template <bool RELEASE, typename Sums>
__device__ __forceinline__ void brick_publish(const Sums &bs, unsigned tag, const double *red) {
  if (threadIdx.x >= 32) return;
  const double y = brick_cta_sum(red);
  if (threadIdx.x < 4) {
    if (RELEASE) __threadfence();
    st_packet(bs.of(tag) + bs.block() * 4 + threadIdx.x, y, tag);
  }
}

// The fixed-order total of sum number `tag` in every thread: thread t polls value t & 3
// of CTA t / 4 (and of CTA t / 4 + 128), warps and then the CTA add them up.  `ok`
// (this thread's waits so far) is combined over the CTA; false = a wait gave up and
// the kernel must unwind.
__device__ __forceinline__ bool brick_gather(const BrickSums &bs, unsigned tag, double (&out)[4],
                                             double *red, bool ok) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Packet *const slot = bs.of(tag) + threadIdx.x;
  const int mine = bs.nblocks * 4 - static_cast<int>(threadIdx.x);
  RawPacket r0, r1;
  BoundedWait w;
  for (;;) {
    r0.ld(mine > 0, slot, tag);
    r1.ld(mine > kBT, slot + kBT, tag);
    if (r0.has(tag) & r1.has(tag)) break;
    if (!w.again(bs.abort_flag, bs.timeout_ns)) {
      ok = false;
      break;
    }
  }
  double x = r0.value() + r1.value();
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  x += __shfl_xor_sync(0xffffffffu, x, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 16);
  if (lane < 4) red[warp * 4 + lane] = x;
  const bool all = __syncthreads_and(ok ? 1 : 0) != 0;
  const double y = brick_cta_sum(red);
#pragma unroll
  for (int a = 0; a < 4; ++a) out[a] = __shfl_sync(0xffffffffu, y, a);
  return all;
}
static_assert(2 * kBT >= 4 * 160, "two polls per thread cover every CTA");

// ---- geometry ----------------------------------------------------------------
template <int BX_>
struct BrickShape {
  static constexpr int BX = BX_, BY = kBT / BX_;
  static constexpr int SX = BX + 2, SXY = SX * (BY + 2);  // shared plane with its side ring
  static constexpr int kSide = 2 * (BX + BY);             // side ring cells per plane
  static constexpr int kLanes = kBT / kSide;              // planes the ring threads cover at once
  static constexpr int kXLanes = kBT / (2 * BY);          // planes the x-face senders cover at once
  // Offsets at which the CG kernels send face values (-1: not sent), from those of
  // BrickFaces: a y face's plane m, the n-th staged x value of thread t; and whether a
  // thread's n-th side ring cell is waited for.  In a queue a CTA sends exactly what is
  // waited for: a packet that nobody reads could land after its receiver has gone on to
  // another system and cleared its inbox for that one.  A launch with one system has no
  // such next one, and sends its last chunk's padding planes and the rows past the grid as
  // well: tests of every plane cost it 3 % of an iteration of 128^3 (mixed 9 %), the test of
  // the rows alone 2 % of mixed 36 x 52 x 36.  A queue tests a whole chunk first
  // (the 48 plumes, 4 steps, tests of every plane -> this: 46.5 -> 45.4 ms).
  static __host__ __device__ __forceinline__ int y_at(int ydst, int m, int nzb) {
    return ydst >= 0 && m < nzb ? ydst + m * kSide : -1;
  }
  template <bool QUEUED>
  static __host__ __device__ __forceinline__ int x_at(int xdst, int t, int n, int cz, int nzb) {
    return xdst >= 0 && t / (2 * BY) + n * kXLanes < (QUEUED ? nzb : cz)
               ? xdst + n * kXLanes * kSide : -1;
  }
  static __host__ __device__ __forceinline__ bool side_on(int n, int side_lim) {
    return n * kLanes < side_lim;
  }
};

// Packets of one CTA's inbox for one parity: kSide per plane (x-, x+, y-, y+
// faces), then the z- and the z+ face.  czp = cz rounded up to 4.
__host__ __device__ inline int brick_inbox_packets(int side, int czp) {
  return side * czp + 2 * kBT;
}

// A thread's column.
template <typename S>
struct BrickCells {
  int bx, by, bz;        // the brick
  int i, j, z0, nzb;     // column; first plane; planes of the brick inside the grid
  bool in_ij;
  int c0;                // global index of the column's cell in plane 0
  __host__ __device__ __forceinline__ BrickCells(const Dims &g, int nbx, int nby, int cz, int t,
                                                 int block) {
    bx = block % nbx;
    const int q = block / nbx;
    by = q % nby;
    bz = q / nby;
    i = bx * S::BX + t % S::BX;
    j = by * S::BY + t / S::BX;
    z0 = bz * cz;
    nzb = cz < g.nz - z0 ? cz : g.nz - z0;
    in_ij = i < g.nx && j < g.ny;
    c0 = (z0 * g.ny + j) * g.nx + i;
  }
  __device__ __forceinline__ bool column_interior(const Dims &g) const {
    return i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2;
  }
  // the operator's diagonal at a cell of the column with both z neighbours
  __device__ __forceinline__ int diag2(const Dims &g) const {
    return int(i > 1) + int(i + 2 < g.nx) + int(j > 1) + int(j + 2 < g.ny) + 2;
  }
};

// Where a thread sends face values, and the ring cells it looks after: side
// ring position t % kSide in every kLanes-th plane from t / kSide, and the
// cells below and above its own column.  Offsets are packets from the start of
// the inboxes (-1: no neighbour there).  The y and z faces are sent by the
// columns' own threads as they are computed; the x faces, which only the first
// and the last lane of a row hold, are staged in shared memory ([plane][x-
// rows, x+ rows]) and sent by all threads: thread t sends staged row
// t % (2 * BY) of every kXLanes-th plane.
// QUEUED: rows past the grid have no x face (BrickShape::x_at).
template <typename S, bool QUEUED = false>
struct BrickFaces {
  int xstage;         // this column's staged row (-1: not on an x face)
  int xdst;           // where the thread's first staged value goes; kSide packets per plane
  int xcol;           // where plane 0 of an x-face column goes when it is sent directly
  int ydst;           // plane 0 of the column; kSide packets further per plane
  int zlo_dst, zhi_dst;
  int own;            // this CTA's inbox
  int side_lim;       // the thread's n-th side ring cell exists when n * kLanes < side_lim
  int side_d;         // its shared index in D for n = 0
  int si, sj;         // column of the side ring position
  __host__ __device__ __forceinline__ BrickFaces(const Dims &g, const BrickCells<S> &cl, int nbx,
                                                 int nby, int nbz, int czp, int t) {
    const int ii = t % S::BX, jj = t / S::BX;
    const int per = brick_inbox_packets(S::kSide, czp);
    auto box = [&](int dx, int dy, int dz) {
      return per * (((cl.bz + dz) * nby + cl.by + dy) * nbx + cl.bx + dx);
    };
    const int zface = S::kSide * czp;
    own = box(0, 0, 0);
    ydst = zlo_dst = zhi_dst = -1;
    xstage = ii == 0 ? jj : ii == S::BX - 1 ? S::BY + jj : -1;
    {
      const int xs = t % (2 * S::BY), m0 = t / (2 * S::BY) * S::kSide;
      xdst = xs < S::BY ? (cl.bx > 0 ? box(-1, 0, 0) + S::BY + xs + m0 : -1)
                        : (cl.bx + 1 < nbx ? box(1, 0, 0) + xs - S::BY + m0 : -1);
      if (QUEUED && cl.by * S::BY + xs % S::BY >= g.ny) xdst = -1;
    }
    xcol = -1;
    if (cl.in_ij) {
      if (ii == 0 && cl.bx > 0) xcol = box(-1, 0, 0) + S::BY + jj;
      if (ii == S::BX - 1 && cl.bx + 1 < nbx) xcol = box(1, 0, 0) + jj;
      if (jj == 0 && cl.by > 0) ydst = box(0, -1, 0) + 2 * S::BY + S::BX + ii;
      if (jj == S::BY - 1 && cl.by + 1 < nby) ydst = box(0, 1, 0) + 2 * S::BY + ii;
      if (cl.bz > 0) zlo_dst = box(0, 0, -1) + zface + kBT + t;
      if (cl.bz + 1 < nbz) zhi_dst = box(0, 0, 1) + zface + t;
    }
    const int s = t % S::kSide, m0 = t / S::kSide;
    int ri, rj;  // ring position relative to the brick
    bool have;
    if (s < S::BY) {
      ri = -1; rj = s; have = cl.bx > 0;
    } else if (s < 2 * S::BY) {
      ri = S::BX; rj = s - S::BY; have = cl.bx + 1 < nbx;
    } else if (s < 2 * S::BY + S::BX) {
      ri = s - 2 * S::BY; rj = -1; have = cl.by > 0;
    } else {
      ri = s - 2 * S::BY - S::BX; rj = S::BY; have = cl.by + 1 < nby;
    }
    si = cl.bx * S::BX + ri;
    sj = cl.by * S::BY + rj;
    side_lim = m0 < S::kLanes && have && si < g.nx && sj < g.ny ? cl.nzb - m0 : 0;
    side_d = m0 * S::SXY + (rj + 1) * S::SX + ri + 1;
  }
};

// ---- plan ---------------------------------------------------------------------
inline int brick_cz_class(int cz) { return cz <= 4 ? 4 : cz <= 8 ? 8 : cz <= 16 ? 16 : 32; }

template <int BX>
size_t brick_smem(int cz) {
  using S = BrickShape<BX>;
  const int c = brick_cz_class(cz);
  const int rows = (c + S::kLanes - 1) / S::kLanes;  // side ring cells per thread
  return sizeof(double) *
         (static_cast<size_t>(c + 1) * S::SXY + 3 * kBT + rows * S::kLanes * S::kSide +
          c * 2 * S::BY) +
         sizeof(int) * 6 * kBT;
}

template <int BX>
void consider(const Dims &g, int sms, BrickPlan *best, bool *found) {
  using S = BrickShape<BX>;
  const int nbx = (g.nx + S::BX - 1) / S::BX, nby = (g.ny + S::BY - 1) / S::BY;
  if (nbx * nby > sms) return;
  int nbz = sms / (nbx * nby);
  const int cz = (g.nz + nbz - 1) / nbz;
  // a 64-wide brick of more than 16 planes does not fit shared memory
  if (cz > (S::BX == 64 ? 16 : kBrickMaxPlanes)) return;
  nbz = (g.nz + cz - 1) / cz;
  // fewest planes per thread first (0.17 us an iteration each above 4 planes;
  // below, 36 to 144 CTAs measured the same), then fewest CTAs
  if (*found && (best->cz < cz || (best->cz == cz && best->ctas() <= nbx * nby * nbz))) return;
  *best = BrickPlan{S::BX, nbx, nby, nbz, cz, brick_smem<BX>(cz),
                    2 * sizeof(Packet) * static_cast<size_t>(nbx * nby * nbz) *
                        brick_inbox_packets(S::kSide, (cz + 3) / 4 * 4)};
  *found = true;
}

// afl_launch.h, plan_brick, on a chip of sms SMs with smem bytes of shared memory per CTA.
inline bool plan_brick_on(const Dims &g, int sms, int smem, BrickPlan *plan) {
  if (sms > 160) sms = 160;  // the sums' polls cover 160 CTAs
  bool found = false;
  consider<32>(g, sms, plan, &found);
  consider<16>(g, sms, plan, &found);
  consider<64>(g, sms, plan, &found);
  constexpr size_t kStatic = 2048;  // reduction scratch and scalars, rounded up
  return found && plan->smem_bytes + kStatic <= static_cast<size_t>(smem);
}

// ---- several systems in one launch ---------------------------------------------------
// Bricks are kQueueBX wide for every system, and an inbox belongs to a CTA, not to a
// system: a CTA leaves a system only after it has read every packet sent to it (none is
// sent that is not waited for: BrickShape::y_at, x_at), and clears its inbox before the
// next one's first sum.
constexpr int kQueueBX = 16;

template <typename Args>
struct BrickJob {
  Args a;
  BrickSums bs;
  int begin;  // the system's first CTA
};

template <typename Args>
struct BrickQueue {
  const BrickJob<Args> *jobs;
  const int *first, *list;
};

// Where the parts of the queue's scratch start.
struct QueueLayout {
  size_t first, list, slots, inbox, bytes;
  QueueLayout(const BrickQueuePlan &q, size_t job_bytes, size_t packet_bytes) {
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    first = up(job_bytes * q.plan.size());
    list = first + sizeof(int) * q.first.size();
    slots = up(list + sizeof(int) * q.list.size());
    inbox = up(slots + sizeof(Packet) * 8 * static_cast<size_t>(q.total));
    czp = q.cz_class;
    bytes = inbox + 2 * packet_bytes * per() * static_cast<size_t>(q.ctas);
  }
  int czp = 0;
  size_t per() const {
    return static_cast<size_t>(brick_inbox_packets(BrickShape<kQueueBX>::kSide, czp));
  }
};

// The jobs and lists on the device; fill(m, args) sets system m's own arguments.
template <typename Args, typename Mem, typename Fill>
cudaError_t write_queue(const BrickQueuePlan &q, void *scratch, int *abort_flag,
                        unsigned long long timeout_ns, Fill fill) {
  using Job = BrickJob<Args>;
  const QueueLayout at(q, sizeof(Job), sizeof(Mem));
  auto *const base = static_cast<unsigned char *>(scratch);
  std::vector<Job> jobs(q.plan.size());
  size_t slot = 0;
  for (size_t m = 0; m < jobs.size(); ++m) {
    const BrickPlan &p = q.plan[m];
    Args &a = jobs[m].a;
    fill(m, a);
    a.nbx = p.nbx;
    a.nby = p.nby;
    a.nbz = p.nbz;
    a.cz = p.cz;
    a.czp = q.cz_class;
    a.inbox = reinterpret_cast<Mem *>(base + at.inbox) + at.per() * static_cast<size_t>(q.begin[m]);
    a.parity = static_cast<int>(at.per() * static_cast<size_t>(q.ctas));
    jobs[m].bs = BrickSums{reinterpret_cast<Packet *>(base + at.slots) + 8 * slot, p.ctas(),
                           abort_flag, timeout_ns};
    jobs[m].begin = q.begin[m];
    slot += static_cast<size_t>(p.ctas());
  }
  auto put = [&](size_t off, const void *src, size_t bytes) {
    return cudaMemcpy(base + off, src, bytes, cudaMemcpyHostToDevice);
  };
  cudaError_t err = put(0, jobs.data(), sizeof(Job) * jobs.size());
  if (err == cudaSuccess) err = put(at.first, q.first.data(), sizeof(int) * q.first.size());
  if (err == cudaSuccess) err = put(at.list, q.list.data(), sizeof(int) * q.list.size());
  return err;
}

template <typename Args, typename Mem, typename Fn>
int launch_queue(Fn fn, size_t smem, const BrickQueuePlan &q, void *scratch, cudaStream_t st) {
  const QueueLayout at(q, sizeof(BrickJob<Args>), sizeof(Mem));
  auto *const base = static_cast<unsigned char *>(scratch);
  const void *const f = reinterpret_cast<const void *>(fn);
  cudaError_t err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
  if (err != cudaSuccess) return -static_cast<int>(err);
  cudaMemsetAsync(base + at.slots, 0, sizeof(Packet) * 8 * static_cast<size_t>(q.total), st);
  BrickQueue<Args> a{reinterpret_cast<const BrickJob<Args> *>(base),
                     reinterpret_cast<const int *>(base + at.first),
                     reinterpret_cast<const int *>(base + at.list)};
  void *params[] = {&a};
  err = cudaLaunchCooperativeKernel(f, dim3(q.ctas), dim3(kBT), params, smem, st);
  return err == cudaSuccess ? q.ctas : -static_cast<int>(err);
}

// This CTA's systems in order: solve(args, sums) of each, from shared memory.
template <typename Args, typename Solve>
__device__ __forceinline__ void run_queue(const BrickQueue<Args> &q, Args &a, QueuedSums &bs,
                                          Solve solve) {
  const int end = q.first[blockIdx.x + 1];
  for (int n = q.first[blockIdx.x]; n < end; ++n) {
    __syncthreads();  // the previous system's shared memory is free
    if (threadIdx.x == 0) {
      const BrickJob<Args> &job = q.jobs[q.list[n]];
      a = job.a;
      static_cast<BrickSums &>(bs) = job.bs;
      bs.vblock = static_cast<int>(blockIdx.x) - job.begin;
    }
    __syncthreads();
    solve();
  }
}

// ---- tensor memory as per-thread storage -------------------------------------------
// Everything below starts with __syncwarp(): the .sync.aligned forms need the whole
// warp converged, and a branch that only some lanes took just before does not
// promise that (an illegal instruction otherwise).
// 128 lanes x 512 columns of 32 bits beside the register file and shared
// memory.  Warp w reaches lanes 32*(w%4) .. +31 and owns a quarter of the
// allocated columns; 32x32b loads and stores move a thread's own columns.
template <int COLS>
__device__ __forceinline__ void brick_tm_alloc(unsigned *dst_smem) {  // one whole warp
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(dst_smem));
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa),
               "n"(COLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS>
__device__ __forceinline__ void brick_tm_dealloc(unsigned taddr) {  // the allocating warp
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(COLS)
               : "memory");
}
__device__ __forceinline__ void brick_tm_sync_threads() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 8 columns; asynchronous: brick_tm_wait_st before the next load of them.
__device__ __forceinline__ void brick_tm_st8(unsigned taddr, const unsigned (&v)[8]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
      : "memory");
}
__device__ __forceinline__ void brick_tm_wait_st() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 16 columns; the registers are valid after brick_tm_wait_ld on them.
__device__ __forceinline__ void brick_tm_ld16(unsigned taddr, unsigned (&v)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// Names the registers, so that no use of them moves above the wait.
__device__ __forceinline__ void brick_tm_wait_ld(unsigned (&v)[16]) {
  __syncwarp();
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]),
                 "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]),
                 "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               :
               : "memory");
}
__device__ __forceinline__ void put_double(unsigned (&v)[8], int e, double x) {
  v[2 * e] = static_cast<unsigned>(__double2loint(x));
  v[2 * e + 1] = static_cast<unsigned>(__double2hiint(x));
}
template <int N>
__device__ __forceinline__ double get_double(const unsigned (&v)[N], int at) {
  return __hiloint2double(static_cast<int>(v[at + 1]), static_cast<int>(v[at]));
}

}  // namespace
}  // namespace afl
