// CG2D solves with the whole iteration state on chip.
//
// A team of CTAs (one per SM) holds one instance's r, s and z/q in its shared memory for the whole solve; the
// instance's rows are split over the team in contiguous runs of work units. Per pass only three things move:
//   - the coefficients (L1 / L2 hits or one read from HBM) and x (own points, read and written by one thread);
//   - the halo: the points a neighbouring CTA's stencil reads, of z after pass X and of q after pass S;
//   - one partial sum per work unit.
// r and s at halo cells are kept by the reader: it applies the owner's update to them with the owner's values of
// q and z, so they are the owner's values bit for bit.
//
// Halo points and partial sums travel as 16-byte messages {value, tag} written and read with single 128-bit accesses
// (st / ld.relaxed.gpu.b128, which are single-copy atomic): a reader polls the message itself until its tag is the
// step's, so a pass needs no barrier, no fence and no counter, and its latency is one store and one successful load
// through L2. Every CTA reads all partial sums of its instance and forms the sums itself in the fixed order (blocks of a
// tile in order, tiles in order from 0), so every CTA of the team takes the same branch. Two message buffers
// alternate: a CTA sends the sums of exchange p + 1 only after it has those of p, so everybody has read p - 1; and it
// sends the halo values h + 2 only after an exchange that every reader of h has entered having read h.
//
// Teams never wait for one another. An instance is as large as its team's shared memory (team_plan); what does not
// fit runs in cg2d_solver.cu, which streams the state. Groups of a call have a launch each (cg2d_team) or share one on parts
// of the CTAs (cg2d_team_groups). The arithmetic, the sum order and the results are those of
// cg2d_solver.cu bit for bit, in every precision and sum order.
//
// What bounds it. One LLC90 FP64 solve: 2.3 ms, 4.6 us a pass (6.9 ms and 14 us when streamed): the message latency (an
// all-to-all of 148 CTAs takes 1.3 us when every CTA's sums have 128-byte lines of their own, 3.2 us when CTAs share
// lines), the block barriers and short dependent steps between the phases. Batches: the shared-memory / L1 pipe. With 11
// teams of 13 CTAs (mixed pairs) it is busy 53 % of the time, DRAM 2 %, issue slots 37 %; 64 mixed pairs take 31 ms (48
// streamed), 64 FP64 solves 29 ms (52). One LLC270 FP64 solve: 16 ms (54); nothing is near its peak (shared-memory / L1 pipe
// 46 %, issue slots 32 %, DRAM 2 %), warps wait at block barriers (24 rows over 16 warps) and for shared memory.
// Two CTAs of 8 warps per SM, so that one team computes while another waits, measured the same (16 FP64 solves 8.7 ms
// either way) and fit fewer teams.

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "cg2d_device.cuh"
#include "cg2d_internal.cuh"

namespace cg2d {
namespace {

using u64 = unsigned long long;

// ------------------------------------------------------------------------------------------------
// vector elements: the NS right-hand sides of a point

template <bool MIXED, int NS> struct El;
template <> struct El<false, 1> { using T = double; using C = double; };
template <> struct El<false, 2> { using T = double2; using C = double; };
template <> struct El<true, 1> { using T = float; using C = float; };
template <> struct El<true, 2> { using T = float2; using C = float; };

// the coefficients of a point: west, south and north faces and the centre (the east face is the next point's west face)
// Packed rows of n + 1 points: FP32 16 bytes a point; FP64 (west, south) of every point, then (north, centre) of every
// point, so that a warp's 16-byte loads are contiguous in both.
struct __align__(16) D4 { double w, s, n, c; };
struct __align__(16) F4 { float w, s, n, c; };
template <class C> struct Four;
template <> struct Four<double> { using V = D4; };
template <> struct Four<float> { using V = F4; };
__device__ __forceinline__ D4 load4(const D4* row, int n1, int i) {
  const double2* p = reinterpret_cast<const double2*>(row);
  const double2 a = p[i], b = p[n1 + i];
  return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ F4 load4(const F4* row, int, int i) {
  const float4 a = *reinterpret_cast<const float4*>(row + i);
  return {a.x, a.y, a.z, a.w};
}
__device__ __forceinline__ double load_w(const D4* row, int i) { return reinterpret_cast<const double2*>(row)[i].x; }
__device__ __forceinline__ float load_w(const F4* row, int i) { return row[i].w; }
__device__ __forceinline__ void store4(D4* row, int n1, int i, double w, double s, double n, double c) {
  double2* p = reinterpret_cast<double2*>(row);
  p[i] = make_double2(w, s);
  p[n1 + i] = make_double2(n, c);
}
__device__ __forceinline__ void store4(F4* row, int, int i, float w, float s, float n, float c) {
  *reinterpret_cast<float4*>(row + i) = make_float4(w, s, n, c);
}

__device__ __forceinline__ double get(double v, int) { return v; }
__device__ __forceinline__ double get(float v, int) { return (double)v; }
__device__ __forceinline__ double get(double2 v, int s) { return s == 0 ? v.x : v.y; }
__device__ __forceinline__ double get(float2 v, int s) { return (double)(s == 0 ? v.x : v.y); }
__device__ __forceinline__ void put(double& v, int, double a) { v = a; }
__device__ __forceinline__ void put(float& v, int, double a) { v = (float)a; }
__device__ __forceinline__ void put(double2& v, int s, double a) { if (s == 0) v.x = a; else v.y = a; }
__device__ __forceinline__ void put(float2& v, int s, double a) { if (s == 0) v.x = (float)a; else v.y = (float)a; }

// c + a b with the solver's rounding (Ar), per right-hand side
__device__ __forceinline__ double vmadd(double a, double b, double c) { return Ar<false>::madd(a, b, c); }
__device__ __forceinline__ float vmadd(float a, float b, float c) { return Ar<true>::madd(a, b, c); }
__device__ __forceinline__ double2 vmadd(double2 a, double2 b, double2 c) {
  return make_double2(vmadd(a.x, b.x, c.x), vmadd(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 vmadd(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ double2 vneg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ double st5(double c0, double c1, double c2, double c3, double c4, double v0, double v1,
                                      double v2, double v3, double v4) {
  return stencil5<false, double>(c0, c1, c2, c3, c4, v0, v1, v2, v3, v4);
}
__device__ __forceinline__ float st5(float c0, float c1, float c2, float c3, float c4, float v0, float v1, float v2,
                                     float v3, float v4) {
  return stencil5<true, float>(c0, c1, c2, c3, c4, v0, v1, v2, v3, v4);
}
__device__ __forceinline__ double2 st5(double c0, double c1, double c2, double c3, double c4, double2 v0, double2 v1,
                                       double2 v2, double2 v3, double2 v4) {
  return make_double2(st5(c0, c1, c2, c3, c4, v0.x, v1.x, v2.x, v3.x, v4.x),
                      st5(c0, c1, c2, c3, c4, v0.y, v1.y, v2.y, v3.y, v4.y));
}
__device__ __forceinline__ float2 st5(float c0, float c1, float c2, float c3, float c4, float2 v0, float2 v1,
                                      float2 v2, float2 v3, float2 v4) {
  return stencil5p(c0, c1, c2, c3, c4, v0, v1, v2, v3, v4);
}

// ------------------------------------------------------------------------------------------------
// messages

struct Msg { u64 v, tag; };   // 16 bytes, 16-byte aligned
__device__ __forceinline__ void st_msg(void* p, u64 v, u64 tag) {
  asm volatile("{\n\t.reg .b128 m;\n\tmov.b128 m, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], m;\n\t}" ::"l"(p),
               "l"(v), "l"(tag)
               : "memory");
}
__device__ __forceinline__ Msg ld_msg(const void* p) {
  Msg m;
  asm volatile("{\n\t.reg .b128 m;\n\tld.relaxed.gpu.global.b128 m, [%2];\n\tmov.b128 {%0, %1}, m;\n\t}"
               : "=l"(m.v), "=l"(m.tag)
               : "l"(p)
               : "memory");
  return m;
}

// a vector element as halo messages (mixed: both right-hand sides in one; FP64: one per right-hand side, at message
// kind s) and back
__device__ __forceinline__ u64 bits_of(double v) { return (u64)__double_as_longlong(v); }
__device__ __forceinline__ u64 bits_of(float v) { return (u64)__float_as_uint(v); }
__device__ __forceinline__ u64 bits_of(float2 v) {
  return (u64)__float_as_uint(v.x) | ((u64)__float_as_uint(v.y) << 32);
}
__device__ __forceinline__ void send(char* buf, long long nslots, long long slot, u64 tag, double v) {
  st_msg(buf + slot * 16, bits_of(v), tag);
}
__device__ __forceinline__ void send(char* buf, long long nslots, long long slot, u64 tag, float v) {
  st_msg(buf + slot * 16, bits_of(v), tag);
}
__device__ __forceinline__ void send(char* buf, long long nslots, long long slot, u64 tag, float2 v) {
  st_msg(buf + slot * 16, bits_of(v), tag);
}
__device__ __forceinline__ void send(char* buf, long long nslots, long long slot, u64 tag, double2 v) {
  st_msg(buf + slot * 16, bits_of(v.x), tag);
  st_msg(buf + (nslots + slot) * 16, bits_of(v.y), tag);
}
__device__ __forceinline__ void got(double& v, int, u64 b) { v = __longlong_as_double((long long)b); }
__device__ __forceinline__ void got(float& v, int, u64 b) { v = __uint_as_float((unsigned)b); }
__device__ __forceinline__ void got(float2& v, int, u64 b) {
  v = make_float2(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}
__device__ __forceinline__ void got(double2& v, int s, u64 b) { put(v, s, __longlong_as_double((long long)b)); }

// ------------------------------------------------------------------------------------------------
// a CTA's view of its instance

// CG scalars of the instance, the same in every CTA of the team
struct Scalars {
  double alpha[2], beta[2], eta[2], eta_prev[2], rr[2], rn[2], nrm[2], total[2 * kTeamKinds];
  u64 vmax[2];
  int act[2], k_done[2], nrep[2], rep[2];
  int run, any_rep;
  u64 tm[kProfSlots];   // phase times of thread 0 (profiling)
};
// where the team's dynamic shared memory starts after the scalars
constexpr unsigned kScalBytes = 384;
static_assert(sizeof(Scalars) <= kScalBytes, "Scalars");

// one row of a CTA: its column 0 in the ring arrays, its row t nj + j of the instance, and the first row past its run (the
// CTA's consecutive rows of one tile)
struct __align__(16) RowEnt { int ring, grow, end, unused; };
struct __align__(8) HaloEnt { int elem, slot; };   // ring element (-1: never written); message slot of its source
struct __align__(8) SendEnt { int point, slot; };  // point lr ni + i that a neighbouring CTA reads; its message slot

extern __shared__ __align__(128) unsigned char team_smem[];

template <class T>
__device__ __forceinline__ T* smem_at(unsigned off) { return reinterpret_cast<T*>(team_smem + off); }

// first row (of the instance's T nj rows) of work unit u
__device__ __forceinline__ int unit_row(const TeamDev& t, int nj, int u) {
  const int tile = u / t.nblk, blk = u - tile * t.nblk;
  return tile * nj + min(nj, blk * t.rpb);
}
// message slot of boundary point (row grow = t nj + j, column i): the west and east points of every row have their own
// slots; another point's slot is that of its work unit's first or last row
__device__ __forceinline__ long long row_slot(const TeamDev& t, const TopoDev& tp, int grow) {
  const int tile = grow / tp.nj, j = grow - tile * tp.nj, blk = j / t.rpb;
  const int which = j == blk * t.rpb ? 0 : 1;
  return 2ll * tp.T * tp.nj + ((long long)(tile * t.nblk + blk) * 2 + which) * tp.ni;
}
__device__ __forceinline__ long long point_slot(const TeamDev& t, const TopoDev& tp, int grow, int i) {
  if (i == 0) return 2ll * grow;
  if (i == tp.ni - 1) return 2ll * grow + 1;
  return row_slot(t, tp, grow) + i;
}

template <bool MIXED, int NS, bool SERIAL, int STEPS>
struct Team {
  using T = typename El<MIXED, NS>::T;
  using C = typename El<MIXED, NS>::C;
  using A = Ar<MIXED>;
  using C4 = typename Four<C>::V;
  static constexpr int MS = MIXED ? 1 : NS;              // halo messages per point

  const TeamParams& kp;   // (the kernel's parameter: every field is a constant-bank operand)
  int rank, inst;
  int u0, nunits, row0, nrows, nhalo, nsend;
  int lrA, lrB;           // this warp's rows
  char* msg;
  double* x;
  C4* coef;               // this CTA's packed coefficients [2 operators][rows][ni]
  unsigned htag, stag;    // tags of the last halo values and of the last sums sent by this team
  bool fail;

  __device__ __forceinline__ Team(const TeamParams& kp_, int team, int rank_)
      : kp(kp_), rank(rank_), inst(0), nhalo(0), nsend(0), htag(0), stag(0), fail(false) {
    const TeamDev& td = kp.t;
    const int nj = kp.g.tp.nj;
    u0 = td.ub[rank];
    nunits = td.ub[rank + 1] - u0;
    row0 = unit_row(td, nj, u0);
    nrows = unit_row(td, nj, u0 + nunits) - row0;
    const int warp = threadIdx.x >> 5;
    lrA = warp * nrows / kTeamWarps;
    lrB = (warp + 1) * nrows / kTeamWarps;
    msg = td.msg + (long long)team * td.msg_stride;
    x = td.x + (long long)team * td.x_stride;
    coef = reinterpret_cast<C4*>(td.coef) + (long long)(team * td.G + rank) * 2 * td.max_rows * (kp.g.tp.ni + 1);
    if (threadIdx.x < kProfSlots) sc().tm[threadIdx.x] = 0ull;
  }

  __device__ __forceinline__ int ni() const { return kp.g.tp.ni; }
  __device__ __forceinline__ int P() const { return kp.g.tp.ni + 2; }
  __device__ __forceinline__ Scalars& sc() const { return *smem_at<Scalars>(0); }
  __device__ __forceinline__ RowEnt* rows() const { return smem_at<RowEnt>(kp.t.o_rows); }
  __device__ __forceinline__ HaloEnt* halo() const { return smem_at<HaloEnt>(kp.t.o_halo); }
  __device__ __forceinline__ SendEnt* sends() const { return smem_at<SendEnt>(kp.t.o_send); }
  __device__ __forceinline__ int* unit_msg() const { return smem_at<int>(kp.t.o_umsg); }
  __device__ __forceinline__ int* unit_rows() const { return smem_at<int>(kp.t.o_units); }
  __device__ __forceinline__ T* hval() const { return smem_at<T>(kp.t.o_hval); }
  __device__ __forceinline__ double* rowsum() const { return smem_at<double>(kp.t.o_rowsum); }
  __device__ __forceinline__ double* psum() const { return smem_at<double>(kp.t.o_psum); }
  __device__ __forceinline__ double* tsum() const { return smem_at<double>(kp.t.o_tsum); }
  __device__ __forceinline__ T* R() const { return smem_at<T>(kp.t.o_r); }
  __device__ __forceinline__ T* S() const { return smem_at<T>(kp.t.o_s); }
  __device__ __forceinline__ T* Q() const { return smem_at<T>(kp.t.o_q); }   // q after pass S, z after pass X
  __device__ __forceinline__ int rid(int s) const { return kp.g.rhs_base + inst * NS + s; }
  __device__ __forceinline__ char* halo_buf() const { return msg + (htag & 1) * (MS * kp.t.nslots * 16); }
  __device__ __forceinline__ char* sum_buf() const {
    return msg + (2 * MS * kp.t.nslots + (long long)(int)(stag & 1) * (kp.t.G * kp.t.sum_block)) * 16;
  }
  __device__ __forceinline__ double* hist(int s, int kind, int k) const {
    return kp.hist + ((size_t)rid(s) * H_NKIND + kind) * (size_t)kp.hist_len + k;
  }

  // halo cell h of the CTA: the point (t, j, i) it stands for, -1 <= j <= nj, -1 <= i <= ni. First, per run of rows, the
  // row below and the row above it, then the west and east cells of every row.
  __device__ __forceinline__ void halo_point(int h, int tile0, int& t, int& j, int& i) const {
    const int nj = kp.g.tp.nj, n = ni(), nwe = nhalo - 2 * nrows;
    if (h < nwe) {
      const int seg = h / (2 * n), rem = h - seg * 2 * n, top = rem / n;
      t = tile0 + seg;
      i = rem - top * n;
      j = (top ? min(row0 + nrows, (t + 1) * nj) : max(row0, t * nj) - 1) - t * nj;
    } else {
      const int q = h - nwe, grow = row0 + (q >> 1);
      t = grow / nj;
      j = grow - t * nj;
      i = (q & 1) ? n : -1;
    }
  }

  // tables of the CTA's rows, units and halo cells (the same for every instance of the group)
  __device__ void tables() {
    const TeamDev& td = kp.t;
    const TopoDev& tp = kp.g.tp;
    const int nj = tp.nj, ni = tp.ni, tile0 = row0 / nj;
    for (int lr = threadIdx.x; lr < nrows; lr += kTeamThreads) {
      const int grow = row0 + lr, tile = grow / nj;
      RowEnt e;
      e.ring = (lr + 1 + 2 * (tile - tile0)) * P() + 1;
      e.grow = grow;
      e.end = min(nrows, (tile + 1) * nj - row0);
      e.unused = 0;
      rows()[lr] = e;
    }
    for (int u = threadIdx.x; u <= nunits; u += kTeamThreads) unit_rows()[u] = unit_row(td, nj, u0 + u) - row0;
    // halo cells; a cell whose source the exchange does not write keeps 0: elem -1
    const int nseg = (row0 + nrows - 1) / nj - tile0 + 1;
    nhalo = nseg * 2 * ni + nrows * 2;
    for (int h = threadIdx.x; h < nhalo; h += kTeamThreads) {
      int t, j, i;
      halo_point(h, tile0, t, j, i);
      // its ring row: that of the run's rows continued by one below and above
      const int elem = (t * nj + j - row0 + 1 + 2 * (t - tile0)) * P() + 1 + i;
      const int src = source(t, j, i);
      HaloEnt e;
      e.elem = src >= 0 ? elem : -1;
      e.slot = src >= 0 ? (int)point_slot(td, tp, src / ni, src % ni) : 0;
      halo()[h] = e;
    }
    // points to send: the west and east point of every row, and the rest of each run's first and last row
    nsend = nrows * 2 + nseg * 2 * (ni - 2);
    for (int h = threadIdx.x; h < nsend; h += kTeamThreads) {
      int lr, i;
      if (h < nrows * 2) {
        lr = h >> 1;
        i = (h & 1) ? ni - 1 : 0;
      } else {
        const int q = h - nrows * 2, seg = q / (2 * (ni - 2)), rem = q - seg * 2 * (ni - 2);
        const int top = rem / (ni - 2), tile = tile0 + seg;
        lr = (top ? min(row0 + nrows, (tile + 1) * nj) - 1 : max(row0, tile * nj)) - row0;
        i = 1 + rem - top * (ni - 2);
      }
      SendEnt e;
      e.point = lr * ni + i;
      e.slot = (int)point_slot(td, tp, row0 + lr, i);
      sends()[h] = e;
    }
    // where the sum of unit u lies among the sum messages of an exchange: every CTA has 128-byte lines of its own
    for (int u = threadIdx.x; u < td.units; u += kTeamThreads) {
      int c = 0, z = td.G;            // the CTA with ub[c] <= u < ub[c + 1]
      while (z - c > 1) {
        const int m = (c + z) >> 1;
        if (td.ub[m] <= u) c = m;
        else z = m;
      }
      unit_msg()[u] = c * td.sum_block + u - td.ub[c];
    }
  }
  // send the points of `src` (their values by point index lr ni + i) that neighbours read, as step htag
  template <class F>
  __device__ __forceinline__ void send_points(F value) {
    char* hb = halo_buf();
    for (int h = threadIdx.x; h < nsend; h += kTeamThreads) {
      const SendEnt e = sends()[h];
      send(hb, kp.t.nslots, e.slot, htag, value(e.point));
    }
  }
  __device__ __forceinline__ void send_ring(const T* v) {   // from a ring array
    send_points([&](int pt) -> T {
      const int lr = pt / ni();
      return v[rows()[lr].ring + pt - lr * ni()];
    });
  }

  // wait until the message at p carries `tag`; false when the time limit ran out or another CTA reported an error
  __device__ __forceinline__ bool poll(const char* p, u64 tag, Msg& m) {
    if (m.tag == tag) return true;
    u64 t0 = 0;
    for (unsigned n = 1;; ++n) {
      m = ld_msg(p);
      if (m.tag == tag) return true;
      if ((n & 255u) == 0u) {
        if (t0 == 0) t0 = globaltimer();
        if (ld_relaxed(&kp.gs[1]) != 0u) return false;
        if (globaltimer() - t0 > kp.timeout_ns) {
          note_timeout(kp.gs, 1u, 0u);
          return false;
        }
      }
    }
  }

  // halo messages of step htag into hval; nsum > 0: also the sums of exchange stag, [nsum][units], into psum.
  // A thread takes messages tid, tid + threads, ...; two loads are in flight before the first is tested. acquire: what the
  // senders had written to memory when they sent (after a fence of theirs) is visible to the CTA afterwards.
  __device__ __forceinline__ void receive(bool with_halo, int nsum, bool acquire = false) {
    const int nh = with_halo ? nhalo * MS : 0, n = nh + nsum * kp.t.units;
    const char* hb = halo_buf();
    const char* sb = sum_buf();
    const u64 ht = htag, ts = stag;
    bool ok = true;
    auto at = [&](int e) -> const char* {
      if (e < nh) {
        const int h = MS == 1 || e < nhalo ? e : e - nhalo;
        const HaloEnt he = halo()[h];
        return he.elem >= 0 ? hb + ((MS == 1 || e < nhalo ? 0 : kp.t.nslots) + he.slot) * 16 : nullptr;
      }
      if (e >= n) return nullptr;
      int u = e - nh, q = 0;
      while (u >= kp.t.units) { u -= kp.t.units; ++q; }
      return sb + (long long)(unit_msg()[u] + q * kp.t.max_units) * 16;
    };
    auto take = [&](int e, const char* p, Msg& m) {
      if (!p) return;
      ok = poll(p, e < nh ? ht : ts, m) && ok;
      if (e < nh) got(hval()[MS == 1 || e < nhalo ? e : e - nhalo], MS == 1 || e < nhalo ? 0 : 1, m.v);
      else psum()[e - nh] = __longlong_as_double((long long)m.v);
    };
    for (int e = threadIdx.x; e < n && ok; e += 2 * kTeamThreads) {
      const int f = e + kTeamThreads;
      const char *p = at(e), *r = at(f);
      Msg m{}, w{};
      if (p) m = ld_msg(p);
      if (r) w = ld_msg(r);
      take(e, p, m);
      take(f, r, w);
    }
    if (acquire) __threadfence();
    fail = __syncthreads_or(!ok) || fail;
  }

  // send the CTA's unit sums [nk kinds][NS][units] of the next exchange from the row sums (block barrier before): warp q
  // takes sum q, its lanes the units. FORTRAN order: serial_sums has formed the unit sums.
  __device__ __forceinline__ void send_sums(int nk) {
    ++stag;
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (q < nk * NS) {
      char* b = sum_buf() + ((long long)rank * kp.t.sum_block + q * kp.t.max_units) * 16;
      const double* rs = rowsum() + q * kp.t.max_rows;
      for (int lu = lane; lu < nunits; lu += 32) {
        double v;
        if constexpr (SERIAL) {
          v = rs[lu];
        } else {
          const int z = unit_rows()[lu + 1];
          v = 0.0;
          for (int lr = unit_rows()[lu]; lr < z; lr += 8) {
            double r[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) r[c] = lr + c < z ? rs[lr + c] : 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (lr + c < z) v = add(v, r[c]);
          }
        }
        st_msg(b + (long long)lu * 16, bits_of(v), stag);
      }
    }
  }

  // the total of each of the n sums from psum, in fixed order: tile sums by all threads, then (warp 0) the totals into
  // sc().total
  __device__ __forceinline__ void fold(int n) {
    const int nb = kp.t.nblk, nt = kp.g.tp.T;
    for (int e = threadIdx.x; e < n * nt; e += kTeamThreads) {
      const double* p = psum() + e * nb;   // [sum][T][nblk]
      double a = 0.0;
      for (int b = 0; b < nb; b += 6) {
        double v[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = b + c < nb ? p[b + c] : 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c)
          if (b + c < nb) a = add(a, v[c]);
      }
      tsum()[e] = a;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      if ((int)threadIdx.x < n) {
        const double* p = tsum() + threadIdx.x * nt;
        double a = 0.0;
        for (int t = 0; t < nt; t += 13) {
          double v[13];
#pragma unroll
          for (int c = 0; c < 13; ++c) v[c] = t + c < nt ? p[t + c] : 0.0;
#pragma unroll
          for (int c = 0; c < 13; ++c)
            if (t + c < nt) a = add(a, v[c]);
        }
        sc().total[threadIdx.x] = a;
      }
      __syncwarp();
    }
  }

  __device__ __forceinline__ long long pad_of(int grow, int i) const {
    const TopoDev& tp = kp.g.tp;
    const int t = grow / tp.nj, j = grow - t * tp.nj;
    return (long long)inst * kp.g.pad_elems + ((long long)t * tp.npy + j + tp.OLy) * tp.npx + tp.OLx + i;
  }
  // f(lr, row entry, i) for every point of this warp's rows; after(lr) closes a row (set-up and closing steps)
  template <class F, class E>
  __device__ __forceinline__ void each_point(F f, E after) const {
#pragma unroll 1
    for (int lr = lrA; lr < lrB; ++lr) {
      const RowEnt e = rows()[lr];
#pragma unroll 1
      for (int i = threadIdx.x & 31; i < ni(); i += 32) f(lr, e, i);
      after(lr);
    }
  }

  // the row sums first .. first + nk - 1 of row lr (xor butterflies over the lanes)
  __device__ __forceinline__ void row_sum(int lr, int nk, const double (&acc)[2][NS], int first) const {
    const int lane = threadIdx.x & 31, mr = kp.t.max_rows;
    double* rs = rowsum() + first * NS * mr + lr;
    if (nk == 1 && NS == 1) {
      const double v = butterfly(acc[0][0]);
      if (lane == 0) rs[0] = v;
    } else if (nk * NS == 2) {
      const double v = NS == 2 ? butterfly2(acc[0][0], acc[0][NS - 1]) : butterfly2(acc[0][0], acc[1][0]);
      if ((lane & 15) == 0) rs[(lane >> 4) * mr] = v;
    } else {
      const double v = butterfly4(acc[0][0], acc[0][NS - 1], acc[1][0], acc[1][NS - 1]);
      if ((lane & 7) == 0) rs[(lane >> 3) * mr] = v;
    }
  }

  // ---- FORTRAN order: sum kind q of right-hand side s over each of the CTA's tiles, every product in j, i order, one
  // after the other (cg2d.py:141-161), one warp per (tile, sum)
  template <bool M>
  __device__ __forceinline__ void serial_sums(const T* v) {
    const int warp = threadIdx.x >> 5;
    constexpr int nk = M ? 2 : 1;
    for (int task = warp; task < nunits * nk * NS; task += kTeamWarps) {
      const int q = task / (nunits * NS), rem = task % (nunits * NS), s = rem / nunits, lu = rem % nunits;
      const int lr = unit_rows()[lu];
      const T* a = v + rows()[lr].ring;
      const T* b = M && q == 0 ? a : Q() + lr * ni();
      const double sum = chain(a, b, M && q == 0 ? P() : ni(), s, ni(), kp.g.tp.nj, P());
      if ((threadIdx.x & 31) == 0) rowsum()[(q * NS + s) * kp.t.max_rows + lu] = sum;
    }
  }
  // the sum of the products a b of nj rows of n points in order, rows ap and bp elements apart, by one warp: the lanes form
  // 32 consecutive products and every lane adds them in order from
  // shuffles, which do not depend on the additions. 14 cycles a product with two chains on an SM (a dependent addition takes
  // 8.7; the rest, not shown by measurement, likely goes to the products' loads and addresses between the blocks of 32).
  // A function of its own: inlined into the pass, the compiler issues each shuffle only behind the addition before it, for
  // want of registers (32 cycles a product). Zeros past the end leave the sum as it is (it starts at +0, so it never is -0).
  __device__ __noinline__ static double chain(const T* a, const T* b, int bp, int s, int n, int nj, int ap) {
    const int lane = threadIdx.x & 31, total = n * nj;
    int i = lane, e = lane;       // this lane's column and product
    while (i >= n) { i -= n; a += ap; b += bp; }
    T va{}, vb{};
    auto next = [&]() {   // the operands of this lane's next product
      if (e < total) { va = a[i]; vb = b[i]; }
      i += 32;
      while (i >= n) { i -= n; a += ap; b += bp; }
    };
    auto product = [&]() -> double {
      const double v = e < total ? mul(get(va, s), get(vb, s)) : 0.0;
      e += 32;
      return v;
    };
    next();
    double sum = 0.0, cur = product();
    next();
#pragma unroll 1
    for (int c = 0; c < total; c += 32) {
      // operands two steps ahead, product one step ahead: neither is waited for
      const double nxt = product();
      next();
#pragma unroll
      for (int k = 0; k < 32; ++k) sum = add(sum, __shfl_sync(0xffffffffu, cur, k));
      cur = nxt;
    }
    return sum;
  }

  // ---- the second half of a pass: out = (M or A) v from the shared vector, kept in Q, with the pass's row sums.
  // M (pass X): z = M r, sums r.r and z.r; A (pass S): q = A s, sum s.q. One warp per row, lanes over the columns.
  // The latency of the coefficients (L2) and the shared-memory / L1 accesses bound it. So a point's coefficients are one
  // packed load (two in FP64), its east face coming from the next lane; a row's are loaded a row ahead, the first row's
  // before the pass's first half (prefetch); and a warp marches down its rows, two of the three vector rows staying in
  // registers (STEPS = 1, 2, 3: the column steps of 32 of a row). Rows of more than 96 points, and two FP64 right-hand
  // sides, do not leave the registers for that (STEPS = 0).
  static constexpr int NC = STEPS > 0 ? STEPS : (!MIXED && NS == 2) ? 1 : 3;   // column steps whose loads are issued together
  struct Coefs { C4 k[NC]; C w; };   // w: the west face past the last of these columns
  // the coefficients of row lr, columns c + lane + 32 m (past the row: its end column n)
  __device__ __forceinline__ void load(Coefs& f, const C4* cf, int lr, int c) const {
    const int lane = threadIdx.x & 31, n = ni();
    const C4* p = cf + (long long)lr * (n + 1);
#pragma unroll
    for (int m = 0; m < NC; ++m) f.k[m] = load4(p, n + 1, m < STEPS - 1 ? 32 * m + lane : min(c + 32 * m + lane, n));
    if (STEPS == 0 || n == 32 * STEPS) f.w = load_w(p, min(c + 32 * NC, n));
  }
  // the east face at column step m: the next lane's west face, in lane 31 the next step's
  __device__ __forceinline__ C east(const Coefs& f, int m) const {
    const int lane = threadIdx.x & 31;
    const C next = m + 1 < NC ? f.k[m + 1 < NC ? m + 1 : m].w : f.w;
    return __shfl_sync(0xffffffffu, lane == 0 ? next : f.k[m].w, (lane + 1) & 31);
  }
  template <bool M>
  __device__ __forceinline__ const C4* coefs() const { return coef + (M ? (long long)kp.t.max_rows * (ni() + 1) : 0ll); }
  template <bool M>
  __device__ __forceinline__ void prefetch(Coefs& f) const {
    f.w = (C)0;
    if (lrA < lrB) load(f, coefs<M>(), lrA, 0);
  }

  __device__ __forceinline__ void row_done(int lr, bool M, double (&acc)[2][NS]) const {
    if constexpr (!SERIAL) {
      row_sum(lr, M ? 2 : 1, acc, 0);
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[0][s] = acc[1][s] = 0.0;
    }
  }
  template <bool M>
  __device__ __forceinline__ static T apply(const C4& k, C east, T w, T e, T s, T n, T c) {
    if constexpr (M) return st5(k.c, k.w, east, k.s, k.n, c, w, e, s, n);
    else return st5(k.w, east, k.s, k.n, k.c, w, e, s, n, c);
  }
  template <bool M>
  __device__ __forceinline__ static void dots(T v, T o, double (&acc)[2][NS]) {
    if constexpr (!SERIAL) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double a = get(v, s), b = get(o, s);
        if constexpr (M) {
          acc[0][s] = A::dot(a, a, acc[0][s]);
          acc[1][s] = A::dot(b, a, acc[1][s]);
        } else {
          acc[0][s] = A::dot(a, b, acc[0][s]);
        }
      }
    }
  }
  // f: the first row's coefficients (prefetch)
  template <bool M>
  __device__ __forceinline__ void stencil(Coefs& f, double* ck) {
    const T* v = M ? R() : S();
    T* out = Q();
    const int lane = threadIdx.x & 31, n = ni(), p = P();
    const C4* cf = coefs<M>();
    double acc[2][NS] = {};
    if constexpr (STEPS == 0) {
#pragma unroll 1
      for (int lr = lrA; lr < lrB; ++lr) {
        const T* a = v + rows()[lr].ring;
#pragma unroll 1
        for (int c = 0; c < n; c += 32 * NC) {
          // the next step's coefficients
          int lr1 = lr, c1 = c + 32 * NC;
          if (c1 >= n) { c1 = 0; ++lr1; }
          Coefs f1;
          load(f1, cf, min(lr1, lrB - 1), c1);
#pragma unroll
          for (int m = 0; m < NC; ++m) {
            const int i = c + 32 * m + lane;
            const T* b = a + min(i, n - 1);
            const T v0 = b[0];
            const T o = apply<M>(f.k[m], east(f, m), b[-1], b[1], b[-p], b[p], v0);
            if (i < n) {
              out[lr * n + i] = o;
              dots<M>(v0, o, acc);
            }
          }
          f = f1;
        }
        row_done(lr, M, acc);
      }
    } else {
      // the lane's columns lane + 32 m; past the row, its last column (whose values are not used there)
      constexpr int L = STEPS - 1;
      const int last = min(32 * L + lane, n - 1) - lane;
      const bool in_last = 32 * L + lane < n;
#pragma unroll 1
      for (int lr = lrA; lr < lrB;) {
        const RowEnt e = rows()[lr];
        const int end = min(lrB, e.end);
        const T* a = v + e.ring + lane;
        T* o = out + lr * n + lane;
        T vs[STEPS], vc[STEPS];
#pragma unroll
        for (int m = 0; m < STEPS; ++m) {
          const int x = m < L ? 32 * m : last;
          vs[m] = a[x - p];
          vc[m] = a[x];
        }
#pragma unroll 1
        for (; lr < end; ++lr) {
          Coefs f1 = f;
          if (lr + 1 < lrB) load(f1, cf, lr + 1, 0);
#pragma unroll
          for (int m = 0; m < STEPS; ++m) {
            const int x = m < L ? 32 * m : last;
            const T vn = a[x + p];
            const T r = apply<M>(f.k[m], east(f, m), a[x - 1], a[x + 1], vs[m], vn, vc[m]);
            if (m < L || in_last) {
              o[x] = r;
              dots<M>(vc[m], r, acc);
            }
            vs[m] = vc[m];
            vc[m] = vn;
          }
          row_done(lr, M, acc);
          a += p;
          o += n;
          f = f1;
        }
      }
    }
    if constexpr (!MIXED) {
      // checkpoints of r or s (the rows this warp has just read)
      if (ck)
        each_point([&](int, const RowEnt& e, int i) { ck[pad_of(e.grow, i)] = get(v[e.ring + i], 0); }, [](int) {});
    }
    __syncthreads();
    ++htag;
    send_points([&](int pt) -> T { return out[pt]; });
    if constexpr (SERIAL) {
      serial_sums<M>(v);
      __syncthreads();
    }
  }

  // the first half: r -= alpha q (coef = -alpha; pass X) or s = z + beta s (PASS_S), own rows and halo cells
  template <bool PASS_S>
  __device__ __forceinline__ void update(T* vec, T coef) {
    const T* q = Q();
    const int lane = threadIdx.x & 31, n = ni(), p = P();
#pragma unroll 1
    for (int lr = lrA; lr < lrB;) {
      const RowEnt e = rows()[lr];
      const int end = min(lrB, e.end);
      T* a = vec + e.ring;
      const T* b = q + lr * n;
      // two rows at a time (the second one again the first past the end)
#pragma unroll 1
      for (; lr < end; lr += 2, a += 2 * p, b += 2 * n) {
        const bool two = lr + 1 < end;
        const int da = two ? p : 0, db = two ? n : 0;
#pragma unroll 1
        for (int i = lane; i < n; i += 96) {
          T va[2][3], vb[2][3];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int x = min(i + 32 * m, n - 1);
            va[0][m] = a[x];
            vb[0][m] = b[x];
            va[1][m] = a[x + da];
            vb[1][m] = b[x + db];
          }
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int x = i + 32 * m;
            if (x < n) {
              a[x] = PASS_S ? vmadd(coef, va[0][m], vb[0][m]) : vmadd(coef, vb[0][m], va[0][m]);
              if (two) a[x + p] = PASS_S ? vmadd(coef, va[1][m], vb[1][m]) : vmadd(coef, vb[1][m], va[1][m]);
            }
          }
        }
      }
      lr = end;
    }
    for (int h = threadIdx.x; h < nhalo; h += kTeamThreads) {
      const int el = halo()[h].elem;
      if (el >= 0) vec[el] = PASS_S ? vmadd(coef, vec[el], hval()[h]) : vmadd(coef, hval()[h], vec[el]);
    }
  }

  // x += alpha s for the right-hand sides that took the iteration (cg2d.py:254)
  __device__ __forceinline__ void update_x() {
    const T* sv = S();
    const Scalars& q = sc();
    const int lane = threadIdx.x & 31, n = ni();
    const double a0 = q.alpha[0], a1 = NS == 2 ? q.alpha[NS - 1] : 0.0;
    const bool on0 = q.act[0] != 0, on1 = NS == 2 && q.act[NS - 1] != 0;
    // rows two at a time, so that six loads from L2 are in flight per lane
#pragma unroll 1
    for (int lr = lrA; lr < lrB; lr += 2) {
      const bool two = lr + 1 < lrB;
      const RowEnt e = rows()[lr], f = rows()[two ? lr + 1 : lr];
      double* xr[2] = {x + (long long)e.grow * n * NS, x + (long long)f.grow * n * NS};
      const T* sr[2] = {sv + e.ring, sv + f.ring};
#pragma unroll 1
      for (int c = lane; c < n; c += 96) {
        double xv[2][3][NS];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int i = min(c + 32 * m, n - 1);
            if constexpr (NS == 2) {
              const double2 t = __ldcg(reinterpret_cast<const double2*>(xr[r]) + i);
              xv[r][m][0] = t.x;
              xv[r][m][NS - 1] = t.y;
            } else {
              xv[r][m][0] = __ldcg(xr[r] + i);
            }
          }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int i = c + 32 * m;
            if (i < n && (r == 0 || two)) {
              const T s0 = sr[r][i];
              if (on0) xv[r][m][0] = A::madd(a0, get(s0, 0), xv[r][m][0]);
              if constexpr (NS == 2) {
                if (on1) xv[r][m][1] = A::madd(a1, get(s0, 1), xv[r][m][1]);
                __stcg(reinterpret_cast<double2*>(xr[r]) + i, make_double2(xv[r][m][0], xv[r][m][1]));
              } else {
                __stcg(xr[r] + i, xv[r][m][0]);
              }
            }
          }
      }
    }
  }

  // compact index of the neighbour (j, i) of a point of tile t, -1 <= j <= nj, -1 <= i <= ni, or -1 (unwritten)
  __device__ __forceinline__ int source(int t, int j, int i) const {
    const TopoDev& tp = kp.g.tp;
    if (i >= 0 && i < tp.ni && j >= 0 && j < tp.nj) return (t * tp.nj + j) * tp.ni + i;
    if (i < 0) return tp.nbr[t * tp.nj + j];
    if (i >= tp.ni) return tp.nbr[tp.T * tp.nj + t * tp.nj + j];
    if (j < 0) return tp.nbr[2 * tp.T * tp.nj + t * tp.ni + i];
    return tp.nbr[2 * tp.T * tp.nj + tp.T * tp.ni + t * tp.ni + i];
  }
  // (A v) at point (grow, i), p its padded index with the instance, in FP64 from the caller's arrays; val(src, halo): v at
  // compact source src, or at padded halo point `halo` of the instance when src < 0
  template <class F>
  __device__ __forceinline__ double apply_f64(int grow, int i, long long p, F val) const {
    const TopoDev& tp = kp.g.tp;
    const int t = grow / tp.nj, j = grow - t * tp.nj;
    auto nb = [&](int jj, int ii) -> double {
      return val(source(t, jj, ii), ((long long)t * tp.npy + jj + tp.OLy) * tp.npx + ii + tp.OLx);
    };
    const double* const* a = kp.g.a64;
    return op_A<double>(__ldg(a[0] + p), __ldg(a[0] + p + 1), __ldg(a[1] + p), __ldg(a[1] + p + tp.npx),
                        __ldg(a[2] + p), nb(j, i - 1), nb(j, i + 1), nb(j - 1, i), nb(j + 1, i), nb(j, i));
  }
  // rhsMax = max |b cg2dNorm| (cg2d.py:221-225) of every right-hand side, through an exchange
  __device__ void rhs_max() {
    Scalars& q = sc();
    if (threadIdx.x < NS) {
      q.nrm[threadIdx.x] = kp.g.norm_arr ? kp.g.norm_arr[inst] : kp.g.norm;
      q.vmax[threadIdx.x] = 0ull;
    }
    __syncthreads();
    u64 m[NS] = {};
    each_point(
        [&](int, const RowEnt& e, int i) {
          const long long p = pad_of(e.grow, i);
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const u64 v = bits_of(fabs(mul(__ldg(kp.g.b[s] + p), q.nrm[s])));   // cg2d.py:222-223
            m[s] = v > m[s] ? v : m[s];
          }
        },
        [](int) {});
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      for (int o = 16; o > 0; o >>= 1) {
        const u64 y = __shfl_xor_sync(0xffffffffu, m[s], o);
        m[s] = y > m[s] ? y : m[s];
      }
      if ((threadIdx.x & 31) == 0) atomicMax(&q.vmax[s], m[s]);
    }
    __syncthreads();
    ++stag;
    for (int e = threadIdx.x; e < NS * nunits; e += kTeamThreads)
      st_msg(sum_buf() + ((long long)rank * kp.t.sum_block + (e / nunits) * kp.t.max_units + e % nunits) * 16,
             q.vmax[e / nunits], stag);
    // (the test of the time limit: a tag that nobody sends)
    if (kp.test_missing) stag += 1u << 30;
    receive(false, NS);
    if (fail) return;
    u64 a[NS] = {};
    for (int u = threadIdx.x; u < kp.t.units; u += kTeamThreads)
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const u64 v = bits_of(psum()[s * kp.t.units + u]);
        a[s] = v > a[s] ? v : a[s];
      }
#pragma unroll
    for (int s = 0; s < NS; ++s)
      if (a[s]) atomicMax(&q.vmax[s], a[s]);
    __syncthreads();
    if (threadIdx.x < NS) {
      const double rhsMax = __longlong_as_double((long long)q.vmax[threadIdx.x]);
      q.rn[threadIdx.x] = rhsMax != 0.0 ? __ddiv_rn(1.0, rhsMax) : 1.0;
    }
    __syncthreads();
  }

  // after an exchange that ends an iteration (k iterations done): totals into the scalars and the stop rule before
  // the next one (cg2d.py:238-248), by warp 0
  __device__ __forceinline__ void next_iteration(int k, bool start) {
    Scalars& q = sc();
    const int s = threadIdx.x;
    bool on = false;
    if (s < NS) {
      const double tol = kp.g.tol[s];
      // (a right-hand side that has stopped keeps its last sums)
      if (start || q.k_done[s] < 0) {
        q.rr[s] = q.total[s];
        q.eta[s] = q.total[NS + s];
        if (rank == 0) {
          if (start) {
            *hist(s, H_RRR, 0) = q.total[s];
            *hist(s, H_ETAZ, 0) = q.total[NS + s];
            *hist(s, H_SUM, 0) = q.total[2 * NS + s];
          } else {
            *hist(s, H_RRX, k) = q.total[s];
            *hist(s, H_ETAX, k) = q.total[NS + s];
          }
        }
      }
      if (start) {
        q.eta_prev[s] = 1.0;
        q.k_done[s] = -1;
        q.nrep[s] = 0;
      }
      q.act[s] = 0;
      if (q.k_done[s] < 0) {
        if (!(k < kp.g.max_iters[s]) || q.rr[s] < tol * tol) {     // cg2d.py:219, 241
          q.k_done[s] = k;
        } else {
          q.act[s] = 1;
          on = true;
          q.beta[s] = __ddiv_rn(q.eta[s], q.eta_prev[s]);          // cg2d.py:247
          q.eta_prev[s] = q.eta[s];                                 // cg2d.py:248
        }
      }
    }
    const unsigned any = __ballot_sync(0xffffffffu, on);
    if (s == 0) q.run = any != 0u;
  }

  // after pass S: alpha (cg2d.py:252-253) and whether the true residual replaces the carried one
  __device__ __forceinline__ void step_length(int k) {
    Scalars& q = sc();
    const int s = threadIdx.x;
    bool rep = false;
    if (s < NS) {
      if (q.act[s]) {
        if (rank == 0) *hist(s, H_SQ, k) = q.total[s];
        q.alpha[s] = __ddiv_rn(q.eta[s], q.total[s]);
        if (MIXED && kp.replace_every > 0 && ((k + 1) % kp.replace_every) == 0) {
          const double lim = kp.replace_above * kp.g.tol[s];
          rep = q.rr[s] > lim * lim;
        }
      }
      q.rep[s] = rep;
      if (rep) ++q.nrep[s];
    }
    const unsigned any = __ballot_sync(0xffffffffu, rep);
    if (s == 0) q.any_rep = any != 0u;
  }

  __device__ __forceinline__ T coef_of(const double (&a)[2]) const {
    T v;
#pragma unroll
    for (int s = 0; s < NS; ++s) put(v, s, a[s]);
    return v;
  }

  // the true residual b - A x of the right-hand sides in sc().rep, in FP64 (MIXED), into the shared r; x is current. Its
  // neighbours are read from L2 after an exchange that makes every CTA's x visible: the threads that send it fence after the
  // barrier behind the CTA's stores of x, the threads that poll it fence before the barrier in front of the reads
  __device__ void true_residual() {
    Scalars& q = sc();
    for (int lr = threadIdx.x; lr < nrows; lr += kTeamThreads)
      for (int s = 0; s < NS; ++s) rowsum()[s * kp.t.max_rows + lr] = 0.0;
    __syncthreads();
    __threadfence();
    send_sums(1);
    receive(false, NS, true);
    if (fail) return;
    const TopoDev& tp = kp.g.tp;
    const int n = ni(), nj = tp.nj, lane = threadIdx.x & 31, tile0 = row0 / nj;
    const int nwe = nhalo - 2 * nrows;   // halo cells before the west / east ones
    T* r = R();
    double* hx = smem_at<double>(kp.t.o_hval);
    const double* const* a64 = kp.g.a64;
    // x at the halo cells [cell][NS]: an unwritten one keeps the first guess
    for (int h = threadIdx.x; h < nhalo; h += kTeamThreads) {
      int t, j, i;
      halo_point(h, tile0, t, j, i);
      const int src = source(t, j, i);
      const long long o = (long long)inst * kp.g.pad_elems + ((long long)t * tp.npy + j + tp.OLy) * tp.npx + i + tp.OLx;
#pragma unroll
      for (int s = 0; s < NS; ++s)
        hx[h * NS + s] = src >= 0 ? __ldcg(x + (long long)src * NS + s) : __ldg(kp.g.x0[s] + o);
    }
    __syncthreads();
#pragma unroll 1
    for (int lr = lrA; lr < lrB; ++lr) {
      const RowEnt e = rows()[lr];
      const int t = e.grow / nj, j = e.grow - t * nj, seg = t - tile0;
      const long long p0 = pad_of(e.grow, 0);
      const double* xr = x + (long long)e.grow * n * NS;
      // the rows below and above, from x or, at the ends of the run, from the halo
      const bool lo = lr > 0 && j > 0, hi = lr + 1 < e.end;
      const double *hs = hx + seg * 2 * n * NS, *hn = hs + n * NS, *hw = hx + (nwe + 2 * lr) * NS;
#pragma unroll 3
      for (int i = lane; i < n; i += 32) {
        const long long p = p0 + i;
        const double aw = __ldg(a64[0] + p), ae = __ldg(a64[0] + p + 1), as = __ldg(a64[1] + p),
                     an = __ldg(a64[1] + p + tp.npx), ac = __ldg(a64[2] + p);
        const int iw = i > 0 ? i - 1 : 0, ie = i < n - 1 ? i + 1 : i;
        T* rp = r + e.ring + i;
        T rv = *rp;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const double xc = __ldcg(xr + i * NS + s), xw = __ldcg(xr + iw * NS + s), xe = __ldcg(xr + ie * NS + s);
          const double xd = lo ? __ldcg(xr + (i - n) * NS + s) : hs[i * NS + s];
          const double xu = hi ? __ldcg(xr + (i + n) * NS + s) : hn[i * NS + s];
          const double bn = mul(mul(__ldg(kp.g.b[s] + p), q.nrm[s]), q.rn[s]);
          const double ax = op_A<double>(aw, ae, as, an, ac, i > 0 ? xw : hw[s], i < n - 1 ? xe : hw[NS + s], xd, xu, xc);
          if (q.rep[s]) put(rv, s, sub(bn, ax));
        }
        *rp = rv;
      }
    }
    halo_r();
  }

  // exchange the halo of r (the start, and after a true residual)
  __device__ __forceinline__ void halo_r() {
    T* r = R();
    __syncthreads();
    ++htag;
    send_ring(r);
    receive(true, 0);
    for (int h = threadIdx.x; h < nhalo; h += kTeamThreads) {
      const int el = halo()[h].elem;
      if (el >= 0) r[el] = hval()[h];
    }
    __syncthreads();
  }

  // the coefficients of the CTA's rows, in the solver's precision, as the passes read them: [operator][row][ni + 1], the
  // last column's west face being the row's last east face
  __device__ void pack() {
    const int n = ni(), npx = kp.g.tp.npx;
#pragma unroll 1
    for (int w = threadIdx.x >> 5; w < 2 * nrows; w += kTeamWarps) {
      const int op = w >= nrows, lr = w - op * nrows;
      const long long p = pad_of(row0 + lr, 0);
      C4* o = coef + ((long long)op * kp.t.max_rows + lr) * (n + 1);
      const double *aw = kp.g.a64[3 * op] + p, *as = kp.g.a64[3 * op + 1] + p, *ac = kp.g.a64[3 * op + 2] + p;
#pragma unroll 2
      for (int i = threadIdx.x & 31; i <= n; i += 32)
        store4(o, n + 1, i, (C)__ldg(aw + i), (C)__ldg(as + i), (C)__ldg(as + npx + i), (C)__ldg(ac + i));
    }
  }

  // x = x0 rhsNorm, r = b - A x, s = 0 (cg2d.py:226-236); row sums of b in place 2
  __device__ void start() {
    Scalars& q = sc();
    T* r = R();
    T zero;
#pragma unroll
    for (int s = 0; s < NS; ++s) put(zero, s, 0.0);
    for (unsigned e = threadIdx.x; e < kp.t.ring_elems; e += kTeamThreads) { r[e] = zero; S()[e] = zero; }
    __syncthreads();
    double acc[2][NS] = {};
    each_point(
        [&](int lr, const RowEnt& e, int i) {
          const long long p = pad_of(e.grow, i);
          T rv;
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const double* x0 = kp.g.x0[s] + (long long)inst * kp.g.pad_elems;
            const double rn = q.rn[s];
            // the first guess: scaled where it is (or the exchange supplies it from) an interior point (cg2d.py:227-228)
            auto guess = [&](int src, long long h) -> double {
              return src >= 0 ? mul(__ldg(x0 + cmp_to_pad(kp.g.tp, src)), rn) : __ldg(x0 + h);
            };
            const double bn = mul(mul(__ldg(kp.g.b[s] + p), q.nrm[s]), rn);              // cg2d.py:221, 226
            put(rv, s, sub(bn, apply_f64(e.grow, i, p, guess)));                          // cg2d.py:232
            __stcg(x + ((long long)e.grow * ni() + i) * NS + s, mul(__ldg(kp.g.x0[s] + p), rn));
            if constexpr (!SERIAL) acc[0][s] = add(acc[0][s], bn);
          }
          r[e.ring + i] = rv;
        },
        [&](int lr) {
          if constexpr (!SERIAL) {
            row_sum(lr, 1, acc, 2);
#pragma unroll
            for (int s = 0; s < NS; ++s) acc[0][s] = 0.0;
          }
        });
    if constexpr (SERIAL) {   // the sum of b
      const int warp = threadIdx.x >> 5;
      for (int task = warp; task < nunits * NS; task += kTeamWarps) {
        const int s = task / nunits, lu = task % nunits;
        double sum = 0.0;
        for (int lr = unit_rows()[lu]; lr < unit_rows()[lu + 1]; ++lr) {
          const double* row = kp.g.b[s] + pad_of(rows()[lr].grow, 0);
          for (int c = 0; c < ni(); c += 32) {
            const double bn = mul(mul(__ldg(row + min(c + (int)(threadIdx.x & 31), ni() - 1)), q.nrm[s]), q.rn[s]);
            for (int k = 0; k < 32 && c + k < ni(); ++k) sum = add(sum, __shfl_sync(0xffffffffu, bn, k));
          }
        }
        if ((threadIdx.x & 31) == 0) rowsum()[(2 * NS + s) * kp.t.max_rows + lu] = sum;
      }
    }
    halo_r();
  }

  // x_out, x_fortran and diag of the solved instance
  __device__ void finish() {
    const TopoDev& tp = kp.g.tp;
    Scalars& q = sc();
    each_point(
        [&](int, const RowEnt& e, int i) {
          const long long p = pad_of(e.grow, i);
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const double xf = __ddiv_rn(__ldcg(x + ((long long)e.grow * ni() + i) * NS + s), q.rn[s]);   // cg2d.py:266
            kp.g.x_out[s][p] = xf;
            if (kp.g.x_fortran[s]) kp.g.x_fortran[s][p] = xf;
          }
        },
        [](int) {});
    // halo points: x_out 0; x_fortran = exchanged normalised first guess, unwritten points keep cg2d_x
    // (cg2d.py:208-210, 227-228)
    const int plane = tp.npy * tp.npx;
    const long long per = kp.g.pad_elems, o = (long long)inst * per;
    auto interior = [&](int a, int b) { return a >= tp.OLy && a < tp.OLy + tp.nj && b >= tp.OLx && b < tp.OLx + tp.ni; };
    for (int p = rank * kTeamThreads + threadIdx.x; p < per; p += kp.t.G * kTeamThreads) {
      const int in_tile = p % plane, jj = in_tile / tp.npx, ii = in_tile - jj * tp.npx;
      if (interior(jj, ii)) continue;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        kp.g.x_out[s][o + p] = 0.0;
        if (kp.g.x_fortran[s]) {
          const double* x0 = kp.g.x0[s] + o;
          double v = __ldg(x0 + p);
          if (tp.map_comp[p] == 1) {
            const int sp = tp.map_src[p], spl = sp % plane;
            v = __ldg(x0 + sp);
            if (interior(spl / tp.npx, spl % tp.npx)) v = mul(v, q.rn[s]);
          }
          kp.g.x_fortran[s][o + p] = v;
        }
      }
    }
    if (rank == 0 && threadIdx.x < NS) write_diag(threadIdx.x, true);
  }
  __device__ void write_diag(int s, bool ok) {
    const Scalars& q = sc();
    const double rr = q.rr[s], tol = kp.g.tol[s];
    cg2d_diag_t d;
    d.firstResidual = sqrt(*hist(s, H_RRR, 0));
    d.lastResidual = sqrt(rr);
    d.sumRHS = *hist(s, H_SUM, 0);
    d.rhsMax = __longlong_as_double((long long)q.vmax[s]);
    d.numIters = q.k_done[s];
    d.replacements = q.nrep[s];
    d.reserved = 0;
    const unsigned err = ld_relaxed(&kp.gs[1]);
    if (!ok || err != 0u) d.status = err != 0u ? (int)err : CG2D_BARRIER_TIMEOUT;
    else if (rr != rr) d.status = CG2D_NAN;
    else if (!(rr < tol * tol)) d.status = CG2D_NOT_CONVERGED;
    else d.status = CG2D_OK;
    if (!ok) {
      d.firstResidual = d.lastResidual = d.sumRHS = __longlong_as_double(0x7ff8000000000000LL);
      d.numIters = 0;
      d.replacements = 0;
    }
    kp.g.diag[s][inst] = d;
  }

  // phase times of thread 0 (cg2d_params_t.profile)
  __device__ __forceinline__ u64 clock() const { return kp.prof && threadIdx.x == 0 ? globaltimer() : 0ull; }
  __device__ __forceinline__ void lap(int phase, u64& t) const {
    if (kp.prof && threadIdx.x == 0) {
      const u64 now = globaltimer();
      sc().tm[phase] += now - t;
      t = now;
    }
  }

  // one exchange: the sums of the pass just computed out, its halo values and everybody's sums in, totals by warp 0.
  // `meanwhile` runs between sending and receiving.
  template <class F, class W>
  __device__ __forceinline__ void exchange(int nk, F meanwhile, W scalars) {
    u64 t = clock();
    send_sums(nk);
    lap(PR_ISSUE, t);
    meanwhile();
    lap(PR_DIRECT, t);
    receive(true, nk * NS);
    lap(PR_BAR, t);
    if (fail) return;
    fold(nk * NS);
    if (threadIdx.x < 32) scalars();
    __syncthreads();
    lap(PR_FIN, t);
  }

  __device__ __forceinline__ void solve() {
    Scalars& q = sc();
    pack();
    rhs_max();
    if (fail) return;
    start();
    if (fail) return;
    Coefs f;
    prefetch<true>(f);
    stencil<true>(f, nullptr);
    exchange(3, [] {}, [&] { next_iteration(0, true); });
    if (fail) return;
    int k = 0;
    while (q.run) {
      // s = z + beta s (cg2d.py:249), q = A s (cg2d.py:251)
      u64 t = clock();
      const bool ck = !MIXED && kp.ck_r && ((k + 1) % kp.ck_every) == 0;
      const long long cko = ck ? (long long)((k + 1) / kp.ck_every) * kp.ck_stride : 0;
      prefetch<false>(f);
      update<true>(S(), coef_of(q.beta));
      __syncthreads();
      lap(PR_CTRL, t);
      stencil<false>(f, ck ? kp.ck_s + cko : nullptr);
      lap(PR_COMP, t);
      exchange(1, [] {}, [&] { step_length(k); });
      if (fail) return;
      // r -= alpha q (cg2d.py:255), z = M r (cg2d.py:245); x += alpha s while the sums travel
      t = clock();
      prefetch<true>(f);
      update<false>(R(), vneg(coef_of(q.alpha)));
      const bool rep = MIXED && q.any_rep;
      if (rep) update_x();
      __syncthreads();
      if (rep) {
        true_residual();
        if (fail) return;
      }
      lap(PR_CTRL, t);
      stencil<true>(f, ck ? kp.ck_r + cko : nullptr);
      lap(PR_COMP, t);
      ++k;
      exchange(
          2, [&] { if (!rep) update_x(); }, [&] { next_iteration(k, false); });
      if (fail) return;
    }
    finish();
  }
};

// CTA `cta` of a group's CTAs
template <bool MIXED, int NS, bool SERIAL, int STEPS>
__device__ __forceinline__ void run_team(const TeamParams& kp, unsigned cta) {
  const u64 t_begin = kp.prof && threadIdx.x == 0 ? globaltimer() : 0ull;
  const int team = cta / kp.t.G, rank = cta - team * kp.t.G;
  Team<MIXED, NS, SERIAL, STEPS> tm(kp, team, rank);
  tm.tables();
  __syncthreads();
  bool fail = false;
  for (int in = team; in < kp.g.count; in += kp.t.nteams) {
    tm.inst = in;
    if (!fail) {
      tm.solve();
      fail = tm.fail;
      __syncthreads();
    }
    // the time limit ran out: this instance and the team's later ones have no result
    if (fail && rank == 0 && threadIdx.x < NS) tm.write_diag(threadIdx.x, false);
  }
  if (kp.prof && threadIdx.x == 0 && blockIdx.x < kMaxCtas) {
    u64* o = kp.prof + 1 + (size_t)blockIdx.x * kProfSlots;
    const u64 tot = globaltimer() - t_begin;
    u64 sum = 0;
    for (int i = 0; i < kProfSlots; ++i) sum += tm.sc().tm[i];
    for (int i = 0; i < kProfSlots; ++i) o[i] += tm.sc().tm[i];
    o[PR_OTHER] += tot > sum ? tot - sum : 0ull;
    o[PR_TOTAL] += tot;
    atomicMax(kp.prof, (u64)gridDim.x);
  }
}

template <bool MIXED, int NS, bool SERIAL, int STEPS>
__global__ void __launch_bounds__(kTeamThreads, 1) cg2d_team(const __grid_constant__ TeamParams kp) {
  run_team<MIXED, NS, SERIAL, STEPS>(kp, blockIdx.x);
}

// Several groups side by side, each on CTAs of its own. Alone, a group that is bound by latency leaves most of the chip idle, and
// the times of launches one after the other add up: four LLC90 FP64 solves of 40 iterations, one a group, 1722 us as four
// launches and 762 us as one; in the FORTRAN order 23.3 ms and 6.3 ms. A kernel of its own, because the group's parameters are
// indexed here and constants of the launch in cg2d_team. (FORTRAN order: the additions bound a pass, so the general row path
// serves every width.)
template <bool MIXED, int NS, bool SERIAL>
__global__ void __launch_bounds__(kTeamThreads, 1) cg2d_team_groups(const __grid_constant__ TeamGroups kg) {
  int g = 0;
  while (g + 1 < kg.n && (int)blockIdx.x >= kg.first[g + 1]) ++g;
  const TeamParams& kp = kg.p[g];
  const unsigned cta = blockIdx.x - kg.first[g];
  if constexpr (!SERIAL && (MIXED || NS == 1)) {
    const int ni = kp.g.tp.ni;
    if (ni <= 32) run_team<MIXED, NS, SERIAL, 1>(kp, cta);
    else if (ni <= 64) run_team<MIXED, NS, SERIAL, 2>(kp, cta);
    else if (ni <= 96) run_team<MIXED, NS, SERIAL, 3>(kp, cta);
    else run_team<MIXED, NS, SERIAL, 0>(kp, cta);
  } else {
    run_team<MIXED, NS, SERIAL, 0>(kp, cta);
  }
}

template <bool MIXED, int NS, bool SERIAL>
const void* team_fn_of(int ni) {
  if constexpr (MIXED || NS == 1) {
    if (ni <= 32) return (const void*)cg2d_team<MIXED, NS, SERIAL, 1>;
    if (ni <= 64) return (const void*)cg2d_team<MIXED, NS, SERIAL, 2>;
    if (ni <= 96) return (const void*)cg2d_team<MIXED, NS, SERIAL, 3>;
  }
  return (const void*)cg2d_team<MIXED, NS, SERIAL, 0>;
}
const void* team_fn(int mixed, int serial, int nrhs, int ni) {
  if (mixed) {
    if (serial) return nrhs == 2 ? team_fn_of<true, 2, true>(ni) : team_fn_of<true, 1, true>(ni);
    return nrhs == 2 ? team_fn_of<true, 2, false>(ni) : team_fn_of<true, 1, false>(ni);
  }
  if (serial) return nrhs == 2 ? team_fn_of<false, 2, true>(ni) : team_fn_of<false, 1, true>(ni);
  return nrhs == 2 ? team_fn_of<false, 2, false>(ni) : team_fn_of<false, 1, false>(ni);
}

const void* team_groups_fn(int mixed, int serial, int nrhs) {
  if (mixed) {
    if (serial) return nrhs == 2 ? (const void*)cg2d_team_groups<true, 2, true> : (const void*)cg2d_team_groups<true, 1, true>;
    return nrhs == 2 ? (const void*)cg2d_team_groups<true, 2, false> : (const void*)cg2d_team_groups<true, 1, false>;
  }
  if (serial) return nrhs == 2 ? (const void*)cg2d_team_groups<false, 2, true> : (const void*)cg2d_team_groups<false, 1, true>;
  return nrhs == 2 ? (const void*)cg2d_team_groups<false, 2, false> : (const void*)cg2d_team_groups<false, 1, false>;
}

// first row of unit u (host)
int unit_row_h(const TeamDev& t, int nj, int u) {
  const int tile = u / t.nblk, blk = u - tile * t.nblk;
  return tile * nj + (nj < blk * t.rpb ? nj : blk * t.rpb);
}
// contiguous runs of at most `cap` rows: the CTAs it takes (at most `most` + 1 are counted), boundaries in ub
int runs_of(const TeamDev& t, int nj, int cap, int most, unsigned short* ub) {
  int n = 0, u = 0;
  ub[0] = 0;
  while (u < t.units) {
    if (n == most) return most + 1;
    const int row = unit_row_h(t, nj, u);
    // the last unit boundary at or below row + cap
    const int lim = row + cap;
    int tile = lim / nj, v;
    const int rem = lim - tile * nj;
    v = tile * t.nblk + rem / t.rpb;
    if (v > t.units) v = t.units;
    if (v <= u) return most + 1;
    u = v;
    ub[++n] = (unsigned short)u;
  }
  return n;
}

}  // namespace

size_t team_msg_bytes(const TopoDev& tp, int nrhs, int mixed, const TeamDev& t) {
  const size_t ms = mixed ? 1 : nrhs;
  return 2 * (ms * (size_t)t.nslots + (size_t)t.G * t.sum_block) * 16;
}
size_t team_coef_bytes(const TopoDev& tp, int mixed, const TeamDev& t) {
  return (size_t)t.G * 2 * t.max_rows * (tp.ni + 1) * 4 * (mixed ? sizeof(float) : sizeof(double));
}

namespace {

// the shared memory of a CTA with at most `rows` rows, `ring` ring rows, `halo` halo cells and `units` units: the layout into c
size_t smem_layout(const TopoDev& tp, int nrhs, int mixed, int rows, int ring, int halo, int units, TeamDev* c) {
  const unsigned es = (mixed ? 4u : 8u) * nrhs;
  const int ni = tp.ni;
  size_t o = kScalBytes;
  auto take = [&](size_t bytes) { const size_t p = o; o += (bytes + 127) & ~size_t(127); return (unsigned)p; };
  c->o_rows = take(sizeof(RowEnt) * (size_t)rows);
  c->o_halo = take(sizeof(HaloEnt) * (size_t)halo);
  c->o_send = take(sizeof(SendEnt) * (size_t)halo);   // (at most as many as halo cells)
  c->o_umsg = take(sizeof(int) * (size_t)c->units);
  c->o_hval = take((size_t)8 * nrhs * halo);   // (also x at the halo cells, FP64)
  c->o_units = take(sizeof(int) * ((size_t)units + 1));
  c->o_rowsum = take(sizeof(double) * (size_t)kTeamKinds * nrhs * rows);
  c->o_psum = take(sizeof(double) * (size_t)kTeamKinds * nrhs * c->units);
  c->o_tsum = take(sizeof(double) * (size_t)kTeamKinds * nrhs * tp.T);
  c->ring_elems = (unsigned)ring * (unsigned)(ni + 2);
  c->o_r = take((size_t)es * c->ring_elems);
  c->o_s = take((size_t)es * c->ring_elems);
  c->o_q = take((size_t)es * rows * ni);
  return o;
}

// Time of a pass in units of an exchange (4.2 us with its fixed steps); only splits of one launch and the groups of one call
// are compared. From rows alone: 1 + kRowCost per row of the largest CTA's warps and 32 columns, whatever the precision and
// the right-hand sides. Fitted to LLC90 FP64: 4.6 us at 8 rows a CTA, 9.1 us at 66, 10.6 us at 90.
double row_cost(const TopoDev& tp, int rows) {
  const double kRowCost = 0.09;
  return 1.0 + kRowCost * ((rows + kTeamWarps - 1) / kTeamWarps) * ((tp.ni + 31) / 32);
}
// In the FORTRAN order with the ordered additions, too. A CTA's n sums (two kinds in pass X, one in pass S) run side by side on
// its warps, at 15.6 cycles an addition until their shuffles fill the SM at 2.28 cycles an addition and sum. Fitted to 288
// workloads of 2 to 128 instances with tiles of 8 to 96 points, in two splits each, to 2.3 % (root mean square).
double pass_cost(const TopoDev& tp, int nrhs, int mixed, int serial, int rows, int units) {
  if (!serial) return row_cost(tp, rows);
  const double steps = (tp.ni + 31) / 32, per_warp = (rows + kTeamWarps - 1) / kTeamWarps;
  auto chains = [&](int n) {   // cycles an addition of n sums takes
    const int rem = n % kTeamWarps;
    double c = n / kTeamWarps * 2.28 * kTeamWarps;
    if (rem) c += 2.28 * rem > 15.6 ? 2.28 * rem : 15.6;
    return c;
  };
  const double row = mixed ? (nrhs == 2 ? 0.34 : 0.28) : (nrhs == 2 ? 0.57 : 0.33);
  const double us = 3.3 + 0.0096 * nrhs * tp.T + per_warp * (0.44 + row * steps) +
                    (double)tp.ni * tp.nj * (chains(2 * nrhs * units) + chains(nrhs * units)) / 2 / 1920.0;
  return us / 4.2;
}

}  // namespace

size_t team_plan(const TopoDev& tp, int count, int nrhs, int mixed, int serial, int ctas, TeamDev* t, double* cost) {
  if (ctas > kTeamMaxCtas) ctas = kTeamMaxCtas;
  if (t->units > 65535) return 0;
  const int nj = tp.nj, ni = tp.ni, rows = tp.T * nj;
  t->nslots = (2ll * rows + 2ll * t->units * ni + 7) & ~7ll;   // (whole 128-byte lines)
  if (t->nslots > (1ll << 30)) return 0;
  // The split with the least rounds x pass time is taken: 16 ROWBLOCK solves run 8 teams of 18 CTAs, 64 run 11 teams of 13.
  // FORTRAN order: the split that is the best by rows, unless the estimate with the ordered additions has another one at
  // least kSure faster (it is good to 2 or 3 %). 64 mixed LLC90 solves run 21 teams of 7 in 4 rounds (14.0 ms for 20
  // iterations), not the 11 teams of 13 in 6 that the rows alone give (19.0 ms; 16.3 streamed).
  const double kSure = 0.96;
  double rows_best = 0.0, rows_pass = 0.0;
  size_t rows_smem = 0;
  TeamDev by_rows;
  double best = 0.0;
  size_t best_smem = 0;
  TeamDev cand = *t;
  int last_G = -1;
  for (int nt = 1; nt <= count && nt <= ctas; ++nt) {
    int G = ctas / nt;
    if (G > t->units) G = t->units;
    if (G == last_G) continue;   // the same teams, or more of them than fit
    last_G = G;
    // the smallest largest run (a run leaves less than a unit of its rows unused)
    int lo = (rows + G - 1) / G, hi = lo + t->rpb - 1;
    unsigned short tmp[kTeamMaxCtas + 2];
    if (lo < 1) lo = 1;
    while (runs_of(cand, nj, hi, G, tmp) > G) hi += nj;
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (runs_of(cand, nj, mid, G, tmp) <= G) hi = mid;
      else lo = mid + 1;
    }
    const int used = runs_of(cand, nj, hi, G, cand.ub);
    int max_rows = 0, max_ring = 0, max_halo = 0, max_units = 0;
    for (int c = 0; c < used; ++c) {
      const int a = unit_row_h(cand, nj, cand.ub[c]), b = unit_row_h(cand, nj, cand.ub[c + 1]);
      const int nseg = (b - 1) / nj - a / nj + 1;
      const int nr = b - a;
      if (nr > max_rows) max_rows = nr;
      if (nr + 2 * nseg > max_ring) max_ring = nr + 2 * nseg;
      if (2 * nseg * ni + 2 * nr > max_halo) max_halo = 2 * nseg * ni + 2 * nr;
      if (cand.ub[c + 1] - cand.ub[c] > max_units) max_units = cand.ub[c + 1] - cand.ub[c];
    }
    cand.G = used;
    cand.nteams = ctas / used < count ? ctas / used : count;
    cand.max_rows = max_rows;
    cand.max_units = max_units;
    cand.sum_block = (kTeamKinds * nrhs * max_units + 7) & ~7;   // messages: whole 128-byte lines
    const size_t o = smem_layout(tp, nrhs, mixed, max_rows, max_ring, max_halo, max_units, &cand);
    if (o > (size_t)kSmemLimit) continue;
    const int rounds = (count + cand.nteams - 1) / cand.nteams;
    const double c = rounds * pass_cost(tp, nrhs, mixed, serial, max_rows, max_units);
    if (best_smem == 0 || c < best) {
      best = c;
      best_smem = o;
      *t = cand;
    }
    const double r = rounds * row_cost(tp, max_rows);
    if (rows_smem == 0 || r < rows_best) {
      rows_best = r;
      rows_pass = c;
      rows_smem = o;
      by_rows = cand;
    }
  }
  if (rows_smem != 0 && best > kSure * rows_pass) {
    best = rows_pass;
    best_smem = rows_smem;
    *t = by_rows;
  }
  *cost = best;
  return best_smem;
}

// (a run of r rows: over at most (r - 2) / nj + 2 tiles; whole tiles in the FORTRAN order)
int team_least_ctas(const TopoDev& tp, int nrhs, int mixed, int serial, const TeamDev& t) {
  TeamDev c = t;
  const int rows = tp.T * tp.nj;
  auto fits = [&](int r) {
    const int nseg = serial ? r / tp.nj : (r - 2 + tp.nj) / tp.nj + 1;
    return smem_layout(tp, nrhs, mixed, r, r + 2 * nseg, 2 * nseg * tp.ni + 2 * r, (r + t.rpb - 1) / t.rpb + nseg, &c) <=
           (size_t)kSmemLimit;
  };
  int lo = 0, hi = (rows + t.rpb - 1) / t.rpb;   // units: lo fit, hi + 1 need not
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (fits(mid * t.rpb)) lo = mid;
    else hi = mid - 1;
  }
  if (lo == 0) return 0;
  return (t.units + lo - 1) / lo;
}

double team_cost(const TopoDev& tp, int count, int nrhs, int mixed, int serial, int least, int ctas, const TeamDev& t) {
  if (ctas > kTeamMaxCtas) ctas = kTeamMaxCtas;
  double best = 0.0;
  for (int nt = 1; nt <= count && nt * least <= ctas; ++nt) {
    const int G = ctas / nt < t.units ? ctas / nt : t.units;
    const int units = (t.units + G - 1) / G, nteams = ctas / G < count ? ctas / G : count;
    int rows = (tp.T * tp.nj + G - 1) / G + (G < t.units ? t.rpb / 2 : 0);   // (runs end at units)
    if (serial || rows > units * t.rpb) rows = units * t.rpb;
    const double c = (count + nteams - 1) / nteams * pass_cost(tp, nrhs, mixed, serial, rows, units);
    if (best == 0.0 || c < best) best = c;
  }
  return best;
}

cudaError_t launch_team(const TeamParams& kp, int mixed, int serial, size_t smem, cudaStream_t stream) {
  const int nrhs = kp.g.nrhs, grid = kp.t.G * kp.t.nteams;
  const void* fn = team_fn(mixed, serial, nrhs, kp.g.tp.ni);
  // The limit belongs to the function, which every thread and stream of the context shares: always the largest, so that no
  // call lowers it between another one's setting and launch.
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<TeamParams*>(&kp)};
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kTeamThreads), args, smem, stream);
}

cudaError_t launch_team_groups(const TeamGroups& kg, int mixed, int serial, size_t smem, cudaStream_t stream) {
  const void* fn = team_groups_fn(mixed, serial, kg.p[0].g.nrhs);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);   // (as launch_team)
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<TeamGroups*>(&kg)};
  return cudaLaunchCooperativeKernel(fn, dim3(kg.first[kg.n]), dim3(kTeamThreads), args, smem, stream);
}

}  // namespace cg2d
