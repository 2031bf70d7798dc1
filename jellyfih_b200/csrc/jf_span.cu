// Batched path, spans: the grid rows of all instances, one instance after the
// other, are cut into contiguous spans of about equal cost at every re-sort, one
// per SM where there are four rows for each, and one cooperative launch per
// chunk of substeps advances them all, one CTA per span.  A CTA owns the bands
// of rows (one per instance that its span touches) and keeps them, plus a halo,
// in shared memory for the whole chunk.
//
// Why spans and not one thread-block cluster per instance: clusters are placed
// per GPC, so that at one CTA per SM only 33 clusters of 4, 15 of 8 or 7 of 16
// fit a B200 (cudaOccupancyMaxActiveClusters): 32 instances use 128 of the 148
// SMs, and 16 instances on clusters of 8 or 8 on clusters of 16 take two
// waves.  Spans use every SM from 592 rows on (five tanks of 128; one tank
// takes 32), and an instance may share an SM with the next one.
//
// One pass over a CTA's particles fuses G2P of substep s-1 with P2G of substep
// s (mpm_sim.py:312-333 then :168-271).  Neighbouring bands of an instance
// overlap in the four rows around their cut (the stencil's reach plus one row
// of drift either way).  After a pass each side writes its partial sums of
// those rows to global memory and takes the other's, and updates the rows for
// itself: the same two terms, so the same bits.  A node travels as one 16-byte
// word of its sums and the substep's tag, written and read whole, so that the
// reader polls the data itself and no fence stands in its way.  Beside it the
// instance's CTAs count their arrivals, which keeps them within a substep of
// one another.  The rows between are updated while the words travel.
//
// A particle whose stencil has drifted out of its CTA's window (more than a
// row since the last re-sort) adds to a spill grid in global memory, and its
// CTA's arrival carries a drift mark; the instance's CTAs then add the spill to
// their rows, publish their updated rows and meet a second time, so that the
// particle can gather them in the next pass.  The result does not depend on
// the re-sort interval.
//
// Every wait counts its polls and gives up after spin_limit of them: the CTA
// raises the abort flag, which ends the waits of the others, sets kJfErrAbort on
// the instances of its bands, frees its tensor memory and returns.  The abort
// flag stays up until jf_clear_error_flags: what is queued behind the chunk
// returns at once, so that the time of a run whose waits run out is bounded by
// one of them, and sets the same error flag on the instances it leaves alone.
#include <cuda.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "jf_chunk.cuh"

namespace {

constexpr int kMaxSeg = 8;        // bands of one CTA
constexpr int kMinRows = 4;       // rows of a band: the overlaps of its two cuts stay apart
constexpr int kOverlap = 4;       // rows around a cut that both sides hold
// CTA size where the caller asks for none: 16 warps with the node blocks in
// registers beat 24 with the blocks in TMEM at every batch size since the
// packed arithmetic (us per substep, 80K-slot tanks on 128^2: 32 instances 81.9
// against 86.2, 16: 45.8 against 48.7).
constexpr int kSpanThreads = 512;
constexpr int kScanThreads = 1024;
constexpr int kMoveThreads = 256;
// What a pass costs, in units of 1/128 of a warp's iteration over its 32 cells:
// the cell cap minimises, and the spans balance, 128 for every iteration of a
// segment's fullest cell up to the cap, kOverCost for a particle beyond it
// (scattered with atomics of its own), and for the spans also kSegCost for a
// segment's flush, kRowCost for a row's grid update and kSolidCostHalves / 2
// for a non-water particle.  Swept on running batches, us per substep: overflow
// 4 / 6 / 10 / 14 / 24 / 64: 48 uneven beside 16 tall 431 / 242 / 218 / 212 /
// 216 / 217, 32 tanks of 80,000 slots 148 / 74.1 / 74.2 / 74.1 / 74.0 / 73.9;
// segment 0 / 64 / 128 / 192: 32 tanks 76.2 / 74.4 / 74.1 / 74.0.
constexpr int kCapCandidates = 16;
constexpr int kNoCap = 1 << 30;
constexpr int kOverCost = 14;
constexpr int kSegCost = 128;
constexpr int kRowCost = 80;
constexpr int kSolidCostHalves = 5;
constexpr uint32_t kSpinLimit = 20000000;  // default: polls of about 0.7 us each, some 14 seconds
constexpr size_t kMaxSmem = 227 * 1024;
constexpr size_t kStaticSmem = 3072;  // static shared variables of the kernel, rounded up
// Shared memory and L1 share an SM's 256 KB: larger windows slow the particle
// loads, so that larger batches run as several groups of instances, one launch
// after the other, whose equal shares of the rows stay within this size.  A
// window may take 8/5 of the largest share, as bands of equal cost differ in
// rows; up to all of shared memory where one instance's share is already over
// the size, or where the rows do not fit their CTAs otherwise.
// Measured on 48 instances of 40K to 120K particles on 128^2 beside 16 of 128K
// on 128x256 (us per substep; shares of 200, 109, 80 and 65 KB): 1 group 325,
// 2: 293, 3: 273, 4: 287; at 5/4 of the share 302 and 282 for 2 and 3 (some
// re-sorts fell back to spans of equal windows).  With the cost model below 2, 3
// and 4 groups take 216, 220 and 232.
constexpr size_t kSoftSmem = 96 * 1024;

struct SpanGroup {
  int32_t m0, m1;    // instances
  int32_t row0, rows;  // rows of those instances in the concatenation of all
  int32_t n_cta;
  int32_t pad;
};

}  // namespace

// Device and host state of the span path of one engine.
struct JfSpan {
  std::vector<SpanGroup> groups;
  int32_t threads = 0;     // threads of a CTA
  int32_t n_cta = 0;       // CTAs of a launch (table stride)
  int32_t total_rows = 0;
  int32_t cap_nodes = 0;   // window nodes of a CTA
  size_t smem = 0;
  void* pool = nullptr;    // holds every array below
  SpanGroup* d_groups = nullptr;
  int32_t* d_rowoff = nullptr;    // M + 1: first row of each instance
  int32_t* d_rowcost = nullptr;   // total_rows
  unsigned long long* d_rowpre = nullptr;  // total_rows: inclusive prefix of the costs within a group
  int32_t* d_ovrow = nullptr;     // total_rows + M: overflow list starts per row (ny + 1 per instance)
  int32_t* d_ovcur = nullptr;     // total_rows: cursors of the rows' overflow lists
  int32_t* d_fallback = nullptr;  // groups x (n_cta + 1): cuts by window size alone
  int4* d_seg = nullptr;          // groups x n_cta x kMaxSeg: (instance, first row, end row, 0)
  int32_t* d_nseg = nullptr;      // groups x n_cta
  int32_t* d_nbar = nullptr;      // M: CTAs that hold a band of the instance
  // 3 M: arrivals of even and of odd substeps (drift marks in the upper half), of drift meetings
  unsigned long long* d_bar = nullptr;
  int32_t* d_drift = nullptr;     // M: bit s % 3: the spill grid of substep s is in use; kDriftUnknown
  uint32_t* d_tag = nullptr;      // tag of the next chunk's first substep
  int32_t* d_abort = nullptr;     // a wait gave up: nothing runs until it is cleared
  uint32_t spin_limit = kSpinLimit;
  float4* d_spill = nullptr;      // 3 x total nodes
  // n_cta x 2 sides x 2 parities x kOverlap x nx_max nodes (twice that, the hoop
  // sums in the second half, in the axisymmetric variant)
  uint4* d_slot = nullptr;
};

namespace {

struct SpanArgs {
  JfInst I;                   // the constants that follow from n_grid, dt and the flags: the same for every instance
  const JfInst* inst;
  const JfParams* params;
  JfMaterials mats;
  float4* xv;
  float4* C;
  float4* F;
  const int32_t* mat;
  float* Jp;
  const float2* fiber;
  float* glow;
  const float* rref;
  const int32_t* cell_start;  // M x stride: start of each bin's run (relative to p_off)
  const int32_t* cap;
  const int32_t* ovlist;      // overflow positions (relative to p_off), grouped by row
  const int32_t* ovrow;
  const int32_t* rowoff;
  const int4* seg;            // of this group
  const int32_t* nseg;
  const int32_t* nbar;
  unsigned long long* bar;
  int32_t* drift;
  int32_t* abort;
  uint32_t spin_limit;        // polls after which a wait gives up
  const uint32_t* tag;        // counter of the substeps run so far
  uint32_t tag_add;           // of the groups launched before this one in the chunk
  float4* spill;
  uint4* slot;
  float4* grid;               // grid of the chunk's last substep, node = g_off + j * nx + i
  int32_t* err;
  unsigned long long* path;
  const float* t_dev;
  int64_t nodes;              // nodes of all instances (stride of the spill grids)
  int32_t M;
  int32_t stride;
  int32_t K;
  float dt;
};

// A band as its CTA holds it.
struct SpanSeg {
  JfInst I;
  JfParams P;
  int m, lo, hi;
  int off;               // first node of its window in the CTA's planes
  int segs;              // 32-cell segments of a row
  int cap;
  int n_bar;             // CTAs of the instance
  int n_meet2;           // drift meetings so far
  int drifted;           // this CTA scattered into the spill grid in the current pass
  unsigned marks[2];     // drift marks of even and odd substeps so far
  int ov_beg, n_ov;      // its part of the overflow list
  int oor_beg, n_oor;    // live particles outside every stencil range (the instance's last band takes them)
  int gen0, n_gen;       // generic tasks: first, count
  int cell0;             // first cell task
  __device__ __forceinline__ bool lower() const { return lo > 0; }
  __device__ __forceinline__ bool upper() const { return hi < I.ny; }
  // window rows that the band updates by itself: the others overlap a neighbour
  __device__ __forceinline__ int in_lo() const { return lower() ? kOverlap : kHaloLo; }
  __device__ __forceinline__ int in_hi() const { return hi - lo + (upper() ? 0 : kHaloLo); }
};

// The window of a band; rows outside it are reached through the published
// grid and the spill grid.
struct SpanWindow : JfWindow {
  const SpanArgs& a;
  SpanSeg& S;
  const int& s;  // the substep
  __device__ __forceinline__ float2 far_gather(int i, int j) const {
    const float4 g = __ldcg(a.grid + S.I.g_off + (int64_t)j * S.I.nx + i);
    return make_float2(g.x, g.y);
  }
  __device__ __forceinline__ void far_scatter(int i, int j, float3 c, float h, bool) const {
    atomicAdd(a.spill + (s % 3) * a.nodes + S.I.g_off + (int64_t)j * S.I.nx + i, make_float4(c.x, c.y, c.z, h));
    *(volatile int*)&S.drifted = 1;
  }
};

constexpr unsigned long long kMark = 1ull << 40;  // a drift mark in an arrival count
constexpr int kDriftUnknown = 8;  // beside the drift bits: a CTA gave up, any of the spill grids may be in use

__device__ __forceinline__ void arrive(unsigned long long* p, unsigned long long n) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(n) : "memory");
}

// One poll of a wait; false when the wait gave up or another CTA did.
__device__ __forceinline__ bool keep_polling(uint32_t& n, const SpanArgs& a) {
  if (++n >= a.spin_limit) {
    atomicExch(a.abort, 1);
    return false;
  }
  return (n & 63u) != 0u || *(volatile int32_t*)a.abort == 0;
}

// Waits until the arrivals at *p have reached `target` (they only grow within a
// launch); *seen is the count with its marks.
__device__ __forceinline__ bool wait_for(const unsigned long long* p, unsigned long long target, const SpanArgs& a,
                                         unsigned long long* seen) {
  for (uint32_t n = 0;;) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    *seen = v;
    if ((v & (kMark - 1)) >= target) return true;
    if (!keep_polling(n, a)) return false;
  }
}

// A 16-byte word written and read as one access: three values and a tag.
__device__ __forceinline__ void send(uint4* p, float a, float b, float c, uint32_t tag) {
  asm volatile(
      "{\n\t.reg .b128 w;\n\t.reg .b64 l, h;\n\tmov.b64 l, {%1, %2};\n\tmov.b64 h, {%3, %4};\n\t"
      "mov.b128 w, {l, h};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
      "f"(a), "f"(b), "f"(c), "r"(tag)
      : "memory");
}
__device__ __forceinline__ bool receive(const uint4* p, uint32_t tag, const SpanArgs& a, float3* v) {
  for (uint32_t n = 0;;) {
    uint32_t t;
    asm volatile(
        "{\n\t.reg .b128 w;\n\t.reg .b64 l, h;\n\tld.relaxed.gpu.global.b128 w, [%4];\n\tmov.b128 {l, h}, w;\n\t"
        "mov.b64 {%0, %1}, l;\n\tmov.b64 {%2, %3}, h;\n\t}"
        : "=f"(v->x), "=f"(v->y), "=f"(v->z), "=r"(t)
        : "l"(p)
        : "memory");
    if (t == tag) return true;
    if (!keep_polling(n, a)) return false;
  }
}

// kTmem: the node blocks live in TMEM (544 .. 768 threads); otherwise in
// registers (up to 512 threads, the default).  What bounds the pass is the
// latency and the issue rate of the particles' FP32 chains at 16 warps per SM,
// not memory: the state of the batch lives in L2.  Measured (us per substep,
// 80K-slot tanks on 128^2) against one cluster per instance with the particle
// code of the day: 32 instances 92.6 -> 82.6, 16: 91 -> 46, 8: 63 -> 27, 1: 35 ->
// 21; now 75.9, 41, 24.4 and 16.0.
template <bool kTmem, bool kAxisym, bool kGlow>
__global__ void __launch_bounds__(kTmem ? kTmemThreads : 512, 1) span_kernel(const __grid_constant__ SpanArgs a) {
  extern __shared__ float4 smem4[];
  __shared__ SpanSeg s_seg[kMaxSeg];
  __shared__ float s_pressure[2][kMaxSeg];  // double-buffered: substep s + 1's are set while s is finished
  __shared__ int s_next_task[2];
  __shared__ int s_drift[2][kMaxSeg];
  __shared__ int s_tot[4];                  // generic tasks, all tasks, window nodes, a wait gave up
  __shared__ unsigned s_path[4];
  __shared__ uint32_t s_tmem;

  const int cta = blockIdx.x;
  const int nseg = a.nseg[cta];
  if (nseg == 0) return;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, n_warps = nth >> 5;
  if (tid < nseg) {
    SpanSeg& S = s_seg[tid];
    const int4 q = a.seg[cta * kMaxSeg + tid];
    S.m = q.x;
    S.lo = q.y;
    S.hi = q.z;
    S.I = a.inst[q.x];
    S.P = a.params[q.x];
    S.segs = (S.I.nx + 31) >> 5;
    S.cap = a.cap[q.x];
    S.n_bar = a.nbar[q.x];
    S.n_meet2 = 0;
    S.drifted = 0;
    S.marks[0] = S.marks[1] = 0u;
    const int32_t* ovr = a.ovrow + a.rowoff[q.x] + q.x;
    S.ov_beg = ovr[q.y];
    S.n_ov = ovr[q.z] - S.ov_beg;
    S.oor_beg = 0;
    S.n_oor = 0;
    if (q.z == S.I.ny) {
      const int32_t* cs = a.cell_start + (int64_t)q.x * a.stride + S.I.nx * S.I.ny;
      S.oor_beg = cs[0];
      S.n_oor = cs[1] - cs[0];
    }
    S.n_gen = (S.n_ov + S.n_oor + 31) >> 5;
    s_drift[0][tid] = s_drift[1][tid] = 0;
  }
  if (tid < 4) s_path[tid] = 0u;
  if (tid == 0) s_tot[3] = *(volatile int32_t*)a.abort;
  __syncthreads();
  if (s_tot[3]) {
    if (tid < nseg) atomicOr(a.err + s_seg[tid].m, kJfErrAbort);
    return;
  }
  float t = *a.t_dev;
  const uint32_t tag0 = *a.tag + a.tag_add;
  if (tid == 0) {
    int gen = 0, cell = 0, off = 0;
    for (int q = 0; q < nseg; ++q) {
      SpanSeg& S = s_seg[q];
      S.gen0 = gen;
      S.cell0 = cell;
      S.off = off;
      gen += S.n_gen;
      cell += (S.hi - S.lo) * S.segs;
      off += (S.hi - S.lo + kHalo) * S.I.nx;
    }
    s_tot[0] = gen;
    s_tot[1] = gen + cell;
    s_tot[2] = off;
    s_next_task[0] = n_warps;
  }
  if (tid < nseg)
    s_pressure[0][tid] = s_seg[tid].P.actuation * jf_activation(s_seg[tid].P.freq, s_seg[tid].P.contraction, t);
  uint32_t tm_cols = 32, tm_base = 0, ta = 0;
  if constexpr (kTmem) {
    // one CTA per SM (its registers fill it), so the allocation never waits for another CTA's
    const int per_quad = (n_warps + 3) >> 2;
    while (tm_cols < (uint32_t)(48 * per_quad)) tm_cols <<= 1;
    if (warp == 0) tm_alloc(&s_tmem, tm_cols);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if constexpr (kTmem) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tm_base = s_tmem;
    ta = tm_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(48 * (warp >> 2));
  }
  const int n_gen = s_tot[0], n_tasks = s_tot[1], WN = s_tot[2];
  float2* const G = reinterpret_cast<float2*>(smem4);
  float* const Ax = reinterpret_cast<float*>(smem4) + 2 * WN;
  float* const Ay = Ax + WN;
  float* const Am = Ay + WN;
  float* const Ah = Am + WN;  // a sixth plane exists only in the axisymmetric variant
  for (int n = tid; n < (kAxisym ? 6 : 5) * WN; n += nth) reinterpret_cast<float*>(smem4)[n] = 0.0f;
  __syncthreads();

  const int nx = a.I.nx;
  const int64_t slot_n = (int64_t)kOverlap * nx * (kAxisym ? 2 : 1), slot_half = (int64_t)kOverlap * nx;

  for (int s = 0; s <= a.K; ++s) {
    const bool do_g2p = s > 0;
    const bool do_p2g = s < a.K;

    // a warp claims tasks from a shared counter: groups of 32 generic particles
    // first, lanes far apart in the list, then the 32-cell row segments
    for (int task = warp; task < n_tasks;) {
      const bool generic = task < n_gen;
      int q = 0;
      if (generic) {
        while (q + 1 < nseg && task >= s_seg[q + 1].gen0) ++q;
      } else {
        while (q + 1 < nseg && task - n_gen >= s_seg[q + 1].cell0) ++q;
      }
      SpanSeg& S = s_seg[q];
      // kernel parameters where the instances agree: operands of the arithmetic that take no registers
      JfInst I = a.I;
      I.axisym = kAxisym;
      I.ny = S.I.ny;
      I.y_hi = S.I.y_hi;
      const JfEnv<SpanArgs> E{I, a, S.P.payload_density, kGlow};
      const SpanWindow w{{G + S.off, Ax + S.off, Ay + S.off, Am + S.off, Ah + S.off, I.nx, S.lo - kHaloLo,
                          S.hi - S.lo + kHalo},
                         a, S, s};
      const float pressure = s_pressure[s & 1][q];
      bool nonfinite = false;
      // the lane's particles, as engine positions
      int beg = 0, end = 0, cy = 0, seg0 = 0;
      const int p0 = (int)S.I.p_off;
      if (generic) {
        const int e = task - S.gen0 + lane * S.n_gen;
        if (e < S.n_ov + S.n_oor) {
          const bool over = e < S.n_ov;
          beg = p0 + (over ? a.ovlist[p0 + S.ov_beg + e] : S.oor_beg + e - S.n_ov);
          end = beg + 1;
          atomicAdd(&s_path[over ? 3 : 1], 1u);
        }
      } else {
        const int c = task - n_gen - S.cell0;
        const int row = c / S.segs;
        cy = S.lo + row;
        seg0 = (c - row * S.segs) << 5;
        if (seg0 + lane < I.nx) {
          const int32_t* cs = a.cell_start + (int64_t)S.m * a.stride + cy * I.nx + seg0 + lane;
          beg = p0 + cs[0];
          end = p0 + cs[1];
          if (end - beg > S.cap) end = beg + S.cap;  // the rest of the cell is overflow
        }
      }
      run_task<kTmem>(E, w, !generic, beg, end, cy, seg0, ta, do_g2p, do_p2g, pressure, s_path, nonfinite);
      if (__any_sync(0xffffffffu, nonfinite) && lane == 0) atomicOr(a.err + S.m, 1);
      int nt = 0;
      if (lane == 0) nt = atomicAdd(&s_next_task[s & 1], 1);
      task = __shfl_sync(0xffffffffu, nt, 0);
    }
    __syncthreads();
    if (!do_p2g) break;
    const uint32_t tag = tag0 + (uint32_t)s;
    if (tid < nseg) {
      SpanSeg& S = s_seg[tid];
      if (S.n_bar > 1) {
        unsigned long long n = 1;
        // the spill is there for whoever sees the mark, and rows cleared in the
        // substep before are clear for the next to use that grid
        if (S.drifted || s_drift[s & 1][tid]) __threadfence();
        if (S.drifted) {
          S.drifted = 0;
          atomicOr(a.drift + S.m, 1 << (s % 3));
          n += kMark;
        }
        arrive(a.bar + (s & 1) * a.M + S.m, n);
      }
    }
    // partial sums of the rows around the cuts, for the other side
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const SpanSeg& S = s_seg[side ? nseg - 1 : 0];
      if (!(side ? S.upper() : S.lower())) continue;
      const int n0 = S.off + (side ? S.hi - S.lo : 0) * nx;
      uint4* const to = a.slot + ((cta * 2 + side) * 2 + (s & 1)) * slot_n;
      for (int n = tid; n < kOverlap * nx; n += nth) {
        send(to + n, Ax[n0 + n], Ay[n0 + n], Am[n0 + n], tag);
        if (kAxisym) send(to + slot_half + n, Ah[n0 + n], 0.0f, 0.0f, tag);
      }
    }
    // the next substep's pressures, by the last warp while the words travel
    t = t + a.dt;
    if (tid >= nth - 32 && lane < nseg)
      s_pressure[(s + 1) & 1][lane] =
          s_seg[lane].P.actuation * jf_activation(s_seg[lane].P.freq, s_seg[lane].P.contraction, t);

    // grid update of one node of band S from its sums; `publish`: into global
    // memory too, which only follows the meeting: until then another CTA of the
    // instance may be in this pass, whose drifted particles gather the rows that
    // the substep before published
    auto update_node = [&](const SpanSeg& S, int wr, int i, float mx, float my, float mm, float mh, bool publish) {
      const int j = S.lo - kHaloLo + wr;
      const float2 u = jf_grid_node(S.I, i, j, mx, my, mm, mh);
      G[S.off + wr * nx + i] = u;
      if (publish) a.grid[S.I.g_off + (int64_t)j * nx + i] = make_float4(u.x, u.y, mm, 0.0f);
    };
    // Rows that no neighbour shares, then the rows around the cuts from both
    // sides' sums.  The sums stay until the meeting is over: a spill may come in.
    for (int q = 0; q < nseg; ++q) {
      const SpanSeg& S = s_seg[q];
      const int n0 = S.in_lo() * nx, n1 = S.in_hi() * nx;
      for (int n = n0 + tid; n < n1; n += nth) {
        const int wr = n / nx, o = S.off + n;
        update_node(S, wr, n - wr * nx, Ax[o], Ay[o], Am[o], kAxisym ? Ah[o] : 0.0f, false);
      }
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const SpanSeg& S = s_seg[side ? nseg - 1 : 0];
      if (!(side ? S.upper() : S.lower())) continue;
      const int wr0 = side ? S.hi - S.lo : 0;
      const int other = side ? cta + 1 : cta - 1;
      const uint4* const from = a.slot + ((other * 2 + (side ^ 1)) * 2 + (s & 1)) * slot_n;
      for (int n = tid; n < kOverlap * nx; n += nth) {
        const int r = n / nx, i = n - r * nx;
        const int o = S.off + wr0 * nx + n;
        float3 b, h = make_float3(0.0f, 0.0f, 0.0f);
        if (!receive(from + n, tag, a, &b) || (kAxisym && !receive(from + slot_half + n, tag, a, &h))) {
          s_tot[3] = 1;
          break;
        }
        // both sides' sums, kept for a spill
        const float mx = Ax[o] + b.x, my = Ay[o] + b.y, mm = Am[o] + b.z;
        const float mh = kAxisym ? Ah[o] + h.x : 0.0f;
        Ax[o] = mx;
        Ay[o] = my;
        Am[o] = mm;
        if (kAxisym) Ah[o] = mh;
        update_node(S, wr0 + r, i, mx, my, mm, mh, false);
      }
    }
    if (tid < nseg) {
      SpanSeg& S = s_seg[tid];
      int drift = 0;
      if (S.n_bar > 1) {
        unsigned long long seen;
        if (!wait_for(a.bar + (s & 1) * a.M + S.m, (unsigned long long)(s / 2 + 1) * S.n_bar, a, &seen)) s_tot[3] = 1;
        const unsigned marks = (unsigned)(seen >> 40);
        drift = marks != S.marks[s & 1];
        S.marks[s & 1] = marks;
        if (drift || s_drift[0][tid] || s_drift[1][tid]) __threadfence();
      }
      s_drift[s & 1][tid] = drift;
    }
    if (tid == 0) s_next_task[(s + 1) & 1] = n_warps;
    __syncthreads();
    if (s_tot[3]) break;

    // the spill of this substep where there is one
    bool any_drift = false;
    for (int q = 0; q < nseg; ++q) {
      const SpanSeg& S = s_seg[q];
      const int rows = S.hi - S.lo;
      if (s_drift[s & 1][q]) {
        any_drift = true;
        const int n0 = max(kHaloLo - S.lo, 0) * nx, n1 = min(rows + kHalo, S.I.ny - S.lo + kHaloLo) * nx;
        for (int n = n0 + tid; n < n1; n += nth) {
          const int wr = n / nx, i = n - wr * nx, o = S.off + n;
          const float4 e = __ldcg(a.spill + (s % 3) * a.nodes + S.I.g_off + (int64_t)(S.lo - kHaloLo + wr) * nx + i);
          update_node(S, wr, i, Ax[o] + e.x, Ay[o] + e.y, Am[o] + e.z, kAxisym ? Ah[o] + e.w : 0.0f,
                      wr >= kHaloLo && wr < kHaloLo + rows);
        }
      } else if (s == a.K - 1) {  // the chunk's last grid, of the rows it owns
        for (int n = kHaloLo * nx + tid; n < (kHaloLo + rows) * nx; n += nth) {
          const float2 u = G[S.off + n];
          a.grid[S.I.g_off + (int64_t)(S.lo - kHaloLo) * nx + n] = make_float4(u.x, u.y, Am[S.off + n], 0.0f);
        }
      }
      // the spill of the substep before has been read by everyone: its rows are cleared by their owners
      if (s > 0 && s_drift[(s - 1) & 1][q]) {
        float4* const old = a.spill + ((s - 1) % 3) * a.nodes + S.I.g_off + (int64_t)S.lo * nx;
        for (int n = tid; n < rows * nx; n += nth) __stcg(old + n, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        if (tid == 0 && S.lo == 0) atomicAnd(a.drift + S.m, ~(1 << ((s - 1) % 3)));
      }
    }
    if (any_drift) {  // the published rows are there for everyone after a second meeting
      __syncthreads();
      if (tid < nseg && s_drift[s & 1][tid]) {
        SpanSeg& S = s_seg[tid];
        S.n_meet2 += 1;
        __threadfence();
        arrive(a.bar + 2 * a.M + S.m, 1);
        unsigned long long seen;
        if (!wait_for(a.bar + 2 * a.M + S.m, (unsigned long long)S.n_meet2 * S.n_bar, a, &seen)) s_tot[3] = 1;
        __threadfence();
      }
    }
    // clear sums for the next pass (the last one adds none, and the last grid is still being published)
    if (s < a.K - 1)
      for (int n = tid; n < (kAxisym ? 4 : 3) * WN; n += nth) Ax[n] = 0.0f;
    __syncthreads();
    if (any_drift && s_tot[3]) break;
  }
  // all that the CTA's bands belong to is left in the middle of the chunk
  if (s_tot[3] && tid < nseg) {
    atomicOr(a.err + s_seg[tid].m, kJfErrAbort);
    atomicOr(a.drift + s_seg[tid].m, kDriftUnknown);
  }
  // every warp is past its last access: the TMEM allocation is freed
  if constexpr (kTmem) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (kTmem) {
    if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tm_free(tm_base, tm_cols);
    }
  }
  if (tid < 4 && s_path[tid]) atomicAdd(a.path + tid, (unsigned long long)s_path[tid]);
}

// Per instance: the cell cap, the row costs, the overflow list's row starts,
// the exclusive scan of the bins (counts become bin starts), and the span
// kernel's flags and counters cleared.  One warp per 32-cell segment: its
// counts are one coalesced load and the candidates' overflows warp sums.
__global__ void __launch_bounds__(kScanThreads) span_scan_kernel(
    const JfInst* __restrict__ inst, int32_t* __restrict__ counts, int stride, const int32_t* __restrict__ solid,
    const int32_t* __restrict__ rowoff, int32_t* __restrict__ rowcost, int32_t* __restrict__ ovrow,
    int32_t* __restrict__ ovcur, int32_t* __restrict__ cap_out, int fixed_cap, int32_t* __restrict__ band, int CS,
    unsigned long long* __restrict__ bar, int32_t* __restrict__ drift, float4* __restrict__ spill, int64_t nodes,
    int M) {
  constexpr int kWarps = kScanThreads / 32;
  __shared__ int s_cost[32];
  __shared__ int s_row_cost[kJfMaxBandRows];
  __shared__ int s_row_over[kJfMaxBandRows];
  __shared__ int s_warp[kWarps];
  __shared__ int s_cap;
  const unsigned full = 0xffffffffu;
  const int m = blockIdx.x;
  const JfInst I = inst[m];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int32_t* c = counts + (int64_t)m * stride;
  const int segs = (I.nx + 31) >> 5;
  // what a chunk's last substeps may have left in the spill grids
  for (int r = 0; r < 3; ++r)
    if ((drift[m] >> r & 1) || (drift[m] & kDriftUnknown))
      for (int n = tid; n < I.nx * I.ny; n += kScanThreads)
        spill[(int64_t)r * nodes + I.g_off + n] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (tid < 32) s_cost[tid] = 0;
  for (int y = tid; y < I.ny; y += kScanThreads) {
    s_row_cost[y] = kRowCost + (kSolidCostHalves * solid[m * kJfMaxBandRows + y]) / 2;
    s_row_over[y] = 0;
  }
  __syncthreads();
  if (tid == 0) drift[m] = 0;
  if (tid < 3) bar[tid * M + m] = 0ull;

  // lane k sums the cost of candidate k (0 = no cap)
  int cost = 0;
  for (int sg = warp; sg < I.ny * segs; sg += kWarps) {
    const int row = sg / segs, x = ((sg - row * segs) << 5) + lane;
    const int n = x < I.nx ? c[row * I.nx + x] : 0;
    const int mx = (int)__reduce_max_sync(full, (unsigned)n);
    if (mx == 0) continue;
    int ov = 0;
    for (int k = 1; k < min(mx, kCapCandidates); ++k) {
      const int o = (int)__reduce_add_sync(full, (unsigned)max(0, n - k));
      if (lane == k) ov = o;
    }
    cost += 128 * (lane == 0 ? mx : min(mx, lane)) + kOverCost * ov;
  }
  if (lane < kCapCandidates) atomicAdd(&s_cost[lane], cost);
  __syncthreads();
  if (tid == 0) {
    int best = 0;
    for (int k = 1; k < kCapCandidates; ++k)
      if (s_cost[k] < s_cost[best]) best = k;
    if (fixed_cap > 0) best = fixed_cap < kCapCandidates ? fixed_cap : 0;
    s_cap = best == 0 ? kNoCap : best;
    cap_out[m] = s_cap;
  }
  __syncthreads();
  const int cap = s_cap;
  for (int sg = warp; sg < I.ny * segs; sg += kWarps) {
    const int row = sg / segs, x = ((sg - row * segs) << 5) + lane;
    const int n = x < I.nx ? c[row * I.nx + x] : 0;
    const int mx = (int)__reduce_max_sync(full, (unsigned)n);
    const int ov = (int)__reduce_add_sync(full, (unsigned)max(0, n - cap));
    if (lane == 0 && mx) {
      atomicAdd(&s_row_cost[row], kSegCost + 128 * min(mx, cap) + kOverCost * ov);
      if (ov) atomicAdd(&s_row_over[row], ov);
    }
  }
  __syncthreads();

  // block scan of one value per thread
  auto block_exclusive = [&](int v) {
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(full, incl, off);
      if (lane >= off) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = s_warp[lane];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(full, w, off);
        if (lane >= off) w += y;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    const int r = incl - v + (warp > 0 ? s_warp[warp - 1] : 0);
    __syncthreads();
    return r;
  };
  static_assert(kJfMaxBandRows <= kScanThreads, "one row per thread");
  {
    const int over = tid < I.ny ? s_row_over[tid] : 0;
    const int start = block_exclusive(over);
    if (tid < I.ny) {
      const int r = rowoff[m] + tid;
      rowcost[r] = s_row_cost[tid];
      ovrow[r + m] = start;
      ovcur[r] = start;
      if (tid == I.ny - 1) ovrow[r + m + 1] = start + over;
    }
  }
  // bins: each warp takes a run of 32-bin tiles
  const int nbins = I.nx * I.ny + 2;
  const int tiles = (nbins + 31) >> 5, per = (tiles + kWarps - 1) / kWarps;
  const int t0 = min(warp * per, tiles), t1 = min(t0 + per, tiles);
  int sum = 0;
  for (int q = t0; q < t1; ++q) {
    const int b = (q << 5) + lane;
    sum += b < nbins ? c[b] : 0;
  }
  sum = (int)__reduce_add_sync(full, (unsigned)sum);
  const int before = block_exclusive(lane == 0 ? sum : 0);
  int run = __shfl_sync(full, before, 0);
  for (int q = t0; q < t1; ++q) {
    const int b = (q << 5) + lane;
    const int n = b < nbins ? c[b] : 0;
    int incl = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(full, incl, off);
      if (lane >= off) incl += y;
    }
    if (b < nbins) c[b] = run + incl - n;
    if (b == nbins - 1) band[m * (CS + 1) + CS] = (int32_t)I.p_off + run + incl - n;  // first dead slot
    run += __shfl_sync(full, incl, 31);
  }
}

// One block per group: the costs' prefix over the group's rows, cut into spans
// of equal cost, each cut moved so that every band has at least kMinRows rows
// and every CTA's windows fit (where that cannot be had, the cuts by window
// size alone), and the CTAs' band table.
__global__ void __launch_bounds__(kScanThreads) span_cut_kernel(
    const SpanGroup* __restrict__ groups, const JfInst* __restrict__ inst, const int32_t* __restrict__ rowoff,
    const int32_t* __restrict__ rowcost, unsigned long long* __restrict__ rowpre, int cap_nodes, int n_cta_max, int n_warps,
    const int32_t* __restrict__ fallback, int4* __restrict__ seg, int32_t* __restrict__ nseg,
    int32_t* __restrict__ nbar) {
  __shared__ unsigned long long s_sum[kScanThreads / 32];
  __shared__ int s_cut[kScanThreads + 1];
  __shared__ int s_off[kScanThreads + 1];
  __shared__ int s_used;
  const SpanGroup g = groups[blockIdx.x];
  // row starts of the group's instances, near at hand for the serial walk below
  const int n_inst = g.m1 - g.m0;
  const bool near = n_inst <= kScanThreads;
  if (near)
    for (int q = threadIdx.x; q <= n_inst; q += kScanThreads) s_off[q] = rowoff[g.m0 + q] - g.row0;
  auto row_start = [&](int m) { return near ? s_off[m - g.m0] : rowoff[m] - g.row0; };
  const int nx = inst[g.m0].nx;  // the same for every instance
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned full = 0xffffffffu;
  const int32_t* row_cost = rowcost + g.row0;
  // Where equal shares give every warp at most one segment and a row more would
  // give some a second, the rows count and not their cost: one tank of 80,000
  // slots, 4 rows on 16 warps, 18.7 -> 16.1 us per substep, four 19.3 -> 17.4
  // (with a row to spare, 32^2, the cost still does better: 10.2 against 13.0).
  const int share = (g.rows + g.n_cta - 1) / g.n_cta, segs = (nx + 31) >> 5;
  const bool thin = share * segs <= n_warps && (share + 1) * segs > n_warps;
  auto cost = [&](int r) { return thin ? 2u : (unsigned)row_cost[r]; };
  unsigned long long* pre = rowpre + g.row0;
  const int per = (g.rows + kScanThreads - 1) / kScanThreads;
  const int r0 = min(tid * per, g.rows), r1 = min(r0 + per, g.rows);
  unsigned long long sum = 0;
  for (int r = r0; r < r1; ++r) sum += cost(r);
  unsigned long long incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long y = __shfl_up_sync(full, incl, off);
    if (lane >= off) incl += y;
  }
  if (lane == 31) s_sum[warp] = incl;
  for (int m = g.m0 + tid; m < g.m1; m += kScanThreads) nbar[m] = 0;
  __syncthreads();
  unsigned long long run = incl - sum, total = 0;
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) run += s_sum[w];
    total += s_sum[w];
  }
  for (int r = r0; r < r1; ++r) {
    run += cost(r);
    pre[r] = run;
  }
  __syncthreads();
  // span c starts where the cost before it reaches c / n_cta of the total
  if (tid > 0 && tid < g.n_cta) {
    const unsigned long long target = total * (unsigned)tid / (unsigned)g.n_cta;
    int lo = 0, hi = g.rows;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (pre[mid] - cost(mid) / 2 < target) lo = mid + 1;
      else hi = mid;
    }
    s_cut[tid] = lo;
  }
  __syncthreads();
  if (tid == 0) {
    int prev = 0, used = 0, m = g.m0;
    bool ok = true;
    for (int q = 1; q <= g.n_cta && prev < g.rows; ++q) {
      int y = q < g.n_cta ? s_cut[q] : g.rows;
      // instance of the span's first row, its rows [b, e) in the group
      int b = row_start(m), e = row_start(m + 1);
      while (prev >= e) {
        ++m;
        b = e;
        e = row_start(m + 1);
      }
      if (y < prev + kMinRows) y = prev + kMinRows;
      // walk its bands while they fit
      int at = prev, mm = m, bb = b, ee = e, room = cap_nodes, left = kMaxSeg;
      for (;;) {
        int stop = min(y, ee);
        // a cut leaves at least kMinRows rows on either side within an instance
        if (stop < ee && ee - stop < kMinRows) stop = ee;
        if (stop < ee && stop - bb < kMinRows) stop = at > prev ? at : bb + kMinRows;
        if (left == 0) stop = at;
        if (stop > at && (stop - at + kHalo) * nx > room) {
          stop = at + room / nx - kHalo;
          if (ee - stop < kMinRows) stop = ee - kMinRows;
          if (stop - at < kMinRows) stop = at;
        }
        if (stop > at) {
          room -= (stop - at + kHalo) * nx;
          --left;
        }
        at = stop;
        if (at < ee || at >= y || at >= g.rows) break;
        ++mm;
        bb = ee;
        ee = row_start(mm + 1);
      }
      if (at <= prev) {
        ok = false;
        break;
      }
      s_cut[used++] = prev;  // span `used`: s_cut[used] is read above only for larger q
      prev = at;
    }
    if (prev < g.rows) ok = false;
    s_used = ok ? used : -1;
    if (ok) s_cut[used] = g.rows;
  }
  __syncthreads();
  const int used = s_used;
  const int32_t* fb = fallback + blockIdx.x * (n_cta_max + 1);
  for (int q = tid; q < n_cta_max; q += kScanThreads) {
    const int lo = used >= 0 ? (q < used ? s_cut[q] : g.rows) : fb[q];
    const int hi = used >= 0 ? (q < used ? s_cut[q + 1] : g.rows) : fb[q + 1];
    int n = 0;
    if (lo < hi) {
      int m = g.m0, top = g.m1;  // instance of row lo
      while (top - m > 1) {
        const int mid = (m + top) >> 1;
        if (row_start(mid) <= lo) m = mid;
        else top = mid;
      }
      for (int at = lo; at < hi; ++m) {
        const int b = row_start(m), e = row_start(m + 1);
        const int stop = min(hi, e);
        seg[((int64_t)blockIdx.x * n_cta_max + q) * kMaxSeg + n] = make_int4(m, at - b, stop - b, 0);
        atomicAdd(nbar + m, 1);
        ++n;
        at = stop;
      }
    }
    nseg[blockIdx.x * n_cta_max + q] = n;
  }
}

// Moves every particle to bin start + rank; particles of a cell beyond the
// cap are also listed in their row's part of the overflow list.
__global__ void __launch_bounds__(kMoveThreads) span_move_kernel(
    const JfInst* __restrict__ inst, const int32_t* __restrict__ keys, const int32_t* __restrict__ rank,
    const int32_t* __restrict__ starts, int stride, const int32_t* __restrict__ cap,
    const int32_t* __restrict__ rowoff, int32_t* __restrict__ ovcur, int32_t* __restrict__ ovlist, JfParticles src,
    JfParticles dst) {
  const int m = blockIdx.y;
  const JfInst I = inst[m];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= I.n_slots) return;
  const int64_t g = I.p_off + k;
  const int key = keys[g];
  const int rk = rank[g];
  const int32_t rel = starts[(int64_t)m * stride + key] + rk;
  const int64_t d = I.p_off + rel;
  if (key < I.nx * I.ny && rk >= cap[m])
    ovlist[I.p_off + atomicAdd(ovcur + rowoff[m] + key / I.nx, 1)] = rel;
  dst.xv[d] = src.xv[g];
  dst.C[d] = src.C[g];
  dst.F[d] = src.F[g];
  dst.mat[d] = src.mat[g];
  dst.fiber[d] = src.fiber[g];
  dst.Jp[d] = src.Jp[g];
  dst.glow[d] = src.glow[g];
  dst.slot[d] = src.slot[g];
  dst.rref[d] = src.rref[g];
}

using SpanKernel = void (*)(const SpanArgs);

// the instantiation for the launch's CTA size and the engine's flags
SpanKernel span_kernel_for(const jf_engine* e, int threads) {
  const bool axisym = e->flags & JF_FLAG_AXISYM, glow = e->flags & JF_FLAG_GLOW;
  if (threads > 512)
    return axisym ? (glow ? span_kernel<true, true, true> : span_kernel<true, true, false>)
                  : (glow ? span_kernel<true, false, true> : span_kernel<true, false, false>);
  return axisym ? (glow ? span_kernel<false, true, true> : span_kernel<false, true, false>)
                : (glow ? span_kernel<false, false, true> : span_kernel<false, false, false>);
}

// SMs that kernels on the engine's stream may use: fewer than the device's
// where the stream belongs to a green context.
int sms_of_stream(const jf_engine* e) {
  int n_sm = 0;
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, e->device);
  CUresult (*of_stream)(CUstream, CUgreenCtx*) = nullptr;
  CUresult (*resource)(CUgreenCtx, CUdevResource*, CUdevResourceType) = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPointByVersion("cuStreamGetGreenCtx", (void**)&of_stream, 12040, cudaEnableDefault, &found) !=
          cudaSuccess || !of_stream ||
      cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", (void**)&resource, 12040, cudaEnableDefault,
                                       &found) != cudaSuccess || !resource) {
    cudaGetLastError();  // a driver older than green contexts
    return n_sm;
  }
  CUgreenCtx green = nullptr;
  CUdevResource r;
  if (of_stream((CUstream)e->stream, &green) != CUDA_SUCCESS || !green ||
      resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
    return n_sm;
  return std::min(n_sm, (int)r.sm.smCount);
}

// Spans of the group by window size alone; false when n_cta spans do not do.
bool fill_cuts(const jf_engine* e, const SpanGroup& g, const std::vector<int32_t>& rowoff, int cap_nodes,
               std::vector<int32_t>& cuts) {
  cuts.assign(1, 0);
  int room = cap_nodes, left = kMaxSeg;
  for (int m = g.m0; m < g.m1; ++m) {
    const int nx = e->inst[m].nx, ny = e->inst[m].ny, b = rowoff[m] - g.row0;
    int y = 0;
    while (y < ny) {
      int rows = left > 0 ? std::min(room / nx - kHalo, ny - y) : 0;
      if (ny - y - rows > 0 && ny - y - rows < kMinRows) rows = ny - y - kMinRows;
      if (rows < kMinRows) {
        if (cuts.back() == b + y) return false;  // an empty span: a band does not fit
        cuts.push_back(b + y);
        room = cap_nodes;
        left = kMaxSeg;
        continue;
      }
      room -= (rows + kHalo) * nx;
      --left;
      y += rows;
    }
  }
  if ((int)cuts.size() > g.n_cta) return false;
  cuts.resize(g.n_cta + 1, g.rows);
  return true;
}

}  // namespace

void jf_span_free(jf_engine* e) {
  JfSpan* s = e->span;
  if (!s) return;
  cudaFree(s->pool);
  delete s;
  e->span = nullptr;
}

// Sets the span path up (e->span), or leaves it off where the batch does not
// suit it: grids taller than the row tables, instances of different n_grid
// (the kernel's constants are launch parameters), rows too wide for a band of
// 4 rows and its halo, or a device without cooperative launches.
cudaError_t jf_span_setup(jf_engine* e, int threads) {
  int n_sm = sms_of_stream(e), coop = 0;
  e->span_threads = threads;
  e->span_sms = n_sm;
  if (threads == 0) threads = kSpanThreads;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, e->device);
  if (!coop || n_sm < 1) return cudaSuccess;
  n_sm = std::min(n_sm, kScanThreads);
  std::vector<int32_t> rowoff(1, 0);
  int nx_max = 0;
  for (const JfInst& I : e->inst) {
    if (I.ny > kJfMaxBandRows || I.nx != e->inst[0].nx) return cudaSuccess;
    if (rowoff.back() > (1 << 28)) return cudaSuccess;
    rowoff.push_back(rowoff.back() + I.ny);
    nx_max = std::max(nx_max, I.nx);
  }
  const size_t node_bytes = sizeof(float) * ((e->flags & JF_FLAG_AXISYM) ? 6 : 5);
  const int64_t hard = (int64_t)((kMaxSmem - kStaticSmem) / node_bytes);
  const int64_t soft = std::min<int64_t>(hard, (int64_t)(kSoftSmem / node_bytes));

  // as few groups of consecutive instances as keep a CTA's share of the rows
  // within the soft size
  std::vector<SpanGroup> groups;
  int64_t need = 0;
  for (int n_groups = 1; n_groups <= e->M; n_groups = n_groups < 8 ? n_groups + 1 : n_groups * 2) {
    groups.clear();
    need = 0;
    int m = 0;
    for (int k = 0; k < n_groups && m < e->M; ++k) {
      SpanGroup g = {};
      g.m0 = m;
      const int64_t upto = rowoff[e->M] * (int64_t)(k + 1) / n_groups;
      do ++m;
      while (m < e->M && (k == n_groups - 1 || rowoff[m + 1] <= upto));
      g.m1 = m;
      g.row0 = rowoff[g.m0];
      g.rows = rowoff[m] - g.row0;
      g.n_cta = std::max(1, std::min(n_sm, g.rows / kMinRows));
      int64_t nodes = 0;
      for (int q = g.m0; q < g.m1; ++q) nodes += (int64_t)e->inst[q].nx * e->inst[q].ny;
      // a CTA's share and its halo, twice where its span holds the end of one instance and the start of the next
      const int64_t share = nodes / g.n_cta + (g.m1 - g.m0 > 1 ? 2 : 1) * kHalo * nx_max;
      need = std::max(need, share);
      groups.push_back(g);
    }
    if (need <= soft) break;
  }
  int64_t cap = std::max<int64_t>(need + need * 3 / 5, (int64_t)(4 * kMinRows + kHalo) * nx_max);
  cap = std::min(cap, hard);
  std::vector<int32_t> table, cuts;
  int n_cta = 0;
  for (const SpanGroup& g : groups) n_cta = std::max(n_cta, g.n_cta);
  for (const SpanGroup& g : groups) {
    if (!fill_cuts(e, g, rowoff, (int)cap, cuts)) {
      cap = hard;
      if (!fill_cuts(e, g, rowoff, (int)cap, cuts)) return cudaSuccess;
    }
    cuts.resize(n_cta + 1, g.rows);
    table.insert(table.end(), cuts.begin(), cuts.end());
  }
  const size_t smem = node_bytes * (size_t)cap;
  const void* k = (const void*)span_kernel_for(e, threads);
  // the attribute belongs to the kernel, not to the engine: the most any engine may take
  cudaError_t err =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMaxSmem - kStaticSmem));
  int blocks = 0;
  if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, threads, smem);
  if (err != cudaSuccess) return err;
  if (blocks < 1) return cudaSuccess;

  JfSpan* s = new JfSpan();
  e->span = s;
  s->threads = threads;
  s->groups = groups;
  s->n_cta = n_cta;
  s->total_rows = rowoff[e->M];
  s->cap_nodes = (int32_t)cap;
  s->smem = smem;
  const size_t slots = (size_t)n_cta * 4 * kOverlap * nx_max * ((e->flags & JF_FLAG_AXISYM) ? 2 : 1);
  const size_t ng = groups.size(), rows = (size_t)s->total_rows, M = (size_t)e->M;
  // one allocation for all of it: engines are made anew by callers that change shapes
  size_t bytes = 0;
  std::vector<std::pair<void**, size_t>> parts;
  auto part = [&](auto** p, size_t n) {
    parts.emplace_back((void**)p, bytes);
    bytes += (sizeof(**p) * std::max<size_t>(n, 1) + 255) / 256 * 256;
  };
  part(&s->d_spill, 3 * (size_t)e->total_nodes);  // the first five are cleared
  part(&s->d_slot, slots);
  part(&s->d_drift, M);
  part(&s->d_abort, 1);
  part(&s->d_nseg, ng * n_cta);
  const size_t zero_end = bytes;
  part(&s->d_groups, ng);
  part(&s->d_rowoff, M + 1);
  part(&s->d_fallback, table.size());
  part(&s->d_tag, 1);
  part(&s->d_rowcost, rows);
  part(&s->d_rowpre, rows);
  part(&s->d_ovrow, rows + M);
  part(&s->d_ovcur, rows);
  part(&s->d_seg, ng * n_cta * kMaxSeg);
  part(&s->d_nbar, M);
  part(&s->d_bar, 3 * M);
  if ((err = cudaMalloc(&s->pool, bytes))) {
    jf_span_free(e);
    return err;
  }
  for (auto& p : parts) *p.first = (char*)s->pool + p.second;
  const uint32_t first_tag = 1;  // the slots start at 0
  if ((err = cudaMemsetAsync(s->pool, 0, zero_end, e->stream)) ||
      (err = cudaMemcpyAsync(s->d_groups, groups.data(), sizeof(SpanGroup) * ng, cudaMemcpyHostToDevice, e->stream)) ||
      (err = cudaMemcpyAsync(s->d_rowoff, rowoff.data(), sizeof(int32_t) * (M + 1), cudaMemcpyHostToDevice,
                             e->stream)) ||
      (err = cudaMemcpyAsync(s->d_fallback, table.data(), sizeof(int32_t) * table.size(), cudaMemcpyHostToDevice,
                             e->stream)) ||
      (err = cudaMemcpyAsync(s->d_tag, &first_tag, sizeof(first_tag), cudaMemcpyHostToDevice, e->stream)) ||
      (err = cudaStreamSynchronize(e->stream)))
    jf_span_free(e);  // no half-made layout is left to a later launch
  return err;
}

// One CTA per SM is what the waits between CTAs stand on, so that a stream with
// other SMs takes spans of its own (or clusters, where these do not fit it).
cudaError_t jf_span_follow_stream(jf_engine* e) {
  if (sms_of_stream(e) == e->span_sms) return cudaSuccess;
  uint32_t limit = kSpinLimit;
  int32_t abort = 0;
  cudaError_t err = cudaSuccess;
  if (e->span) {
    limit = e->span->spin_limit;
    if ((err = cudaMemcpy(&abort, e->span->d_abort, sizeof(abort), cudaMemcpyDeviceToHost))) return err;
  }
  if (e->graph_exec) cudaGraphExecDestroy(e->graph_exec);  // its launches are those of the old layout
  e->graph_exec = nullptr;
  jf_span_free(e);
  e->sorted = false;
  if ((err = jf_span_setup(e, e->span_threads)) || !e->span) return err;
  e->span->spin_limit = limit;
  return abort ? cudaMemcpy(e->span->d_abort, &abort, sizeof(abort), cudaMemcpyHostToDevice) : cudaSuccess;
}

// The part of a re-sort after the cell keys: bins, spans, and the particles
// moved into the other buffer set.
cudaError_t jf_span_sort(jf_engine* e) {
  JfSpan* s = e->span;
  const int stride = e->max_cells + 2;
  span_scan_kernel<<<e->M, kScanThreads, 0, e->stream>>>(
      e->d_inst, e->d_counts, stride, e->d_solid, s->d_rowoff, s->d_rowcost, s->d_ovrow, s->d_ovcur, e->d_cap,
      e->cell_cap, e->d_band, e->cluster, s->d_bar, s->d_drift, s->d_spill, e->total_nodes, e->M);
  span_cut_kernel<<<(int)s->groups.size(), kScanThreads, 0, e->stream>>>(
      s->d_groups, e->d_inst, s->d_rowoff, s->d_rowcost, s->d_rowpre, s->cap_nodes, s->n_cta, s->threads / 32,
      s->d_fallback, s->d_seg, s->d_nseg, s->d_nbar);
  if (e->max_slots > 0) {
    const dim3 grid((e->max_slots + kMoveThreads - 1) / kMoveThreads, e->M);
    span_move_kernel<<<grid, kMoveThreads, 0, e->stream>>>(e->d_inst, e->d_keys, e->d_rank, e->d_counts, stride,
                                                          e->d_cap, s->d_rowoff, s->d_ovcur, e->d_ovlist, e->p, e->q);
  }
  return cudaGetLastError();
}

// K substeps of every instance: one cooperative launch per group.
cudaError_t jf_span_launch(jf_engine* e, int K) {
  JfSpan* s = e->span;
  SpanArgs a;
  a.I = e->inst[0];
  a.inst = e->d_inst;
  a.params = e->d_params;
  a.mats = jf_materials();
  a.xv = e->p.xv;
  a.C = e->p.C;
  a.F = e->p.F;
  a.mat = e->p.mat;
  a.Jp = e->p.Jp;
  a.fiber = e->p.fiber;
  a.glow = e->p.glow;
  a.rref = e->p.rref;
  a.cell_start = e->d_counts;
  a.cap = e->d_cap;
  a.ovlist = e->d_ovlist;
  a.ovrow = s->d_ovrow;
  a.rowoff = s->d_rowoff;
  a.nbar = s->d_nbar;
  a.bar = s->d_bar;
  a.drift = s->d_drift;
  a.abort = s->d_abort;
  a.spin_limit = s->spin_limit;
  a.tag = s->d_tag;
  a.spill = s->d_spill;
  a.slot = s->d_slot;
  a.grid = e->d_grid;
  a.err = e->d_err;
  a.path = e->d_path;
  a.t_dev = e->d_time;
  a.nodes = e->total_nodes;
  a.M = e->M;
  a.stride = e->max_cells + 2;
  a.K = K;
  a.dt = (float)e->dt;
  for (size_t g = 0; g < s->groups.size(); ++g) {
    a.seg = s->d_seg + g * s->n_cta * kMaxSeg;
    a.nseg = s->d_nseg + g * s->n_cta;
    a.tag_add = (uint32_t)(g * K);  // the groups share the slots
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s->groups[g].n_cta, 1, 1);
    cfg.blockDim = dim3(s->threads, 1, 1);
    cfg.dynamicSmemBytes = s->smem;
    cfg.stream = e->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, span_kernel_for(e, s->threads), a);
    if (err != cudaSuccess) return err;
    e->launches += 1;
  }
  return cudaSuccess;
}

// Device counter of the substeps run so far, which tags their words, and what a
// chunk of K substeps adds to it after its last launch.
uint32_t* jf_span_tag(const jf_engine* e) { return e->span->d_tag; }
uint32_t jf_span_tag_step(const jf_engine* e, int K) { return (uint32_t)(e->span->groups.size() * K); }

// The poll count after which a wait gives up, 0 for the default.
void jf_span_set_wait_limit(jf_engine* e, uint32_t polls) { e->span->spin_limit = polls ? polls : kSpinLimit; }

// Lets chunks run again after a wait has given up.
cudaError_t jf_span_clear_abort(jf_engine* e) {
  return cudaMemsetAsync(e->span->d_abort, 0, sizeof(int32_t), e->stream);
}

// The layout: launches, CTAs, threads and window nodes, and the bands of the latest re-sort.
cudaError_t jf_span_info(jf_engine* e, int32_t* info, std::vector<int32_t>& bands) {
  const JfSpan* s = e->span;
  info[0] = (int32_t)s->groups.size();
  info[1] = s->n_cta;
  info[2] = s->threads;
  info[3] = s->cap_nodes;
  const size_t n = s->groups.size() * s->n_cta;
  std::vector<int32_t> nseg(n);
  std::vector<int4> seg(n * kMaxSeg);
  cudaError_t err;
  if ((err = cudaMemcpyAsync(nseg.data(), s->d_nseg, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, e->stream)) ||
      (err = cudaMemcpyAsync(seg.data(), s->d_seg, sizeof(int4) * n * kMaxSeg, cudaMemcpyDeviceToHost, e->stream)) ||
      (err = cudaStreamSynchronize(e->stream)))
    return err;
  for (size_t c = 0; c < n; ++c)
    for (int k = 0; k < nseg[c]; ++k) {
      const int4 q = seg[c * kMaxSeg + k];
      bands.insert(bands.end(), {(int32_t)(c / s->n_cta), (int32_t)(c % s->n_cta), q.x, q.y, q.z});
    }
  return cudaSuccess;
}
