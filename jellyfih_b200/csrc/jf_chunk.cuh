// What the two batched chunk kernels share: the shared-memory window's layout,
// the cell lanes' node blocks (in registers or in tensor memory) and the tasks
// of one pass over an instance's particles, written for either kernel's window
// type.  A window W has the fields G, Ax, Ay, Am, Ah, nx, win0 and VR of
// JfWindow, and two members for grid rows outside it: far_gather(i, j), the
// updated velocity of a node, and far_scatter(i, j, c, h), which adds a
// contribution to a node.
#pragma once
#include "jf_engine.h"

namespace {

constexpr int kHaloLo = 1;  // window rows below the band (drift of one row)
constexpr int kHaloHi = 3;  // rows above: the stencil's +2 plus one row of drift
constexpr int kHalo = kHaloLo + kHaloHi;
// CTA size of the TMEM variant of the chunk kernels (24 warps per SM)
constexpr int kTmemThreads = 768;

// Shared-memory window of a band: grid rows [win0, win0 + VR) of its instance:
// the updated velocity G as float2 pairs (one 64-bit load per node in G2P),
// then planar accumulators (momentum Ax, Ay, mass Am and, axisymmetric only,
// the hoop sum Ah).
struct JfWindow {
  float2* G;
  float *Ax, *Ay, *Am, *Ah;
  int nx, win0;
  int VR;  // rows in use: the band's rows plus the halo
};

// Two rows of a lane's 4x4 node block as packed pairs: entries 0 .. 7 are the
// nodes' (x, y) momentum, node (row, column i) at 4 row + i, entries 8 .. 11
// their masses, columns (2 h, 2 h + 1) at 8 + 2 row + h.
constexpr int kHalfBlock = 12;

// Tensor memory (TMEM) variant of the cell lanes' node block.  With more than
// 16 warps per SM the 48-float block no longer fits in registers beside one
// particle's state, so between the particles of its cell a lane keeps the
// block in TMEM: warp w of the CTA uses TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31
// (its threads' own lanes, the quadrant a warp may access) and the 48 columns
// starting at 48 (w / 4) of the CTA's allocation.  Each access starts at a
// multiple of its width in columns.  A load first waits for the thread's
// earlier stores (tcgen05.wait::st; the second half needs none of its own,
// see the cell loop) and waits for its data inside the same asm statement, so
// its outputs cannot be read before they arrive.
#define JF_TM_OUT16(b)                                                                                   \
  "=r"(r[b + 0]), "=r"(r[b + 1]), "=r"(r[b + 2]), "=r"(r[b + 3]), "=r"(r[b + 4]), "=r"(r[b + 5]),        \
      "=r"(r[b + 6]), "=r"(r[b + 7]), "=r"(r[b + 8]), "=r"(r[b + 9]), "=r"(r[b + 10]), "=r"(r[b + 11]), \
      "=r"(r[b + 12]), "=r"(r[b + 13]), "=r"(r[b + 14]), "=r"(r[b + 15])
#define JF_TM_IN16(b)                                                                                             \
  "r"(r[b + 0]), "r"(r[b + 1]), "r"(r[b + 2]), "r"(r[b + 3]), "r"(r[b + 4]), "r"(r[b + 5]), "r"(r[b + 6]),      \
      "r"(r[b + 7]), "r"(r[b + 8]), "r"(r[b + 9]), "r"(r[b + 10]), "r"(r[b + 11]), "r"(r[b + 12]), "r"(r[b + 13]), \
      "r"(r[b + 14]), "r"(r[b + 15])
#define JF_TM_OUT8(b) \
  "=r"(r[b + 0]), "=r"(r[b + 1]), "=r"(r[b + 2]), "=r"(r[b + 3]), "=r"(r[b + 4]), "=r"(r[b + 5]), "=r"(r[b + 6]), "=r"(r[b + 7])
#define JF_TM_IN8(b) \
  "r"(r[b + 0]), "r"(r[b + 1]), "r"(r[b + 2]), "r"(r[b + 3]), "r"(r[b + 4]), "r"(r[b + 5]), "r"(r[b + 6]), "r"(r[b + 7])

// `cols` TMEM columns (a power of two >= 32) for the CTA, the address of the
// first into *out; by one whole warp, which also frees them.
__device__ __forceinline__ void tm_alloc(uint32_t* out, uint32_t cols) {
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(out)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_free(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

// columns 0 .. 47 of the warp's block set to zero (a task's start)
__device__ __forceinline__ void tm_zero48(uint32_t ta) {
  const uint32_t z = 0u;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3};\n\t"
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%1], {%3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3};\n\t"
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%2], {%3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3, %3};"
      :
      : "r"(ta), "r"(ta + 16u), "r"(ta + 32u), "r"(z)
      : "memory");
}
// columns 0 .. 23 (block rows 0 and 1): 16 at 0, 8 at 16
__device__ __forceinline__ void tm_load_rows01(uint32_t ta, f2* acc) {
  uint32_t r[24];
  asm volatile(
      "tcgen05.wait::st.sync.aligned;\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%25];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : JF_TM_OUT16(0), JF_TM_OUT8(16)
      : "r"(ta), "r"(ta + 16u)
      : "memory");
#pragma unroll
  for (int q = 0; q < kHalfBlock; ++q) acc[q] = f2_pack(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
}
__device__ __forceinline__ void tm_store_rows01(uint32_t ta, const f2* acc) {
  uint32_t r[24];
#pragma unroll
  for (int q = 0; q < kHalfBlock; ++q) {
    const float2 v = f2_get(acc[q]);
    r[2 * q] = __float_as_uint(v.x);
    r[2 * q + 1] = __float_as_uint(v.y);
  }
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17};\n\t"
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%1], {%18, %19, %20, %21, %22, %23, %24, %25};"
      :
      : "r"(ta), "r"(ta + 16u), JF_TM_IN16(0), JF_TM_IN8(16)
      : "memory");
}
// columns 24 .. 47 (block rows 2 and 3): 8 at 24, 16 at 32.  No wait for
// earlier stores: the last store to these columns came before the wait of the
// rows-0/1 load that precedes every use.
__device__ __forceinline__ void tm_load_rows23(uint32_t ta, f2* acc) {
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23}, [%25];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : JF_TM_OUT8(0), JF_TM_OUT16(8)
      : "r"(ta + 24u), "r"(ta + 32u)
      : "memory");
#pragma unroll
  for (int q = 0; q < kHalfBlock; ++q) acc[q] = f2_pack(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
}
__device__ __forceinline__ void tm_store_rows23(uint32_t ta, const f2* acc) {
  uint32_t r[24];
#pragma unroll
  for (int q = 0; q < kHalfBlock; ++q) {
    const float2 v = f2_get(acc[q]);
    r[2 * q] = __float_as_uint(v.x);
    r[2 * q + 1] = __float_as_uint(v.y);
  }
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%2, %3, %4, %5, %6, %7, %8, %9};\n\t"
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%1], {%10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25};"
      :
      : "r"(ta + 24u), "r"(ta + 32u), JF_TM_IN8(0), JF_TM_IN16(8)
      : "memory");
}
#undef JF_TM_OUT16
#undef JF_TM_IN16
#undef JF_TM_OUT8
#undef JF_TM_IN8

// Adds a particle's 3x3 stencil into rows J0 and J0 + 1 of the lane's 4x4 node
// block, shifted by (di, dj) = stencil base - (cell - 1), both 0 or 1.
// Branch-free: the weights are shifted into 4-wide vectors with zeros outside
// the stencil, so lanes with different shifts run the same instructions.
// Contributions are formed separably, weight_x * (m v + A (x_i - x_p)) per
// column and then weight_y per row, a re-association of mpm_sim.py:256-271 that
// moves results by rounding only.
template <int J0>
__device__ __forceinline__ void accumulate_rows(f2* acc, const JfInst& I, const JfStencil& st, const JfScatter& sc,
                                                int di, int dj) {
  const bool sx = di != 0, sy = dj != 0;
  const float wx4[4] = {sx ? 0.0f : st.wx0, sx ? st.wx0 : st.wx1, sx ? st.wx1 : st.wx2, sx ? st.wx2 : 0.0f};
  const float wy4[4] = {sy ? 0.0f : st.wy0, sy ? st.wy0 : st.wy1, sy ? st.wy1 : st.wy2, sy ? st.wy2 : 0.0f};
  // node offsets from the particle: (I - di - fx0) dx; di + fx0 is exact
  const f2 ex = f2_dup(-((float)di + st.fx0)), ey = f2_dup(-((float)dj + st.fx1));
  const f2 dx = f2_dup(I.dx), mv = f2_pack(sc.mv0, sc.mv1);
  const f2 a0 = f2_pack(sc.af00, sc.af10), a1 = f2_pack(sc.af01, sc.af11);
  f2 P[4], Q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const f2 d0 = f2_mul(f2_add(f2_dup((float)i), ex), dx);
    P[i] = f2_dup(wx4[i]);
    Q[i] = f2_mul(P[i], f2_fma(a0, d0, mv));
  }
  const f2 ms = f2_dup(sc.mass);
  const f2 M0 = f2_mul(f2_pack(wx4[0], wx4[1]), ms), M1 = f2_mul(f2_pack(wx4[2], wx4[3]), ms);
#pragma unroll
  for (int jj = 0; jj < 2; ++jj) {
    const int j = J0 + jj;
    const f2 r = f2_mul(a1, f2_mul(f2_add(f2_dup((float)j), ey), dx));
    const f2 w = f2_dup(wy4[j]);
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[4 * jj + i] = f2_fma(w, f2_fma(P[i], r, Q[i]), acc[4 * jj + i]);
    acc[8 + 2 * jj] = f2_fma(w, M0, acc[8 + 2 * jj]);
    acc[9 + 2 * jj] = f2_fma(w, M1, acc[9 + 2 * jj]);
  }
}

// Adds rows J0 and J0 + 1 of a warp's 4x4 node blocks to the window.  Lane l
// owns cell column cx = seg0 + l and covers node columns cx-1 .. cx+2; node
// column cx collects block column 1 of lane l, 0 of lane l+1, 2 of lane l-1 and
// 3 of lane l-2, so each lane issues one atomic per (row, component).  The
// three columns that stick out of the segment (seg0 - 1 from lane 0, seg0 + 32
// and seg0 + 33 from lanes 30 and 31) go to lanes 3 (3 row + component) + column
// of one further atomic for all of them: an FP32 shared-memory atomic is a
// compare-and-swap loop, and one divergent site costs as much as a full one.
template <int J0, class Win>
__device__ __forceinline__ void flush_rows(const f2* acc, const Win& w, int lane, int cx, int cy, int seg0, int nx) {
  const unsigned full = 0xffffffffu;
  float edge = 0.0f;
#pragma unroll
  for (int jj = 0; jj < 2; ++jj) {
    const int rowo = (cy - 1 + J0 + jj - w.win0) * nx;
    const float2 n0 = f2_get(acc[4 * jj]), n1 = f2_get(acc[4 * jj + 1]);
    const float2 n2 = f2_get(acc[4 * jj + 2]), n3 = f2_get(acc[4 * jj + 3]);
    const float2 m0 = f2_get(acc[8 + 2 * jj]), m1 = f2_get(acc[9 + 2 * jj]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      float* A = q == 0 ? w.Ax : (q == 1 ? w.Ay : w.Am);
      const float a0 = q == 0 ? n0.x : (q == 1 ? n0.y : m0.x), a1 = q == 0 ? n1.x : (q == 1 ? n1.y : m0.y);
      const float a2 = q == 0 ? n2.x : (q == 1 ? n2.y : m1.x), a3 = q == 0 ? n3.x : (q == 1 ? n3.y : m1.y);
      // rotations: the lanes that wrap around carry the columns that stick out
      const float r0 = __shfl_sync(full, a0, lane + 1);
      const float r2 = __shfl_sync(full, a2, lane + 31);
      const float r3 = __shfl_sync(full, a3, lane + 30);
      float col = a1;
      col += lane <= 30 ? r0 : 0.0f;
      col += lane >= 1 ? r2 : 0.0f;
      col += lane >= 2 ? r3 : 0.0f;
      if (cx < nx && col != 0.0f) atomicAdd(A + rowo + cx, col);
      // lane 31: r0 = column seg0 - 1; lanes 0 and 1: columns seg0 + 32 and + 33
      const float out = lane == 31 ? r0 : (lane == 0 ? r2 + r3 : r3);
      const int first = 3 * (3 * jj + q);
      const float e = __shfl_sync(full, out, lane == first ? 31 : lane - first - 1);
      if (lane >= first && lane < first + 3) edge = e;
    }
  }
  if (lane < 18 && edge != 0.0f) {
    const int g = lane / 3, c = lane - 3 * g, jj = g / 3, q = g - 3 * jj;
    const int col = c == 0 ? seg0 - 1 : seg0 + 31 + c;
    float* A = q == 0 ? w.Ax : (q == 1 ? w.Ay : w.Am);
    if (col >= 0 && col < nx) atomicAdd(A + (cy - 1 + J0 + jj - w.win0) * nx + col, edge);
  }
}

// One instance as the tasks of a pass see it: its constants, its payload
// density and the engine's particle arrays.  Particles are indexed by engine
// position, so that the array bases stay kernel parameters and cost no
// registers.
template <class Args>
struct JfEnv {
  const JfInst& I;
  const Args& a;  // the kernel's parameters: xv, C, F, mat, Jp, fiber, glow, rref, mats
  float pdens;
  bool do_glow;
};

template <class Win>
__device__ __forceinline__ float2 gather_node(const Win& w, int i, int j) {
  const int wr = j - w.win0;
  if (wr >= 0 && wr < w.VR) return w.G[wr * w.nx + i];
  return w.far_gather(i, j);
}

// Scatter of one particle's 9 stencil contributions with atomics, into the
// window where it holds the rows, else to the rows' owner.
template <class Win>
__device__ __forceinline__ void scatter_particle(const Win& w, const JfInst& I, const JfStencil& st,
                                                 const JfScatter& sc) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int row = st.by + j;
    const int wr = row - w.win0;
    if (wr >= 0 && wr < w.VR) {
      const int rn = wr * w.nx + st.bx;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float3 c = jf_node_contrib(I, st, sc, i, j);
        atomicAdd(w.Ax + rn + i, c.x);
        atomicAdd(w.Ay + rn + i, c.y);
        atomicAdd(w.Am + rn + i, c.z);
        if (I.axisym) atomicAdd(w.Ah + rn + i, jf_w(st, 0, i) * jf_w(st, 1, j) * sc.hoop);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i)
        w.far_scatter(st.bx + i, row, jf_node_contrib(I, st, sc, i, j),
                      I.axisym ? jf_w(st, 0, i) * jf_w(st, 1, j) * sc.hoop : 0.0f, I.axisym);
    }
  }
}

// A task of a pass: each lane of the warp runs its particles beg .. end - 1
// (engine positions) through G2P of the previous substep and P2G of this one.
// In a cell task the lanes own 32 consecutive cells of row cy from column seg0
// on, lane l the cell of column cx = seg0 + l, and add the particles whose
// stencil lies in their cell's node block to that block, which the warp then
// flushes into the window.  In a group of single particles (`cells` false)
// every particle is scattered on its own.  The node blocks of kTmem live in
// TMEM from column `ta` of the warp's lanes.  s_path: the CTA's path counters.
template <bool kTmem, class Args, class Win>
__device__ __forceinline__ void run_task(const JfEnv<Args>& E, const Win& w, bool cells, int beg, int end, int cy,
                                         int seg0, uint32_t ta, bool do_g2p, bool do_p2g, float pressure,
                                         unsigned* s_path, bool& nonfinite) {
  const JfInst& I = E.I;
  const int nx = I.nx;
  const int lane = threadIdx.x & 31;
  const int cx = seg0 + lane;
  // G2P then P2G of particle k of this lane's cell (nxv / nmt: its
  // prefetched position-velocity and material, replaced by particle
  // k + 1's); returns true when its stencil lies in the lane's 4x4 node
  // block (columns cx-1 .. cx+2, rows cy-1 .. cy+2), with the stencil,
  // the scatter terms and the block offset for the caller to add
  auto cell_particle = [&](int k, float4& nxv, int& nmt, JfStencil& st, JfScatter& sc, int& di,
                           int& dj) -> bool {
    const float4 xv = nxv;
    const int mt = nmt;
    float4 F = E.a.F[k];  // first used by P2G, after the gather
    if (k + 1 < end) {  // next particle of this cell, loaded while this one computes
      nxv = E.a.xv[k + 1];
      nmt = E.a.mat[k + 1];
    }
    float2 x = make_float2(xv.x, xv.y), v = make_float2(xv.z, xv.w);
    float jp = 1.0f;
    if (mt == 2 || E.do_glow) jp = E.a.Jp[k];
    // G2P replaces v and C from the grid (mpm_sim.py:315-327); the stored
    // C is read only where G2P does not run
    float4 C;
    if (do_g2p) {
      JfStencil gs;
      if (!jf_stencil(I, x, gs)) {
        C = E.a.C[k];
      } else {
        const int wr0 = gs.by - w.win0;
        if (wr0 >= 0 && wr0 + 2 < w.VR) {
          const int wb = wr0 * nx + gs.bx;
          jf_g2p_apic(I, gs, v, C, [&](int i, int j) {
            const int n = wb + j * nx + i;
            return w.G[n];
          });
        } else {
          if (cells) atomicAdd(&s_path[2], 1u);
          jf_g2p_apic(I, gs, v, C,
                      [&](int i, int j) { return gather_node(w, gs.bx + i, gs.by + j); });
        }
      }
      jf_g2p_advect(I, x, v);
      if (E.do_glow) E.a.glow[k] = jf_glow(E.a.glow[k], jp);
      nonfinite |= !(isfinite(v.x) && isfinite(v.y));  // the wall clamp leaves x finite whatever it was
      E.a.xv[k] = make_float4(x.x, x.y, v.x, v.y);
      // this pass's P2G takes C from registers and the next pass's G2P
      // recomputes it, so C is stored only by the chunk's last pass and
      // where the particle leaves the stencil range (P2G below)
      if (!do_p2g) E.a.C[k] = C;
    } else {
      C = E.a.C[k];
    }
    if (!do_p2g) return false;
    if (!jf_stencil(I, x, st)) {
      if (do_g2p) E.a.C[k] = C;  // out of range: the next G2P keeps this C
      return false;
    }
    const float2 fb = (mt == 3) ? E.a.fiber[k] : make_float2(0.0f, 1.0f);
    jf_p2g_particle(I, E.a.mats, mt, v, C, F, jp, fb, pressure, E.pdens, sc, x.x,
                    I.axisym ? E.a.rref[k] : 1.0f);
    E.a.F[k] = F;
    if (mt == 2) E.a.Jp[k] = jp;
    di = st.bx - (cx - 1);
    dj = st.by - (cy - 1);
    if (cells && (unsigned)di < 2u && (unsigned)dj < 2u) {
      if (I.axisym) {  // the hoop sum goes straight to the window (rows in it)
        const int hb = (st.by - w.win0) * nx + st.bx;
#pragma unroll
        for (int jj = 0; jj < 3; ++jj)
#pragma unroll
          for (int ii = 0; ii < 3; ++ii)
            atomicAdd(w.Ah + hb + jj * nx + ii, jf_w(st, 0, ii) * jf_w(st, 1, jj) * sc.hoop);
      }
      return true;
    }
    if (cells) atomicAdd(&s_path[1], 1u);
    scatter_particle(w, I, st, sc);
    return false;
  };
  float4 nxv;
  int nmt = -1;
  if (beg < end) {
    nxv = E.a.xv[beg];
    nmt = E.a.mat[beg];
  }
  if constexpr (!kTmem) {
    // the lane's cell runs as a loop of its own length; the block stays in registers
    unsigned n_block = 0;
    f2 acc[2 * kHalfBlock];
#pragma unroll
    for (int q = 0; q < 2 * kHalfBlock; ++q) acc[q] = 0;
    for (int k = beg; k < end; ++k) {
      JfStencil st;
      JfScatter sc;
      int di, dj;
      if (cell_particle(k, nxv, nmt, st, sc, di, dj)) {
        accumulate_rows<0>(acc, I, st, sc, di, dj);
        accumulate_rows<2>(acc + kHalfBlock, I, st, sc, di, dj);
        ++n_block;
      }
    }
    __syncwarp();
    if (do_p2g && cells) {
      flush_rows<0>(acc, w, lane, cx, cy, seg0, nx);
      flush_rows<2>(acc + kHalfBlock, w, lane, cx, cy, seg0, nx);
      const unsigned nb = __reduce_add_sync(0xffffffffu, n_block);
      if (lane == 0 && nb) atomicAdd(&s_path[0], nb);
    }
  } else {
    // the warp steps its cells' particles together (the TMEM accesses are
    // warp-wide) for as many iterations as its fullest cell; the block of
    // each lane is loaded from TMEM, added to and stored back, two rows at
    // a time, once per iteration in which some lane's particle adds to it
    const int iters = (int)__reduce_max_sync(0xffffffffu, (unsigned)(end - beg));
    unsigned n_block = 0;  // the same in every lane of the warp
    __syncwarp();
    if (do_p2g && cells) tm_zero48(ta);
    for (int it = 0; it < iters; ++it) {
      const int k = beg + it;
      JfStencil st;
      JfScatter sc;
      int di = 0, dj = 0;
      const bool blk = k < end && cell_particle(k, nxv, nmt, st, sc, di, dj);
      if (do_p2g) {
        const unsigned bm = __ballot_sync(0xffffffffu, blk);
        if (bm) {
          n_block += (unsigned)__popc(bm);
          f2 half[kHalfBlock];
          tm_load_rows01(ta, half);
          if (blk) accumulate_rows<0>(half, I, st, sc, di, dj);
          __syncwarp();
          tm_store_rows01(ta, half);
          tm_load_rows23(ta, half);
          if (blk) accumulate_rows<2>(half, I, st, sc, di, dj);
          __syncwarp();
          tm_store_rows23(ta, half);
        }
      }
    }
    __syncwarp();
    if (do_p2g && cells) {
      // the last store to columns 24 .. 47 precedes the wait of the first load
      f2 half[kHalfBlock];
      tm_load_rows01(ta, half);
      flush_rows<0>(half, w, lane, cx, cy, seg0, nx);
      tm_load_rows23(ta, half);
      flush_rows<2>(half, w, lane, cx, cy, seg0, nx);
      if (lane == 0 && n_block) atomicAdd(&s_path[0], n_block);
    }
  }
}

}  // namespace
