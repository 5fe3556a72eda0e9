// Immersed-boundary kernels: smoothed indicator, momentum exchange and the
// volume integrals of the particle interiors.
//
// Reference functions restated here (NaokiHori/EllipsesInFlows):
//   suspensions_decide_loop_size   src/suspensions/auxiliary.c:11-17
//   compute_signed_dist            src/suspensions/auxiliary.c:19-47
//   suspensions_s_weight/v_weight  src/suspensions/auxiliary.c:51-59
//   mass, moment of inertia        src/suspensions/auxiliary.c:63-75
//   find_normal_t, compute_ex/ey   src/ellipse.c:7-65
//   kernel_exchange_momentum       src/suspensions/exchange.c:13-88
//   compute_inertia                src/suspensions/inertia.c:9-70
//
// Work decomposition. For every particle the reference visits, for the
// periodic images -1, 0, +1, the cells of a clipped bounding box. Here every
// box row is one task (rows wider than CHUNK cells are cut into segments of
// CHUNK cells); tasks are numbered in the reference's (image, j, i) order. One
// warp evaluates one task (two cells per lane) inside a persistent grid sized
// to the SM count, so particles of any size keep all SMs busy. Per-particle sums are reduced per chunk with warp shuffles and
// then per particle over its chunks in a fixed order: results are
// deterministic. The momentum exchange also stores each box cell's field
// contribution in a scratch buffer; a tile gather then adds, for every cell,
// the contributions of all covering boxes in (particle, image) order, which
// is the reference's accumulation order (exchange.c:71-72), without atomics.
#ifndef EIF_CHECK
#define EIF_CHECK 1
#endif
#include "eif_internal.cuh"
#include <cfloat>
#include <vector>
#include <algorithm>
#include <cmath>

#include "ibm_device.cuh"
#include "particle_device.cuh"

namespace {

// What the table kernels clear for the kernels after them (a clearing node of its own holds
// the branch up for 4 us between two kernels): the bitmap that k_band_marks adds the boxes of
// this build to (to which it adds them again when the lists are built twice from one build),
// and the count of the tasks that the memo does not serve.
struct TableClears {
  unsigned *marks;   // or null: inside a sub-iteration loop, where no lists are built
  int nmarks;
  int *miss;         // or null: double precision
  __device__ __forceinline__ void clear() const {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (miss && t == 0) *miss = 0;
    if (marks)
      for (int k = t; k < nmarks; k += gridDim.x * blockDim.x) marks[k] = 0u;
  }
};

// Stand-alone kernels over the bodies of ibm_device.cuh. Inside the sub-iteration
// loop of a step graph (iter set) the loop counter decides what runs: in the first
// sub-iteration the increments are zero, the positions are X and the boxes and the
// weights built at X before the loop are still in place.
__global__ void __launch_bounds__(32) k_boxes(BoxArgs a) {
  if (a.iter && *a.iter == 0u) return;
  box_part(a, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(TT_WARPS * 32) k_task_table_scan(const int *__restrict__ box, const int *__restrict__ cnt,
                                                                  int *__restrict__ off, int4 *__restrict__ tdesc, int np,
                                                                  Bounds bd, int cap, const unsigned *__restrict__ iter, TableClears z) {
  if (iter && *iter == 0u) return;
  z.clear();
  task_table_block(box, cnt, off, tdesc, np, bd, cap, blockIdx.x);
}

// The double-precision body is the batch stage kernel's instantiation (ordinary loads):
// one function, compiled alike in both translation units, gives both kernels the same
// bits.
__global__ void __launch_bounds__(256, 3) k_ibm_work(WorkArgs a) {
  // per warp: its near cells, their feet and their weights
  __shared__ WorkSlots slot_buf[8];
  const int wmode = a.iter ? (*a.iter == 0u ? 2 : 0) : a.wmode;
  ibm_work_tasks<false>(a, wmode, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
                        slot_buf[threadIdx.x >> 5], nullptr);
}

__global__ void __launch_bounds__(256, 3) k_ibm_work_f(WorkArgs a) {
  __shared__ WorkSlotsF slot_buf[8];
  ibm_work_f_tasks<true>(a, a.wmode, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
                         slot_buf[threadIdx.x >> 5]);
}

// the stage start's evaluation at X (mixed form): memo-served tasks, the rest listed
__global__ void __launch_bounds__(256, 4) k_ibm_memo_f(WorkArgs a) {
  ibm_memo_f_tasks<true>(a, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5);
}

__global__ void __launch_bounds__(256, 4) k_ibm_sum_f(WorkArgs a) {
  ibm_sum_f_tasks<true>(a, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
                        EIF_CHK(a.bd.rec, a.np, a.bd.off, 70) ? __ldg(a.off + a.np) : 0);
}

// Inside a sub-iteration loop: the sums with the weights at X in the first sub-iteration, the
// full evaluation afterwards. One launch: a second one that finds that it is not its turn costs
// each of some hundred sub-iterations of a step 3 us.
__global__ void __launch_bounds__(256, 3) k_ibm_loop_f(WorkArgs a) {
  __shared__ WorkSlotsF slot_buf[8];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
  if (*a.iter == 0u) {
    ibm_sum_f_tasks<true>(a, warp, warps, EIF_CHK(a.bd.rec, a.np, a.bd.off, 70) ? __ldg(a.off + a.np) : 0);
  } else {
    ibm_work_f_tasks<true>(a, 0, warp, warps, slot_buf[threadIdx.x >> 5]);
  }
}

__global__ void k_chunk_reduce(const double *__restrict__ partial, const int *__restrict__ off, double *__restrict__ P,
                               int pcap, int np, int f0, int f1, int f2, Bounds bd) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (n >= np || !EIF_CHK(bd.rec, n + 1, bd.off, 30)) return;
  const double v = chunk_sum_warp(partial, off[n], off[n + 1], bd);
  const int lane = threadIdx.x & 31;
  if (lane < 3 && EIF_CHK(bd.rec, f2 * pcap + n, bd.P, 32)) P[(lane == 0 ? f0 : (lane == 1 ? f1 : f2)) * pcap + n] = v;
}

// save: after an indicator evaluation that stored its weights in the memo
__global__ void k_chunk_reduce_f(const float *__restrict__ partial, const int *__restrict__ off, double *__restrict__ P,
                                 int pcap, int np, int f0, int f1, int f2, Bounds bd, WeightMemo memo, int save,
                                 const float *__restrict__ pf, const int *__restrict__ box) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (n >= np || !EIF_CHK(bd.rec, n + 1, bd.off, 33)) return;
  if (save) memo_particle(memo, pf + (size_t)PF_WORDS * n, box + 12 * (size_t)n, off[n], n);
  const double v = chunk_sum_f_warp(partial, off[n], off[n + 1], bd);
  const int lane = threadIdx.x & 31;
  if (lane < 3 && EIF_CHK(bd.rec, f2 * pcap + n, bd.P, 35)) P[(lane == 0 ? f0 : (lane == 1 ? f1 : f2)) * pcap + n] = v;
}

// The end of a sub-iteration in a loop of kernels: the particles' sums over their tasks and
// their increments, then the residual and the loop's condition (k_chunk_reduce, k_increment).
// One warp sums one particle; the first warp of the block then forms the increments of the
// block's particles, component k of particle q in lane 3 q + k: a lone warp's FP64 instruction
// holds its scheduler 64 cycles for one lane or for all. What the sums do not change is loaded
// before them. 8.2 us with 2048 ellipses and 7.2 with 512; as two kernels 14.1 and 11.1.
constexpr int END_WARPS = 8;
struct EndArgs {
  double *P, *scal;
  const double *partial;
  const int *off, *box;
  const float *pf;
  unsigned long long *res_bits, *total;
  unsigned *counter, *arrivals;   // counter: sub-iterations of the stage before this one
  cudaGraphConditionalHandle handle;
  double gamma, Fr2;
  int pcap, np, mixed, use_handle, save;   // save: see k_chunk_reduce_f; in a loop not the first
  WeightMemo memo;
  Bounds bd;
};
__global__ void __launch_bounds__(END_WARPS * 32) k_sub_end(EndArgs a) {
  __shared__ double sums[3 * END_WARPS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, pc = a.pcap;
  const int q = lane / 3, k = lane - 3 * q, m = blockIdx.x * END_WARPS + q;
  const bool own = w == 0 && q < END_WARPS && m < a.np && EIF_CHK(a.bd.rec, EIF_P_DAZ * pc + m, a.bd.P, 36);
  double *p = a.P + m;
  const double dt = a.scal[0];
  double c0 = 0., c1 = 0., f = 0., i0 = 0., u = 0., du0 = 0., g = 0.;
  if (own) {
    c0 = p[(k == 0 ? EIF_P_CFX0 : (k == 1 ? EIF_P_CFY0 : EIF_P_CTZ0)) * pc];
    c1 = p[(k == 0 ? EIF_P_CFX1 : (k == 1 ? EIF_P_CFY1 : EIF_P_CTZ1)) * pc];
    f = p[(k == 0 ? EIF_P_FUX : (k == 1 ? EIF_P_FUY : EIF_P_TVZ)) * pc];
    i0 = p[(k == 0 ? EIF_P_IUX0 : (k == 1 ? EIF_P_IUY0 : EIF_P_IVZ0)) * pc];
    u = p[(k == 0 ? EIF_P_UX : (k == 1 ? EIF_P_UY : EIF_P_VZ)) * pc];
    du0 = p[(k == 0 ? EIF_P_DUX : (k == 1 ? EIF_P_DUY : EIF_P_DVZ)) * pc];
    if (k == 0) g = gravity_increment(a.gamma, dt, p[EIF_P_DEN * pc], a.Fr2);
  }
  const int n = blockIdx.x * END_WARPS + w;
  if (n < a.np && EIF_CHK(a.bd.rec, n + 1, a.bd.off, 37)) {
    const int t0 = a.off[n], t1 = a.off[n + 1];
    if (a.save && !(a.use_handle && *a.counter == 0u))
      memo_particle(a.memo, a.pf + (size_t)PF_WORDS * n, a.box + 12 * (size_t)n, t0, n);
    const double v = a.mixed ? chunk_sum_f_warp(reinterpret_cast<const float *>(a.partial), t0, t1, a.bd)
                             : chunk_sum_warp(a.partial, t0, t1, a.bd);
    if (lane < 3) sums[3 * w + lane] = v;
  }
  __syncthreads();
  if (w != 0) return;
  // the largest change as bits (non-negative; a NaN does not count, as in fmax)
  long long r = 0ll;
  if (own) {
    const double i1 = sums[lane], hgd = __dmul_rn(0.5 * a.gamma, dt);
    double du = velocity_increment(hgd, dt, c0, c1, f, i0, i1);
    if (k == 0) du = __dadd_rn(du, g);
    const double change = fabs(du - du0);
    if (change > 0.) r = __double_as_longlong(change);
    p[(k == 0 ? EIF_P_IUX1 : (k == 1 ? EIF_P_IUY1 : EIF_P_IVZ1)) * pc] = i1;
    p[(k == 0 ? EIF_P_DUX : (k == 1 ? EIF_P_DUY : EIF_P_DVZ)) * pc] = du;
    p[(k == 0 ? EIF_P_DX : (k == 1 ? EIF_P_DY : EIF_P_DAZ)) * pc] = position_increment(hgd, u, du);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
  if (lane == 0) {
    if (r > 0ll) atomicMax(a.res_bits, (unsigned long long)r);
    // the last block to finish publishes the residual (its maximum is complete)
    __threadfence();
    if (atomicAdd(a.arrivals, 1u) == gridDim.x - 1) {
      __threadfence();
      *a.arrivals = 0u;
      const double res = __longlong_as_double((long long)atomicExch(a.res_bits, 0ull));
      a.scal[1] = res;
      *a.total += 1ull;   // sub-iterations run (eif_counters)
      // the condition of the loop (main.c:40-48): continue while the residual is not below
      // 1e-8 and at most 101 sub-iterations ran
      if (a.use_handle) {
        const unsigned count = ++*a.counter;
        cudaGraphSetConditional(a.handle, (!(res < 1.e-8) && count <= 101u) ? 1u : 0u);
      }
    }
  }
}

// exclusive scan of the chunk counts (one block); off[np] = total
__global__ void k_scan(const int *__restrict__ cnt, int *__restrict__ off, int np, Bounds bd,
                       const unsigned *__restrict__ iter) {
  if (iter && *iter == 0u) return;
  __shared__ int s[1024];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < np; base += 1024) {
    const int t = base + threadIdx.x;
    const int v = (t < np && EIF_CHK(bd.rec, (cnt - off) + 2 * np + t, bd.off, 4)) ? cnt[t] + cnt[np + t] + cnt[2 * np + t] : 0;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const int add = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
      __syncthreads();
      s[threadIdx.x] += add;
      __syncthreads();
    }
    if (t < np && EIF_CHK(bd.rec, t, bd.off, 5)) off[t] = carry + s[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += s[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0 && EIF_CHK(bd.rec, np, bd.off, 6)) off[np] = carry;
}

// Bound on the box cells of one particle over its three images. A box spans at
// most 2r/h + 2 + 2*NEXTRA + 1 cells per direction before clipping; the three
// images are shifted by exactly jtot rows, so their clipped row ranges together
// never exceed the unclipped height.
__host__ __device__ inline size_t tasks_bound(double r, double dx, double dy, int itot, int jtot) {
  const long w = (long)ceil(2. * r / dx) + 2 + 2 * NEXTRA + 2;
  const long h = (long)ceil(2. * r / dy) + 2 + 2 * NEXTRA + 2;
  const long wc = w < itot ? w : itot;
  const long hc = h < 3L * jtot ? h : 3L * jtot;
  return (size_t)hc * (size_t)box_segs((int)wc);
}

// exclusive sums of the bounds (one block of 1024): first task slots of the particles
__global__ void __launch_bounds__(1024) k_task_bases(const double *__restrict__ P, int pcap, int np, double dx, double dy,
                                                     int itot, int jtot, int *__restrict__ base) {
  __shared__ int w[32];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  int run = 0;
  for (int n0 = 0; n0 < np; n0 += 1024) {
    const int n = n0 + threadIdx.x;
    const int v = n < np ? (int)tasks_bound(fmax(P[EIF_P_A * pcap + n], P[EIF_P_B * pcap + n]), dx, dy, itot, jtot) : 0;
    int sc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sc, o);
      if (lane >= o) sc += u;
    }
    if (lane == 31) w[wl] = sc;
    __syncthreads();
    int before = 0, all = 0;
    for (int q = 0; q < 32; q++) {
      before += q < wl ? w[q] : 0;
      all += w[q];
    }
    if (n < np) base[n] = run + before + sc - v;
    run += all;
    __syncthreads();
  }
}

// The task table: one int4 per task (chunk) {particle, row, first column, last
// column * 4 + image + 1}, so that a kernel finds its task's geometry with one
// load instead of a chain of dependent loads (owner, boxes, offsets). One warp
// per particle.
__global__ void k_task_table(const int *__restrict__ box, const int *__restrict__ off, int4 *__restrict__ tdesc,
                             int np, Bounds bd, int cap, const unsigned *__restrict__ iter, TableClears z) {
  if (iter && *iter == 0u) return;
  z.clear();
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (n >= np) return;
  const int4 *b4 = reinterpret_cast<const int4 *>(box + 12 * n);
  const int4 bA = b4[0], bB = b4[1], bC = b4[2];
  const int c0 = off[n], c1 = off[n + 1];
  for (int c = c0 + lane; c < c1; c += 32) {
    RowTask t;
    int4 d = make_int4(-1, 0, 0, 0);
    if (row_task(bA, bB, bC, c - c0, t)) d = make_int4(n, t.j, t.ib, t.ie * 4 + t.img + 1);
    if (EIF_CHK(bd.rec, c, cap, 59)) tdesc[c] = d;
  }
}


// Ordered lists of the (particle, image) boxes that reach each band of GTY rows,
// built once per exchange; entry = 3 * particle + image index, in entry order.
// Step 1 (one thread per particle): every box sets its bit in the bitmap of each
// band it reaches (atomicOr: the result does not depend on the order). Step 2
// (one warp per band): the band's set bits are compacted in index order.
__global__ void k_band_marks(const int *__restrict__ box, const int *__restrict__ off, int np, int jtot,
                             unsigned *__restrict__ marks, int words, int4 *__restrict__ edesc, Bounds bd) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= np) return;
  const int nbands = (jtot + GTY - 1) / GTY;
  const int *bx = box + 12 * n;
  int tasks_q = 0;   // tasks of the earlier images
  const int off_n = off[n];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int bi0 = bx[4 * q], bi1 = bx[4 * q + 1], bj0 = bx[4 * q + 2], bj1 = bx[4 * q + 3];
    const bool nonempty = bi1 >= bi0 && bj1 >= bj0;
    const int e = 3 * n + q;
    // the entry's box and where its rows start in the scratch buffer (a box row
    // occupies segs * CHUNK slots)
    if (EIF_CHK(bd.rec, 2LL * e + 1, 6LL * np, 47)) {
      edesc[2 * e] = nonempty ? make_int4(bi0, bi1, bj0, bj1) : make_int4(1, 0, 1, 0);
      edesc[2 * e + 1] = make_int4(nonempty ? box_segs(bi1 - bi0 + 1) * CHUNK : 0, (off_n + tasks_q) * CHUNK, 0, 0);
    }
    if (!nonempty) continue;
    tasks_q += (bj1 - bj0 + 1) * box_segs(bi1 - bi0 + 1);
    const int b0 = max(0, (bj0 - 1) / GTY), b1 = min(nbands - 1, (bj1 - 1) / GTY);
    for (int b = b0; b <= b1; b++) atomicOr(marks + (size_t)b * words + (e >> 5), 1u << (e & 31));
  }
}

__global__ void k_band_lists(const unsigned *__restrict__ marks, int words, int jtot, int *__restrict__ lists,
                             int *__restrict__ counts, int cap, unsigned *__restrict__ flags) {
  const int lane = threadIdx.x & 31;
  const int band = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nbands = (jtot + GTY - 1) / GTY;
  if (band >= nbands) return;
  int count = 0;
  int *out = lists + (size_t)band * cap;
  const unsigned *row = marks + (size_t)band * words;
  for (int base = 0; base < words; base += 32) {
    const int w = base + lane;
    unsigned bits = w < words ? row[w] : 0u;
    const int m = __popc(bits);
    int sc = m;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sc, o);
      if (lane >= o) sc += v;
    }
    int pos = count + sc - m;
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1u;
      if (pos < cap) out[pos] = 32 * w + b;
      pos++;
    }
    count += __shfl_sync(0xffffffffu, sc, 31);
  }
  if (lane == 0) {
    counts[band] = count;
    if (count > cap) atomicOr(flags, EIF_FLAG_NOCONV);
  }
}

struct GatherArgs {
  const int4 *edesc;   // per (particle, image) entry: box, then row pitch and scratch offset
  const int *lists, *counts;
  int cap;
  const void *wbuf;
  void *dux, *duy;   // double (FP64 form) or float (mixed form) fields with the same pitch
  unsigned *flags;
  int np, itot, jtot, ld;
  Bounds bd;
};

// field response dux/duy (exchange.c:71-72,80-81): per tile, the entries of the
// band's ordered list that reach the tile's columns are compacted in order into
// shared memory, then every cell sums their contributions in that order
template <typename V2, typename Acc>
__global__ void __launch_bounds__(GTHREADS, 6) k_gather(GatherArgs a) {
  const V2 *wbuf = static_cast<const V2 *>(a.wbuf);
  // compacted entries: columns, rows, row pitch and offset of the box in the scratch buffer
  __shared__ int e_i0[LMAX], e_i1[LMAX], e_j0[LMAX], e_j1[LMAX], e_w[LMAX], e_base[LMAX];
  __shared__ int wcount[GTHREADS / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i0 = 1 + blockIdx.x * GTX, j0 = 1 + blockIdx.y * GTY;
  const int i1 = min(i0 + GTX - 1, a.itot), j1 = min(j0 + GTY - 1, a.jtot);
  constexpr int NC = (GTX / GCOLS) * 2;
  Acc acc_x[NC], acc_y[NC];
#pragma unroll
  for (int r = 0; r < NC; r++) { acc_x[r] = 0; acc_y[r] = 0; }
  // cells of this thread: (i0 + lx + GCOLS h, j0 + ly0 + 4 r), cell index 2 h + r
  const int lx = threadIdx.x % GCOLS, ly0 = threadIdx.x / GCOLS;  // GTHREADS / GCOLS = 4 rows per pass
  const int band = blockIdx.y;
  const int L = min(__ldg(a.counts + band), a.cap);
  const int *blist = a.lists + (size_t)band * a.cap;
  for (int base = 0; base < L; base += GTHREADS) {
    const int e = base + threadIdx.x;
    int4 b = make_int4(1, 0, 1, 0), w = make_int4(0, 0, 0, 0);
    if (e < L) {
      const int ent = __ldg(blist + e);
      // entry = 3 * particle + image; anything else is recorded and skipped
      if (EIF_CHK(a.bd.rec, ent, 3LL * a.np, 46)) {
        b = __ldg(a.edesc + 2 * ent);
        w = __ldg(a.edesc + 2 * ent + 1);
      }
    }
    const bool keep = b.y >= b.x && b.x <= i1 && b.y >= i0 && b.z <= j1 && b.w >= j0;
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) wcount[wid] = __popc(mask);
    __syncthreads();
    int pos = __popc(mask & ((1u << lane) - 1u)), cnt = 0;
#pragma unroll
    for (int q = 0; q < GTHREADS / 32; q++) {
      const int wc = wcount[q];
      pos += q < wid ? wc : 0;
      cnt += wc;
    }
    if (keep) {
      e_i0[pos] = b.x; e_i1[pos] = b.y; e_j0[pos] = b.z; e_j1[pos] = b.w; e_w[pos] = w.x; e_base[pos] = w.y;
    }
    __syncthreads();
    for (int k = 0; k < cnt; k++) {
      const int bi0 = e_i0[k], bi1 = e_i1[k], bj0 = e_j0[k], bj1 = e_j1[k], pw = e_w[k];
      const size_t pbase = (size_t)e_base[k];
#pragma unroll
      for (int q = 0; q < NC; q++) {
        const int i = i0 + lx + GCOLS * (q >> 1), j = j0 + ly0 + 4 * (q & 1);
        if (i >= bi0 && i <= bi1 && j >= bj0 && j <= bj1 &&
            EIF_CHK(a.bd.rec, (long long)(pbase + (size_t)(j - bj0) * pw + (i - bi0)),
                    a.bd.wbuf * (long long)(sizeof(double2) / sizeof(V2)), 41)) {
          const V2 v = wbuf[pbase + (size_t)(j - bj0) * pw + (i - bi0)];
          acc_x[q] += v.x;
          acc_y[q] += v.y;
        }
      }
    }
    __syncthreads();
  }
  // write the tile's interior cells (zero where no box covers); the halo rows and
  // ghost columns are filled afterwards by k_ibm_halo from these cells
  const int ld = a.ld;
#pragma unroll
  for (int q = 0; q < NC; q++) {
    const int i = i0 + lx + GCOLS * (q >> 1), j = j0 + ly0 + 4 * (q & 1);
    if (i > i1 || j > j1) continue;
    const int cidx = j * ld + i;
    if (!EIF_CHK(a.bd.rec, cidx, a.bd.field, 42)) continue;
    static_cast<Acc *>(a.dux)[cidx] = acc_x[q];
    static_cast<Acc *>(a.duy)[cidx] = acc_y[q];
  }
}

// Periodic halo rows (j = 0 <- jtot, j = jtot+1 <- 1) and Neumann ghost columns
// (i = 0 <- 1, i = itot+1 <- itot, corners included) of the IBM field response,
// exchange.c:80-81 with the boundary update of the reference. Every thread reads
// one interior cell and writes one halo cell.
template <typename T>
__global__ void k_ibm_halo(T *__restrict__ dux, T *__restrict__ duy, int itot, int jtot, int ld) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nrow = itot + 2;
  int dst, src;
  if (t < 2 * nrow) {
    const int i = t % nrow, top = t / nrow;
    const int ic = i < 1 ? 1 : (i > itot ? itot : i);
    dst = (top ? jtot + 1 : 0) * ld + i;
    src = (top ? 1 : jtot) * ld + ic;
  } else if (t < 2 * nrow + 2 * jtot) {
    const int u = t - 2 * nrow;
    const int j = 1 + u % jtot, right = u / jtot;
    dst = j * ld + (right ? itot + 1 : 0);
    src = j * ld + (right ? itot : 1);
  } else {
    return;
  }
  dux[dst] = dux[src];
  duy[dst] = duy[src];
}

}  // namespace

namespace eif {

static size_t box_tasks_bound(const eif_ctx *c, double r) {
  return tasks_bound(r, c->dx, c->dy, c->itot, c->jtot);
}

// resident CTAs per SM of the IBM work kernels (a host query; done before any graph capture)
int ibm_prepare(eif_ctx *c) {
  int v = 0;
  EIF_CK(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_ibm_work, 256, 0));
  c->ibm_ctas_per_sm[0] = std::max(1, v);
  EIF_CK(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_ibm_work_f, 256, 0));
  c->ibm_ctas_per_sm[1] = std::max(1, v);
  EIF_CK(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_ibm_sum_f, 256, 0));
  c->ibm_ctas_per_sm[2] = std::max(1, v);
  return EIF_OK;
}

// task bound of a particle set, from the radii in the host records (EIF_NFIELDS per particle);
// most: the largest of one particle
size_t ibm_tasks_needed(const eif_ctx *c, const double *rec, int n, size_t *most) {
  size_t chunks = 0;
  *most = 0;
  for (int k = 0; k < n; k++) {
    const size_t b =
        box_tasks_bound(c, std::max(rec[(size_t)k * EIF_NFIELDS + EIF_P_A], rec[(size_t)k * EIF_NFIELDS + EIF_P_B]));
    chunks += b;
    *most = std::max(*most, b);
  }
  return chunks;
}

// the first task slots of the pushed particles (box_tasks_bound summed on the device)
int ibm_task_bases(eif_ctx *c) {
  if (c->np == 0) return EIF_OK;
  k_task_bases<<<1, 1024, 0, c->stream>>>(c->P, c->pcap, c->np, c->dx, c->dy, c->itot, c->jtot, c->task_base);
  EIF_LAUNCH_CK(c);
  return EIF_OK;
}

// tanh_tab's values (tanh rounded to double and 1 minus its square, then where tanh has that
// value), then tanh_mid's (float pairs), formed once in the process: long double
// functions are software on some hosts (1.4 ms for the 2100 of them), so the exponentials are
// products with a constant step, restarted every 16 (an error of some 2^-60 at most).
static const std::vector<double2> &tanh_tables() {
  static const std::vector<double2> tab = [] {
    std::vector<double2> t(2 * TANH_N + (MID_N + 1) / 2);
    auto exps = [](int n, long double z0, int steps, auto put) {   // put(k, exp(-2 (z0 + k / steps)))
      const long double step = expl(-2.L / steps);
      long double e = 0.L;
      for (int k = 0; k < n; k++) {
        e = k % 16 == 0 ? expl(-2.L * (z0 + (long double)k / steps)) : e * step;
        put(k, e);
      }
    };
    exps(TANH_N, 0.L, TANH_STEPS, [&](int k, long double e) {
      // below 1, the place of which is infinite
      const double th = std::min((double)((1.L - e) / (1.L + e)), 1. - 0.5 * DBL_EPSILON);
      t[2 * k] = make_double2(th, (double)((1.L - th) * (1.L + th)));
      t[2 * k + 1] = make_double2((double)(0.5L * logl((1.L + th) / (1.L - th))), 0.);
    });
    float2 *mid = reinterpret_cast<float2 *>(t.data() + 2 * TANH_N);
    exps(MID_N, MID_Z0, MID_STEPS, [&](int k, long double e) {
      const float hi = (float)(2.L * e);
      mid[k] = make_float2(hi, (float)(2.L * e - (long double)hi));
    });
    return t;
  }();
  return tab;
}

int ibm_reserve(eif_ctx *c, size_t chunks) {
  // called after a particle push that changed the particle set: size the task and scratch buffers
  ibm_free(c);
  if (c->np == 0) return EIF_OK;
  c->chunk_cap = (int)chunks;
  c->wcap = chunks * CHUNK;
  EIF_CK(c, cudaMalloc((void **)&c->box, sizeof(int) * 12 * c->np));
  EIF_CK(c, cudaMalloc((void **)&c->chunk_off, sizeof(int) * (4 * (size_t)c->np + 1)));
  EIF_CK(c, cudaMalloc((void **)&c->task_base, sizeof(int) * c->np));
  EIF_CK(c, cudaMalloc((void **)&c->partial, sizeof(double) * 6 * chunks));
  EIF_CK(c, cudaMalloc((void **)&c->wbuf, sizeof(double2) * c->wcap));
  EIF_CK(c, cudaMalloc((void **)&c->wcache, sizeof(double) * c->wcap));
  if (c->cfg.precision == EIF_PREC_MIXED) EIF_CK(c, cudaMalloc((void **)&c->pf, sizeof(float) * PF_WORDS * c->np));
  else EIF_CK(c, cudaMalloc((void **)&c->pd, sizeof(double) * PD_WORDS * c->np));
  if (c->cfg.precision != EIF_PREC_MIXED && !c->tanh_tab) {
    const std::vector<double2> &tab = tanh_tables();
    EIF_CK(c, cudaMalloc((void **)&c->tanh_tab, sizeof(double2) * tab.size()));
    EIF_CK(c, cudaMemcpyAsync(c->tanh_tab, tab.data(), sizeof(double2) * tab.size(), cudaMemcpyHostToDevice, c->stream));
  }
  EIF_CK(c, cudaMalloc((void **)&c->tdesc, sizeof(int4) * (size_t)chunks));
  const int nbands = (c->jtot + GTY - 1) / GTY;
  c->band_cap = 3 * c->np;
  EIF_CK(c, cudaMalloc((void **)&c->band_lists, sizeof(int) * (size_t)nbands * c->band_cap));
  EIF_CK(c, cudaMalloc((void **)&c->band_counts, sizeof(int) * (size_t)nbands));
  EIF_CK(c, cudaMalloc((void **)&c->band_marks, sizeof(unsigned) * (size_t)nbands * ((3 * c->np + 31) / 32)));
  EIF_CK(c, cudaMalloc((void **)&c->edesc, sizeof(int4) * 6 * (size_t)c->np));
  if (c->cfg.precision == EIF_PREC_MIXED) {
    EIF_CK(c, cudaMalloc((void **)&c->memo_w, sizeof(float) * c->wcap));
    EIF_CK(c, cudaMalloc((void **)&c->memo_pf, sizeof(float) * PF_WORDS * c->np));
    EIF_CK(c, cudaMalloc((void **)&c->memo_box, sizeof(int) * 12 * c->np));
    EIF_CK(c, cudaMalloc((void **)&c->memo_off, sizeof(int) * c->np));
    EIF_CK(c, cudaMalloc((void **)&c->memo_valid, sizeof(int)));
    EIF_CK(c, cudaMemsetAsync(c->memo_valid, 0, sizeof(int), c->stream));
    EIF_CK(c, cudaMalloc((void **)&c->memo_miss, sizeof(int) * ((size_t)chunks + 1)));
  }
  return EIF_OK;
}

void ibm_free(eif_ctx *c) {
  if (c->box) cudaFree(c->box);
  if (c->chunk_off) cudaFree(c->chunk_off);
  if (c->task_base) cudaFree(c->task_base);
  c->task_base = nullptr;
  if (c->partial) cudaFree(c->partial);
  if (c->wbuf) cudaFree(c->wbuf);
  if (c->wcache) cudaFree(c->wcache);
  if (c->pf) cudaFree(c->pf);
  if (c->pd) cudaFree(c->pd);
  if (c->tanh_tab) cudaFree(c->tanh_tab);
  if (c->tdesc) cudaFree(c->tdesc);
  if (c->band_lists) cudaFree(c->band_lists);
  if (c->band_counts) cudaFree(c->band_counts);
  if (c->band_marks) cudaFree(c->band_marks);
  if (c->edesc) cudaFree(c->edesc);
  for (void *m : {(void *)c->memo_w, (void *)c->memo_pf, (void *)c->memo_box, (void *)c->memo_off, (void *)c->memo_valid,
                  (void *)c->memo_miss})
    if (m) cudaFree(m);
  c->memo_w = nullptr; c->memo_pf = nullptr; c->memo_box = nullptr; c->memo_off = nullptr; c->memo_valid = nullptr;
  c->memo_miss = nullptr;
  c->band_lists = nullptr; c->band_counts = nullptr; c->band_marks = nullptr; c->edesc = nullptr;
  c->box = nullptr; c->chunk_off = nullptr; c->partial = nullptr; c->wbuf = nullptr; c->wcache = nullptr;
  c->weights_x_valid = false;
  c->pf = nullptr; c->pd = nullptr; c->tanh_tab = nullptr; c->tdesc = nullptr;
  c->chunk_cap = 0; c->wcap = 0;
}

// bitmap over the 3 np (particle, image) boxes, one row of words per band
static int band_mark_words(const eif_ctx *c) { return (c->jtot + GTY - 1) / GTY * ((3 * c->np + 31) / 32); }

static int launch_boxes(eif_ctx *c, bool use_increment) {
  // boxes at the positions X (no increment, or increments known to be zero) are
  // reused until the positions or the particle set change
  const bool x_only = !use_increment || c->incr_zero;
  if (x_only && c->boxes_x_valid) return EIF_OK;
  c->boxes_x_valid = false;
  c->weights_x_valid = false;
  c->bands_x_valid = false;
  BoxArgs b = box_args(c, use_increment);
  b.iter = c->in_loop ? reinterpret_cast<const unsigned *>(c->d_inc + 1) : nullptr;
  int *cnt = b.nchunk;
  EIF_PROF(c, "ibm_boxes", c->np <= TT_MAX_NP ? 2 : 3);
  TableClears z;
  z.marks = c->in_loop ? nullptr : c->band_marks;
  z.nmarks = band_mark_words(c);
  z.miss = c->memo_miss;
  k_boxes<<<dim3((c->np + 31) / 32, BOX_PARTS), 32, 0, c->stream>>>(b);
  EIF_LAUNCH_CK(c);
  if (c->np <= TT_MAX_NP) {
    k_task_table_scan<<<(c->np + TT_WARPS - 1) / TT_WARPS, TT_WARPS * 32, 0, c->stream>>>(
        c->box, cnt, c->chunk_off, c->tdesc, c->np, bounds_of(c), c->chunk_cap, b.iter, z);
    EIF_LAUNCH_CK(c);
  } else {
    k_scan<<<1, 1024, 0, c->stream>>>(cnt, c->chunk_off, c->np, bounds_of(c), b.iter);
    EIF_LAUNCH_CK(c);
    k_task_table<<<(c->np * 32 + 255) / 256, 256, 0, c->stream>>>(c->box, c->chunk_off, c->tdesc, c->np,
                                                                   bounds_of(c), c->chunk_cap, b.iter, z);
    EIF_LAUNCH_CK(c);
  }
  c->memo_miss_zero = !c->in_loop;
  c->boxes_x_valid = x_only;
  return EIF_OK;
}

// store: the mixed form's evaluation that stores its weights in the memo (see launch_sums)
static int launch_work(eif_ctx *c, int mode, int cn, bool *store) {
  WorkArgs w = work_args(c, mode, cn);
  const bool mixed = c->cfg.precision == EIF_PREC_MIXED;
  // weights at the positions X (inertia with zero increments, or the exchange)
  // are stored once and reused while the boxes at X stay valid
  const bool x_only = mode == 1 || c->incr_zero;
  w.count = c->prof.enabled ? c->d_inc + 3 : nullptr;
  if (c->in_loop) {
    w.wmode = 0;
    w.iter = reinterpret_cast<const unsigned *>(c->d_inc + 1);
  } else if (x_only && c->boxes_x_valid && c->weights_x_valid) {
    w.wmode = 2;
  } else if (x_only && c->boxes_x_valid) {
    w.wmode = 1;
    c->weights_x_valid = true;
  } else {
    w.wmode = 0;
  }
  // persistent grid: as many CTAs as are resident at once (queried once per context)
  const int per_sm_idx = c->cfg.precision == EIF_PREC_MIXED ? 1 : 0;
  if (c->ibm_ctas_per_sm[per_sm_idx] == 0) {
    int rc = ibm_prepare(c);
    if (rc) return rc;
  }
  const int per_sm = c->ibm_ctas_per_sm[per_sm_idx];
  const int blocks = std::max(1, std::min(c->sms * per_sm, (c->chunk_cap * 32 + 255) / 256));
  // the weight memo (mixed form): the loop's evaluations with geometry (integrals 1)
  // store their weights in it; the first evaluation at X of a stage (integrals 0,
  // weights stored for the stage) takes them where the geometry is the memo's
  const bool memo_store = mixed && mode == 0 && cn == 1 && (c->in_loop || w.wmode == 0);
  if (mixed && mode == 0 && cn == 0 && w.wmode == 1 && c->memo_on) w.memo_mode = 1;
  {
    // launches that evaluate the indicator geometry are timed as ibm_indicator, those
    // with stored weights (sums and field contributions only) as inertia or exchange,
    // the stage start's evaluation that takes its weights from the memo as
    // ibm_stage_start
    const bool geometry = w.wmode != 2;
    EIF_PROF(c, w.memo_mode == 1 ? "ibm_stage_start" :
                (geometry ? "ibm_indicator" : (mode == 0 ? "ibm_inertia" : "ibm_exchange")),
             w.memo_mode == 1 ? 2 : 1);
    if (w.memo_mode == 1) {
      // the stage start: the memo-served tasks in the light kernel (sums-kernel
      // registers), then the full evaluation of the tasks it listed as not served
      if (!c->memo_miss_zero) EIF_CK(c, cudaMemsetAsync(c->memo_miss, 0, sizeof(int), c->stream));
      c->memo_miss_zero = false;
      WorkArgs wm = w, wf = w;
      wm.miss = c->memo_miss;
      wf.only = c->memo_miss;
      wf.memo_mode = 0;
      k_ibm_memo_f<<<c->sms * c->ibm_ctas_per_sm[2], 256, 0, c->stream>>>(wm);
      EIF_LAUNCH_CK(c);
      k_ibm_work_f<<<blocks, 256, 0, c->stream>>>(wf);
    } else if (mixed && c->in_loop) {
      w.memo_mode = 2;
      k_ibm_loop_f<<<blocks, 256, 0, c->stream>>>(w);
    } else if (mixed && w.wmode == 2) {
      k_ibm_sum_f<<<c->sms * c->ibm_ctas_per_sm[2], 256, 0, c->stream>>>(w);
    } else if (mixed) {
      if (memo_store) w.memo_mode = 2;
      k_ibm_work_f<<<blocks, 256, 0, c->stream>>>(w);
    } else {
      k_ibm_work<<<blocks, 256, 0, c->stream>>>(w);
    }
    EIF_LAUNCH_CK(c);
  }
  *store = memo_store;
  return EIF_OK;
}

// the particles' sums of the last evaluation of mode and cn
static int launch_sums(eif_ctx *c, int mode, int cn, bool memo_store) {
  const bool mixed = c->cfg.precision == EIF_PREC_MIXED;
  const double *partial = partial_of(c, mode);
  const int f0 = mode == 0 ? EIF_P_IUX0 + cn : EIF_P_FUX;
  const int f1 = mode == 0 ? EIF_P_IUY0 + cn : EIF_P_FUY;
  const int f2 = mode == 0 ? EIF_P_IVZ0 + cn : EIF_P_TVZ;
  EIF_PROF(c, "ibm_reduce", 1);
  if (mixed) {
    k_chunk_reduce_f<<<(c->np * 32 + 255) / 256, 256, 0, c->stream>>>(
        reinterpret_cast<const float *>(partial), c->chunk_off, c->P, c->pcap, c->np, f0, f1, f2, bounds_of(c),
        memo_of(c), memo_store ? 1 : 0, c->pf, c->box);
  } else {
    k_chunk_reduce<<<(c->np * 32 + 255) / 256, 256, 0, c->stream>>>(partial, c->chunk_off, c->P, c->pcap, c->np, f0, f1,
                                                                      f2, bounds_of(c));
  }
  EIF_LAUNCH_CK(c);
  return EIF_OK;
}

int launch_inertia(eif_ctx *c, int cn) {
  if (c->np == 0) return EIF_OK;
  int rc = launch_boxes(c, true);
  bool store = false;
  if (rc || (rc = launch_work(c, 0, cn, &store))) return rc;
  return launch_sums(c, 0, cn, store);
}

int launch_inertia_tasks(eif_ctx *c) {
  int rc = launch_boxes(c, true);
  bool store = false;
  return rc ? rc : launch_work(c, 0, 0, &store);
}
int launch_inertia_sums(eif_ctx *c) { return launch_sums(c, 0, 0, false); }

int launch_inertia_increment(eif_ctx *c, int rk, bool beside) {
  int rc = launch_boxes(c, true);
  bool store = false;
  if (rc || (rc = launch_work(c, 0, 1, &store))) return rc;
  if (beside && (rc = join_collision(c))) return rc;
  c->incr_zero = false;
  EndArgs a;
  a.P = c->P; a.scal = c->d_scal; a.partial = partial_of(c, 0);
  a.off = c->chunk_off; a.box = c->box; a.pf = c->pf;
  a.res_bits = c->d_inc; a.total = c->d_inc + 2;
  a.counter = reinterpret_cast<unsigned *>(c->d_inc + 1);
  a.arrivals = a.counter + 1;
  a.handle = c->loop_handle;
  a.gamma = rk_coef(rk).gamma; a.Fr2 = c->cfg.Fr * c->cfg.Fr;
  a.pcap = c->pcap; a.np = c->np;
  a.mixed = c->cfg.precision == EIF_PREC_MIXED ? 1 : 0;
  a.use_handle = c->in_loop ? 1 : 0;
  a.save = store ? 1 : 0;
  a.memo = memo_of(c);
  a.bd = bounds_of(c);
  k_sub_end<<<(c->np + END_WARPS - 1) / END_WARPS, END_WARPS * 32, 0, c->stream>>>(a);
  EIF_LAUNCH_CK(c);
  return EIF_OK;
}

int launch_exchange_tasks(eif_ctx *c) {
  int rc = launch_boxes(c, false);
  bool store = false;
  return rc ? rc : launch_work(c, 1, 0, &store);
}
int launch_exchange_sums(eif_ctx *c) { return launch_sums(c, 1, 0, false); }

static int band_lists_of_boxes(eif_ctx *c);

// ordered box lists per band of GTY rows for the gather, from the boxes at X
int launch_band_lists(eif_ctx *c) {
  if (c->np == 0) return EIF_OK;
  int rc = launch_boxes(c, false);
  if (rc) return rc;
  return band_lists_of_boxes(c);
}

// the band lists of the boxes currently built
static int band_lists_of_boxes(eif_ctx *c) {
  const int nbands = (c->jtot + GTY - 1) / GTY;
  const int words = (3 * c->np + 31) / 32;
  EIF_PROF(c, "ibm_band_lists", 2);
  k_band_marks<<<(c->np + 127) / 128, 128, 0, c->stream>>>(c->box, c->chunk_off, c->np, c->jtot, c->band_marks,
                                                           words, c->edesc, bounds_of(c));
  EIF_LAUNCH_CK(c);
  k_band_lists<<<(nbands * 32 + 255) / 256, 256, 0, c->stream>>>(c->band_marks, words, c->jtot, c->band_lists,
                                                                   c->band_counts, c->band_cap, c->d_flags);
  EIF_LAUNCH_CK(c);
  c->bands_x_valid = c->boxes_x_valid;
  return EIF_OK;
}

int launch_exchange(eif_ctx *c) {
  if (c->np == 0) {
    EIF_PROF(c, "ibm_gather", 0);
    EIF_CK(c, cudaMemsetAsync(c->dux, 0, sizeof(double) * c->nfield, c->stream));
    EIF_CK(c, cudaMemsetAsync(c->duy, 0, sizeof(double) * c->nfield, c->stream));
    return EIF_OK;
  }
  int rc;
  if ((rc = launch_exchange_tasks(c)) || (rc = launch_exchange_sums(c))) return rc;
  if (!(c->boxes_x_valid && c->bands_x_valid) && (rc = launch_band_lists(c))) return rc;
  return launch_gather(c);
}

// the field response from the tasks' contributions and the band lists
int launch_gather(eif_ctx *c) {
  GatherArgs g;
  g.edesc = c->edesc; g.wbuf = c->wbuf;
  g.dux = c->dux; g.duy = c->duy; g.flags = c->d_flags;
  g.np = c->np; g.itot = c->itot; g.jtot = c->jtot; g.ld = c->ld;
  g.bd = bounds_of(c);
  g.lists = c->band_lists; g.counts = c->band_counts; g.cap = c->band_cap;
  dim3 grid((c->itot + GTX - 1) / GTX, (c->jtot + GTY - 1) / GTY);
  EIF_PROF(c, "ibm_gather", 2);
  const int nhalo = 2 * (c->itot + 2) + 2 * c->jtot;
  if (c->cfg.precision == EIF_PREC_MIXED) {
    k_gather<float2, float><<<grid, GTHREADS, 0, c->stream>>>(g);
    EIF_LAUNCH_CK(c);
    k_ibm_halo<float><<<(nhalo + 255) / 256, 256, 0, c->stream>>>(reinterpret_cast<float *>(c->dux),
                                                                  reinterpret_cast<float *>(c->duy), c->itot,
                                                                  c->jtot, c->ld);
  } else {
    k_gather<double2, double><<<grid, GTHREADS, 0, c->stream>>>(g);
    EIF_LAUNCH_CK(c);
    k_ibm_halo<double><<<(nhalo + 255) / 256, 256, 0, c->stream>>>(c->dux, c->duy, c->itot, c->jtot, c->ld);
  }
  EIF_LAUNCH_CK(c);
  return EIF_OK;
}

}  // namespace eif

// ---------------------------------------------------------------------------
// Transposed box evaluations for the discrete adjoint (double precision).
//
// The inertia integrals I = sum_cells w_v(D) (u_c, r x u_c) dxdy / (m, I_z)
// (inertia.c:41-52) and the exchange sums F = -sum_cells w_s(D) (U_r - u_c) dxdy
// / (dt m, dt I_z) with the field response dux = sum w_s (U_r - u_c)
// (exchange.c:61-76) depend on the cell velocities u_c (face averages), on the
// particle velocities U, Omega, and on the centre and angle through the lever arm
// r = x - X and the signed distance D = d/h of the cell centre. With q = R(-az) r
// the body-frame offset and the distance computed through the normal foot
// (ellipse.c:30-65), dD/dq at the foot is minus the outward unit normal over h
// (the foot parameter is stationary, so it does not contribute), hence
//   dD/dX = -g,   dD/daz = g_x r_y - g_y r_x,   g = R(az) dD/dq.
// w_v = (1 + tanh(2D))/2 has dw_v/dD = w_s, and w_s = 1 - tanh^2(2D) has
// dw_s/dD = -4 tanh(2D) w_s.
//
// One warp per box row task as in k_ibm_work. Per cell the kernel writes the cell
// cotangent of the face-averaged velocity into the scratch buffer (gathered per
// cell afterwards in the fixed order of the forward exchange) and sums per task the
// cotangents of (X, Y, az) and (U, V, Omega). Boxes are those of the forward
// evaluation (the loop bounds are piecewise constant in the positions).
namespace {

struct AdjWorkArgs {
  const double *P;
  const double *pd;         // per-particle parameters at the boxes' positions (PD_WORDS each)
  const double2 *tanh_tab;
  const double *ux, *uy, *xc, *yc, *dt;
  const int *off;
  const int4 *tdesc;
  const double *bar;        // 3 x np: inertia cotangent (mode 0) or force cotangent (mode 1)
  const double *gx, *gy;    // mode 1: cell cotangents of the field response
  double *part;             // 6 per task
  double2 *wbuf;
  double *geom;             // geo 1/2: per task slot th, gwx, gwy (3 x slots, by component)
  long long nslot;
  int geo;
  int pcap, np, ld, mode;
  double dx, dy, ly;
  Bounds bd;
};

__global__ void __launch_bounds__(256) k_ibm_adj(AdjWorkArgs a) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int total = EIF_CHK(a.bd.rec, a.np, a.bd.off, 70) ? __ldg(a.off + a.np) : 0;
  const double dxdy = a.dx * a.dy;
  const double kdt = a.mode == 1 ? dxdy / __ldg(a.dt) : 0.;
  const int pc = a.pcap, ld = a.ld;
  for (int c = warp; c < total; c += nwarps) {
    if (!EIF_CHK(a.bd.rec, 6LL * c + 5, 6LL * (a.bd.partial / 3), 71)) continue;
    const int4 dsc = __ldg(a.tdesc + c);
    const int n = dsc.x;
    if (!EIF_CHK(a.bd.rec, n, a.np, 72)) continue;
    RowTask t;
    const bool task = task_of(dsc, a.np, t) && EIF_CHK(a.bd.rec, t.j, a.bd.yc - 1, 73);
    const double *P = a.P;
    const double *pd = a.pd + (size_t)PD_WORDS * n;
    const float *pdf = reinterpret_cast<const float *>(pd + PD_F);
    const double px = __ldg(pd + PD_X), py_ = __ldg(pd + PD_Y) + a.ly * (task ? t.img : 0);
    const double rpm = __ldg(pd + PD_RPM), rpim = __ldg(pd + PD_RPIM);
    const double pux = __ldg(P + EIF_P_UX * pc + n), puy = __ldg(P + EIF_P_UY * pc + n), pvz = __ldg(P + EIF_P_VZ * pc + n);
    // cotangents per unit mass and moment of inertia
    const double kf = a.mode == 1 ? kdt : 1.;
    const double b0 = __ldg(a.bar + n) * (kf * rpm), b1 = __ldg(a.bar + a.np + n) * (kf * rpm),
                 b2 = __ldg(a.bar + 2 * a.np + n) * (kf * rpim);
    const double cz = __ldg(pd + PD_CZ), sz = __ldg(pd + PD_SZ), pa = __ldg(pd + PD_A), pb = __ldg(pd + PD_B);
    EllF ef;
    ef.a = __ldg(pdf + PDF_A); ef.b = __ldg(pdf + PDF_B); ef.kex = __ldg(pdf + PDF_KEX); ef.key = __ldg(pdf + PDF_KEY);
    ef.cz = eifd::d2f(cz); ef.sz = eifd::d2f(sz);
    const int j = task ? t.j : 1;
    const double y = __ldg(a.yc + j);
    const double ry = y - py_;
    float olo, ohi, ilo, ihi;
    row_chords(__ldg(pdf + PDF_AL), __ldg(pdf + PDF_KA), __ldg(pdf + PDF_DE), __ldg(pdf + PDF_SO2), __ldg(pdf + PDF_SI2),
               __ldg(pdf + PDF_RO2), eifd::d2f(ry), olo, ohi, ilo, ihi);
    double sX = 0., sY = 0., sA = 0., sU = 0., sV = 0., sW = 0.;
#pragma unroll 1
    for (int half = 0; half < CHUNK / 32; half++) {
      const int i = (task ? t.ib : 1) + half * 32 + lane;
      bool in = task && i <= t.ie;
      if (in) {
        in = EIF_CHK(a.bd.rec, i, a.bd.xc - 1, 74) && EIF_CHK(a.bd.rec, j * ld + i, a.bd.field, 75) &&
             EIF_CHK(a.bd.rec, (j + 1) * ld + i, a.bd.field, 76) && EIF_CHK(a.bd.rec, j * ld + (i - 1), a.bd.field, 77);
      }
      double2 contrib = make_double2(0., 0.);
      if (in) {
        const double x = __ldg(a.xc + i);
        const double rx = x - px;
        double th, gwx = 0., gwy = 0.;
        const long long slot = (long long)c * CHUNK + half * 32 + lane;
        const bool cached = a.geo == 2 && EIF_CHK(a.bd.rec, slot, a.nslot, 81);
        if (cached) {
          th = a.geom[slot];
          gwx = a.geom[a.nslot + slot];
          gwy = a.geom[2 * a.nslot + slot];
        } else {
          // far cells (row_chords): tanh(2D) is +-1 in double precision and both weights'
          // derivatives vanish
          const float Xf = eifd::d2f(rx);
          const int side = !(Xf > olo && Xf < ohi) ? -1 : ((Xf >= ilo && Xf <= ihi) ? 1 : 0);
          if (side != 0) {
            th = side > 0 ? 1. : -1.;
          } else {
            // g = R(az) dD/dq, dD/dq = -n / h with the outward normal n at the foot; cz and
            // sz carry the factor BETA / h
            double nx, ny;
            float c0, s0, d0;
            const double qx = fma(cz, rx, -(sz * ry)), qy = fma(sz, rx, cz * ry);
            foot_f(ef, eifd::d2f(fabs(qx)), eifd::d2f(fabs(qy)), c0, s0, d0);
            th = indicator_d<true>(pa, pb, ef.a * ef.b, c0, s0, qx, qy, a.tanh_tab, nx, ny);
            gwx = (-1. / BETA) * fma(cz, nx, sz * ny);
            gwy = (-1. / BETA) * fma(cz, ny, -(sz * nx));
          }
        }
        if (a.geo == 1 && EIF_CHK(a.bd.rec, slot, a.nslot, 82)) {
          a.geom[slot] = th;
          a.geom[a.nslot + slot] = gwx;
          a.geom[2 * a.nslot + slot] = gwy;
        }
        const double ws = 0.5 * BETA * (1. - th * th);
        const double uxf = 0.5 * (__ldg(a.ux + j * ld + (i - 1)) + __ldg(a.ux + j * ld + i));
        const double uyf = 0.5 * (__ldg(a.uy + j * ld + i) + __ldg(a.uy + (j + 1) * ld + i));
        const double dDdaz = gwx * ry - gwy * rx;
        if (a.mode == 0) {
          const double wv = 0.5 * (1. + th);
          const double cx = b0, cy = b1, cw = b2;
          contrib = make_double2(wv * dxdy * (cx - cw * ry), wv * dxdy * (cy + cw * rx));
          const double sv = dxdy * (cx * uxf + cy * uyf + cw * (-ry * uxf + rx * uyf));
          const double dw = ws * sv;
          sX += -dw * gwx - wv * dxdy * cw * uyf;
          sY += -dw * gwy + wv * dxdy * cw * uxf;
          sA += dw * dDdaz;
        } else {
          const int cc = j * ld + i;
          const double urx = pux - pvz * ry, ury = puy + pvz * rx;
          const double ex = urx - uxf, ey = ury - uyf;
          const double Cx = __ldg(a.gx + cc) - b0 + b2 * ry;
          const double Cy = __ldg(a.gy + cc) - b1 - b2 * rx;
          const double Ex = ws * Cx, Ey = ws * Cy;
          contrib = make_double2(-Ex, -Ey);
          sU += Ex;
          sV += Ey;
          sW += -ry * Ex + rx * Ey;
          const double dw = (ex * Cx + ey * Cy) * (-2. * BETA * th * ws);
          sX += -dw * gwx - pvz * Ey + b2 * ws * ey;
          sY += -dw * gwy + pvz * Ex - b2 * ws * ex;
          sA += dw * dDdaz;
        }
      }
      if (EIF_CHK(a.bd.rec, (long long)c * CHUNK + half * 32 + lane, a.bd.wbuf, 78))
        a.wbuf[(size_t)c * CHUNK + half * 32 + lane] = contrib;
    }
    sX = eifd::warp_sum(sX);
    sY = eifd::warp_sum(sY);
    sA = eifd::warp_sum(sA);
    sU = eifd::warp_sum(sU);
    sV = eifd::warp_sum(sV);
    sW = eifd::warp_sum(sW);
    if (lane == 0) {
      double *q = a.part + 6 * (size_t)c;
      q[0] = sX; q[1] = sY; q[2] = sA; q[3] = sU; q[4] = sV; q[5] = sW;
    }
  }
}

// per-particle sums of the task cotangents in task order: out[k * np + n]
__global__ void k_adj_chunk_reduce(const double *__restrict__ part, const int *__restrict__ off,
                                   double *__restrict__ out, int np, Bounds bd) {
  const int lane = threadIdx.x & 31;
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (n >= np) return;
  if (!EIF_CHK(bd.rec, n + 1, bd.off, 79)) return;
  const int c0 = off[n], c1 = off[n + 1];
  double s[6] = {0., 0., 0., 0., 0., 0.};
  for (int c = c0 + lane; c < c1; c += 32) {
    if (!EIF_CHK(bd.rec, 6LL * c + 5, 6LL * (bd.partial / 3), 80)) break;
#pragma unroll
    for (int k = 0; k < 6; k++) s[k] += part[6 * (size_t)c + k];
  }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double v = eifd::warp_sum(s[k]);
    if (lane == 0) out[(size_t)k * np + n] = v;
  }
}

}  // namespace

namespace eif {

int launch_adj_pass(eif_ctx *c, const AdjPass &p) {
  if (c->np == 0) return EIF_OK;
  if (p.use_increment) c->incr_zero = false;
  int rc = launch_boxes(c, p.use_increment);
  if (rc) return rc;
  AdjWorkArgs w;
  w.P = c->P; w.pd = c->pd; w.tanh_tab = c->tanh_tab; w.ux = p.ux; w.uy = p.uy; w.xc = c->xc; w.yc = c->yc; w.dt = c->d_scal;
  w.off = c->chunk_off; w.tdesc = c->tdesc;
  w.bar = p.bar; w.gx = p.gx; w.gy = p.gy;
  w.part = p.part;
  w.wbuf = reinterpret_cast<double2 *>(c->wbuf);
  w.geom = p.geom;
  w.nslot = (long long)c->wcap;
  w.geo = p.geom ? p.geo : 0;
  w.pcap = c->pcap; w.np = c->np; w.ld = c->ld; w.mode = p.mode;
  w.dx = c->dx; w.dy = c->dy; w.ly = c->ly;
  w.bd = bounds_of(c);
  const int blocks = std::max(1, std::min(c->sms * 8, (c->chunk_cap * 32 + 255) / 256));
  k_ibm_adj<<<blocks, 256, 0, c->stream>>>(w);
  EIF_LAUNCH_CK(c);
  k_adj_chunk_reduce<<<(c->np * 32 + 255) / 256, 256, 0, c->stream>>>(p.part, c->chunk_off, p.out, c->np,
                                                                        bounds_of(c));
  EIF_LAUNCH_CK(c);
  if ((rc = band_lists_of_boxes(c))) return rc;
  GatherArgs g;
  g.edesc = c->edesc; g.wbuf = c->wbuf;
  g.dux = p.fx; g.duy = p.fy; g.flags = c->d_flags;
  g.np = c->np; g.itot = c->itot; g.jtot = c->jtot; g.ld = c->ld;
  g.bd = bounds_of(c);
  g.lists = c->band_lists; g.counts = c->band_counts; g.cap = c->band_cap;
  dim3 grid((c->itot + GTX - 1) / GTX, (c->jtot + GTY - 1) / GTY);
  k_gather<double2, double><<<grid, GTHREADS, 0, c->stream>>>(g);
  EIF_LAUNCH_CK(c);
  return EIF_OK;
}

int adj_chunk_cap(const eif_ctx *c) { return c->chunk_cap; }
size_t adj_slot_cap(const eif_ctx *c) { return c->wcap; }

}  // namespace eif
