// Sub-iterations of the particles (src/main.c:36-50) in one persistent kernel per RK stage:
// of one suspension (eif_advance) or of many (a batch, batch.cu, whose stage fronts join
// before the kernel and fork after it).
//
// The kernel's CTAs (all resident: a cooperative launch) loop over the sub-iterations. The
// work of one is a list of units, the collision forces of PAIR_WARPS particles each, and for
// every particle ns slices of the row tasks of its inertia integrals:
//  * a slice forms the boxes and parameters of its particle at X + dX in shared memory
//    (box_warps) and runs its share of the particle's tasks, a warp per task; in the first
//    sub-iteration, where the increments are zero, it runs the
//    stage front's tasks with their stored weights;
//  * every unit counts itself at its particles; the last one of a particle sums the tasks,
//    forms the increments (increment.c) and raises the suspension's residual.
// Nothing else orders the units of a sub-iteration: the new increments go to the records, the
// centres that the collisions of other particles may still be reading are a list of their own
// (two, alternating). One grid barrier ends the sub-iteration; every CTA then evaluates the
// stopping rule of each suspension (main.c:40-48: go on while the residual is not below 1e-8
// and at most 101 sub-iterations ran) from the same residuals, so all agree on the set still
// iterating. When none is left the kernel updates every suspension's particles (update.c) and,
// before stages 1 and 2, resets their increments (reset.c).
//
// As a loop of kernels (boxes, task table, indicator, sums, collisions, increments: a
// conditional node of the step graph) a sub-iteration was eight launches in a row of 2 to 7 us
// each, about 30 us before any real work.
//
// Every body is the one of the stand-alone kernels (ibm_device.cuh, particle_device.cuh) with
// the same decomposition per task and particle, so each suspension gets the same bits as from
// those.
//
// The grid barrier is an arrival counter per stage, zeroed with the particles' counters by a
// memset node at the start of every step and polled with acquire loads. A poll gives up after
// 2^22 tries: the CTA sets the plan's error word, which makes the others give up at their next
// poll, and every suspension's EIF_FLAG_TIMEOUT, and the CTAs return. Data that one CTA writes
// and another reads is read with ordinary loads, not through the read-only path. For the tests
// of that bounded wait, EIF_TEST_HOLD_BARRIER=1 in the environment when a batch's graph is
// built keeps CTA 0 of the first stage's kernel from arriving at its first barrier: the other
// CTAs give up, and the step reports it.
//
// Where a context alone cannot have the kernel (no cooperative launch, no room for its grid or its
// buffers) its steps run the loops of kernels, with the same results (stage_off). For the tests of
// that, EIF_TEST_NO_STAGE_KERNEL=1 in the environment makes subiter_plan_create fail.
#ifndef EIF_CHECK
#define EIF_CHECK 1
#endif
#include "eif_internal.cuh"
#include "ibm_device.cuh"
#include "particle_device.cuh"
#include <algorithm>
#include <cstdlib>

namespace {

// one suspension's sub-iteration loop in one RK stage
struct SubDesc {
  BoxArgs box;     // boxes at X + dX
  WorkArgs work;   // inertia integrals at X + dX (mode 0, integrals 1)
  double *P;
  int pcap, np, ns, mixed;       // ns: slices per particle
  int *cnt, *off;                // tasks at X + dX, first tasks at X
  const int *base;               // first task slots at X + dX (fixed, from the radii)
  double2 *pos[2];               // centres X + dX
  float4 *near[2];               // the same for the partner search (pair_prefilter)
  unsigned *arr;                 // units of the particle that are done
  double ly, lx, gamma, Fr2;
  double *scal;                  // [0] dt, [1] residual
  unsigned *flags, *counter;     // error flags, the stage's sub-iteration count
  unsigned long long *total;     // sub-iterations run (eif_counters)
};

struct StageArgs {
  const SubDesc *d;
  int n;
  int reset_next;               // the particles' increments are reset for a following stage
  int hold;                     // a CTA that does not arrive at the first barrier (tests), or -1
  unsigned *sync;               // [0] arrivals, [1] error, [2..4] units taken (by sub-iteration mod 3)
  unsigned long long *res;      // three residual words per suspension (by sub-iteration mod 3)
  double *tape;                 // dX after sub-iteration m to tape + 3 np m (one suspension), or null
  int *contact;                 // with tape: set where a collision force is not zero
};

constexpr int SUB_THREADS = 256;
constexpr int SUB_WARPS = SUB_THREADS / 32;
constexpr int SUB_MAX = (int)eif::SUBITER_MAX;
constexpr unsigned SUB_CAP = 102;      // the stopping rule ends every loop by the 102nd sub-iteration
constexpr unsigned SPIN_MAX = 1u << 22;
constexpr int SYNC_WORDS = 32;         // per stage (arrivals, error word, unit counters; padded)
static_assert(PAIR_WARPS == SUB_WARPS, "units of the sub-iterations");

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// adds 1, ordering what this thread has seen and written before with what it does after
__device__ __forceinline__ unsigned atom_acq_rel(unsigned *p) {
  unsigned v;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// grid barrier number idx (0, 1, ...) of this launch; false when it gave up. arrive:
// the CTA counts itself (false only for the tests of the bounded wait)
__device__ bool grid_barrier(unsigned *sync, unsigned idx, bool arrive) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = gridDim.x * (idx + 1u);
    int good = arrive && atom_acq_rel(sync) + 1u >= target;
    for (unsigned k = 0; !good && k < SPIN_MAX; k++) {
      good = ld_acquire(sync) >= target;
      if (!good && k % 16u == 15u) {
        if (ld_acquire(sync + 1) != 0u) break;
        __nanosleep(64);
      }
    }
    if (!good) atomicOr(sync + 1, 1u);
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// per suspension, in shared memory: the loop control, so that the units are found without
// loading the descriptors; running numbers of the units, collisions first, then slices
enum { ST_NP, ST_NS, ST_CEND, ST_SEND, ST_WORDS };

// a warp counts a unit of particle n as done; true (for all lanes) when it was the last one
__device__ __forceinline__ bool unit_done(const SubDesc &d, int n, int lane) {
  unsigned last = 0u;
  __syncwarp();
  if (lane == 0) {
    last = atom_acq_rel(d.arr + n) == (unsigned)d.ns ? 1u : 0u;   // ns slices and the collisions
    if (last) d.arr[n] = 0u;
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  __syncwarp();
  return last != 0u;
}

// What a particle's increments need and no unit of the sub-iteration writes, component k in
// lane k < 3 (x, y, rotation): loaded before the units are counted, so that the loads and the
// gravity's division are in flight with the counter's round trip.
struct FinishIn {
  double c0, f, i0, u, du, x, g, dt;
};
__device__ __forceinline__ FinishIn finish_load(const SubDesc &d, int n) {
  const int k = min(threadIdx.x & 31u, 2u);
  const double *p = d.P + n;
  const int pc = d.pcap;
  FinishIn v;
  v.c0 = p[(k == 0 ? EIF_P_CFX0 : (k == 1 ? EIF_P_CFY0 : EIF_P_CTZ0)) * pc];
  v.f = p[(k == 0 ? EIF_P_FUX : (k == 1 ? EIF_P_FUY : EIF_P_TVZ)) * pc];
  v.i0 = p[(k == 0 ? EIF_P_IUX0 : (k == 1 ? EIF_P_IUY0 : EIF_P_IVZ0)) * pc];
  v.u = p[(k == 0 ? EIF_P_UX : (k == 1 ? EIF_P_UY : EIF_P_VZ)) * pc];
  v.du = p[(k == 0 ? EIF_P_DUX : (k == 1 ? EIF_P_DUY : EIF_P_DVZ)) * pc];
  v.x = p[(k == 1 ? EIF_P_Y : EIF_P_X) * pc];
  v.dt = d.scal[0];
  v.g = k == 0 ? gravity_increment(d.gamma, v.dt, p[EIF_P_DEN * pc], d.Fr2) : 0.;
  return v;
}

// the particle's sums over its tasks q0 .. q1 - 1 and its increments (one warp), after its last unit
__device__ __forceinline__ void finish_particle(const SubDesc &d, int n, unsigned it, int q0, int q1,
                                                unsigned long long *res, const FinishIn &v, double *tape, int *contact) {
  const int lane = threadIdx.x & 31, k = min(lane, 2), pc = d.pcap;
  double *p = d.P + n;
  const double c1 = p[(k == 0 ? EIF_P_CFX1 : (k == 1 ? EIF_P_CFY1 : EIF_P_CTZ1)) * pc];
  const double i1 = d.mixed ? chunk_sum_f_warp(reinterpret_cast<const float *>(d.work.partial), q0, q1, d.box.bd)
                            : chunk_sum_warp(d.work.partial, q0, q1, d.box.bd);
  const double hgd = __dmul_rn(0.5 * d.gamma, v.dt);
  double du = velocity_increment(hgd, v.dt, v.c0, c1, v.f, v.i0, i1);
  if (k == 0) du = __dadd_rn(du, v.g);
  const double dx = position_increment(hgd, v.u, du);
  const double at = __dadd_rn(v.x, dx);
  // the largest change of the three as bits (non-negative; a NaN does not count, as in fmax)
  const double change = fabs(du - v.du);
  long long r = change > 0. ? __double_as_longlong(change) : 0ll;
  if (lane < 3) {
    p[(k == 0 ? EIF_P_IUX1 : (k == 1 ? EIF_P_IUY1 : EIF_P_IVZ1)) * pc] = i1;
    p[(k == 0 ? EIF_P_DUX : (k == 1 ? EIF_P_DUY : EIF_P_DVZ)) * pc] = du;
    p[(k == 0 ? EIF_P_DX : (k == 1 ? EIF_P_DY : EIF_P_DAZ)) * pc] = dx;
    const unsigned o = (it + 1u) & 1u;
    // the centre, rounded as load_pv forms it from the records, and pair_prefilter's values of it
    if (k < 2) {
      reinterpret_cast<double *>(d.pos[o] + n)[k] = at;
      reinterpret_cast<float *>(d.near[o] + n)[k] = eifd::d2f(at);
    } else {
      reinterpret_cast<float *>(d.near[o] + n)[2] = eifd::d2f(fmax(p[EIF_P_A * pc], p[EIF_P_B * pc]));
    }
    if (tape) {
      tape[(size_t)3 * d.np * (it + 1u) + (size_t)k * d.np + n] = dx;
      if (v.c0 != 0. || c1 != 0.) *contact = 1;
    }
  }
  r = max(r, max(__shfl_sync(0xffffffffu, r, 1), __shfl_sync(0xffffffffu, r, 2)));
  if (lane == 0 && r > 0ll) atomicMax(res, (unsigned long long)r);
}

__global__ void __launch_bounds__(SUB_THREADS, 2) k_subiterations(StageArgs s) {
  __shared__ unsigned act[SUB_MAX / 32];   // suspensions still iterating
  __shared__ WorkSlots slot_d[SUB_WARPS];   // of the double-precision form, or the mixed form's cells
  __shared__ __align__(16) int bx[12];
  __shared__ __align__(16) float pf[PF_WORDS];
  __shared__ __align__(16) double pd[PD_WORDS];
  __shared__ int unit[2];                  // suspension and unit within it
  // the descriptor of the suspension at hand: read in nearly every instruction of the units,
  // and from global memory again after every acquire (which empties L1)
  __shared__ __align__(16) unsigned sd_words[(sizeof(SubDesc) + 15) / 16 * 4];
  const SubDesc &d = *reinterpret_cast<const SubDesc *>(sd_words);
  int have = -1;
  extern __shared__ int stab[];            // ST_WORDS per suspension
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int G = gridDim.x, n = s.n;
  for (int q = threadIdx.x; q < SUB_MAX / 32; q += SUB_THREADS) {
    const int lo = 32 * q;
    act[q] = lo >= n ? 0u : (n - lo >= 32 ? 0xffffffffu : ((1u << (n - lo)) - 1u));
  }
  for (int j = threadIdx.x; j < n; j += SUB_THREADS) {
    stab[ST_WORDS * j + ST_NP] = s.d[j].np;
    stab[ST_WORDS * j + ST_NS] = s.d[j].ns;
  }
  __syncthreads();
  unsigned bar = 0;
  auto barrier = [&]() {
    const bool arrive = bar != 0u || (int)blockIdx.x != s.hold;
    return grid_barrier(s.sync, bar++, arrive);
  };
  bool ok = true;
  auto active = [&](int j) { return ((act[j >> 5] >> (j & 31)) & 1u) != 0u; };
  int ncoll = 0, units = 0;
  bool changed = true;
  for (unsigned it = 0; it < SUB_CAP; it++) {
    if (changed) {
      // the units of the suspensions still iterating
      if (threadIdx.x < 32) {
        int run = 0;
        for (int pass = 0; pass < 2; pass++) {
          for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + lane;
            int v = 0;
            if (j < n && active(j)) {
              const int np = stab[ST_WORDS * j + ST_NP];
              v = pass == 0 ? (np + PAIR_WARPS - 1) / PAIR_WARPS : np * stab[ST_WORDS * j + ST_NS];
            }
            int sc = v;
            for (int o = 1; o < 32; o <<= 1) {
              const int w = __shfl_up_sync(0xffffffffu, sc, o);
              if (lane >= o) sc += w;
            }
            if (j < n) stab[ST_WORDS * j + (pass == 0 ? ST_CEND : ST_SEND)] = run + sc;
            run += __shfl_sync(0xffffffffu, sc, 31);
          }
        }
      }
      __syncthreads();
      ncoll = stab[ST_WORDS * (n - 1) + ST_CEND];
      units = stab[ST_WORDS * (n - 1) + ST_SEND];
    }
    const unsigned m3 = it % 3u;
    // words of the next sub-iteration: last used two barriers ago
    if (blockIdx.x == 0) {
      for (int j = threadIdx.x; j < n; j += SUB_THREADS) s.res[3 * j + (it + 1u) % 3u] = 0ull;
      if (threadIdx.x == 0) s.sync[2 + (it + 1u) % 3u] = 0u;
    }
    // units in order: the first by the CTA's number, the next ones as CTAs come free
    int next = blockIdx.x;
    for (;;) {
      // with a CTA for every unit a CTA keeps its unit as long as the set does not change
      const bool kept = units <= G && !changed;
      if (!kept && threadIdx.x == 0) {
        const int u = next;
        if (units > G) next = G + (int)atomicAdd(s.sync + 2 + m3, 1u);
        else next = units;
        // the first suspension whose running number is above u
        const int col = u < ncoll ? ST_CEND : ST_SEND;
        int lo = 0, hi = n - 1;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (stab[ST_WORDS * mid + col] > u) hi = mid;
          else lo = mid + 1;
        }
        unit[0] = u < units ? lo : -1;
        unit[1] = u - (lo > 0 ? stab[ST_WORDS * (lo - 1) + col] : (col == ST_SEND ? ncoll : 0)) +
                  (col == ST_CEND ? (1 << 30) : 0);
      }
      if (!kept) __syncthreads();
      const int j = unit[0];
      if (j < 0) break;
      const bool coll = unit[1] >= (1 << 30);
      const int q = unit[1] & ((1 << 30) - 1);
      if (j != have) {
        const unsigned *src = reinterpret_cast<const unsigned *>(s.d + j);
        for (int w = threadIdx.x; w < (int)(sizeof(SubDesc) / sizeof(unsigned)); w += SUB_THREADS) sd_words[w] = src[w];
        have = j;
        __syncthreads();
      }
      unsigned long long *res = s.res + 3 * j + m3;
      if (coll) {
        collision_block(it > 0 ? Places{d.pos[it & 1u], d.near[it & 1u], false} : Places{nullptr, nullptr, true}, d.P, d.pcap, d.np, 1, d.ly, d.lx, d.flags, q);
        const int k = q * PAIR_WARPS + wl;
        if (k < d.np) {
          const FinishIn in = finish_load(d, k);
          const int c0 = it == 0 ? d.off[k] : d.base[k];
          if (unit_done(d, k, lane))
            finish_particle(d, k, it, c0, it == 0 ? d.off[k + 1] : c0 + d.cnt[k], res, in, s.tape, s.contact);
        }
      } else {
        const int p = q / d.ns, sl = q - p * d.ns;
        FinishIn in;
        if (wl == SUB_WARPS - 1) in = finish_load(d, p);
        int c0, cnt;
        if (it == 0) {
          c0 = d.off[p];
          cnt = d.off[p + 1] - c0;
          const int r0 = (int)((long long)cnt * sl / d.ns), r1 = (int)((long long)cnt * (sl + 1) / d.ns);
          if (d.mixed) {
            ibm_sum_f_tasks<false>(d.work, c0 + r0 + wl, SUB_WARPS, c0 + r1);
          } else {
            const OneParticle one{nullptr, nullptr, nullptr, p, 0, c0 + r1};
            ibm_work_tasks<false>(d.work, 2, c0 + r0 + wl, SUB_WARPS, slot_d[wl], &one);
          }
        } else {
          if (wl < 4) box_warps(d.box, p, wl, bx, d.mixed ? pf : nullptr, pd);
          __syncthreads();
          c0 = d.base[p];
          cnt = box_tasks(bx);
          const int r0 = (int)((long long)cnt * sl / d.ns), r1 = (int)((long long)cnt * (sl + 1) / d.ns);
          const OneParticle one{reinterpret_cast<const int4 *>(bx), pf, pd, p, c0, r1};
          if (d.mixed) {
            ibm_work_f_tasks<false, true>(d.work, 0, r0 + wl, SUB_WARPS, reinterpret_cast<WorkSlotsF &>(slot_d[wl]), &one);
            if (sl == 0 && wl == SUB_WARPS - 2 && d.work.memo_mode == 2) memo_particle(d.work.memo, pf, bx, one.base, p);
          } else {
            ibm_work_tasks<false>(d.work, 0, r0 + wl, SUB_WARPS, slot_d[wl], &one);
          }
          if (threadIdx.x == 0) d.cnt[p] = cnt;
        }
        __syncthreads();
        if (wl == SUB_WARPS - 1 && unit_done(d, p, lane)) finish_particle(d, p, it, c0, c0 + cnt, res, in, s.tape, s.contact);
      }
      if (units <= G) break;
    }
    if (!(ok = barrier())) break;
    // the stopping rule of every suspension, evaluated alike by all CTAs
    bool stop = false;
    for (int j = threadIdx.x; j < n; j += SUB_THREADS) {
      if (!active(j)) continue;
      const double r = __longlong_as_double((long long)*reinterpret_cast<volatile unsigned long long *>(s.res + 3 * j + m3));
      const unsigned count = it + 1u;
      if (!(!(r < 1.e-8) && count <= 101u)) {
        atomicAnd(&act[j >> 5], ~(1u << (j & 31)));
        stop = true;
      }
      if (blockIdx.x == 0) {
        const SubDesc &e = s.d[j];
        e.scal[1] = r;
        *e.counter = count;
        *e.total += 1ull;
      }
    }
    changed = __syncthreads_or(stop);
    bool any = false;
    for (int q = 0; q < SUB_MAX / 32; q++) any |= act[q] != 0u;
    if (!any) break;
  }
  if (!ok) {
    if (threadIdx.x == 0)
      for (int j = 0; j < n; j++) atomicOr(s.d[j].flags, EIF_FLAG_TIMEOUT);
    return;
  }
  // the particle update of the stage (update.c:8-34) and, before a following stage, the
  // reset of the increments (reset.c:7-18); the last increments were written before the
  // last grid barrier
  const int T = G * SUB_THREADS;
  int at = blockIdx.x * SUB_THREADS + threadIdx.x;
  for (int j = 0; j < n; j++) {
    const int np = stab[ST_WORDS * j + ST_NP];
    if (at < np) {
      const SubDesc &e = s.d[j];
      for (int m = at; m < np; m += T) {
        update_particle(e.P, e.pcap, m, e.ly);
        if (s.reset_next) reset_particle(e.P, e.pcap, m);
      }
    }
    at = (at + T - np % T) % T;   // the suspensions' particles spread over all CTAs
  }
}

}  // namespace

namespace eif {

struct SubiterPlan {
  int n = 0, grid = 0;
  std::vector<SubDesc> h;               // 3 stages x n (x 2 buffer indices, launch_stage_kernel)
  SubDesc *d_desc = nullptr;
  // zeroed at the start of every step: residuals (3 stages x 3n), then barriers and counters
  // (3 stages x SYNC_WORDS), then the particles' unit counters
  unsigned long long *d_res = nullptr;
  unsigned *d_sync = nullptr;
  size_t zero_words = 0;
  double2 *d_pos = nullptr;             // two lists of centres of all particles
  float4 *d_near = nullptr;             // the same for the partner search
  std::vector<int> first;               // first particle of every suspension in these arrays
  std::vector<int> ns;                  // slices per particle
  int np = 0;
  int hold = -1;                        // EIF_TEST_HOLD_BARRIER: CTA 0 of stage 0 held back
};

bool subiter_joinable(const eif_ctx *c) { return c->np <= TT_MAX_NP; }

// One suspension's loops in stage kernels: while every unit has a CTA of its own, np + np / 8 of
// them on two CTAs an SM, so up to 270 particles on 152 SMs. There the loop of kernels takes 1.05
// to 1.75 times as long; as soon as some CTAs have a second unit, a sub-iteration of the stage
// kernel takes two units' time, while the stand-alone indicator has 24 warps on an SM (16 here, for
// the registers of the fits) and no CTA-wide steps. Passes of some steps, loop over stage kernel:
//   256 x 512, 16 / 160 ellipses   double precision 1.34 / 1.17, mixed 1.75 / 1.37
//   512 x 1024, 270 / 340          1.17 / 0.94 (4.81 and 4.11 ms / 5.50 and 5.83), 1.18 / 0.99
//   768 x 1536, 270 / 320 / 640    1.10 / 0.90 / 0.97, 1.15 / 0.99 / 0.80
//   1024 x 2048, 256 / 320 / 768   1.06 / 0.91 / 0.98, 1.16 / 0.97 / 0.85
bool subiter_alone(const eif_ctx *c) {
  return c->np > 0 && !c->stage_off && c->np + (c->np + PAIR_WARPS - 1) / PAIR_WARPS <= 2 * c->sms;
}

void subiter_plan_destroy(SubiterPlan *p) {
  if (!p) return;
  if (p->d_desc) cudaFree(p->d_desc);
  if (p->d_res) cudaFree(p->d_res);
  if (p->d_pos) cudaFree(p->d_pos);
  if (p->d_near) cudaFree(p->d_near);
  delete p;
}

static int plan_fail(std::string *err, const char *what, cudaError_t e) {
  *err = std::string(what) + ": " + cudaGetErrorString(e);
  return EIF_ERR_CUDA;
}

int subiter_plan_create(eif_ctx *const *ctx, int n, SubiterPlan **out, std::string *err, int sets) {
  *out = nullptr;
  if (n <= 0 || n > SUB_MAX) {
    *err = "a stage kernel takes 1 to " + std::to_string(SUB_MAX) + " suspensions";
    return EIF_ERR_ARG;
  }
  const char *none = std::getenv("EIF_TEST_NO_STAGE_KERNEL");
  if (none && none[0] == '1') {
    *err = "EIF_TEST_NO_STAGE_KERNEL is set";
    return EIF_ERR_CUDA;
  }
  int coop = 0, occ = 0;
  cudaError_t e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx[0]->device);
  if (e != cudaSuccess) return plan_fail(err, "cudaDeviceGetAttribute", e);
  if (!coop) {
    *err = "the device has no cooperative launch";
    return EIF_ERR_CUDA;
  }
  // the loop-control table in dynamic shared memory: ST_WORDS ints per suspension
  e = cudaFuncSetAttribute(k_subiterations, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(sizeof(int) * ST_WORDS * SUB_MAX));
  if (e != cudaSuccess) return plan_fail(err, "cudaFuncSetAttribute", e);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_subiterations, SUB_THREADS, sizeof(int) * ST_WORDS * n);
  if (e != cudaSuccess) return plan_fail(err, "cudaOccupancyMaxActiveBlocksPerMultiprocessor", e);
  if (occ < 1) {
    *err = "the stage kernel does not fit on an SM";
    return EIF_ERR_CUDA;
  }
  SubiterPlan *p = new (std::nothrow) SubiterPlan;
  if (!p) return EIF_ERR_NOMEM;
  p->n = n;
  // slices: as many as give every CTA of the GPU a unit when the particles are few, none
  // without four tasks, one for each scheduler of an SM
  const int most = occ * ctx[0]->sms;
  long long units = 0;
  for (int j = 0; j < n; j++) {
    p->first.push_back(p->np);
    p->np += ctx[j]->np;
  }
  for (int j = 0; j < n; j++) {
    // a CTA to an SM where that leaves a warp a task: a second one would share the FP64 pipe of
    // the boxes (216 x 430 with 24 ellipses: boxes 6100 cycles with, 3700 without)
    const int np = std::max(1, p->np), sms = ctx[0]->sms;
    const int by_sm = (sms - (np + PAIR_WARPS - 1) / PAIR_WARPS) / np;
    const int by_gpu = by_sm >= 1 && ctx[j]->max_tasks <= by_sm * SUB_WARPS ? by_sm : std::max(1, most / np);
    const int by_tasks = std::max(1, (ctx[j]->max_tasks + 3) / 4);
    p->ns.push_back(std::min(by_gpu, by_tasks));
    units += (long long)ctx[j]->np * p->ns[j] + (ctx[j]->np + PAIR_WARPS - 1) / PAIR_WARPS;
  }
  p->zero_words = (size_t)18 * n + 3 * SYNC_WORDS + p->np;
  p->grid = (int)std::max<long long>(1, std::min<long long>(most, units));
  p->h.assign((size_t)3 * sets * n, SubDesc{});
  if ((e = cudaMalloc((void **)&p->d_desc, sizeof(SubDesc) * p->h.size())) != cudaSuccess ||
      (e = cudaMalloc((void **)&p->d_pos, sizeof(double2) * std::max(1, 2 * p->np))) != cudaSuccess ||
      (e = cudaMalloc((void **)&p->d_near, sizeof(float4) * std::max(1, 2 * p->np))) != cudaSuccess ||
      (e = cudaMalloc((void **)&p->d_res, sizeof(unsigned) * p->zero_words)) != cudaSuccess) {
    subiter_plan_destroy(p);
    return plan_fail(err, "cudaMalloc", e);
  }
  p->d_sync = reinterpret_cast<unsigned *>(p->d_res + (size_t)9 * n);
  *out = p;
  return EIF_OK;
}

static void describe(SubiterPlan *p, SubDesc &d, int rk, int j, const eif_ctx *c) {
  d.box = box_args(c, true);
  d.work = work_args(c, 0, 1);
  // the evaluations with geometry (sub-iterations after the first) store their weights
  if (c->cfg.precision == EIF_PREC_MIXED) d.work.memo_mode = 2;
  d.P = c->P;
  d.pcap = c->pcap;
  d.np = c->np;
  d.ns = p->ns[j];
  d.base = c->task_base;
  for (int k = 0; k < 2; k++) {
    d.pos[k] = p->d_pos + (size_t)k * p->np + p->first[j];
    d.near[k] = p->d_near + (size_t)k * p->np + p->first[j];
  }
  d.arr = p->d_sync + 3 * SYNC_WORDS + p->first[j];
  d.mixed = c->cfg.precision == EIF_PREC_MIXED ? 1 : 0;
  d.cnt = c->np > 0 ? c->chunk_off + (c->np + 1) : nullptr;
  d.off = c->chunk_off;
  d.ly = c->ly;
  d.lx = c->lx;
  d.gamma = rk_coef(rk).gamma;
  d.Fr2 = c->cfg.Fr * c->cfg.Fr;
  d.scal = c->d_scal;
  d.flags = c->d_flags;
  d.counter = c->d_sub + rk;
  d.total = c->d_inc + 2;
}

void subiter_describe(SubiterPlan *p, int rk, int j, const eif_ctx *c) {
  describe(p, p->h[(size_t)rk * p->n + j], rk, j, c);
}

void subiter_test_hold(SubiterPlan *p) {
  const char *hold = std::getenv("EIF_TEST_HOLD_BARRIER");
  p->hold = hold && hold[0] == '1' ? 0 : -1;
}

int subiter_add_reset(SubiterPlan *p, cudaGraph_t g, cudaGraphNode_t *node, std::string *err) {
  cudaMemsetParams m = {};
  m.dst = p->d_res;
  m.value = 0;
  m.elementSize = sizeof(unsigned);
  m.width = p->zero_words;
  m.height = 1;
  const cudaError_t e = cudaGraphAddMemsetNode(node, g, nullptr, 0, &m);
  return e == cudaSuccess ? EIF_OK : plan_fail(err, "cudaGraphAddMemsetNode", e);
}

// arguments of stage rk's kernel with the descriptors d
static StageArgs stage_args(SubiterPlan *p, int rk, const SubDesc *d) {
  StageArgs a;
  a.d = d;
  a.n = p->n;
  a.sync = p->d_sync + SYNC_WORDS * rk;
  a.res = p->d_res + (size_t)3 * p->n * rk;
  a.reset_next = rk < 2 ? 1 : 0;
  a.hold = rk == 0 ? p->hold : -1;
  a.tape = nullptr;
  a.contact = nullptr;
  return a;
}

int subiter_add_stage(SubiterPlan *p, int rk, cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps,
                      cudaGraphNode_t *node, std::string *err) {
  StageArgs a = stage_args(p, rk, p->d_desc + (size_t)rk * p->n);
  void *args[] = {&a};
  cudaKernelNodeParams k = {};
  k.func = reinterpret_cast<void *>(k_subiterations);
  k.gridDim = dim3(p->grid);
  k.blockDim = dim3(SUB_THREADS);
  k.sharedMemBytes = (unsigned)(sizeof(int) * ST_WORDS * p->n);
  k.kernelParams = args;
  cudaError_t e = cudaGraphAddKernelNode(node, g, deps.data(), deps.size(), &k);
  if (e != cudaSuccess) return plan_fail(err, "cudaGraphAddKernelNode", e);
  cudaKernelNodeAttrValue v = {};
  v.cooperative = 1;
  e = cudaGraphKernelNodeSetAttribute(*node, cudaKernelNodeAttributeCooperative, &v);
  return e == cudaSuccess ? EIF_OK : plan_fail(err, "cudaGraphKernelNodeSetAttribute (cooperative)", e);
}

// The kernels that read the descriptors run on streams that do not wait for the null stream, and a
// copy from pageable memory may return before it has reached the device: it is waited for here.
int subiter_upload(SubiterPlan *p, std::string *err) {
  cudaError_t e = cudaMemcpy(p->d_desc, p->h.data(), sizeof(SubDesc) * p->h.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  return e == cudaSuccess ? EIF_OK : plan_fail(err, "cudaMemcpy (stage descriptors)", e);
}

int stage_kernel_prepare(eif_ctx *c) {
  std::string err;
  int rc;
  if (c->stage_plan && c->stage_gen != c->buf_gen) {
    subiter_plan_destroy(c->stage_plan);
    c->stage_plan = nullptr;
  }
  if (!c->stage_plan) {
    SubiterPlan *p = nullptr;
    if (subiter_plan_create(&c, 1, &p, &err, 2)) {
      cudaGetLastError();
      c->stage_off = true;
      return EIF_OK;
    }
    const int cur = c->cur;
    for (int k = 0; k < 6; k++) {
      c->cur = k / 3;
      describe(p, p->h[k], k % 3, 0, c);
    }
    c->cur = cur;
    if ((rc = subiter_upload(p, &err))) {
      subiter_plan_destroy(p);
      return fail(c, rc, "stage kernel: %s", err.c_str());
    }
    c->stage_plan = p;
    c->stage_gen = c->buf_gen;
  }
  return EIF_OK;
}

int launch_stage_kernel(eif_ctx *c, int rk, double *tape, int *contact) {
  SubiterPlan *p = c->stage_plan;
  EIF_CK(c, cudaMemsetAsync(p->d_res, 0, sizeof(unsigned) * p->zero_words, c->stream));
  StageArgs a = stage_args(p, rk, p->d_desc + 3 * c->cur + rk);
  a.reset_next = 0;
  a.tape = tape;
  a.contact = contact;
  void *args[] = {&a};
  EIF_CK(c, cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_subiterations), dim3(p->grid), dim3(SUB_THREADS), args,
                                        sizeof(int) * ST_WORDS, c->stream));
  EIF_LAUNCH_CK(c);
  c->incr_zero = false;
  c->boxes_x_valid = false;
  c->weights_x_valid = false;
  return EIF_OK;
}

}  // namespace eif
