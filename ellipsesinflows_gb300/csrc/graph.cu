// Step graphs: one time step of eif_advance as a single CUDA graph.
//
// The graph holds, in launch order, the dt decision and for each RK stage the
// stage kernels and one persistent kernel for its particle sub-iterations and the
// particle update (subiter.cu; src/main.c:13-53). Work that the stage driver puts on the side
// stream is captured as a parallel branch of the same graph. A step needs
// no host round trip; the host synchronises once per step to read dt and the
// error flags. The kernels' bodies and their order are those of the host-driven path
// (rk_stage), so both paths give bit-identical results. Contexts of many particles
// (subiter_alone) have a conditional WHILE node per stage whose body is one
// sub-iteration; the last block of k_sub_end sets its condition.
//
// The stage kernels swap the double-buffered velocity and source arrays, so the
// buffers a step touches depend on the buffer indices at its start; one graph
// is kept per starting pair of indices (at most two occur). Graphs are rebuilt
// after the particle buffers are reallocated.
#include "eif_internal.cuh"
#include <string>
#include <vector>

namespace eif {

namespace {

int end_capture(eif_ctx *c, std::vector<cudaGraphNode_t> *sinks) {
  if (sinks) {
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t *deps = nullptr;
    size_t n = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(c->stream, &st, nullptr, nullptr, &deps, nullptr, &n);
    if (e == cudaSuccess) sinks->assign(deps, deps + n);
    cudaGraph_t g = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(c->stream, &g);
    if (e != cudaSuccess) return check_cuda(c, e, "cudaStreamGetCaptureInfo");
    if (e2 != cudaSuccess) return check_cuda(c, e2, "cudaStreamEndCapture");
    return EIF_OK;
  }
  cudaGraph_t g = nullptr;
  EIF_CK(c, cudaStreamEndCapture(c->stream, &g));
  return EIF_OK;
}

// abandon a capture after an error, leaving the streams usable
void abort_capture(eif_ctx *c) {
  for (cudaStream_t s : {c->stream, c->side}) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (s && cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(s, &g);
      if (g) cudaGraphDestroy(g);
    }
  }
  cudaGetLastError();
  c->in_loop = false;
}

}  // namespace

// Host state of c before the capture of a step: the graph must not depend on boxes
// computed before it, so it starts without them.
int step_capture_begin(eif_ctx *c) {
  int rc = ibm_prepare(c);
  if (rc) return rc;
  c->boxes_x_valid = false;
  c->weights_x_valid = false;
  c->incr_zero = false;
  return EIF_OK;
}

// Host state of c after the capture of a step (or after a failed capture): nothing
// has run yet, so the step starts from the buffers (cur0, scur0); the step ends with
// new positions, so no boxes are valid after it.
void step_capture_end(eif_ctx *c, int cur0, int scur0) {
  abort_capture(c);
  c->cur = cur0;
  c->scur = scur0;
  c->boxes_x_valid = false;
  c->weights_x_valid = false;
}

// Captures part `part` of one time step of c into g after the nodes deps (none: an
// independent branch) and returns its last nodes in sinks. Part 0 is the dt decision
// and the front of RK stage 0 (src/main.c:14-35), parts 1 and 2 the particle update
// of the stage before (main.c:51-53) and the front of the next stage, part 3 the
// particle update of stage 2. The sub-iteration loops (main.c:36-50) go between the
// parts: a conditional node per context (capture_subiteration_loop), or one kernel (for
// all the suspensions of a batch), which then also updates the particles at the end of the
// stage and resets the increments for the next (particles_in_stage_kernel: those launches
// are left out of parts 1-3). fields_event: ev_fields is recorded once the fields are final.
// with_dt: false leaves the dt decision out (eif_integrate).
int capture_step_part(eif_ctx *c, cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps, int part,
                      std::vector<cudaGraphNode_t> *sinks, bool particles_in_stage_kernel, bool fields_event, bool with_dt) {
  cudaError_t e = cudaStreamBeginCaptureToGraph(c->stream, g, deps.data(), nullptr, deps.size(),
                                                cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaStreamBeginCaptureToGraph");
  int rc;
  if (part > 0) {
    // after a sub-iteration loop: the increments are not zero and the boxes of the
    // loop's last positions are not those at X
    c->incr_zero = false;
    c->boxes_x_valid = false;
    c->weights_x_valid = false;
    c->bands_x_valid = false;
    if (!particles_in_stage_kernel && (rc = launch_update_particles(c))) return rc;
  }
  if (part < 3) {
    c->reset_in_stage_kernel = particles_in_stage_kernel && part > 0;
    rc = rk_stage_front(c, part, part == 0 && with_dt);
    c->reset_in_stage_kernel = false;
    if (rc) return rc;
  }
  if (part == 2 && fields_event && c->ev_fields) {
    // the last stage's projection is done: the fields are final for this step
    // (eif_advance_pull copies them to the host beside the particle work that follows)
    const cudaError_t e = cudaEventRecordWithFlags(c->ev_fields, c->stream, cudaEventRecordExternal);
    if (e != cudaSuccess) return check_cuda(c, e, "cudaEventRecordWithFlags (fields)");
  }
  return end_capture(c, sinks);
}

// The sub-iteration loop of RK stage rk of c as a conditional WHILE node after the
// nodes deps (its counter reset before it); sinks = {the loop node}. The last block
// of k_sub_end sets the loop condition on the device. Without particles one
// sub-iteration is all there is: no loop.
int capture_subiteration_loop(eif_ctx *c, cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps, int rk,
                              std::vector<cudaGraphNode_t> *sinks) {
  std::vector<cudaGraphNode_t> tail;
  cudaError_t e = cudaStreamBeginCaptureToGraph(c->stream, g, deps.data(), nullptr, deps.size(),
                                                cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaStreamBeginCaptureToGraph");
  // the sub-iteration counter starts at zero for every stage
  e = cudaMemsetAsync(reinterpret_cast<unsigned *>(c->d_inc + 1), 0, sizeof(unsigned), c->stream);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaMemsetAsync");
  int rc = c->np == 0 ? sub_iteration(c, rk) : EIF_OK;
  if (rc || (rc = end_capture(c, &tail))) return rc;
  if (c->np == 0) {
    *sinks = tail;
    return EIF_OK;
  }
  cudaGraphConditionalHandle h;
  e = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaGraphConditionalHandleCreate");
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t loop = nullptr;
  e = cudaGraphAddNode(&loop, g, tail.data(), nullptr, tail.size(), &p);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaGraphAddNode (while)");
  cudaGraph_t body = p.conditional.phGraph_out[0];
  e = cudaStreamBeginCaptureToGraph(c->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaStreamBeginCaptureToGraph (body)");
  c->in_loop = true;
  c->loop_handle = h;
  // the body runs repeatedly with changing increments: it always computes its boxes
  c->incr_zero = false;
  c->boxes_x_valid = false;
  if ((rc = sub_iteration(c, rk))) return rc;
  c->in_loop = false;
  if ((rc = end_capture(c, nullptr))) return rc;
  sinks->assign(1, loop);
  return EIF_OK;
}

// the loop's count to the stage's place in d_sub
int capture_loop_count(eif_ctx *c, cudaGraph_t g, int rk, std::vector<cudaGraphNode_t> *tail) {
  cudaGraphNode_t n = nullptr;
  const cudaError_t e = cudaGraphAddMemcpyNode1D(&n, g, tail->data(), tail->size(), c->d_sub + rk, c->d_inc + 1,
                                                 sizeof(unsigned), cudaMemcpyDeviceToDevice);
  if (e != cudaSuccess) return check_cuda(c, e, "cudaGraphAddMemcpyNode1D");
  tail->assign(1, n);
  return EIF_OK;
}

// Captures one time step of c into g (appended as an independent branch: its first
// nodes have no dependences) and returns the buffer indices the step ends with. The
// host state of c is left as before the capture; on failure g may hold a partial
// branch and should be discarded.
int capture_step(eif_ctx *c, cudaGraph_t g, int *cur1, int *scur1, SubiterPlan **plan, bool with_dt) {
  int rc = step_capture_begin(c);
  if (rc) return rc;
  const int cur0 = c->cur, scur0 = c->scur;
  bool stage_kernels = plan && subiter_alone(c);
  SubiterPlan *p = nullptr;
  std::string err;
  std::vector<cudaGraphNode_t> tail;
  cudaGraphNode_t reset = nullptr;
  auto failed = [&](int code, bool stage) {
    subiter_plan_destroy(p);
    step_capture_end(c, cur0, scur0);
    return stage ? fail(c, code, "stage kernel: %s", err.c_str()) : code;
  };
  if (stage_kernels && subiter_plan_create(&c, 1, &p, &err)) {
    cudaGetLastError();
    c->stage_off = true;
    stage_kernels = false;
  }
  if (stage_kernels && (rc = subiter_add_reset(p, g, &reset, &err))) return failed(rc, true);
  for (int part = 0; part < 4; part++) {
    if ((rc = capture_step_part(c, g, tail, part, &tail, stage_kernels, true, with_dt))) return failed(rc, false);
    if (part == 3) break;
    if (stage_kernels) {
      subiter_describe(p, part, 0, c);
      if (part == 0) tail.push_back(reset);
      cudaGraphNode_t node = nullptr;
      if ((rc = subiter_add_stage(p, part, g, tail, &node, &err))) return failed(rc, true);
      tail.assign(1, node);
    } else if ((rc = capture_subiteration_loop(c, g, tail, part, &tail)) ||
               (!with_dt && c->np > 0 && (rc = capture_loop_count(c, g, part, &tail)))) {
      return failed(rc, false);
    }
  }
  if (stage_kernels && (rc = subiter_upload(p, &err))) return failed(rc, true);
  *cur1 = c->cur;
  *scur1 = c->scur;
  step_capture_end(c, cur0, scur0);
  if (plan) *plan = p;
  return EIF_OK;
}

namespace {

int build(eif_ctx *c, eif_ctx::StepGraph &sg, bool with_dt) {
  cudaGraph_t g = nullptr;
  EIF_CK(c, cudaGraphCreate(&g, 0));
  int cur1 = 0, scur1 = 0;
  SubiterPlan *plan = nullptr;
  int rc = capture_step(c, g, &cur1, &scur1, &plan, with_dt);
  if (rc) {
    cudaGraphDestroy(g);
    return rc;
  }
  cudaGraphExec_t exec = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    subiter_plan_destroy(plan);
    if (plan && e == cudaErrorCooperativeLaunchTooLarge) {
      cudaGetLastError();
      c->stage_off = true;
      return build(c, sg, with_dt);
    }
    return check_cuda(c, e, "cudaGraphInstantiate");
  }
  sg.graph = g;
  sg.exec = exec;
  sg.plan = plan;
  sg.cur0 = c->cur;
  sg.scur0 = c->scur;
  sg.cur1 = cur1;
  sg.scur1 = scur1;
  return EIF_OK;
}

}  // namespace

static void free_graphs(eif_ctx::StepGraph (&graphs)[2]) {
  for (auto &sg : graphs) {
    if (sg.exec) cudaGraphExecDestroy(sg.exec);
    if (sg.graph) cudaGraphDestroy(sg.graph);
    subiter_plan_destroy(sg.plan);
    sg = eif_ctx::StepGraph{};
  }
}

void graphs_free(eif_ctx *c) {
  free_graphs(c->graphs);
  free_graphs(c->igraphs);
  subiter_plan_destroy(c->stage_plan);
  c->stage_plan = nullptr;
}

// A launch of a captured step moves the particles and leaves the increments of its last
// stage, without the launch functions that keep the host's record of what the buffers hold:
// nothing formed before it is valid after it.
void step_graph_ran(eif_ctx *c) {
  c->boxes_x_valid = false;
  c->weights_x_valid = false;
  c->bands_x_valid = false;
  c->incr_zero = false;
  c->memo_miss_zero = false;
}

int step_graph_launch(eif_ctx *c, bool with_dt) {
  auto &graphs = with_dt ? c->graphs : c->igraphs;
  eif_ctx::StepGraph *sg = nullptr;
  for (auto &g : graphs) {
    if (g.exec && g.cur0 == c->cur && g.scur0 == c->scur) sg = &g;
  }
  if (!sg) {
    for (auto &g : graphs) {
      if (!g.exec) { sg = &g; break; }
    }
    if (!sg) {
      free_graphs(graphs);
      sg = &graphs[0];
    }
    int rc = build(c, *sg, with_dt);
    if (rc) return rc;
  }
  const cudaError_t e = cudaGraphLaunch(sg->exec, c->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge && sg->plan) {
    // fewer resident CTAs than the occupancy query gave (another limit on the SMs): nothing ran
    cudaGetLastError();
    c->stage_off = true;
    free_graphs(c->graphs);
    free_graphs(c->igraphs);
    return step_graph_launch(c, with_dt);
  }
  if (e != cudaSuccess) return check_cuda(c, e, "cudaGraphLaunch");
  c->cur = sg->cur1;
  c->scur = sg->scur1;
  step_graph_ran(c);
  return EIF_OK;
}

}  // namespace eif
