// Mixed precision (GF_PREC_MIXED) of Shell_1 structures: K_AA factored in FP32 by
// the multifrontal LU (gf_front.cu), the solution refined in FP64 until the
// corrections stop shrinking, r = b - K x formed from the element matrices; a
// solve that does not reach the FP64 level is done again in FP64.
//
// Bound by the latency of the sweep's launches, a height of the tree at a time down
// and up: the 24x24x2 plate's step, 177 ms with the FP32 wide-band LU and a residual
// from the FP64 band, 10.5 ms here.
#include <cuda_runtime.h>

#include <cfloat>
#include <vector>

#include "gf_kernels.cuh"
#include "gf_types.h"

namespace gf {

namespace {

__device__ __forceinline__ bool wide_active(const Batch& b, int s) {
  const StructState& st = b.state[s];
  return st.phase == PH_ITER && st.need_solve && (!b.sh.fp64_pass || st.ir_fb);
}

}  // namespace

// Start of a mixed solve: the Newton right-hand side saved in FP64 (ir_rhs) and
// rounded into r32, the slot's refinement state reset.
__global__ void __launch_bounds__(256) k_ir_begin(Batch b) {
  const int z = blockIdx.y, s = b.sh.wide_structs[z];
  if (!wide_active(b, s)) return;
  const StructInfo& inf = b.info[s];
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, dt = (int64_t)gridDim.x * blockDim.x;
  const double* P = b.P + inf.dof_off;
  for (int64_t i = t0; i < inf.n_free; i += dt) {
    b.sh.ir_rhs[inf.dof_off + i] = P[i];
    b.sh.r32[inf.dof_off + i] = __double2float_rn(P[i]);
  }
  if (t0 == 0) {
    WideIr& q = b.sh.ir[z];
    q.dn = 0;
    q.xn = 0;
    q.dprev = 0.0;
    q.k = 0;
    q.done = 0;
    b.state[s].ir_fb = 0;
  }
}

// y_e = K_e x_e in FP64 into ir_fe, x in P: a warp per element, lane r < 27 row r.
__global__ void __launch_bounds__(128) k_ir_elements(Batch b) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= b.sh.n_shells) return;
  const int s = b.sh.sstruct[e];
  if (!wide_active(b, s) || b.sh.ir[b.sh.wide_slot[s]].done) return;
  const int off = b.info[s].dof_off;
  const int* nd = b.sh.snodes + 6 * e;
  double x = 0.0;
  if (lane < 27) {
    const int node = lane < 18 ? nd[lane / 3] : nd[3 + (lane - 18) / 3];
    const int g = b.gl[(int64_t)node * 6 + (lane < 18 ? lane % 3 : 3 + (lane - 18) % 3)];
    if (g >= 0) x = b.P[off + g];
  }
  const double* K = b.sh.Ke + (int64_t)e * 729 + lane;
  double y0 = 0.0, y1 = 0.0;
#pragma unroll
  for (int q = 0; q < 26; q += 2) {
    const double k0 = lane < 27 ? K[27 * q] : 0.0, k1 = lane < 27 ? K[27 * q + 27] : 0.0;
    y0 = fma(k0, __shfl_sync(0xffffffffu, x, q), y0);
    y1 = fma(k1, __shfl_sync(0xffffffffu, x, q + 1), y1);
  }
  y0 = fma(lane < 27 ? K[27 * 26] : 0.0, __shfl_sync(0xffffffffu, x, 26), y0);
  if (lane < 27) b.sh.ir_fe[(int64_t)e * 27 + lane] = y0 + y1;
}

// r = b - K x, b in ir_rhs: a thread per DOF takes its elements' y_e in colour order
// and the nodal load stiffness' share; r rounded into r32 for the FP32 solve.  (A
// launch per colour that subtracts in place, and one to start r, took 41 us a sweep on
// the 24x24x2 plate; these two take 9.6.)
__global__ void k_ir_round(Batch b) {
  const int s = b.sh.wide_structs[blockIdx.y];
  if (!wide_active(b, s) || b.sh.ir[blockIdx.y].done) return;
  const StructInfo& inf = b.info[s];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x) {
    double r = b.sh.ir_rhs[inf.dof_off + i];
    const int n6 = b.dof_node6[inf.dof_off + i], k = n6 % 6;
    const int64_t node = n6 / 6;
    const int o0 = b.sh.nref_off[node], o1 = b.sh.nref_off[node + 1];
    for (int o = o0; o < o1; o += 4) {
      double y[4];
      bool in[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = o + q < o1 ? b.sh.nref[o + q] : 0, x = shell_dof(t & 7, k);
        in[q] = o + q < o1 && x >= 0;
        y[q] = in[q] ? b.sh.ir_fe[(int64_t)(t >> 3) * 27 + x] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (in[q]) r -= y[q];
    }
    if (inf.n_loads && k >= 3) {
      for (int j = 0; j < 3; ++j) {
        const int gj = b.gl[node * 6 + 3 + j];
        if (gj >= 0) r -= b.nodeK[node * 9 + (k - 3) * 3 + j] * b.P[inf.dof_off + gj];
      }
    }
    b.sh.r32[inf.dof_off + i] = __double2float_rn(r);
  }
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// x += d in FP64 (d: the FP32 correction, in the fronts' order; first: x = d, the
// first solve); the sweep's largest |d| and |x| raise the slot's maxima (FP64 bits of
// non-negative values order like the values, so the maxima do not depend on the
// CTAs' order, and take no FP64 comparison).  A non-finite entry counts as an
// infinite |d|.
__global__ void __launch_bounds__(256) k_ir_correct(Batch b, int first) {
  const int z = blockIdx.y, s = b.sh.wide_structs[z];
  if (!wide_active(b, s) || b.sh.ir[z].done) return;
  const StructInfo& inf = b.info[s];
  double* x = b.P + inf.dof_off;
  const float* d = reinterpret_cast<const float*>(b.sh.mf.x);
  const int* pos = b.sh.mf.pos + inf.dof_off;
  unsigned long long dm = 0, xm = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x) {
    const double di = (double)d[pos[i]], xi = first ? di : x[i] + di;
    x[i] = xi;
    const unsigned long long db = (unsigned long long)__double_as_longlong(di) & 0x7fffffffffffffffull;
    const unsigned long long xb = (unsigned long long)__double_as_longlong(xi) & 0x7fffffffffffffffull;
    dm = max(dm, xb < 0x7ff0000000000000ull ? db : 0x7ff0000000000000ull);
    xm = max(xm, xb);
  }
  __shared__ unsigned long long red[2][8];
  dm = warp_max(dm);
  xm = warp_max(xm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red[0][warp] = dm;
    red[1][warp] = xm;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
      dm = max(dm, red[0][q]);
      xm = max(xm, red[1][q]);
    }
    WideIr& q = b.sh.ir[z];
    if (dm) atomicMax(&q.dn, dm);
    if (xm) atomicMax(&q.xn, xm);
  }
}

// After a correction, per slot: converged (|d| <= 2^-52 |x|), stalled
// (|d| > |d_prev| / 2: at the FP64 floor, or a factor too poor to refine),
// or out of sweeps (ir_max).  A stall above 2^-30 |x|, the sweep limit, a
// non-finite value or a failed FP32 pivot hand the solve to the FP64
// fallback (ir_fb).  ir_more[0]: a slot refines on (inside a captured pass
// also the refinement loop's condition h); ir_more[1]: a slot takes the
// fallback; ir_more[2] counts the sweeps run (sweep: called after one).
__global__ void k_ir_check(Batch b, cudaGraphConditionalHandle h, int use_h, int sweep) {
  __shared__ int more, fb;
  if (threadIdx.x == 0) {
    more = 0;
    fb = 0;
  }
  __syncthreads();
  for (int z = threadIdx.x; z < b.sh.n_wide; z += blockDim.x) {
    const int s = b.sh.wide_structs[z];
    if (!wide_active(b, s)) continue;
    WideIr& q = b.sh.ir[z];
    StructState& st = b.state[s];
    if (!q.done) {
      const double dn = __longlong_as_double((long long)q.dn), xn = __longlong_as_double((long long)q.xn);
      q.dn = 0;
      q.xn = 0;
      bool stop = false, bad = false;
      if (st.ir_fb || !(dn <= DBL_MAX) || !(xn <= DBL_MAX)) {
        stop = true;
        bad = true;
      } else if (q.k > 0) {
        st.ir_sweeps += 1;
        if (dn <= 0x1p-52 * xn) {
          stop = true;
        } else if (dn > 0.5 * q.dprev) {
          stop = true;
          bad = dn > 0x1p-30 * xn;
        } else if (q.k >= b.sh.ir_max) {
          stop = true;
          bad = true;
        }
      }
      q.dprev = dn;
      q.k += 1;
      if (stop) {
        q.done = 1;
        if (bad) {
          st.ir_fb = 1;
          st.ir_fallbacks += 1;
        }
      }
    }
    if (!q.done) atomicOr(&more, 1);
    if (st.ir_fb) atomicOr(&fb, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    b.sh.ir_more[0] = more;
    b.sh.ir_more[1] = fb;
    if (sweep) b.sh.ir_more[2] += 1;
    if (use_h) cudaGraphSetConditional(h, more ? 1u : 0u);
  }
}

// The FP64 fallback's condition: a slot whose refinement did not finish.
__global__ void k_ir_fb_cond(Batch b, cudaGraphConditionalHandle h) {
  cudaGraphSetConditional(h, b.sh.ir_more[1] ? 1u : 0u);
}

// The FP64 fallback's right-hand side: P = the saved Newton right-hand side
// (b: the fallback's view, so only structures with ir_fb are active);
// ir_more[3] counts the fallbacks run.
__global__ void k_ir_restore(Batch b) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) b.sh.ir_more[3] += 1;
  const int z = blockIdx.y, s = b.sh.wide_structs[z];
  if (!wide_active(b, s)) return;
  const StructInfo& inf = b.info[s];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x)
    b.P[inf.dof_off + i] = b.sh.ir_rhs[inf.dof_off + i];
}

namespace {
// A conditional handle on the graph that st captures into, its value reset
// to dflt at every launch of the graph.
cudaError_t make_cond(cudaStream_t st, cudaGraphConditionalHandle* h, unsigned dflt) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr, nullptr);
  if (e != cudaSuccess) return e;
  return cudaGraphConditionalHandleCreate(h, g, dflt, cudaGraphCondAssignDefault);
}

// Appends a conditional node of the given type on handle h to the capture
// of st and returns its body graph, into which the caller captures the body.
cudaError_t add_cond(cudaStream_t st, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                     cudaGraph_t* body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, nullptr, &nd);
  if (e != cudaSuccess) return e;
  std::vector<cudaGraphNode_t> dv(deps, deps + nd);
  cudaGraphNodeParams np{};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = h;
  np.conditional.type = type;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  if ((e = cudaGraphAddNode(&node, g, dv.data(), nullptr, dv.size(), &np)) != cudaSuccess) return e;
  *body = np.conditional.phGraph_out[0];
  return cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies);
}

}  // namespace

// The first error of a mixed solve's capture step on this thread (a failed
// conditional node or body capture), which the capturing caller reports:
// capture_error() returns it and clears it.
static thread_local cudaError_t g_capture_error = cudaSuccess;
static void capture_fail(cudaError_t e) {
  if (e != cudaSuccess && g_capture_error == cudaSuccess) g_capture_error = e;
}
cudaError_t wide_capture_error() {
  const cudaError_t e = g_capture_error;
  g_capture_error = cudaSuccess;
  return e;
}

// One refinement sweep: the FP64 residual into r32, the forward and backward
// substitution with the FP32 factor, x += d and the check, which sets the
// refinement loop's condition h when use_h.
static void ir_sweep(const Batch& b, cudaStream_t st, cudaGraphConditionalHandle h, int use_h, LaunchProf* prof) {
  const ShellData& sd = b.sh;
  const dim3 dofs(2 * 152, sd.n_wide);
  {
    ProfScope q(prof, st, KC_WIDE_REFINE);
    k_ir_elements<<<(sd.n_shells + 3) / 4, 128, 0, st>>>(b);
    k_ir_round<<<dofs, 256, 0, st>>>(b);
  }
  {
    ProfScope q(prof, st, KC_WIDE_SUBST);
    launch_front_resolve32(b, st);
  }
  {
    ProfScope q(prof, st, KC_WIDE_REFINE);
    k_ir_correct<<<dofs, 256, 0, st>>>(b, 0);
    k_ir_check<<<1, 128, 0, st>>>(b, h, use_h, 1);
  }
}

// The FP32 LU of K_AA, its solve, then FP64 iterative refinement until the
// corrections stop shrinking; a structure whose refinement does not reach the
// FP64 level is solved again by the FP64 LU.  Inside a captured pass the
// refinement loop is a WHILE node and the fallback an IF node, so the pass needs
// no host round trip; otherwise the host reads the loop's flags after each
// sweep.
static void wide_solve_mixed(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  const ShellData& sd = b.sh;
  const dim3 dofs(2 * 152, sd.n_wide);
  Batch fb = b;  // the FP64 fallback's view
  fb.sh.fp64_pass = 1;
  { ProfScope q(prof, st, KC_WIDE_REFINE); k_ir_begin<<<dofs, 256, 0, st>>>(b); }
  launch_front_solve32(b, st, prof);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const bool capturing = !prof && cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusActive;
  if (capturing) {
    // the bodies are captured on a stream of their own, which the pass's
    // capture has not forked into; a failed step is recorded for the capturing
    // caller
    cudaStream_t sr = sd.ir_stream;
    cudaGraphConditionalHandle h, hf;
    cudaGraph_t body, done;
    cudaError_t e;
    if ((e = make_cond(st, &h, 0)) != cudaSuccess) return capture_fail(e);
    k_ir_correct<<<dofs, 256, 0, st>>>(b, 1);
    k_ir_check<<<1, 128, 0, st>>>(b, h, 1, 0);
    if ((e = add_cond(st, h, cudaGraphCondTypeWhile, &body)) != cudaSuccess) return capture_fail(e);
    if ((e = cudaStreamBeginCaptureToGraph(sr, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
      return capture_fail(e);
    ir_sweep(b, sr, h, 1, nullptr);
    if ((e = cudaStreamEndCapture(sr, &done)) != cudaSuccess) return capture_fail(e);
    if ((e = make_cond(st, &hf, 0)) != cudaSuccess) return capture_fail(e);
    k_ir_fb_cond<<<1, 1, 0, st>>>(b, hf);
    if ((e = add_cond(st, hf, cudaGraphCondTypeIf, &body)) != cudaSuccess) return capture_fail(e);
    if ((e = cudaStreamBeginCaptureToGraph(sr, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
      return capture_fail(e);
    k_ir_restore<<<dofs, 256, 0, sr>>>(fb);
    launch_front_solve(fb, sr);
    if ((e = cudaStreamEndCapture(sr, &done)) != cudaSuccess) return capture_fail(e);
    return;
  }
  {
    ProfScope q(prof, st, KC_WIDE_REFINE);
    k_ir_correct<<<dofs, 256, 0, st>>>(b, 1);
    k_ir_check<<<1, 128, 0, st>>>(b, 0, 0, 0);
  }
  int more[2] = {0, 0};
  for (int k = 0; k <= sd.ir_max; ++k) {
    if (cudaMemcpyAsync(more, sd.ir_more, sizeof(more), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess || !more[0])
      break;
    ir_sweep(b, st, 0, 0, prof);
  }
  if (cudaMemcpyAsync(more, sd.ir_more, sizeof(more), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return;
  if (more[1]) {
    k_ir_restore<<<dofs, 256, 0, st>>>(fb);
    launch_front_solve(fb, st, prof);
  }
}

void launch_shell_solve(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  if (b.sh.n_wide == 0) return;
  if (b.mixed) wide_solve_mixed(b, st, prof);
  else launch_front_solve(b, st, prof);
}

// Kernel launches per Newton pass; the mixed path adds its start, check and the
// fallback's condition (its first correction takes the place of k_mf_out), and its sweeps and
// fallbacks come on top (refine_launches).
int shell_solve_launches(const Batch& b) { return front_launches(b) + (b.sh.n_wide && b.mixed ? 3 : 0); }

// Launches of `sweeps` refinement sweeps and `fallbacks` FP64 fallbacks.
long long refine_launches(const Batch& b, long long sweeps, long long fallbacks) {
  return sweeps * (4 + front_resolve_launches(b)) + fallbacks * (1 + front_launches(b));
}

}  // namespace gf
