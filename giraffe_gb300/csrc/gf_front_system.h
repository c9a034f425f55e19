// One standalone system on the multifrontal LU: its plan, and the batch of one
// structure around it that the kernels of gf_front.cu take.  Everything lives
// in one block of the context's device workspace, its host data sent by one copy
// from pinned staging.  Internal to libgiraffe_gpu.so.
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

#include "gf_front.h"
#include "gf_host_internal.h"
#include "gf_kernels.cuh"

namespace gfh {

struct FrontSystem {
  gf::Batch b{};
  FrontBuild fb;
  // parts of the block: offset and, for host data, the source
  struct Part {
    size_t off, bytes;
    const void* src;
  };
  std::vector<Part> parts;
  size_t sent = 0, total = 0;
  char* dev = nullptr;
  struct {
    gf::StructState st;
    int bad;  // the solution's backward error passes the limit
  } state{};
  gf::StructInfo info{};
  double *xs = nullptr, *r = nullptr;  // solution and residual (device)
  int zero = 0;
  int p_state = 0, p_rhs = 0;

  // A host array to send (before any device-only part) or a device-only part.
  int send(const void* src, size_t bytes) {
    parts.push_back({sent, bytes, src});
    sent += (bytes + 255) / 256 * 256;
    return (int)parts.size() - 1;
  }
  template <typename T> T* at(int p) const { return reinterpret_cast<T*>(dev + parts[p].off); }

  // plan: the system's fronts; extra: more arrays sent with it (their parts'
  // numbers come back in order).  rhs: n doubles.
  int init(gf_ctx* ctx, const FrontPlan& plan, int n, const double* rhs,
           const std::vector<std::pair<const void*, size_t>>& extra, std::vector<int>* extra_parts) {
    join_fronts({&plan}, {0}, {0}, 1, n, ctx->wide_update == GF_WIDE_TENSOR, fb);
    info.n_free = n;
    info.wide = 1;
    state.st.phase = gf::PH_ITER;
    state.st.need_solve = 1;
    auto vec = [&](const auto& v) { return send(v.data(), v.size() * sizeof(v[0])); };
    const int p_fr = vec(fb.fronts), p_bnd = vec(fb.bnd), p_kids = vec(fb.kids),
              p_inv = vec(fb.inv), p_list = vec(fb.list),
              p_ext = vec(fb.ext_jobs), p_sch = vec(fb.schur_jobs), p_t5 = vec(fb.t5), p_t5j = vec(fb.t5_jobs), p_pos = vec(fb.pos), p_df = vec(fb.dof_front),
              p_base = vec(fb.base), p_size = vec(fb.size), p_da = vec(fb.dof_at);
    const int p_info = send(&info, sizeof(info)), p_ws = send(&zero, sizeof(int));
    p_state = send(&state, sizeof(state));
    p_rhs = send(rhs, sizeof(double) * (size_t)n);
    for (const auto& x : extra) extra_parts->push_back(send(x.first, x.second));
    auto after = [](size_t at, size_t bytes) { return at + (bytes + 255) / 256 * 256; };
    const size_t off_F = sent, off_x = after(off_F, (size_t)fb.total * sizeof(double));
    const size_t off_oz = after(off_x, sizeof(double) * (size_t)n), off_km = after(off_oz, (size_t)fb.oz * 2);
    const size_t off_ex = after(off_km, (size_t)fb.oz_kmax * sizeof(unsigned long long));
    const size_t off_xs = after(off_ex, (size_t)fb.oz_exp * sizeof(int)), off_r = after(off_xs, sizeof(double) * (size_t)n);
    total = off_r + sizeof(double) * (size_t)n;
    dev = static_cast<char*>(ctx->device_work(total));
    if (!dev) {
      set_err(ctx, "linear solve: allocation of %zu device bytes failed", total);
      return GF_ERR_CUDA;
    }
    // through the context's pinned staging; from pageable memory, a part at a time, where
    // there is none or the parts are too large to keep page-locked
    if (char* pin = sent <= gf_ctx::kStagePin ? static_cast<char*>(ctx->pinned(sent)) : nullptr) {
      for (const Part& p : parts)
        if (p.bytes) std::memcpy(pin + p.off, p.src, p.bytes);
      GF_CK(cudaMemcpyAsync(dev, pin, sent, cudaMemcpyHostToDevice, ctx->stream));
    } else {
      for (const Part& p : parts)
        if (p.bytes) GF_CK(cudaMemcpyAsync(dev + p.off, p.src, p.bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    b.n_struct = 1;
    b.n_free = n;
    b.info = at<gf::StructInfo>(p_info);
    b.state = at<gf::StructState>(p_state);
    b.P = at<double>(p_rhs);
    b.sh.n_wide = 1;
    b.sh.wide_structs = at<int>(p_ws);
    gf::FrontData& d = b.sh.mf;
    d.fronts = at<gf::Front>(p_fr);
    d.bnd = at<int>(p_bnd);
    d.kids = at<int2>(p_kids);
    d.inv = at<int>(p_inv);
    d.list = at<gf::Front>(p_list);
    d.ext_jobs = at<int2>(p_ext);
    d.schur_jobs = at<int2>(p_sch);
    d.pos = at<int>(p_pos);
    d.dof_front = at<int>(p_df);
    d.base = at<int64_t>(p_base);
    d.size = at<int64_t>(p_size);
    d.F = reinterpret_cast<double*>(dev + off_F);
    d.x = reinterpret_cast<double*>(dev + off_x);
    d.t5 = at<gf::FrontT5>(p_t5);
    d.t5_jobs = at<int2>(p_t5j);
    d.oz = reinterpret_cast<__nv_bfloat16*>(dev + off_oz);
    d.oz_kmax = reinterpret_cast<unsigned long long*>(dev + off_km);
    d.oz_exp = reinterpret_cast<int*>(dev + off_ex);
    d.dof_at = at<int>(p_da);
    d.sched = &fb.sched;
    xs = reinterpret_cast<double*>(dev + off_xs);
    r = reinterpret_cast<double*>(dev + off_r);
    return GF_OK;
  }

  // Factorization and solution: assemble(b) puts the matrix into the fronts, check(x,
  // r, bad) forms r = rhs - A x and sets *bad where a row's backward error passes
  // MF_ERROR_LIMIT.  No elimination pivots, so an order of its own can meet pivots that
  // the caller's does not: small ones lose digits without failing.  A solution above the
  // limit is refined with the factor (r as the right-hand side) up to twice; one that is
  // still above it, or a failed pivot, leaves *done false and x as it was, and the caller
  // solves in the natural order.
  template <typename Assemble, typename Check>
  int solve(gf_ctx* ctx, int n, Assemble assemble, Check check, double* x, bool* done) {
    cudaStream_t st = ctx->stream;
    int* bad = reinterpret_cast<int*>(b.state + 1);
    const size_t xb = sizeof(double) * (size_t)n;
    // the staging is free again once the factorization has run
    std::vector<char> pageable;
    char* pin = xb + sizeof(state) <= ctx->pin_bytes ? static_cast<char*>(ctx->pin) : nullptr;
    if (!pin) {
      pageable.resize(xb + sizeof(state));
      pin = pageable.data();
    }
    assemble(b);
    gf::launch_front_lu(b, xs, st);
    *done = false;
    for (int sweep = 0;; ++sweep) {
      check(xs, r, bad);
      GF_CK(cudaGetLastError());
      GF_CK(cudaMemcpyAsync(pin, xs, xb, cudaMemcpyDeviceToHost, st));
      GF_CK(cudaMemcpyAsync(pin + xb, b.state, sizeof(state), cudaMemcpyDeviceToHost, st));
      GF_CK(cudaStreamSynchronize(st));
      std::memcpy(&state, pin + xb, sizeof(state));
      if (state.st.info_fail || !state.bad) {
        *done = !state.st.info_fail;
        break;
      }
      if (sweep == 2) break;
      GF_CK(cudaMemsetAsync(bad, 0, sizeof(int), st));
      gf::launch_front_refine(b, n, r, xs, st);
    }
    if (*done) std::memcpy(x, pin, xb);
    ctx->trim_work();
    return GF_OK;
  }
};

}  // namespace gfh
