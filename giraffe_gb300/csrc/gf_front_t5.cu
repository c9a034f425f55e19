// The Schur complements C -= L21 U12 of the largest fronts on the 5th-generation
// tensor cores, FP64 products from exact bf16 slices (see k_wb_update_tc's comment
// in gf_wideband.cu for the slicing and its error: a row's power of two holds for 64
// pivots).
//   k_mf_kmax    largest entry of every pivot's column of L21 and row of U12
//   k_mf_slice   the slices, every pivot balanced by a power of two
//   k_mf_t5      128 x 64 tiles of C
// FP64 FMA bounds the factorization of large plates (2.7 of the 3.7 G multiply-adds
// of a 64x64x2 plate are in these fronts): its pass takes 5.5 ms with FP64 tiles, 4.2
// with these.  A tile's 192 KB of slices per 64 pivots, from L2 at about 6 TB/s over
// the chip (10,000 cycles), bound the tiles now; the products take 5,000.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gf_kernels.cuh"
#include "gf_oz.cuh"
#include "gf_types.h"

namespace gf {

namespace {

constexpr int SL_ROWS = 32;  // rows (columns) a CTA slices

__device__ __forceinline__ bool mf_active(const Batch& b, int s) {
  const StructState& st = b.state[s];
  return st.phase == PH_ITER && st.need_solve && (!b.sh.fp64_pass || st.ir_fb);
}
// Slice 0 of 64 pivots `sub` of operand op (0: L21, 1: U12); slice q is q rows * 64
// further.
__device__ __forceinline__ __nv_bfloat16* t5_slices(const FrontData& d, const FrontT5& T, int s, int op, int sub) {
  return d.oz + T.slices + (int64_t)(op * ((s + OZ_K - 1) / OZ_K) + sub) * OZ_S * T.rows * OZ_K;
}
__device__ __forceinline__ int* t5_exps(const FrontData& d, const FrontT5& T, int s, int op, int sub) {
  return d.oz_exp + T.exps + (op * ((s + OZ_K - 1) / OZ_K) + sub) * T.rows;
}

// S 2^k
__device__ __forceinline__ double t5_scaled(long long S, int k) {
  if (S == 0) return 0.0;
  const unsigned long long a = S < 0 ? 0ull - (unsigned long long)S : (unsigned long long)S;
  const int z = __clzll(a);
  // 53 bits, the leading one at bit 52 (a carry of the rounding moves it up, and with it
  // the exponent field it is added to)
  const unsigned long long m = z < 11 ? (a >> (11 - z)) + (a >> (10 - z) & 1) : a << (z - 11);
  const int e = 1023 + 63 - z + k;
  if (e <= 0 || e >= 2046) return ldexp((double)S, k);
  return __longlong_as_double((long long)(((unsigned long long)(e - 1) << 52) + m) | (S & (long long)0x8000000000000000ull));
}

}  // namespace

// Eight pivots of L21 (blockIdx.y = 0: columns, one a warp) or U12 (1: rows, a lane
// in four on each, a thread every 32nd column).
__global__ void __launch_bounds__(256) k_mf_kmax(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const FrontT5 T = d.t5[off + blockIdx.z];
  const Front F = d.fronts[T.front];
  const int s = F.s, ld = F.ld, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (8 * (int)blockIdx.x >= s || !mf_active(b, F.slot)) return;
  const double* G = d.F + F.off;
  unsigned long long m = 0;
  if (blockIdx.y == 0) {
    const int k = 8 * blockIdx.x + warp;
    if (k < s)
#pragma unroll 4
      for (int i = s + lane; i < F.f; i += 32) m = max(m, oz_mag(G[i + (int64_t)k * ld]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && k < s) d.oz_kmax[T.kmax + k] = m;
    return;
  }
  __shared__ unsigned long long part[8][8];
  const int k = 8 * blockIdx.x + (lane & 7);
  if (k < s)
#pragma unroll 4
    for (int c = s + 4 * warp + (lane >> 3); c < F.f; c += 32) m = max(m, oz_mag(G[k + (int64_t)c * ld]));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if (lane < 8) part[warp][lane] = m;
  __syncthreads();
  if (warp == 0 && lane < 8 && k < s) {
#pragma unroll
    for (int q = 1; q < 8; ++q) m = max(m, part[q][lane]);
    d.oz_kmax[T.kmax + s + k] = m;
  }
}

// SL_ROWS rows of L21 (blockIdx.y even) or columns of U12 (odd) over 64 pivots, the
// blockIdx.y / 2-th of them; rows beyond the front and pivots beyond s are zero.  The CTAs
// of L21's first pivots also take the right-hand side of their rows.
__global__ void __launch_bounds__(256) k_mf_slice(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const FrontT5 T = d.t5[off + blockIdx.z];
  const Front F = d.fronts[T.front];
  if (!mf_active(b, F.slot)) return;
  const int op = blockIdx.y & 1, ch = blockIdx.y >> 1, r0 = SL_ROWS * blockIdx.x, s = F.s, ld = F.ld;
  const int kb = OZ_K * ch, kn = min(OZ_K, s - kb);
  if (r0 >= T.rows || kn <= 0) return;
  const int n = F.f - s;  // rows of L21, columns of U12
  double* G = d.F + F.off;
  static_assert(SL_ROWS * OZ_K == 8 * 256, "eight pivots of a row per thread");
  __shared__ double A[SL_ROWS][OZ_K + 1];
  __shared__ int e[SL_ROWS];
  __shared__ double bal[OZ_K];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < OZ_K) {
    // pivot k's column of L21 times 2^-f, its row of U12 times 2^f: the products
    // unchanged, the two maxima within a factor two of each other
    int f = 0;
    if (tid < kn) {
      const unsigned long long ml = d.oz_kmax[T.kmax + kb + tid], mu = d.oz_kmax[T.kmax + s + kb + tid];
      if (ml && mu) f = ((int)(ml >> 52) - (int)(mu >> 52)) >> 1;
      f = max(-1000, min(1000, f));
    }
    bal[tid] = __longlong_as_double((long long)(1023 + (op ? f : -f)) << 52);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < SL_ROWS * OZ_K / 256; ++q) {
    const int x = tid + 256 * q;
    const int i = op ? x / OZ_K : x % SL_ROWS, k = op ? x % OZ_K : x / SL_ROWS;
    const bool live = k < kn && r0 + i < n;
    A[i][k] = live ? G[op ? kb + k + (int64_t)(s + r0 + i) * ld : s + r0 + i + (int64_t)(kb + k) * ld] * bal[k] : 0.0;
  }
  __syncthreads();
  for (int i = warp; i < SL_ROWS; i += 8) {
    unsigned long long m = 0;
#pragma unroll
    for (int q = 0; q < OZ_K / 32; ++q) m = max(m, oz_mag(A[i][lane + 32 * q]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) e[i] = oz_exponent(m);
  }
  __syncthreads();
  // eight pivots of a row per thread: a 16-byte chunk of every slice
  {
    const int i = tid >> 3, k0 = 8 * (tid & 7), r = r0 + i;
    uint32_t w[OZ_S][4];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      uint16_t v[OZ_S];
      oz_split_bits(A[i][k0 + x], e[i], v);
#pragma unroll
      for (int q = 0; q < OZ_S; ++q) w[q][x >> 1] = x & 1 ? w[q][x >> 1] | (uint32_t)v[q] << 16 : v[q];
    }
    // the 128-byte swizzle: 16-byte chunk c of row r at chunk c ^ (r & 7)
    __nv_bfloat16* dst = t5_slices(d, T, s, op, ch) + (int64_t)r * OZ_K + 8 * ((tid & 7) ^ (r & 7));
#pragma unroll
    for (int q = 0; q < OZ_S; ++q)
      *reinterpret_cast<uint4*>(dst + (int64_t)q * T.rows * OZ_K) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
  }
  if (tid < SL_ROWS) t5_exps(d, T, s, op, ch)[r0 + tid] = e[tid];
  if (op || ch || r0 >= n) return;
  // the right-hand side of these rows, in FP64: eight lanes a row
  const int i = tid % SL_ROWS, q = tid / SL_ROWS, r = s + r0 + i;
  double acc = 0.0;
  if (r < F.f)
#pragma unroll 4
    for (int k = q; k < s; k += 8) acc = fma(G[r + (int64_t)k * ld], G[k + (int64_t)F.f * ld], acc);
  __syncthreads();
  A[i][q] = acc;
  __syncthreads();
  if (q == 0 && r < F.f) {
    double t = A[i][0];
#pragma unroll
    for (int x = 1; x < 8; ++x) t += A[i][x];
    G[r + (int64_t)F.f * ld] -= t;
  }
}

// 128 x 64 tiles of C, one after the other, all pivots of a tile, 64 at a time: eight
// accumulators of 64 columns in tensor memory (diagonal q + t of the slice products),
// issued by one thread.  The sixteen slices of 64 pivots (192 KB) are asked for at
// once, as soon as the products of the 64 before have run, of the next tile too, so
// they arrive beside the epilogue.  The tile of C waits in registers (a row and 16
// columns per thread); after every 64 pivots the diagonals are joined in 64-bit
// integers, converted once and subtracted: two FP64 operations an entry for 64 FMA.
// Every wait is bounded; one that gives up fails the solves of its and the CTA's
// later tiles, and the copies in flight are waited for (bounded) before the CTA ends.
constexpr size_t MF_T5_SMEM = 1024 + OZ_S * (T5_B_BYTES + T5_A_BYTES) + 128 + T5_N * sizeof(int);
__global__ void __launch_bounds__(T5_THREADS, 1) k_mf_t5(Batch b, int job0, int n_jobs) {
  const FrontData& d = b.sh.mf;
  auto slot = [&](int job) { return d.fronts[d.t5[d.t5_jobs[job0 + job].x].front].slot; };
  // the first job from `job` on whose structure solves
  auto find = [&](int job) {
    while (job < n_jobs && !mf_active(b, slot(job))) job += gridDim.x;
    return job;
  };
  int job = find(blockIdx.x);
  if (job >= n_jobs) return;
  extern __shared__ __align__(16) unsigned char t5_raw[];
  unsigned char* base = t5_raw + ((1024u - (t5_smem(t5_raw) & 1023u)) & 1023u);
  unsigned char* Bs = base;                   // [slice][64 columns][128 B]
  unsigned char* As = Bs + OZ_S * T5_B_BYTES;  // [slice][128 rows][128 B]
  uint64_t* bars = reinterpret_cast<uint64_t*>(As + OZ_S * T5_A_BYTES);  // fullB, fullA[8], done
  uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 10);
  int* okflag = reinterpret_cast<int*>(holder + 1);
  int* eU = reinterpret_cast<int*>(bars + 16);
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t fullB = t5_smem(bars), fullA = fullB + 8, done = fullA + 8 * OZ_S;
  const uint32_t sA = t5_smem(As), sB = t5_smem(Bs);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(t5_smem(holder)),
                 "r"(T5_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  // the copies of 64 pivots of a job (thread 0)
  auto load = [&](int x, int sub) {
    const int2 J = d.t5_jobs[job0 + x];
    const FrontT5 T = d.t5[J.x];
    const int s = d.fronts[T.front].s;
    const int64_t slice = (int64_t)T.rows * OZ_K;
    const __nv_bfloat16* gU = t5_slices(d, T, s, 1, sub) + (int64_t)T5_N * (J.y >> 16) * OZ_K;
    const __nv_bfloat16* gL = t5_slices(d, T, s, 0, sub) + (int64_t)T5_M * (J.y & 0xFFFF) * OZ_K;
    t5_expect_tx(fullB, OZ_S * T5_B_BYTES);
    for (int q = 0; q < OZ_S; ++q) {
      t5_bulk_load(sB + q * T5_B_BYTES, gU + q * slice, T5_B_BYTES, fullB);
      if (q == 0) {
        t5_expect_tx(fullA, T5_A_BYTES);
        t5_bulk_load(sA, gL, T5_A_BYTES, fullA);
      }
    }
    for (int q = 1; q < OZ_S; ++q) {
      t5_expect_tx(fullA + 8 * q, T5_A_BYTES);
      t5_bulk_load(sA + q * T5_A_BYTES, gL + q * slice, T5_A_BYTES, fullA + 8 * q);
    }
  };
  if (tid == 0) {
    for (int i = 0; i < OZ_S + 2; ++i) t5_mbar_init(fullB + 8 * i, 1);
    *okflag = 1;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    load(job, 0);
  }
  t5_fence_before();
  __syncthreads();
  t5_fence_after();
  const uint32_t tmem = *holder;
  const uint64_t descA = t5_desc(sA), descB = t5_desc(sB);
  const int lg = warp & 3, cb = T5_COLS_PER_WARP * (warp >> 2);  // TMEM lane group, first column of the thread
  bool good = true;
  int phase = 0;  // of the barriers: 64 pivots each, of every job
  while (job < n_jobs && good) {
    const int2 J = d.t5_jobs[job0 + job];
    const FrontT5 T = d.t5[J.x];
    const Front F = d.fronts[T.front];
    const int s = F.s, u = F.f - s, r0 = T5_M * (J.y & 0xFFFF), c0 = T5_N * (J.y >> 16);
    const int nsub = (s + OZ_K - 1) / OZ_K, next = find(job + gridDim.x);
    const int r = r0 + 32 * lg + (tid & 31);  // this thread's row of C, < T.rows
    const bool row_live = r < u;
    double* C = d.F + F.off + s + r + (int64_t)(s + c0 + cb) * F.ld;
    double c22[T5_COLS_PER_WARP];
    for (int sub = 0; sub < nsub; ++sub, phase ^= 1) {
      if (tid < T5_N) eU[tid] = t5_exps(d, T, s, 1, sub)[c0 + tid];
      if (tid == 0) {
        const int kk_n = (min(OZ_K, s - OZ_K * sub) + 15) / 16;
        bool ok = t5_wait(fullB, phase);
        int landed = 0;
#pragma unroll
        for (int q = 0; q < OZ_S; ++q) {
          ok = ok && t5_wait(fullA + 8 * q, phase);
          if (ok) {
            ++landed;
            t5_fence_after();
            // descriptors count 16-byte units: a slice, then 16 pivots (32 bytes)
            const uint64_t da = descA + (uint64_t)(q * (T5_A_BYTES >> 4));
#pragma unroll
            for (int t = 0; t + q < OZ_S; ++t) {
              const uint64_t db = descB + (uint64_t)(t * (T5_B_BYTES >> 4));
              const uint32_t acc = tmem + (uint32_t)((q + t) * T5_N);
              t5_mma(acc, da, db, q == 0 ? 0u : 1u);  // the first products overwrite the accumulators
              if (kk_n > 1) t5_mma(acc, da + 2, db + 2, 1u);
              if (kk_n > 2) t5_mma(acc, da + 4, db + 4, 1u);
              if (kk_n > 3) t5_mma(acc, da + 6, db + 6, 1u);
            }
          }
        }
        t5_commit(done);  // arrives once every product issued so far has run
        if (!ok) {
          // let the copies in flight land before the CTA's shared memory goes
          *okflag = 0;
          t5_wait(fullB, phase);
          for (; landed < OZ_S; ++landed) t5_wait(fullA + 8 * landed, phase);
        }
      }
      if (sub == 0)
#pragma unroll
        for (int c = 0; c < T5_COLS_PER_WARP; ++c) c22[c] = (row_live && c0 + cb + c < u) ? C[(int64_t)c * F.ld] : 0.0;
      const bool ready = t5_wait(done, phase);
      if (!ready && tid == 0) t5_wait(done, phase);  // once more before tensor memory is freed
      good = __syncthreads_and(ready) && *(volatile int*)okflag;
      if (!good) break;
      if (tid == 0) {
        if (sub + 1 < nsub) load(job, sub + 1);
        else if (next < n_jobs) load(next, 0);
      }
      const int eLr = t5_exps(d, T, s, 0, sub)[r];
      t5_fence_after();
      const uint32_t tl = tmem + ((uint32_t)(lg * 32) << 16);
#pragma unroll
      for (int j = 0; j < T5_COLS_PER_WARP / 8; ++j) {
        uint32_t v[OZ_S][8];
#pragma unroll
        for (int q = 0; q < OZ_S; ++q) t5_ld8(tl + (uint32_t)(q * T5_N + cb + 8 * j), v[q]);
        t5_wait_ld();
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) {
          int ci[OZ_S];
#pragma unroll
          for (int q = 0; q < OZ_S; ++q) ci[q] = __float2int_rn(__uint_as_float(v[q][cc]));
          // S = sum_d c_d 2^(7 (7 - d)) with |c_d| <= (d + 1) 2^20, T = floor(S / 2^10) in
          // 64 bits: pairs of diagonals first (|c_d 2^7 + c_(d+1)| < 2^31)
          const int P0 = ci[0] * 128 + ci[1], P1 = ci[2] * 128 + ci[3], P2 = ci[4] * 128 + ci[5];
          const int P3 = (ci[6] * 128 + ci[7]) >> 10;
          const long long S = ((long long)P0 << 32) + ((long long)P1 << 18) + ((long long)P2 << 4) + (long long)P3;
          // S times 2^(e_i + e_j - 2046 - 53) as a double, rounded to 53 bits: by integer
          // operations, an FP64 conversion would take the pipe's 64 cycles
          c22[8 * j + cc] -= t5_scaled(S, eLr + eU[cb + 8 * j + cc] - 2046 - 53);
        }
      }
      t5_fence_before();
      __syncthreads();
      t5_fence_after();
    }
    if (good) {
      if (row_live) {
#pragma unroll
        for (int c = 0; c < T5_COLS_PER_WARP; ++c)
          if (c0 + cb + c < u) C[(int64_t)c * F.ld] = c22[c];
      }
      job = next;
    }
  }
  for (; job < n_jobs; job = find(job + gridDim.x))  // a wait gave up
    if (tid == 0) b.state[slot(job)].info_fail = 1;
  t5_fence_before();
  __syncthreads();
  if (warp == 0) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(T5_TMEM_COLS));
  }
}

void launch_front_t5(const Batch& b, const FrontLevel& V, cudaStream_t st) {
  if (!V.t5_cnt) return;
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_mf_t5, (int)MF_T5_SMEM}});
  for (int q = 0; q < front_grids(V.t5_cnt); ++q) {
    const int n = min(V.t5_cnt - q * MF_GRID_FRONTS, MF_GRID_FRONTS), off = V.t5_off + q * MF_GRID_FRONTS;
    k_mf_kmax<<<dim3((V.t5_s + 7) / 8, 2, n), 256, 0, st>>>(b, off);
    k_mf_slice<<<dim3(V.t5_rows / SL_ROWS, 2 * ((V.t5_s + OZ_K - 1) / OZ_K), n), 256, 0, st>>>(b, off);
  }
  k_mf_t5<<<min(V.t5_job_cnt, 152), T5_THREADS, MF_T5_SMEM, st>>>(b, V.t5_job_off, V.t5_job_cnt);
}

}  // namespace gf
