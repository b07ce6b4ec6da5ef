// solver.cuh -- pieces shared by the CSR (pcg.cu) and node-block (bsr.cu)
// persistent Krylov kernels: block partial sums, the PCG result record and
// the CSR argument pack.
#pragma once

#include "common.cuh"

constexpr int PCG_THREADS = 512;
int pcg_lanes_for(const axia_ctx* ctx, bool fp32, int requested);
constexpr int S_PQ = 0, S_RR = 1, N_SLOTS = 3;  // partial-sum slots: p.q; r.r, r.z

// result of one persistent solve, written by block 0
struct PcgOut {
  long long iters;
  double residual;
  double bnorm;
  int status;
  int updates;
};

template <typename V>
struct PcgArgs {
  int n;
  const int* rowptr;
  const int* col;
  const V* val;
  const V* dinv;
  const V* b;
  V* x;
  V* r;
  V* p;
  V* q;
  double* partials;  // [N_SLOTS][gridDim.x]
  double* totals;    // [N_SLOTS]
  GridBarrier* bar;
  DevStatus* st;
  PcgOut* out;
  double tol;
  long long max_iter;
  unsigned long long limit_ns;
};

template <int L, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-reduce up to two values: emit(k, sum) runs on one warp per value (all
// its lanes hold the sum).
// FP64 values go through shared memory: a warp sum costs every warp five
// dependent FP64 additions per value, and GB300 issues one FP64 warp
// instruction per SM about every 18 cycles, so 16 warps and two values take
// 1.5 us per block; four warps per value adding up a quarter of the warps'
// lanes each, then one warp, need 8 + 3 + 5 instead of 160 of them.  RARE: warp
// sums all the same, for the FP64 sums of a mixed solve (a few in all), where
// 10 KB of shared memory would cost the matrix product L1.
struct SumsScratch {
  double all[2][PCG_THREADS];
  double part[2][4][32];
};
__device__ __forceinline__ SumsScratch& sums_scratch() {  // one for every instantiation
  __shared__ SumsScratch s;
  return s;
}
template <int NV, bool RARE, typename A, typename E>
__device__ __forceinline__ void block_sums(A v0, A v1, E&& emit) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if constexpr (sizeof(A) == sizeof(double) && !RARE) {
    constexpr int Q = 4;
    auto& s_all = sums_scratch().all;
    auto& s_part = sums_scratch().part;
    s_all[0][threadIdx.x] = v0;
    if (NV > 1) s_all[1][threadIdx.x] = v1;
    __syncthreads();
    for (int t = warp; t < Q * NV; t += nw) {
      const int k = t / Q, g = t % Q;
      A a = A(0);
      for (int w = g; w < nw; w += Q) a += s_all[k][32 * w + lane];
      s_part[k][g][lane] = a;
    }
    __syncthreads();
    if (warp < NV)
      emit(warp, warp_sum((s_part[warp][0][lane] + s_part[warp][1][lane]) +
                          (s_part[warp][2][lane] + s_part[warp][3][lane])));
  } else {
    __shared__ A s_red[2][32];
    v0 = warp_sum(v0);
    if (NV > 1) v1 = warp_sum(v1);
    if (lane == 0) {
      s_red[0][warp] = v0;
      s_red[1][warp] = v1;
    }
    __syncthreads();
    if (warp == 0) {
      A a0 = lane < nw ? s_red[0][lane] : A(0);
      A a1 = lane < nw ? s_red[1][lane] : A(0);
      emit(0, (double)warp_sum(a0));
      if (NV > 1) emit(1, (double)warp_sum(a1));
    }
  }
}

// a value's block sum as this block's partial
__device__ __forceinline__ void block_partial(double v, double* partials) {
  block_sums<1, true>(v, 0.0, [&](int, double t) {
    if (threadIdx.x == 0) partials[blockIdx.x] = t;
  });
}

// Barriers and reductions over the co-resident blocks of one system: block
// `rank` of nblk.  reduce() adds up one or two values over all threads and runs
// fn(totals) on thread 0 of every block (the scalars of the iteration, left in
// shared memory).  Every block sees the same totals.
//
// CLUSTER: the blocks are one thread-block cluster (at most CLUSTER_MAX): the
// block sums go to every block's shared memory and the cluster's hardware
// barrier replaces the counter in L2.  A small system is all barriers: at 1,500
// rows in FP64 the three of an iteration took 12 of its 17.5 us.
constexpr int CLUSTER_MAX = 16;
// Systems up to these sizes run as one cluster: 16 SMs against all of them,
// cheap barriers against work.  FP32 node blocks, two-level, us per iteration,
// cluster / whole grid: 14 k blocks 12.5 / 25.0, 52 k 14.9 / 24.3, 120 k 20.4 /
// 24.9, 230 k 31.0 / 24.7.
// FP64 CSR: the entries, and 6.25 for every lane of a row, whose sums and vector
// updates take the FP64 issue slots of 16 SMs (about 8 us + 0.018 per 1,000
// entries + 0.11 per 1,000 rows and lane).  C3D8, 4 lanes: 88 k entries 10.3 / 18.1,
// 240 k 14.2 / 18.0, 430 k (6 k rows) 17.6 / 18.1, 690 k 25.2 / 19.3; 5 and 7
// entries per row: 20 k rows 19.0 / 16.7, 27 k 24.8 / 17.5, 55 k 41.0 / 22.6; 3 per
// row: 40 k rows 26.6 / 17.9, 130 k 69.9 / 24.5.
constexpr int64_t CLUSTER_MAX_BLOCKS = 130000;
constexpr int64_t CLUSTER_MAX_CSR = 550000;
constexpr bool cluster_csr(int64_t nnz, int64_t rows, int lanes) {
  return nnz + rows * lanes * 25 / 4 <= CLUSTER_MAX_CSR;
}

// OUTLINED: the last block's sums in a function of their own.  Measured at C3D8
// 90^3 / 100^3: mixed node blocks with the diagonal 167 us per iteration inline,
// 152 outlined; two-level 53.8 ms against 54.2, 64 cubes 68.4 against 71.4.
template <bool CLUSTER, bool OUTLINED = false>
struct BlockSync {
  GridBarrier* bar;
  DevStatus* st;
  unsigned long long limit_ns;
  double* partials;  // [3][nblk]
  double* totals;    // [3]
  unsigned nblk, rank;
  int parity;

  template <int NV, bool RARE = false, typename A, typename F>
  __device__ __forceinline__ bool reduce(A v0, A v1, int slot0, F&& fn) {
    if constexpr (CLUSTER) {
      // two sets in turn: a block writes set k again only after a barrier that
      // every block reached after reading it
      double (*slots)[2][CLUSTER_MAX] = cluster_slots();
      parity ^= 1;
      block_sums<NV, RARE>(v0, v1, [&](int k, double t) {
        const unsigned lane = threadIdx.x & 31;
        if (lane < nblk) {
          const unsigned mine = (unsigned)__cvta_generic_to_shared(&slots[parity][k][rank]);
          unsigned theirs;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(lane));
          asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(theirs), "d"(t) : "memory");
        }
      });
      sync();
      if (threadIdx.x < 32) {
        double a[2];
#pragma unroll
        for (int k = 0; k < NV; ++k) a[k] = threadIdx.x < nblk ? slots[parity][k][threadIdx.x] : 0.0;
#pragma unroll
        for (int o = CLUSTER_MAX / 2; o > 0; o >>= 1)
#pragma unroll
          for (int k = 0; k < NV; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
        if (threadIdx.x == 0) fn(a);
      }
      __syncthreads();
      return true;
    } else {
      block_sums<NV, RARE>(v0, v1, [&](int k, double t) {
        if ((threadIdx.x & 31) == 0) partials[(slot0 + k) * nblk + rank] = t;
      });
      return group_reduce_apply<OUTLINED>(bar, st, limit_ns, partials, totals, slot0, NV, nblk, fn);
    }
  }
  __device__ __forceinline__ bool sync() {
    if constexpr (CLUSTER) {
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      return true;
    } else {
      return group_sync(bar, st, limit_ns, nblk);
    }
  }
  // before the first reduce() / after the last: no block writes to another's
  // shared memory before it runs or after it has left
  __device__ __forceinline__ void fence_lifetime() {
    if constexpr (CLUSTER) sync();
  }
  static __device__ __forceinline__ double (*cluster_slots())[2][CLUSTER_MAX] {
    __shared__ double s_slots[2][2][CLUSTER_MAX];
    return s_slots;
  }
};

// What one iteration of a persistent CG needs from its reductions, computed
// by thread 0 of each block and read by the block from shared memory.
template <typename A>
struct CgScalars {
  A rz, rzn;                     // r.z of the current direction; of the new r, its diagonal part
  A alpha, beta;
  double bnorm, residual;        // ||b||, ||r|| (mixed: at the last update)
  double rr, limit2;             // r.r; its value that stops (mixed: that triggers an update)
  int status;                    // axia_status that ends the loop
  int update;                    // mixed: replace the residual now
  int stop;                      // converged
};

// The scalar steps of the FP32 CG with FP64 reliable updates, on thread 0 of
// each block.  beta is r.z (new) / r.z (old), with the replaced r after an update.
__device__ __forceinline__ void mixed_limit(CgScalars<float>& S, double tol, double delta) {
  const double r = fmax(delta * S.residual, tol * S.bnorm);
  S.limit2 = r * r;
}
__device__ __forceinline__ void mixed_begin(CgScalars<float>& S, const double* t, double tol, double delta) {
  S.rz = (float)t[1];
  S.bnorm = S.residual = sqrt(t[0]);
  mixed_limit(S, tol, delta);
  S.status = isfinite(t[0]) ? AXIA_OK : AXIA_ERR_NONFINITE;  // a load that is not finite is no zero load
  S.update = 0;
  S.stop = S.bnorm < 1e-30;
  if (S.stop) S.residual = 0.0;
  if (S.status != AXIA_OK) S.stop = 1;
}
__device__ __forceinline__ void mixed_alpha(CgScalars<float>& S, const double* t) {
  const float pq = (float)t[0];
  if (!(fabsf(pq) >= 1e-30f) || !isfinite(pq)) S.status = isfinite(pq) ? AXIA_ERR_ZERO_PIVOT : AXIA_ERR_NONFINITE;
  S.alpha = S.rz / pq;
}
__device__ __forceinline__ void mixed_set_beta(CgScalars<float>& S, float rzn) {
  S.beta = rzn / S.rz;
  S.rz = rzn;
}
__device__ __forceinline__ void mixed_check(CgScalars<float>& S, double rr) {
  if (!isfinite(rr)) S.status = AXIA_ERR_NONFINITE;
  S.update = rr <= S.limit2;
}
__device__ __forceinline__ void mixed_replaced(CgScalars<float>& S, double rr, double tol, double delta) {
  S.residual = sqrt(rr);
  mixed_limit(S, tol, delta);
  if (!isfinite(S.residual)) S.status = AXIA_ERR_NONFINITE;
  S.stop = S.residual <= tol * S.bnorm;
}
// the diagonal part of the new r.z: beta at once with the diagonal
// preconditioner, after the coarse part is known with the two-level one
template <bool COARSE>
__device__ __forceinline__ void mixed_rz(CgScalars<float>& S, float rzn, bool last) {
  if constexpr (COARSE)
    S.rzn = rzn;
  else if (last)
    mixed_set_beta(S, rzn);
}
// The same steps of the one-precision CG (linalg.rs:199-259).
template <typename A>
__device__ __forceinline__ void cg_begin(CgScalars<A>& S, const double* t, double tol) {
  S.rz = (A)t[1];
  S.rr = t[0];
  S.bnorm = sqrt(t[0]);
  S.limit2 = tol * S.bnorm * (tol * S.bnorm);
  S.status = isfinite(t[0]) ? AXIA_OK : AXIA_ERR_NONFINITE;
  S.stop = S.bnorm < 1e-30;
  if (S.stop) S.rr = 0.0;
  if (S.status != AXIA_OK) S.stop = 1;
}
template <typename A>
__device__ __forceinline__ void cg_alpha(CgScalars<A>& S, const double* t) {
  const A pq = (A)t[0];
  if (!(fabs((double)pq) >= 1e-30)) S.status = AXIA_ERR_ZERO_PIVOT;
  S.alpha = S.rz / pq;
}
template <typename A>
__device__ __forceinline__ void cg_beta(CgScalars<A>& S, const double* t) {
  const A rzn = (A)t[1];
  S.rr = t[0];
  if (!isfinite(S.rr)) S.status = AXIA_ERR_NONFINITE;
  S.stop = S.rr <= S.limit2;
  S.beta = rzn / S.rz;
  S.rz = rzn;
}
template <typename A>
__device__ __forceinline__ void cg_out(const CgScalars<A>& S, double residual, PcgOut* out, double tol, long long iters,
                                       int updates) {
  out->iters = iters;
  out->residual = residual;
  out->bnorm = S.bnorm;
  out->status = S.status == AXIA_OK && residual > tol * S.bnorm * 10.0 ? AXIA_ERR_NOT_CONVERGED : S.status;
  out->updates = updates;
}

// ---------------------------------------------------------------------------
// Node-block (3x3) matrix and the mixed-precision argument pack (bsr.cu)
// ---------------------------------------------------------------------------
template <typename V>
struct BsrMat {
  int n_nodes;
  const int* adj_ptr;  // [n_nodes+1]
  const int* adj;      // [nb]
  const V* val;        // [9][nb]
  long long nb;
};

// Symmetric FP32 node-block form (axia_ctx::d_uval ...): upper blocks of row a
// at [uptr[a], uptr[a+1]) as 10 floats each (9 values, column bits), lower
// neighbours of row a at [lptr[a], lptr[a+1]) as (b, position of K_ba).
struct SymMat {
  int n_nodes;
  const int* uptr;
  const float* uval;
  const int* lptr;
  const int2* low;
};

// one system of a multi-mesh solve: its block rows and its blocks
struct MeshGroup {
  int node0, node1;   // block rows [node0, node1)
  int cta0, ncta;     // blocks [cta0, cta0 + ncta) of the launch
  long long part_off; // offset of its partial-sum area
  int chunk0, chunk1; // its restriction chunks (two-level preconditioner)
  int row0, row1;     // its coarse unknowns
  int col0, ldm;      // its block of the coarse inverse: first unknown, padded size
  long long moff;     // element offset of that block
};
constexpr int GROUP_SLOTS = N_SLOTS;  // partial-sum slots per group

constexpr int COARSE_MAX = 4096;    // coarse unknowns (6 per subdomain, padded to 64)
constexpr int COARSE_CHUNK = 256;   // nodes per restriction chunk at most

struct CoarseArgs {
  int n_sub;             // subdomains (0: no coarse space)
  int nc;                // 6 n_sub
  int row0, row1;        // the coarse unknowns whose rows of y = M r_c this launch (group) computes
  int chunk_lo, chunk_hi;  // the restriction chunks this launch (group) handles
  int ncp;               // length of rc / yc (one block: nc rounded up to a multiple of 64)
  int col0, ldm;         // the block of M this launch (group) reads: unknowns col0 .., row stride ldm
  int n_chunks;
  const int* sub_node;   // [n_nodes] nodes by subdomain, ascending within each
  const int4* chunk;     // [n_chunks] (subdomain, first, end) ranges of sub_node
  const int* chunk_ptr;  // [n_sub + 1] chunks of each subdomain
  const float4* geo;     // [n_nodes] (x_a - c_I) / h, .w = bits (I << 3 | free-DOF mask)
  const float* minv;     // this launch's block of M: [rows][ldm], row r at (r - col0) ldm, zero in the padding
  float* part;           // [n_chunks][6] restriction partials
  float* rc;             // [ncp] restricted residual Z^T r (zero in the padding)
  int* cnt;              // [n_sub] chunks of each subdomain done (reset by the last)
  float* yc;             // [ncp] coarse correction y = M r_c
  // 32 load cases at once (batch.cu): [n_chunks][6][32], [ncp][32], [ncp][32]
  float* part_m;
  float* rc_m;
  float* yc_m;
};

struct BsrReliableArgs {
  BsrMat<float> M32;
  SymMat S32;        // the FP32 matrix in symmetric storage (kernels instantiated with SYM)
  BsrMat<double> M64;
  int nd;
  const float* dinv32;
  const double* b;
  double* x;
  float* x32;
  float* r32;
  float* p32;
  float* q32;
  float* z32;
  double* partials;
  double* totals;
  GridBarrier* bar;
  DevStatus* st;
  PcgOut* out;
  double tol;
  double delta;
  long long max_iter;
  unsigned long long limit_ns;
  CoarseArgs C;      // two-level preconditioner (n_sub = 0: Jacobi only)
};

BsrReliableArgs make_reliable_args(axia_ctx* ctx, double rtol, double delta, long long max_iter);
int group_kernel_capacity(axia_ctx* ctx, int lanes, int vec, int* per_sm, bool coarse = false);
void group_layout(const axia_ctx* ctx, int lanes_req, int vec_req, int* lanes, int* vec);
int launch_group_reliable(axia_ctx* ctx, BsrReliableArgs& P, const MeshGroup* groups, const int* cta_group,
                          GridBarrier* bars, double* totals4, PcgOut* outs, int grid, int lanes, int vec, bool coarse = false);
int launch_full_rhs(axia_ctx* ctx, const double* d_f);
int launch_full_reconstruct(axia_ctx* ctx, double* d_u);
int prepare_full_buffers(axia_ctx* ctx);

// Sorted (key, value) pairs and their runs of equal keys (triplets.cu).
struct Runs {
  uint64_t* key = nullptr;  // sorted keys
  double* val = nullptr;    // values in sorted order
  int64_t* head = nullptr;  // first position of each run
  int64_t nv = 0, n_runs = 0;
  void release() {
    dev_free(key);
    dev_free(val);
    dev_free(head);
    n_runs = nv = 0;
  }
};
int sort_runs(axia_ctx* ctx, const uint64_t* dk, const double* dv, int64_t nt, int64_t nv, int end_bit, Runs* out);
int key_bits(uint64_t max_key);
int csr_from_runs(axia_ctx* ctx, int64_t n, const Runs& R, bool fp32);
int vector_from_runs(axia_ctx* ctx, int64_t n, const Runs& R, double* d_out);

// Device copy of a DOF map (T, u0) and the reduced right-hand side (reduce.cu).
struct ReducedSystem {
  int64_t n_full = 0, n_ind = 0;
  int64_t* t_ptr = nullptr;
  int64_t* t_col = nullptr;
  double* t_val = nullptr;
  double* u0 = nullptr;
  double* rhs = nullptr;
  void release() {
    dev_free(t_ptr);
    dev_free(t_col);
    dev_free(t_val);
    dev_free(u0);
    dev_free(rhs);
  }
};
int reduce_system(axia_ctx* ctx, const axia_dofmap* map, int64_t nt, const int64_t* h_i, const int64_t* h_j,
                  const double* h_v, const double* h_f, bool fp32, ReducedSystem* S);
int reconstruct_system(axia_ctx* ctx, const ReducedSystem& S, const double* d_x, double* d_u);

// ---------------------------------------------------------------------------
// Host helpers for the persistent launches
// ---------------------------------------------------------------------------
// Blocks of a cooperative CG launch for `work` threads of one matrix product
// (rows x lanes per row): one block per PCG_THREADS up to one per SM, then a
// multiple of the SM count (a part-filled last round left SMs with twice the
// work of others): a second block per SM from 2.25 blocks of work per SM, as
// many as fit from 12.
// Measured, us per iteration of the FP64 CSR form with 4 lanes: 17 k rows 152
// blocks 19.9, 304 23.4; 71 k 37.6, 304 32.8, 456 38.2; 104 k 51.7, 41.8, 41.1;
// 670 k 247, 164, 154.
// most: blocks per SM at most.
inline int coop_grid(axia_ctx* ctx, const void* kern, int64_t work, int* grid_out, size_t dyn_smem = 0,
                     int most = 1 << 30) {
  int per_sm = 0;
  AXIA_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PCG_THREADS, dyn_smem));
  if (per_sm < 1) return set_error(ctx, AXIA_ERR_CUDA, "PCG kernel does not fit on an SM");
  const int64_t need = std::max<int64_t>(1, (work + PCG_THREADS - 1) / PCG_THREADS);
  const int sms = ctx->sm_count;
  const int rounds = std::min(std::min(per_sm, most), need >= 12 * sms ? per_sm : need >= 9 * sms / 4 ? 2 : 1);
  const int grid = (int)std::min<int64_t>(need, (int64_t)rounds * sms);
  if ((size_t)grid * N_SLOTS > ctx->partial_slots) return set_error(ctx, AXIA_ERR_STATE, "partials buffer too small");
  *grid_out = grid;
  return AXIA_OK;
}


// Blocks of the one-cluster form of a CG launch for `work` threads of one
// matrix product (0: use the cooperative launch, e.g. where the device cannot
// hold such a cluster).  kern is the CLUSTER instantiation.
inline int cluster_blocks(const void* kern, int64_t work) {
  const int64_t need = std::max<int64_t>(1, (work + PCG_THREADS - 1) / PCG_THREADS);
  int blocks = 1;
  while (blocks < need && blocks < CLUSTER_MAX) blocks *= 2;
  if (blocks > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    (void)cudaGetLastError();
    blocks = 8;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(PCG_THREADS);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess || fit < 1) {
    (void)cudaGetLastError();
    return 0;
  }
  return blocks;
}
inline int launch_cluster(axia_ctx* ctx, const void* kern, int blocks, void** params) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(PCG_THREADS);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  AXIA_CUDA(ctx, cudaLaunchKernelExC(&cfg, kern, params));
  ctx->launches++;
  return AXIA_OK;
}

// one persistent launch bracketed by CUDA events on the launching stream
template <typename F>
inline int timed_launch(axia_ctx* ctx, axia_solve_info* info, F&& launch) {
  cudaEvent_t a, b;
  AXIA_CUDA(ctx, cudaEventCreate(&a));
  AXIA_CUDA(ctx, cudaEventCreate(&b));
  cudaEventRecord(a, ctx->stream);
  int st = launch();
  cudaEventRecord(b, ctx->stream);
  if (st == AXIA_OK) {
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    info->ms_pcg_kernel += ms;
    info->pcg_launches += 1;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return st;
}


inline int read_out(axia_ctx* ctx, PcgOut* o) {
  AXIA_CUDA(ctx, cudaMemcpyAsync(o, ctx->d_out, sizeof(PcgOut), cudaMemcpyDeviceToHost, ctx->stream));
  AXIA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  DevStatus hs;
  AXIA_TRY(read_dev_status(ctx, &hs));
  if (hs.timeout) return set_error(ctx, AXIA_ERR_TIMEOUT, "a grid barrier of the PCG kernel ran past its time limit");
  return AXIA_OK;
}


inline int status_error(axia_ctx* ctx, const PcgOut& o) {
  if (o.status == AXIA_ERR_NOT_CONVERGED)
    return set_error(ctx, o.status, "CG did not converge (residual " + std::to_string(o.residual) + " after " +
                                        std::to_string(o.iters) + " iterations)");
  if (o.status == AXIA_ERR_ZERO_PIVOT) return set_error(ctx, o.status, "CG: zero pivot, matrix not positive definite");
  return set_error(ctx, o.status, "CG: non-finite iterate");
}


