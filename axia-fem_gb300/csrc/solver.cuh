// solver.cuh -- pieces shared by the CSR (pcg.cu) and node-block (bsr.cu)
// persistent Krylov kernels: block partial sums, the PCG result record and
// the CSR argument pack.
#pragma once

#include "common.cuh"

constexpr int PCG_THREADS = 512;
int pcg_lanes_for(const axia_ctx* ctx, bool fp32, int requested);
constexpr int S_PQ = 0, S_RR = 1, S_RZ = 2, N_SLOTS = 3;

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

// block-reduce up to two values and store them as this block's partials
// (block `rank` of a group of nblk blocks; the whole grid by default).
// FP64 values go through shared memory: a warp sum costs every warp five
// dependent FP64 additions per value, and GB300 issues one FP64 warp
// instruction per SM about every 18 cycles, so 16 warps and two values take
// 1.5 us per block; four warps per value adding up a quarter of the warps'
// lanes each, then one warp, need 8 + 3 + 5 instead of 160 of them.
template <typename A>
__device__ __forceinline__ void block_partials(A v0, A v1, int nv, double* partials, int slot0, int slot1,
                                               unsigned nblk = 0, unsigned rank = 0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (nblk == 0) {
    nblk = gridDim.x;
    rank = blockIdx.x;
  }
  if constexpr (sizeof(A) == sizeof(double)) {
    constexpr int Q = 4;
    __shared__ A s_all[2][PCG_THREADS];
    __shared__ A s_part[2][Q][32];
    s_all[0][threadIdx.x] = v0;
    if (nv > 1) s_all[1][threadIdx.x] = v1;
    __syncthreads();
    for (int t = warp; t < Q * nv; t += nw) {
      const int k = t / Q, g = t % Q;
      A a = A(0);
      for (int w = g; w < nw; w += Q) a += s_all[k][32 * w + lane];
      s_part[k][g][lane] = a;
    }
    __syncthreads();
    for (int k = warp; k < nv; k += nw) {
      const A a = warp_sum((s_part[k][0][lane] + s_part[k][1][lane]) + (s_part[k][2][lane] + s_part[k][3][lane]));
      if (lane == 0) partials[(k == 0 ? slot0 : slot1) * nblk + rank] = a;
    }
  } else {
    __shared__ A s_red[2][32];
    v0 = warp_sum(v0);
    if (nv > 1) v1 = warp_sum(v1);
    if (lane == 0) {
      s_red[0][warp] = v0;
      s_red[1][warp] = v1;
    }
    __syncthreads();
    if (warp == 0) {
      A a0 = lane < nw ? s_red[0][lane] : A(0);
      A a1 = lane < nw ? s_red[1][lane] : A(0);
      a0 = warp_sum(a0);
      if (nv > 1) a1 = warp_sum(a1);
      if (lane == 0) {
        partials[slot0 * nblk + rank] = (double)a0;
        if (nv > 1) partials[slot1 * nblk + rank] = (double)a1;
      }
    }
  }
}

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

__device__ __forceinline__ double total(const double* totals, int slot) { return __ldcg(totals + slot); }


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
  S.status = AXIA_OK;
  S.update = 0;
  S.stop = S.bnorm < 1e-30;
  if (S.stop) S.residual = 0.0;
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
  S.status = AXIA_OK;
  S.stop = !(S.bnorm >= 1e-30);
  if (S.stop) S.rr = 0.0;
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
constexpr int GROUP_SLOTS = 4;  // partial-sum slots per group: S_PQ, S_RR, S_RZ, S_RC

constexpr int COARSE_MAX = 4096;    // coarse unknowns (6 per subdomain, padded to 64)
constexpr int COARSE_CHUNK = 256;   // nodes per restriction chunk at most
constexpr int S_RC = 3;             // partial-sum slot of r_c . y

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
// work of others), another per SM for about 1.5 PCG_THREADS of work each.
// Measured, us per iteration of the FP64 CSR form with 4 lanes: 17 k rows 152
// blocks 19.9, 304 23.4; 71 k 37.6, 304 32.8, 456 38.2; 104 k 51.7, 41.8, 41.1;
// 670 k 247, 164, 154.
inline int coop_grid(axia_ctx* ctx, const void* kern, int64_t work, int* grid_out, size_t dyn_smem = 0) {
  int per_sm = 0;
  AXIA_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PCG_THREADS, dyn_smem));
  if (per_sm < 1) return set_error(ctx, AXIA_ERR_CUDA, "PCG kernel does not fit on an SM");
  const int64_t need = std::max<int64_t>(1, (work + PCG_THREADS - 1) / PCG_THREADS);
  const int sms = ctx->sm_count;
  const int rounds = (int)std::min<int64_t>(per_sm, std::max<int64_t>(1, (2 * need + 3 * sms / 2) / (3 * sms)));
  const int grid = (int)std::min<int64_t>(need, (int64_t)rounds * sms);
  if ((size_t)grid * N_SLOTS > ctx->partial_slots) return set_error(ctx, AXIA_ERR_STATE, "partials buffer too small");
  *grid_out = grid;
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


