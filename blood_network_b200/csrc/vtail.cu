// The V-cycle's coarse tail in one launch (vtail.cuh).
//
// What bounds it: nothing but latency.  A level of at most some ten thousand
// rows is a chain of small operations (a colour class of a sweep, a residual,
// a transfer), each a row pointer -> index -> x chain of three L2 round trips.
// As kernels of their own each cost 4-5 us in a graph (launch, ramp, chain,
// drain), and a level of 2k rows swept by a single block (a warp per row) 52 us
// a sweep.  One cluster of 16 blocks x 512 threads holds these levels' rows at
// once, and its hardware barrier replaces the launch: 500 cycles, 1240 with
// every thread's store before it (with 1024 threads per block 620 and 1680).
// An operation's matrix data (row pointers, the first entries of each lane, the
// diagonal) does not depend on the operation before, so it is loaded between
// the barrier's arrival and its wait; after the wait only x and b are left to
// fetch.  Measured: 1.6-2 us an operation on a 2k-row level, 2-4 us with hub
// rows; the V-cycle of the 2k network 104 -> 38 us a half, whole solves 2k FP64
// 3.18 -> 1.59 ms, 20k 5.05 -> 3.85, one preconditioner at 75k 1.15 -> 0.95.
//
// The rows of an operation are dealt to groups of 2^lg lanes; rows longer than
// kTailPer entries per lane are taken by a warp each and rows longer than
// kTailLong by a block each, from lists made at setup, so that no lane walks
// a hub row.  x, y and b live in global memory and are read and written
// through L2 (ld.cg): the other blocks of the cluster wrote them before the
// barrier.  Row sums: lane strides, then a fixed shuffle tree, so results do
// not depend on timing.
#include "vtail.cuh"

#include <cooperative_groups.h>

namespace bn {
namespace {

constexpr int kPreShort = 4, kPreMid = 4;  // entries per lane loaded ahead
constexpr int kTailWarps = kTailThreads / 32;

template <class T>
__device__ __forceinline__ T tmul(T a, T b) {
  if constexpr (sizeof(T) == 8) return __dmul_rn(a, b);
  else return __fmul_rn(a, b);
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the leading entries of a row as one lane sees them
template <class T, int U>
struct Entries {
  int k0, k1;  // the row's range; k0 == k1 where there is no row
  int j[U];
  T v[U];
  __device__ __forceinline__ void none() { k0 = k1 = 0; }
  __device__ __forceinline__ void load(const TailOp<T>& op, int lane, int step) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + lane + u * step;
      if (k < k1) {
        j[u] = op.ja[k];
        v[u] = op.a[k];
      }
    }
  }
};

// An operation's vectors and the entries that count: j < jmax and j != skip.
template <class T>
struct TailVec {
  const T* b;
  const T* x;
  T* y;
  int jmax;
};

template <class T>
__device__ __forceinline__ T tail_x(const TailOp<T>& op, const TailVec<T>& vec, int j) {
  const T* p = (unsigned)(j - op.ov0) < (unsigned)op.ovn ? op.ov : vec.x;
  return __ldcg(p + j);
}

template <class T, int U>
__device__ __forceinline__ T tail_sum(const TailOp<T>& op, const TailVec<T>& vec, int skip,
                                      Entries<T, U> e, int lane, int step) {
  T sum = T(0);
  for (;;) {
    T xv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const bool in = e.k0 + lane + u * step < e.k1 && e.j[u] < vec.jmax && e.j[u] != skip;
      xv[u] = in ? tail_x(op, vec, e.j[u]) : T(0);
      if (!in) e.v[u] = T(0);
    }
#pragma unroll
    for (int u = 0; u < U; u++) sum += tmul(e.v[u], xv[u]);
    e.k0 += U * step;
    if (e.k0 + lane >= e.k1) return sum;
    e.load(op, lane, step);  // U entries at once: their latencies overlap
  }
}

// b_i (or y_i for ADD)
template <class T>
__device__ __forceinline__ T tail_rhs(const TailOp<T>& op, const TailVec<T>& vec, int i) {
  if (op.kind == TK_ADD) return __ldcg(vec.y + i);
  return op.kind == TK_Y ? T(0) : __ldcg(vec.b + i);
}

template <class T>
__device__ __forceinline__ void tail_finish(const TailOp<T>& op, const TailVec<T>& vec, int i,
                                            T sum, T bi, T di) {
  T r;
  if (op.kind <= TK_GS) r = (bi - sum) / di;
  else if (op.kind == TK_Y) r = sum;
  else if (op.kind == TK_RES) r = bi - sum;
  else r = bi + sum;
  __stcg(vec.y + i, r);
}

template <class T>
__global__ void __launch_bounds__(kTailThreads, 1)
k_tail(const TailOp<T>* ops, int nops, int top_lev, const T* top_b, T* top_x) {
  BN_PDL_ENTRY();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char tail_mem[];
  __shared__ T red[kTailWarps];
  __shared__ double xs[kTailDenseMax];
  TailOp<T>* prog = reinterpret_cast<TailOp<T>*>(tail_mem);
  {
    const int words = nops * (int)(sizeof(TailOp<T>) / 4);
    const int* src = reinterpret_cast<const int*>(ops);
    int* dst = reinterpret_cast<int*>(prog);
    for (int q = threadIdx.x; q < words; q += kTailThreads) dst[q] = src[q];
  }
  __syncthreads();
  const int rank = (int)cluster.block_rank(), nblk = (int)cluster.num_blocks();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // this thread's first row of an operation, and its warp's first mid row
  Entries<T, kPreShort> es;
  Entries<T, kPreMid> em;
  T ds = T(1);
  int mrow = 0;
  auto ahead = [&](const TailOp<T>& op) {
    es.none();
    em.none();
    if (op.kind == TK_COPY || op.kind == TK_DENSE) return;
    // consecutive groups go to different blocks: small operations use them all
    const int t = (threadIdx.x >> op.lg) * nblk + rank;
    if (t < op.n) {
      const int i = op.r0 + t;
      es.k0 = op.ia[i];
      es.k1 = op.ia[i + 1];
      if (op.kind <= TK_GS) ds = op.d[i];
      es.load(op, threadIdx.x & ((1 << op.lg) - 1), 1 << op.lg);
    }
    // the warps take the mid rows from the far end, those with the fewest short rows first
    const int m = (kTailWarps - 1 - w) * nblk + rank;
    if (m < op.nmid) {
      const int4 q = op.list[m];
      mrow = q.x;
      em.k0 = q.y;
      em.k1 = q.z;
      em.load(op, lane, 32);
    }
  };
  ahead(prog[0]);
  for (int o = 0; o < nops; o++) {
    const TailOp<T>& op = prog[o];
    const bool top = op.lev == top_lev;
    TailVec<T> vec;
    vec.b = top && (op.top & TT_B_IS_B) ? top_b : op.b;
    vec.x = op.x;
    if (top && (op.top & TT_X_IS_X)) vec.x = top_x;
    if (top && (op.top & TT_X_IS_B)) vec.x = top_b;
    vec.y = top && (op.top & TT_Y_IS_X) ? top_x : op.y;
    vec.jmax = op.kind == TK_GS0 ? op.r0 : 0x7fffffff;
    if (op.kind == TK_COPY) {
      for (int t = rank * kTailThreads + threadIdx.x; t < op.n; t += nblk * kTailThreads)
        __stcg(vec.y + op.r0 + t, __ldcg(vec.x + op.r0 + t));
    } else if (op.kind == TK_DENSE) {  // a warp per row, FP64 accumulation
      for (int k = threadIdx.x; k < op.n; k += kTailThreads) xs[k] = (double)__ldcg(vec.x + k);
      __syncthreads();
      for (int i = w * nblk + rank; i < op.n; i += kTailWarps * nblk) {
        const double* row = op.dense + (size_t)i * op.n;
        double s = 0.0;
        for (int k0 = 0; k0 < op.n; k0 += 512) {
          double a[16];  // the row's loads in flight together
#pragma unroll
          for (int q = 0; q < 16; q++) {
            const int k = k0 + q * 32 + lane;
            a[q] = k < op.n ? row[k] : 0.0;
          }
#pragma unroll
          for (int q = 0; q < 16; q++) {
            const int k = k0 + q * 32 + lane;
            if (k < op.n) s += a[q] * xs[k];
          }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) __stcg(vec.y + i, (T)s);
      }
      __syncthreads();
    } else {
      const bool gs = op.kind <= TK_GS;
      const int G = 1 << op.lg, gl = threadIdx.x & (G - 1);
      const int stride = (kTailThreads >> op.lg) * nblk;
      const int mid_len = op.nmid + op.nlong > 0 ? kTailPer << op.lg : 0x7fffffff;
      if (op.ovn > 0)
        for (int t = rank * kTailThreads + threadIdx.x; t < op.ovn; t += nblk * kTailThreads)
          __stcg(const_cast<T*>(vec.x) + op.ov0 + t, __ldcg(op.ov + op.ov0 + t));
      for (int base = rank; base < op.n; base += stride) {  // uniform in the block
        const int t = base + (threadIdx.x >> op.lg) * nblk;
        const int i = op.r0 + t;
        const bool row = t < op.n && es.k1 - es.k0 <= mid_len;
        T bi = T(0), sum = T(0);
        if (row) {
          bi = tail_rhs(op, vec, i);
          sum = tail_sum(op, vec, gs ? i : -1, es, gl, G);
        }
        for (int off = G >> 1; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (row && gl == 0) tail_finish(op, vec, i, sum, bi, ds);
        const int tn = t + stride;
        if (base + stride < op.n) {
          es.none();
          if (tn < op.n) {
            es.k0 = op.ia[op.r0 + tn];
            es.k1 = op.ia[op.r0 + tn + 1];
            if (gs) ds = op.d[op.r0 + tn];
            es.load(op, gl, G);
          }
        }
      }
      for (int m = (kTailWarps - 1 - w) * nblk + rank; m < op.nmid;) {
        const T bi = tail_rhs(op, vec, mrow);
        const T di = gs ? op.d[mrow] : T(1);
        T sum = tail_sum(op, vec, gs ? mrow : -1, em, lane, 32);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) tail_finish(op, vec, mrow, sum, bi, di);
        m += kTailWarps * nblk;
        if (m < op.nmid) {
          const int4 q = op.list[m];
          mrow = q.x;
          em.k0 = q.y;
          em.k1 = q.z;
          em.load(op, lane, 32);
        }
      }
      for (int m = rank; m < op.nlong; m += nblk) {  // uniform in the block
        const int4 q = op.list[op.n - 1 - m];
        Entries<T, kPreShort> el;
        el.k0 = q.y;
        el.k1 = q.z;
        el.load(op, threadIdx.x, kTailThreads);
        T sum = tail_sum(op, vec, gs ? q.x : -1, el, threadIdx.x, kTailThreads);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) red[w] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
          T t = T(0);
          for (int k = 0; k < kTailWarps; k++) t += red[k];
          tail_finish(op, vec, q.x, t, tail_rhs(op, vec, q.x), gs ? op.d[q.x] : T(1));
        }
        __syncthreads();
      }
    }
    __syncwarp();
    cluster_arrive();
    if (o + 1 < nops) ahead(prog[o + 1]);
    __syncwarp();
    cluster_wait();
  }
}

template <class T>
__global__ void __launch_bounds__(256) k_tail_lists(TailOp<T>* ops) {
  TailOp<T>& op = ops[blockIdx.x];
  __shared__ int cm, cl;
  if (threadIdx.x == 0) cm = cl = 0;
  __syncthreads();
  int4* list = const_cast<int4*>(op.list);
  if (list)
    for (int t = threadIdx.x; t < op.n; t += blockDim.x) {
      const int i = op.r0 + t, k0 = op.ia[i], k1 = op.ia[i + 1];
      if (k1 - k0 <= (kTailPer << op.lg)) continue;
      const int at = k1 - k0 > kTailLong ? op.n - 1 - atomicAdd(&cl, 1) : atomicAdd(&cm, 1);
      list[at] = make_int4(i, k0, k1, 0);
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    op.nmid = cm;
    op.nlong = cl;
  }
}

template <class T>
int cluster_size() {
  // one of 16 blocks needs the non-portable attribute and a GPC with that many
  // free SMs
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = sizeof(TailOp<T>) * kTailMaxOps;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int nc = 0;
  if (cudaOccupancyMaxActiveClusters(&nc, k_tail<T>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    nc = 0;
  }
  return nc > 0 ? 16 : 8;
}

}  // namespace

template <class T>
static void tail_attributes() {
  BN_CUDA(cudaFuncSetAttribute(k_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(sizeof(TailOp<T>) * kTailMaxOps)));
  BN_CUDA(cudaFuncSetAttribute(k_tail<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

int tail_cluster() {
  tail_attributes<double>();
  tail_attributes<float>();
  const int a = cluster_size<double>(), b = cluster_size<float>();
  return a < b ? a : b;
}

template <class T>
void tail_lists(TailOp<T>* ops, int nops, cudaStream_t s) {
  if (nops > 0) BN_LAUNCH(k_tail_lists<T>, nops, 256, 0, s, ops);
}

template <class T>
void tail_run(const TailOp<T>* ops, int op0, int op1, int top_lev, const T* top_b, T* top_x,
              int nblk, cudaStream_t s) {
  if (op1 <= op0) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = sizeof(TailOp<T>) * (size_t)(op1 - op0);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nblk;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  g_launch_count++;
  BN_CUDA(cudaLaunchKernelEx(&cfg, k_tail<T>, ops + op0, op1 - op0, top_lev, top_b, top_x));
}

#define BN_TAIL_INST(T)                                     \
  template void tail_lists<T>(TailOp<T>*, int, cudaStream_t); \
  template void tail_run<T>(const TailOp<T>*, int, int, int, const T*, T*, int, cudaStream_t);
BN_TAIL_INST(double)
BN_TAIL_INST(float)

}  // namespace bn
