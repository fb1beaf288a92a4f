// IC(0) triangular sweeps, owner form: the sync-free sweep with every row
// given to a warp that keeps it, so that most values never cross the chip.
//
// What bounds a sweep is its chain of dependency levels.  Dealing 32-row
// chunks of each level round-robin to the grid (k_tri_flags) makes every level
// of the chain a store to L2 and a poll of L2 (870 cycles one way) by a warp
// among thousands that poll: 0.83 us per level on 2k rows, 1.2-1.4 us on
// 300k-4M rows.  A flag in shared memory takes 160 cycles.  So:
//  * each block owns a range of consecutive rows and keeps the value of every
//    one of them in shared memory, the value doubling as its ready flag; only
//    dependencies on other blocks are polled in the output vector (on a
//    capillary lattice the next row, line and mostly plane are the block's);
//  * the block's rows go in steps, at most 32 rows of one level, dealt in level
//    order to its warps in turn: while one warp computes a step the others
//    have loaded the rows of the next ones and poll;
//  * a row is computed and published in the polling iteration in which its last
//    value arrives (waiting for the warp's slowest row: 1225 us against 1077 at
//    4M rows FP64);
//  * codes, values and diagonals sit in step order, four entries a row.
// Levels packed into a narrow range of rows (the generations of a
// heap-numbered tree) would all fall to few blocks: such a level is dealt to
// all of them by rank (kDealt).
//
// Two sweeps (forward and backward), chunked form -> this one, microseconds:
//   rows      2k      20k      75k      300k     2M       4M
//   FP64   61 -> 40  159 -> 121  249 -> 182  434 -> 299  820 -> 641  1095 -> 1077
//   FP32   63 -> 48  143 -> 98   223 -> 149  398 -> 252  742 -> 515   978 -> 692
// What is left is 0.7-0.8 us a level: the load-poll-divide-store of a step
// (about 1,500 cycles at 16 warps, FP64 divide 210 of them) and, from some
// 20,000 rows a block on, the crossings between blocks.  Tried without gain:
// a warp owning a few lattice lines, its rows staged by cp.async four steps
// ahead and its own values in a small ring, the rest through L2 (2k 73, 4M
// FP64 2066); the same with register prefetch (the loads of several steps
// share scoreboards, so each step still waited for the newest).
//
// Progress: all blocks are co-resident (cooperative launch, one per SM); a
// block's steps are in level order, each warp takes its own in order, and a
// row waits only on rows of lower levels, so the lowest unfinished level always
// has its inputs.  Every wait is bounded (flags.cuh).  Arithmetic per row: the
// input minus the products in entry order, then one division, as every other
// form (bit-identical).
#include "ichol.cuh"
#include "flags.cuh"

#include <atomic>
#include <cstdlib>
#include <cub/cub.cuh>

namespace bn {
namespace {

// Threads of a block: with fewer blocks than SMs 8 warps (few warps leave the
// one on the chain the issue slots: 300k rows FP64 299 us, 16 warps 324), else
// 16, in FP32 32 (4M rows: 850 us with 16, 692 with 32).  FP64 takes 68 registers
// a thread, so 28 warps are the most that fit; its two sweeps in microseconds at
// 2M / 3M / 4M rows: 16 warps 637 / 830 / 1081, 24 warps 679 / 885 / 1212, 28
// warps 604 / 775 / 1258 (the chunked form 797 / 1018 / 1069).
constexpr int kOwnFew = 256, kOwnMany64 = 512, kOwnMany32 = 1024;
constexpr int kOwnLanes = 4;         // rows of one level per warp that the block count aims at
constexpr int kOwnSlack = 640;       // rows per block kept free for uneven shares
constexpr int kDealt = 512;          // rows of one level in a block's range: above, deal the level
// Rows per block up to which the form is used, chunked form -> this one:
// FP64 820 -> 641 us at 13,600 (2M rows), 1046 -> 835 at 20,300 (3M),
// 1095 -> 1077 at 27,000 (4M); FP32 978 -> 692 at 27,000, 1240 -> 812 at
// 40,700 (6M), 1356 -> 1520 at 54,200 (8M).  The blocks are counted by the levels
// and the shared memory (own_build), so a deep, narrow factor can pass the line
// with SMs left over; it keeps the chunked form.
constexpr int kOwnRows64 = 22000, kOwnRows32 = 45000;
constexpr int kNoEntry = (int)0x80000000;

template <class T>
struct OwnArgs {
  const int* step;        // first position of each step (and one past the last)
  const int2* steps;      // per block: [first step, end step)
  const int* base;        // per block: its first position
  const int4* code;       // per position: four dependencies, ~slot of the block or vector index
  const T* val;           // four values per position
  const T* diag;
  const int2* rec;        // {vector row, first further entry or -1}
  const int* xcode;       // entries past the fourth, kNoEntry after a row's last
  const T* xval;
  const T* in;
  T* out;
  T* clear;
  WaitCtl wc;
};

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <class U> struct ValueOf;
template <> struct ValueOf<unsigned> { using T = float; };
template <> struct ValueOf<unsigned long long> { using T = double; };
template <class U>
__device__ __forceinline__ U lds_word(unsigned at) {
  U v;
  if constexpr (sizeof(U) == 8)
    asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(at) : "memory");
  else
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
// Polls between two looks at the abort word and the clock.
constexpr int kOwnLook = 512;
__device__ __forceinline__ bool own_give_up(const WaitCtl& w, int it, unsigned long long& t0,
                                            bool* ran_out) {
  if (ld_relaxed_i32(w.rec) != 0) {
    *ran_out = false;
    return true;
  }
  const unsigned long long t = global_ns();
  if (t0 == 0) t0 = t;
  *ran_out = t - t0 > w.limit_ns || it >= kSpinHardCap;
  return *ran_out;
}

// Waits until get() returns a value (bounded; NaN when the wait is abandoned).
// The record takes the dependency's code as it is: naming its row here, cold as
// the path is, made the sweep 9 % slower (1.43M rows FP32: 76 us, 83), so the
// host does (own_dep_row).
template <class U, class F>
__device__ __forceinline__ U own_wait(U u, int dep, F get, const WaitCtl& wc, int row) {
  using W = WordOf<typename ValueOf<U>::T>;
  unsigned long long t0 = 0;
  for (int it = 1; u == W::kPending; it++) {
    bool ran_out = false;
    if ((it & (kOwnLook - 1)) == 0 && own_give_up(wc, it, t0, &ran_out)) {
      if (ran_out) wait_give_up(wc, row, dep, global_ns() - t0);
      return W::kNaN;
    }
    u = get();
  }
  return u;
}

template <class T, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_tri_own(OwnArgs<T> a) {
  using W = WordOf<T>;
  using U = typename W::U;
  extern __shared__ __align__(16) unsigned char own_mem[];
  __shared__ unsigned long long s_zero;
  U* sv = reinterpret_cast<U*>(own_mem);
  const int lane = threadIdx.x & 31;
  const int base = a.base[blockIdx.x];
  const int2 ws = a.steps[blockIdx.x];
  U* o = reinterpret_cast<U*>(a.out);
  const int mine = a.base[blockIdx.x + 1] - base;
  for (int q = threadIdx.x; q < mine; q += THREADS) sv[q] = W::kPending;
  if (threadIdx.x == 0) s_zero = 0;
  __syncthreads();
  const unsigned sv0 = (unsigned)__cvta_generic_to_shared(sv);
  const unsigned zero0 = (unsigned)__cvta_generic_to_shared(&s_zero);
  auto sub = [&](T s, T v, U u) -> T {
    if constexpr (sizeof(T) == 8) return xsub(s, xmul(v, word_value(u)));
    else return xsubf(s, xmulf(v, word_value(u)));
  };
  for (int k = ws.x + (int)(threadIdx.x >> 5); k < ws.y; k += THREADS / 32) {
    const int p = a.step[k] + lane;
    if (p < a.step[k + 1]) {
      const int2 rec = a.rec[p];
      const int4 c4 = a.code[p];
      T v[4];
      load4(a.val + 4 * (size_t)p, v);
      const T d = a.diag[p];
      T s = a.in[rec.x];
      if (a.clear) reinterpret_cast<U*>(a.clear)[rec.x] = W::kPending;
      const int c[4] = {c4.x, c4.y, c4.z, c4.w};
      // Own block's values by shared-memory word (the zero word where the entry is
      // missing or another block's), other blocks' in the output vector.
      unsigned at[4];
      U u[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        at[q] = c[q] < 0 && c[q] != kNoEntry ? sv0 + (unsigned)(~c[q]) * (unsigned)sizeof(U) : zero0;
        u[q] = c[q] >= 0 ? ld_relaxed(o + c[q]) : U(0);
      }
      unsigned long long t0 = 0;
      // A row is computed and published inside its own polling loop, in the
      // iteration its last value arrives, not when the warp's slowest row has its.
      for (int it = 1;; it++) {
        U w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = lds_word<U>(at[q]);
        bool far = false;
#pragma unroll
        for (int q = 0; q < 4; q++) far |= u[q] == W::kPending;
        if (far) {
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (u[q] == W::kPending) u[q] = ld_relaxed(o + c[q]);
          far = u[0] == W::kPending || u[1] == W::kPending || u[2] == W::kPending ||
                u[3] == W::kPending;
        }
        bool pend = far || w[0] == W::kPending || w[1] == W::kPending || w[2] == W::kPending ||
                    w[3] == W::kPending;
        if (pend && (it & (kOwnLook - 1)) == 0) {
          bool ran_out = false;
          if (own_give_up(a.wc, it, t0, &ran_out)) {
            int dep = 0;
#pragma unroll
            for (int q = 3; q >= 0; q--) {
              if (w[q] == W::kPending) { dep = c[q]; w[q] = W::kNaN; }
              if (u[q] == W::kPending) { dep = c[q]; u[q] = W::kNaN; }
            }
            if (ran_out) wait_give_up(a.wc, rec.x, dep, global_ns() - t0);
            pend = false;
          }
        }
        if (pend) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) s = sub(s, v[q], c[q] < 0 ? w[q] : u[q]);
        if (rec.y >= 0) {
          for (int e = rec.y; a.xcode[e] != kNoEntry; e++) {
            const int cx = a.xcode[e];
            const unsigned ax = sv0 + (unsigned)(~cx) * (unsigned)sizeof(U);
            auto get = [&] { return cx >= 0 ? ld_relaxed(o + cx) : lds_word<U>(ax); };
            const U ux = own_wait(get(), cx, get, a.wc, rec.x);
            s = sub(s, a.xval[e], ux);
          }
        }
        U res = value_word(s / d);
        if (res == W::kPending) res = W::kNaN;
        *reinterpret_cast<volatile U*>(sv + (p - base)) = res;
        st_relaxed(o + rec.x, res);
        break;
      }
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------ schedule
// dealt[l] = 1 where a window of R consecutive rows holds more than kDealt rows
// of level l (rows of a level are in index order)
__global__ void k_own_dense_levels(const int* __restrict__ rows, const int* __restrict__ lev, int n,
                                   int R, int* __restrict__ dealt) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t + kDealt < n; t += gridDim.x * blockDim.x)
    if (lev[t] == lev[t + kDealt] && rows[t] / R == rows[t + kDealt] / R) dealt[lev[t]] = 1;
}
__global__ void k_own_deal(const int* __restrict__ rows, const int* __restrict__ lev,
                           const int* __restrict__ lptr, const int* __restrict__ dealt, int n,
                           int nown, int* __restrict__ owner, int* __restrict__ flag) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int l = lev[t], i = rows[t];
    const bool d = dealt[l] != 0;
    flag[i] = d ? 0 : 1;
    if (d)
      owner[i] = (int)((long long)(t - lptr[l]) * nown / (lptr[l + 1] - lptr[l]));
  }
}
// rank: exclusive scan of flag (n + 1 entries)
__global__ void k_own_range(const int* __restrict__ rank, int n, long long m, int nown,
                            int* __restrict__ owner) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (rank[i + 1] != rank[i]) owner[i] = (int)((long long)rank[i] * nown / m);
}
__global__ void k_own_key(const int* __restrict__ rows, const int* __restrict__ owner, int n,
                          int* __restrict__ key, int* __restrict__ ids) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    key[t] = owner[rows[t]];
    ids[t] = t;
  }
}
// position of the first row of p's (block, level) run, where p starts one
__global__ void k_own_runs(const int* __restrict__ perm, const int* __restrict__ key,
                           const int* __restrict__ lev, const int* __restrict__ rows, int n,
                           int* __restrict__ start, int* __restrict__ newpos) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const bool first =
        p == 0 || key[p] != key[p - 1] || lev[perm[p]] != lev[perm[p - 1]];
    start[p] = first ? p : 0;
    newpos[rows[perm[p]]] = p;
  }
}
__global__ void k_own_heads(const int* __restrict__ start, int n, int* __restrict__ head) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
    head[p] = ((p - start[p]) & 31) == 0 ? 1 : 0;
}
// step table, the blocks' step ranges and the blocks' first positions
__global__ void k_own_steps(const int* __restrict__ head, const int* __restrict__ sid,
                            const int* __restrict__ key, int n, int nsteps, int nblk,
                            int* __restrict__ step, int2* __restrict__ range,
                            int* __restrict__ base) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int s = sid[p] - 1;
    if (head[p]) step[s] = p;
    if (p == 0 || key[p] != key[p - 1]) range[key[p]].x = s;
    if (p == n - 1 || key[p] != key[p + 1]) range[key[p]].y = s + 1;
    // blocks after the previous row's up to this one's begin here (empty ones too)
    const int b = key[p], pb = p == 0 ? -1 : key[p - 1];
    for (int q = pb + 1; q <= b; q++) base[q] = p;
    if (p == n - 1) {
      step[nsteps] = n;
      for (int q = b + 1; q <= nblk; q++) base[q] = n;
    }
  }
}
__global__ void k_own_max(const int2* __restrict__ range, int nown, const int* __restrict__ base,
                          int nblk, int* __restrict__ out) {
  int s = 0, r = 0;
  for (int q = threadIdx.x; q < nown; q += blockDim.x) s = max(s, range[q].y - range[q].x);
  for (int q = threadIdx.x; q < nblk; q += blockDim.x) r = max(r, base[q + 1] - base[q]);
  atomicMax(out, s);
  atomicMax(out + 1, r);
}
// slots of the further-entry list: a row of m > 4 entries takes m - 4 + 1
__global__ void k_own_more(const int* __restrict__ perm, const int* __restrict__ tia, int n,
                           int* __restrict__ cnt) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int m = tia[perm[p] + 1] - tia[perm[p]];
    cnt[p] = m > 4 ? m - 3 : 0;
  }
}
__global__ void k_own_pack(const int* __restrict__ perm, const int* __restrict__ rows,
                           const int* __restrict__ tia, const int* __restrict__ tja,
                           const int* __restrict__ owner, const int* __restrict__ newpos,
                           const int* __restrict__ base, const int* __restrict__ more,
                           const int* __restrict__ inv, int n, int4* __restrict__ code,
                           int2* __restrict__ rec, int* __restrict__ xcode) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int t = perm[p], i = rows[t], b = owner[i], b0 = base[b];
    const int k0 = tia[t], m = tia[t + 1] - k0;
    auto of = [&](int k) {
      const int j = tja[k];
      return owner[j] == b ? ~(newpos[j] - b0) : (inv ? inv[j] : j);
    };
    int4 c = make_int4(kNoEntry, kNoEntry, kNoEntry, kNoEntry);
    if (m > 0) c.x = of(k0);
    if (m > 1) c.y = of(k0 + 1);
    if (m > 2) c.z = of(k0 + 2);
    if (m > 3) c.w = of(k0 + 3);
    code[p] = c;
    rec[p] = make_int2(inv ? inv[i] : i, m > 4 ? more[p] : -1);
    if (m > 4) {
      for (int k = 4; k < m; k++) xcode[more[p] + k - 4] = of(k0 + k);
      xcode[more[p] + m - 4] = kNoEntry;
    }
  }
}
// another vector numbering: the rows' own places and other blocks' values
__global__ void k_own_renumber(const int* __restrict__ perm, const int* __restrict__ rows,
                               const int* __restrict__ tia, const int* __restrict__ tja,
                               const int* __restrict__ inv, int n, int4* __restrict__ code,
                               int2* __restrict__ rec, int* __restrict__ xcode) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int t = perm[p], k0 = tia[t], m = tia[t + 1] - k0;
    int4 c = code[p];
    if (c.x >= 0) c.x = inv[tja[k0]];
    if (c.y >= 0) c.y = inv[tja[k0 + 1]];
    if (c.z >= 0) c.z = inv[tja[k0 + 2]];
    if (c.w >= 0) c.w = inv[tja[k0 + 3]];
    code[p] = c;
    rec[p].x = inv[rows[t]];
    for (int k = 4; k < m; k++) {
      int& x = xcode[rec[p].y + k - 4];
      if (x >= 0) x = inv[tja[k0 + k]];
    }
  }
}
template <class T>
__global__ void k_own_values(const int* __restrict__ perm, const int* __restrict__ rows,
                             const int* __restrict__ tia, const int* __restrict__ tsrc,
                             const int* __restrict__ dpos, const double* __restrict__ lval,
                             const int2* __restrict__ rec, int n, T* __restrict__ val,
                             T* __restrict__ diag, T* __restrict__ xval) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int t = perm[p], k0 = tia[t], m = tia[t + 1] - k0;
    diag[p] = (T)lval[dpos[rows[t]]];
#pragma unroll
    for (int q = 0; q < 4; q++) val[4 * (size_t)p + q] = q < m ? (T)lval[tsrc[k0 + q]] : T(0);
    for (int q = 4; q < m; q++) xval[rec[p].y + q - 4] = (T)lval[tsrc[k0 + q]];
  }
}

struct MaxInt {
  __device__ __forceinline__ int operator()(int a, int b) const { return a > b ? a : b; }
};

int own_smem_limit() {
  int dev = 0, v = 0;
  BN_CUDA(cudaGetDevice(&dev));
  BN_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return v - 1024;  // static words
}

}  // namespace

template <class T>
bool IChol::own_ready() const {
  return own_blocks > 0 && (size_t)own_rows * sizeof(T) <= (size_t)own_limit &&
         (sizeof(T) == 8 ? of.val.n > 0 : of.val32.n > 0);
}
template bool IChol::own_ready<double>() const;
template bool IChol::own_ready<float>() const;

// The schedule does not depend on the vector numbering and outlives a change of
// it, as a new smoother's colouring makes (made again, a change took 0.3 ms more
// at 300 rows and 0.4 at 75k and 2M).  One found not to suit the factor is not
// tried again in that precision.
void IChol::own_number(const int* inv, cudaStream_t s) {
  if (own_blocks > 0) {
    for (int dir = 0; dir < 2; dir++) {
      Own& w = dir ? ob : of;
      BN_LAUNCH(k_own_renumber, grid_for(n, 256), 256, 0, s, w.perm.p, dir ? border.p : order.p,
                dir ? bia.p : fia.p, dir ? bja.p : fja.p, inv, n, w.code.p, w.rec.p, w.xcode.p);
    }
  } else if (!(own_unfit & (want_f32 ? 2 : 1))) {
    own_build(inv, s);
    own_values(s);
    if (own_blocks == 0) own_unfit |= want_f32 ? 2 : 1;
  }
}

void IChol::own_drop() {
  own_blocks = own_rows = 0;
  of = Own();
  ob = Own();
  own_of.release();
}

// Partition, schedules and packed entries, in the vector numbering inv.  Left
// unbuilt (own_blocks = 0) where the rows do not fit the blocks' shared
// memory or where many rows have more than four entries.
void IChol::own_build(const int* inv, cudaStream_t s) {
  own_drop();
  if (mode != kSweepFlags || n == 0 || nlevels == 0) return;
  const char* e = getenv("BN_IC_OWN");  // 0: the chunked form throughout
  if (e && atoi(e) == 0) return;
  int dev = 0, sms = 0;
  BN_CUDA(cudaGetDevice(&dev));
  BN_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  own_limit = own_smem_limit();
  const long long cap = own_limit / (want_f32 ? 4 : 8) - kOwnSlack;
  // blocks: all rows of a level get a lane, four of them sharing a warp
  const long long lanes = (long long)nlevels * kOwnLanes * (kOwnFew / 32);
  long long nb = (n + lanes - 1) / lanes;
  if (nb < (n + cap - 1) / cap) nb = (n + cap - 1) / cap;
  if (nb > sms) nb = sms;
  if (n > nb * cap || n > nb * (want_f32 ? kOwnRows32 : kOwnRows64)) return;
  const int nown = (int)nb;
  const int g = grid_for(n, 256);
  DBuf<int> lev(n, s), dealt(nlevels, s), flag((size_t)n + 1, s);
  own_of.alloc(n, s);
  dealt.zero();
  BN_LAUNCH(k_pos_level, g, 256, 0, s, d_lptr.p, nlevels, n, lev.p);
  BN_LAUNCH(k_own_dense_levels, g, 256, 0, s, order.p, lev.p, n, (n + nown - 1) / nown, dealt.p);
  BN_LAUNCH(k_own_deal, g, 256, 0, s, order.p, lev.p, d_lptr.p, dealt.p, n, nown, own_of.p, flag.p);
  const int m = scan_counts(flag.p, n, s);
  if (m > 0) BN_LAUNCH(k_own_range, g, 256, 0, s, flag.p, n, (long long)m, nown, own_of.p);
  int rows = 0, steps = 0;
  for (int dir = 0; dir < 2; dir++) {
    Own& w = dir ? ob : of;
    const int* rw = dir ? border.p : order.p;
    const int* tia = dir ? bia.p : fia.p;
    const int* tja = dir ? bja.p : fja.p;
    DBuf<int> key(n, s), ids(n, s), skey(n, s), start(n, s), run(n, s), head(n, s), sid(n, s),
        newpos(n, s);
    w.perm.alloc(n, s);
    if (dir) BN_LAUNCH(k_pos_level, g, 256, 0, s, d_bptr.p, nlevels, n, lev.p);
    BN_LAUNCH(k_own_key, g, 256, 0, s, rw, own_of.p, n, key.p, ids.p);
    int eb = 1;
    while ((1 << eb) <= nown) eb++;
    size_t t0 = 0, t1 = 0, t2 = 0;
    BN_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t0, key.p, skey.p, ids.p, w.perm.p, n, 0, eb, s));
    BN_CUDA(cub::DeviceScan::InclusiveScan(nullptr, t1, start.p, run.p, MaxInt(), n, s));
    BN_CUDA(cub::DeviceScan::InclusiveSum(nullptr, t2, head.p, sid.p, n, s));
    DBuf<unsigned char> tmp(t0 > t1 ? (t0 > t2 ? t0 : t2) : (t1 > t2 ? t1 : t2), s);
    BN_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, t0, key.p, skey.p, ids.p, w.perm.p, n, 0, eb, s));
    BN_LAUNCH(k_own_runs, g, 256, 0, s, w.perm.p, skey.p, lev.p, rw, n, start.p, newpos.p);
    BN_CUDA(cub::DeviceScan::InclusiveScan(tmp.p, t1, start.p, run.p, MaxInt(), n, s));
    BN_LAUNCH(k_own_heads, g, 256, 0, s, run.p, n, head.p);
    BN_CUDA(cub::DeviceScan::InclusiveSum(tmp.p, t2, head.p, sid.p, n, s));
    const int nsteps = read_scalar(sid.p + (n - 1), s);
    w.step.alloc((size_t)nsteps + 1, s);
    w.range.alloc(nown, s);
    w.range.zero();
    w.base.alloc((size_t)nb + 1, s);
    BN_LAUNCH(k_own_steps, g, 256, 0, s, head.p, sid.p, skey.p, n, nsteps, (int)nb, w.step.p,
              w.range.p, w.base.p);
    DBuf<int> mx(2, s);
    mx.zero();
    BN_LAUNCH(k_own_max, 1, 1024, 0, s, w.range.p, nown, w.base.p, (int)nb, mx.p);
    DBuf<int> more((size_t)n + 1, s);
    BN_LAUNCH(k_own_more, g, 256, 0, s, w.perm.p, tia, n, more.p);
    const int nx = scan_counts(more.p, n, s);
    int h[2];
    mx.download(h, 2);
    BN_CUDA(cudaStreamSynchronize(s));
    steps = steps > h[0] ? steps : h[0];
    rows = rows > h[1] ? rows : h[1];
    if (nx > n / 4 + 1024) {
      own_drop();
      return;
    }
    w.code.alloc(n, s);
    w.rec.alloc(n, s);
    w.xcode.alloc(nx > 0 ? nx : 1, s);
    BN_LAUNCH(k_own_pack, g, 256, 0, s, w.perm.p, rw, tia, tja, own_of.p, newpos.p, w.base.p,
              more.p, inv, n, w.code.p, w.rec.p, w.xcode.p);
  }
  if (trace_on())
    fprintf(stderr, "[bn] IC(0) owner form: %d blocks, %d rows a block, %d levels, %d steps a block\n",
            (int)nb, rows, nlevels, steps);
  if (rows > cap + kOwnSlack) {
    own_drop();
    return;
  }
  own_few = nb < sms;
  own_rows = rows;
  own_blocks = (int)nb;
}

// values in the precisions in use (own_build has run)
void IChol::own_values(cudaStream_t s) {
  if (own_blocks == 0) return;
  const int g = grid_for(n, 256);
  for (int dir = 0; dir < 2; dir++) {
    Own& w = dir ? ob : of;
    const int* rw = dir ? border.p : order.p;
    const int* tia = dir ? bia.p : fia.p;
    const int* src = dir ? bsrc.p : fsrc.p;
    if (!want_f32) {  // a mixed solver sweeps in FP32 only
      w.val.alloc(4 * (size_t)n, s);
      w.diag.alloc(n, s);
      w.xval.alloc(w.xcode.n, s);
      BN_LAUNCH(k_own_values<double>, g, 256, 0, s, w.perm.p, rw, tia, src, dpos.p, L.val.p,
                w.rec.p, n, w.val.p, w.diag.p, w.xval.p);
    }
    if (want_f32) {
      w.val32.alloc(4 * (size_t)n, s);
      w.diag32.alloc(n, s);
      w.xval32.alloc(w.xcode.n, s);
      BN_LAUNCH(k_own_values<float>, g, 256, 0, s, w.perm.p, rw, tia, src, dpos.p, L.val.p,
                w.rec.p, n, w.val32.p, w.diag32.p, w.xval32.p);
    }
  }
}

// After a change of want_f32: the values in that precision, where the schedule
// (made for the precision at the time) serves it and does not have them yet.
void IChol::own_want(cudaStream_t s) {
  const size_t bytes = want_f32 ? sizeof(float) : sizeof(double);
  if (own_blocks == 0 || (want_f32 ? of.val32.n : of.val.n) > 0) return;
  if ((size_t)own_rows * bytes > (size_t)own_limit ||
      n > (long long)own_blocks * (want_f32 ? kOwnRows32 : kOwnRows64))
    return;
  own_values(s);
}

// One sweep; out holds the pending pattern everywhere.
template <class T>
void run_tri_own(const IChol& ic, bool forward, const T* in, T* out, T* clear, WaitCtl wc,
                 cudaStream_t s) {
  const IChol::Own& w = forward ? ic.of : ic.ob;
  const size_t smem = ((size_t)ic.own_rows * sizeof(T) + 15) / 16 * 16;
  const bool few = ic.own_few;
  OwnArgs<T> a;
  a.step = w.step.p;
  a.steps = w.range.p;
  a.base = w.base.p;
  a.code = w.code.p;
  a.rec = w.rec.p;
  a.xcode = w.xcode.p;
  if constexpr (sizeof(T) == 8) {
    a.val = w.val.p;
    a.diag = w.diag.p;
    a.xval = w.xval.p;
  } else {
    a.val = w.val32.p;
    a.diag = w.diag32.p;
    a.xval = w.xval32.p;
  }
  a.in = in;
  a.out = out;
  a.clear = clear;
  a.wc = wc;
  constexpr int many = sizeof(T) == 8 ? kOwnMany64 : kOwnMany32;
  auto kernel = few ? k_tri_own<T, kOwnFew> : k_tri_own<T, many>;
  static std::atomic<unsigned long long> attr_set[2] = {};
  int dev = 0;
  BN_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(attr_set[few].load() & bit)) {
    BN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 own_smem_limit()));
    attr_set[few] |= bit;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ic.own_blocks);
  cfg.blockDim = dim3(few ? kOwnFew : many);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // co-residency: waits always end
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  g_launch_count++;
  BN_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
}
// Vector index of the dependency that a wait record of a sweep holds: itself, or
// for a value of the waiting row's own block the row at that slot of the block.
int IChol::own_dep_row(bool forward, int row, int dep, cudaStream_t s) const {
  const Own& w = forward ? of : ob;
  if (dep >= 0 || own_blocks == 0) return dep;
  std::vector<int2> rec(n);
  std::vector<int> base((size_t)own_blocks + 1);
  w.rec.download(rec.data(), n);
  w.base.download(base.data(), base.size());
  BN_CUDA(cudaStreamSynchronize(s));
  for (int b = 0; b < own_blocks; b++)
    for (int p = base[b]; p < base[b + 1]; p++) {
      const int at = base[b] + ~dep;
      if (rec[p].x == row) return at < base[b + 1] ? rec[at].x : dep;
    }
  return dep;
}

// The give-up path: a factor whose first row is left out of the forward
// schedule.  entries 1: a chain; 5: five rows without dependencies, then rows of
// five, the last of them (past the four that a row keeps at hand) the missing
// row or the row before.  The vector numbering is the reverse of the rows'.
static void own_wait_selftest(int n, int entries, double limit_ms, double* elapsed_ms,
                              cudaStream_t s) {
  BN_REQUIRE(entries == 1 || entries == 5, BN_ERR_ARG, "wait self-test: 1 or 5 entries");
  BN_REQUIRE(n > entries && n <= (entries == 1 ? kOwnRows64 : 256), BN_ERR_ARG,
             "wait self-test: number of rows out of range");
  BN_REQUIRE(limit_ms > 0.0 && limit_ms <= 10000.0, BN_ERR_ARG,
             "wait self-test: limit_ms must be in (0, 10000]");
  std::vector<int> ia(1, 0), ja, inv(n);
  for (int i = 0; i < n; i++) {
    if (i >= entries) {
      for (int q = 1; q < entries; q++) ja.push_back(q);
      ja.push_back(i == entries ? 0 : i - 1);
    }
    ja.push_back(i);
    ia.push_back((int)ja.size());
    inv[i] = n - 1 - i;
  }
  CSR L;
  L.alloc(n, n, (int)ja.size(), s, true);
  L.ia.upload(ia.data(), ia.size());
  L.ja.upload(ja.data(), ja.size());
  const std::vector<double> val(ja.size(), 0.5), in(n, 1.0);
  L.val.upload(val.data(), val.size());
  DBuf<int> dinv(n, s);
  DBuf<double> din(n, s), out(n, s);
  dinv.upload(inv.data(), n);
  din.upload(in.data(), n);
  out.fill_bytes(0xff);
  IChol ic;
  ic.mode = IChol::kSweepFlags;
  ic.load(std::move(L), s);
  ic.remap(dinv.p, s);
  BN_REQUIRE(ic.own_ready<double>(), BN_ERR_ARG, "wait self-test: the owner form is off");
  const int first = 1;  // the first step begins behind its first row
  ic.of.step.upload(&first, 1);
  ic.wait.limit_ns = (unsigned long long)(limit_ms * 1e6);
  cudaEvent_t e0, e1;
  BN_CUDA(cudaEventCreate(&e0));
  BN_CUDA(cudaEventCreate(&e1));
  BN_CUDA(cudaEventRecord(e0, s));
  run_tri_own<double>(ic, true, din.p, out.p, nullptr, ic.wait.ctl(WT_SELFTEST), s);
  BN_CUDA(cudaEventRecord(e1, s));
  BN_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (elapsed_ms) *elapsed_ms = ms;
  std::string msg;
  if (ic.wait.take(s, &msg, [&](int, int row, int dep) { return ic.own_dep_row(true, row, dep, s); }))
    throw Error(BN_ERR_SPIN, "wait self-test: " + msg);
}

template void run_tri_own<double>(const IChol&, bool, const double*, double*, double*, WaitCtl,
                                  cudaStream_t);
template void run_tri_own<float>(const IChol&, bool, const float*, float*, float*, WaitCtl,
                                 cudaStream_t);

}  // namespace bn

// See include/amg_b200.h for the contract.
BN_API int amg_debug_wait_timeout_own(int n, int entries, double limit_ms, double* elapsed_ms) {
  using namespace bn;
  try {
    own_wait_selftest(n, entries, limit_ms, elapsed_ms, cudaStreamPerThread);
    set_last_error(BN_OK, "");
    return BN_OK;
  } catch (const Error& e) {
    set_last_error(e.code, e.what());
    return e.code;
  } catch (const std::exception& e) {
    set_last_error(BN_ERR_CUDA, e.what());
    return BN_ERR_CUDA;
  }
}
