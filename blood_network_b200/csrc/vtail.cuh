// The V-cycle's coarse tail: all levels from the first small one down to the
// dense coarsest solve, run by one thread-block cluster in one launch.
#pragma once
#include "common.cuh"

namespace bn {

// What one operation does with the rows [r0, r0 + n) of its matrix (s_i the
// row's sum over its entries a_ij x_j):
enum TailKind : int {
  TK_GS0 = 0,  // y_i = (b_i - sum_{j < r0} a_ij x_j) / d_i: a class of the first sweep from x = 0
  TK_GS = 1,   // y_i = (b_i - sum_{j != i} a_ij x_j) / d_i; y is x, or (an overflow class, whose
               // rows may be adjacent) another vector that the next operation copies back
  TK_COPY = 2, // y_i = x_i
  TK_Y = 3,    // y_i = s_i
  TK_RES = 4,  // y_i = b_i - s_i
  TK_ADD = 5,  // y_i += s_i
  TK_DENSE = 6 // y = D x, D the dense FP64 inverse of the coarsest operator (n x n)
};

// b / x / y of an operation of the first level of a launch may be the caller's
// vectors instead of the level's own (which level 0 does not have)
enum TailTop : int { TT_B_IS_B = 1, TT_X_IS_X = 2, TT_X_IS_B = 4, TT_Y_IS_X = 8 };

template <class T>
struct TailOp {
  int kind, lev, r0, n;
  int lg;           // 2^lg lanes per row
  int top;          // TailTop bits
  int nmid, nlong;  // rows longer than kTailPer * lanes (a warp each) / kTailLong (a block each)
  // rows [ov0, ov0 + ovn) of x: the operation before left their values in ov;
  // this one reads them there and copies them into x
  int ov0, ovn;
  const int* ia;
  const int* ja;
  const T* a;
  const int4* list;  // n slots {row, first entry, end entry, 0}: the mid rows from the front,
                     // the long rows from the back
  const T* d;
  const T* b;
  const T* x;
  T* y;
  const T* ov;
  const double* dense;
};

constexpr int kTailPer = 8;
constexpr int kTailLong = 256;
constexpr int kTailDenseMax = 1024;  // rows of the coarsest level at most
constexpr int kTailThreads = 512;
constexpr int kTailMaxOps = 300;  // of one launch: its operations are staged in shared memory

// Fills list / nmid / nlong of ops[0..nops) on the device (any order of rows:
// every row is computed by itself).
template <class T>
void tail_lists(TailOp<T>* ops, int nops, cudaStream_t s);

// Blocks of the cluster that runs the tail on the current device (16 where the
// device places such a cluster, else 8).
int tail_cluster();

// Operations [op0, op1) in order, a cluster barrier after each.  top_lev: the
// level whose b / x are top_b / top_x; nblk: blocks of the cluster.
template <class T>
void tail_run(const TailOp<T>* ops, int op0, int op1, int top_lev, const T* top_b, T* top_x,
              int nblk, cudaStream_t s);

}  // namespace bn
