// The small levels of one V-cycle as a single launch of one thread-block
// cluster (k_coarse.cu): pre-sweeps, residual restriction, the dense coarsest
// solve, prolongation and post-sweeps of every level from `top` down.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vfs_common.cuh"

namespace vfs {

constexpr int CV_NT = 512;      // threads of a block
constexpr int CV_Q = 4;         // cells a thread may own of a level (their operator in registers)
constexpr int CV_MAXBLOCKS = 16;
constexpr size_t CV_MAXCELLS = (size_t)CV_MAXBLOCKS * CV_NT * CV_Q;  // largest level
constexpr int CV_MAXLEV = 6;    // levels a launch may hold (the coarsest included)
constexpr int CV_MAXSWEEP = 8;  // smoothing sweeps per level and side
constexpr int CV_DENSE_MAX = 2048;  // largest coarsest level: its right-hand side and solution sit in every block
constexpr size_t CV_SMEM_MAX = 200 * 1024;

struct CvLevel {
  Dims d;
  const float2* ffi;  // face form (OpView)
  const float2* ffk;
  const float* ffj;
  const float* faj;
  const float* lf;       // y-line pivots 1/m
  const float* rw;       // restriction weights to the next coarser level
  const double* nvert;   // of this level (masks its right-hand side when it is a coarse level)
  const uint8_t* pcode;  // prolongation codes from the next coarser level
  int c;                 // k planes per block
  int npre, npost;
  int ox[2], osu, osp, osl, ob;  // offsets in shared memory, in floats
};
struct CvArgs {
  CvLevel lev[CV_MAXLEV];  // [0] the coarsest
  int top, cl;             // top level, blocks of the cluster
  const float* Binv;       // dense inverse of level 0
  int n0;
  int osb, ox0;            // level 0: packed right-hand side, ghosted solution
  float* b0;               // level 0's packed right-hand side on its way between the blocks (global, n0)
  float wpre[2][CV_MAXSWEEP], wpost[2][CV_MAXSWEEP];  // damping: [1] where the top level is the finest, [0] below it
  int topset;              // which set the top level takes
  const float* b;          // right-hand side of the top level (global)
  float* x;                // its solution (global)
  const int* skip;
  int nfloats;             // shared memory of a block
};

// Fills the planes per block, the offsets and nfloats for `cl` blocks from
// the level extents; false when a block would need more than CV_SMEM_MAX.
bool cv_layout(CvArgs& a, int cl);
// Blocks of the cluster this device runs for the arguments (16 or 8; 0: the
// levels stay with their own launches).
int cv_cluster(CvArgs& a);
int launch_coarse_vcycle(const CvArgs& a, cudaStream_t s);

}  // namespace vfs
