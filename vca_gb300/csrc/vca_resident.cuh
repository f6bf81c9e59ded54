// vca_resident.cuh -- whole Lanczos runs in one launch, for sectors whose
// vectors fit the shared memory of a few SMs.
#pragma once

#include "vca_batch.cuh"
#include "vca_fx.cuh"
#include "vca_multi.cuh"

namespace vca {

// A sector as the runs on it see it.
struct RsSpace {
  SectorView sv;   // "up" = the fast index (the larger spin space)
  FxView fv;       // (fixed point only)
  const int* slow_order;  // slow rows by decreasing hop count, or nullptr
  int swap;        // 1: the fast index is the down spin
  int64_t nat_up;  // DimUp of the sector: natural element index iup + idw*DimUp
};

// One run: a Green's function chain, or a sector's ground-state search.
struct RsTask {
  int space;       // its sector in RsParams::spaces
  int ncol;        // columns of the chain (2: re and im of a complex chain on a real H)
  int nlanc;       // steps asked for
  // chain: c^(dag) terms on a stored ground state
  const void* gs;          // natural order
  const int* src_words;    // words of the changed spin in the state's sector, ascending
  int src_dim, src_dimup;  // their number; DimUp of the state's sector
  int spin, dag, nterm;
  int pos[2];
  int cre[2], cim[2];      // coefficients, in {-1, 0, 1}
  double boltz, zeta, Ei;  // prefactor of the chain store
  int isign;
  double2 wfac;
  int store;               // place in the chain store
  // search: deterministic start vector; outputs per task
  int isector;
  double *theta, *svec;    // energy and residual; RS_SVEC doubles
  int* mconv;
  // vector pass: psi = sum_k s_k x_k over mconv steps (same start vector)
  void* psi;               // natural order, zeroed
};

#define RS_NMAX 512        // most steps of a search (the tridiagonal's limit)
#define RS_SVEC (7 * RS_NMAX)  // Ritz coefficients and their LU work, alpha, beta

enum { RS_CHAIN = 0, RS_SEARCH = 1, RS_VECTOR = 2 };

struct RsParams {
  const RsSpace* spaces;
  const RsTask* tasks;
  ChainStore cs;           // RS_CHAIN
  i64* scratch;            // RsShape::own 8-byte words per block of the launch
  size_t scratch_block;
  FxScales fx;             // fixed point
  MixedDiag md;            // FP64
  int split;               // FP64: 2 when an amplitude has both parts, else 1
  int diag_im;             // FP64: a one-body energy has an imaginary part
  uint64_t seed;
  double beta_tol, resid_tol;
  int check_every;
  int mode;
};

// Launch shape: C blocks of T threads in a cluster work on each task, smem
// bytes of shared memory a block.
struct RsShape {
  int C = 0, T = 0;
  size_t smem = 0, own = 0;  // own: elements of a block's rows, at most
};
// extents of `count` tasks on one sector
struct RsDims {
  int df, ds;   // fast and slow dimension
  int wd;       // slow hop width
  int ncol;
  int count;
};
// the launch shape for these tasks (C = 0: none holds them all); es: bytes of
// a vector element, fx: fixed point
RsShape rs_shape(const RsDims* dims, size_t n, int es, bool fx, int split, bool search);
// K: hopping classes (1 or 2; 1 also for none), 0 = FP64
int rs_launch(const RsParams& p, int ntask, const RsShape& s, int K, bool cplx, cudaStream_t st);

}  // namespace vca
