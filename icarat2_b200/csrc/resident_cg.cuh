// Jacobi-PCG with every block's share of the iteration resident on its SM
// (resident_cg.cu).
#pragma once
#include "internal.cuh"

namespace icarat_b200
{

constexpr int kResidentChunk = 512; // iterations per launch unless asked

// Block tiles of BX x BY x (S kc) nodes on a grid of nbx x nby x nbz blocks
// (one per SM); (BX + 1)(BY + 1) element columns times S slabs of kc layers
// are the threads.  blocks = 0: the grid does not fit.
struct ResidentPlan
{
  int BX, BY, S, kc, nbx, nby, nbz, blocks;
  size_t smem;
};

ResidentPlan resident_plan(const GridDev &g, int sms);

// doubles of reduction workspace a launch needs
size_t resident_work(const ResidentPlan &p);

// Iterations of k_cg_spmv, k_cg_update_jacobi and k_cg_pupdate on (x, r, p)
// from the scalars *s until the stop test or `chunk` more.  z and Ap (3 numnp
// each) and work (resident_work() doubles) are scratch.
void resident_cg(cudaStream_t st, const ResidentPlan &p, const GridDev &g,
                 const KhParam<double> &kh, const double *E, const double *invd, double *x,
                 double *r, double *z, double *Ap, double *pv, double *work, CgScalars *s,
                 int chunk);
const void *resident_kernel();

} // namespace icarat_b200
