// mtp_launch.hpp - host launchers of the device kernels (mtp_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include "mtp_device.cuh"

namespace mtp {

constexpr int kReduceBlocks = 256;   // fixed: the reduction order never depends on the GPU

bool eval_variant_exists(bool fp64, bool vglobal, int A);
// How a launch shape of the evaluation kernel fits: blocks per SM (0: not at
// all), the stride of a staging row and a block's dynamic shared memory
// (vglobal: value space in global memory, io.vscratch holding
// blocks * A * v_size values).
struct EvalFit {
  int per_sm = 0, qs = 0;
  size_t smem = 0;
};
EvalFit eval_fit(const DevModel& md, int n_pad, int threads, bool fp64, bool vglobal, int A);
cudaError_t launch_eval(const DevModel& md, const DevIO& io, const EvalFit& fit, int threads, int blocks, bool fp64,
                        bool vglobal, int A, cudaStream_t st);

// Incoming-slot lists: for every atom k, the slots (i, s) whose neighbour is k,
// in any order (launch_force_gather sorts them).  in_ptr [natoms + 1].
// `counted`: in_cnt already holds each atom's number of slots.
cudaError_t launch_incoming(int natoms, int stride, const int* js, const int* jtypes, const int* counts,
                            int* in_cnt, int* in_ptr, int* in_slot, int* block_tmp, bool counted, cudaStream_t st);

// forces[i] = own slot gradients - incoming slot gradients; wown [natoms][6]
// = -sym(sum_s r_is (x) g_is) (LAMMPS order xx,yy,zz,xy,xz,yz); when vatom
// is non-null it receives the half/half split of every pair's virial.  `sort`:
// the incoming lists are fresh and get sorted by slot id.
cudaError_t launch_force_gather(int natoms, int stride, const double* rijs, const int* counts,
                                const double* pair_grad, const int* in_ptr, int* in_slot, bool sort,
                                double* forces, double* wown, double* vatom, cudaStream_t st);

// out[0] = sum site_energy[0..natoms), out[1..6] = sum wown; fixed order.
// out[7] = error flags; out [kTotals] holds a counter that is zero between
// calls.  The totals also go to d_energy [1] and d_virial [6] where given.
constexpr int kTotals = 9;
cudaError_t launch_totals(int natoms, const double* site_energy, const double* wown, double* partials,
                          double* out, const int* err, double* d_energy, double* d_virial, cudaStream_t st);

// Per-configuration energy [nconfig] and reference-convention stress [nconfig][6].
cudaError_t launch_config_totals(int natoms, int nconfig, const int* cfg_ptr, const double* site_energy,
                                 const double* wown, const double* volumes, double* energy, double* stress,
                                 cudaStream_t st);
// cfg_ptr [nconfig + 1] from a non-decreasing cfg_of_atom; flags bad input in err.
cudaError_t launch_config_ptr(int natoms, int nconfig, const int* cfg_of_atom, int* cfg_ptr, int* err,
                              cudaStream_t st);

// Rows [nlocal][stride] (r_ij, owner index, species, count) from positions
// x [nall][3] and candidate lists neigh [nlocal][list_stride]: candidates
// closer than cutoff, in list order; more than stride sets kErrCapacity.
// in_cnt [nlocal] gets the number of slots that point at each atom.
cudaError_t launch_rows_from_positions(int nlocal, int nall, const double* x, const int* species, const int* owner,
                                       int list_stride, const int* neigh, const int* numneigh, double cutoff,
                                       int stride, double* rijs, int* js, int* jtypes, int* counts, int* in_cnt,
                                       int* err, cudaStream_t st);

// FMA-chain peak probe.
cudaError_t measure_fma_peak(double* fp64_tflops, double* fp32_tflops);

}  // namespace mtp
