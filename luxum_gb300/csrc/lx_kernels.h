// lx_kernels.h -- host-side launchers of the kernels in lx_kernels.cu.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "lx_internal.h"

namespace lx {

// What the next `steps` (<= kAhead) steps of a handle stepped alone need that does not depend on
// its fields: step q's TF/SF tables at tab + q * p.tab_total, its source amplitude in srcv[q], its
// max|E|^2 slot ring[q] zeroed.  Step q is ctl->t + q, or p.t + q when ctl is null.
template <class C>
cudaError_t launch_prologue_ahead(const PrologueParams& p, int steps, const StepCtl* ctl, C* tab, double* srcv,
                                  unsigned long long* ring, cudaStream_t s);
// `behind`, of the launches of a step: the stream's last launch was one too, and this one may start
// beside its end.  `lanes`: one of the launches that fill a batch's streams.
// The point source of one step (its amplitude formed ahead), before the step's H update.
template <class T>
cudaError_t launch_source(T* field, long long idx, int kind, const double* v, bool behind, cudaStream_t s);
// ring[q] of the steps q in `mask` appended to the max|E|^2 series from entry `at` (ctl: from
// ctl->series, up to cap); with ctl, the counters then advance by `steps`.
cudaError_t launch_finish(const unsigned long long* ring, unsigned mask, unsigned long long* series, int at, int cap,
                          StepCtl* ctl, int steps, int rows, cudaStream_t s);
cudaError_t launch_set_ctl(StepCtl* ctl, StepCtl v, cudaStream_t s);
template <class T, class C>
cudaError_t launch_step(const StepParams<T, C>& p, bool planar, bool uniform, bool h_half, bool behind, bool lanes,
                        cudaStream_t s);
// Single-sweep planar step (float compute, two state buffers): reads the buffers named in
// p.E, p.H, p.psiH, p.psiE and writes those in p.E1, p.H1, p.psiH1, p.psiE1.
template <class T, class C>
cudaError_t launch_step_sweep2(const StepParams<T, C>& p, bool uniform, bool behind, bool lanes, cudaStream_t s);
// Single-sweep 3-D step (float compute, two state buffers), lx_sweep3d.cu: the same buffer
// convention as launch_step_sweep2.
template <class T, class C>
cudaError_t launch_step_sweep3(const StepParams<T, C>& p, bool uniform, cudaStream_t s);
template <class T>
cudaError_t launch_gather(const T* src, double* dst, const int ext[3], int Ny, int Nzp, double mul, cudaStream_t s);
template <class T>
cudaError_t launch_scatter(const double* src, T* dst, const int ext[3], int Ny, int Nzp, int mode, double a, double dt,
                           double eps0, double scale, cudaStream_t s);
template <class C>
cudaError_t launch_eps_box(C* dst, const int ext[3], int Ny, int Nzp, const int lo[3], const int hi[3], double val,
                           cudaStream_t s);
template <class T>
cudaError_t launch_probes(const ProbeParams& pp, T* const f[6], double* out, bool behind, cudaStream_t s);

template <class T>
cudaError_t launch_dft(const DftParams& d, T* const f[4], cudaStream_t s);

// Batched updates: member m of a group owns blocks [first[m], first[m+1]) of each launch;
// launch_batch_tiles turns that prefix into the per-block tile map the update kernels read.
template <class T, class C>
cudaError_t launch_batch_tiles(const StepParams<T, C>* ps, const int* first, int n, int nblocks, bool planar, int march,
                               int4* tiles, cudaStream_t s);
// row: the step's place in its sequence (the members' tables and slots of that row)
template <class T, class C>
cudaError_t launch_batch_step(const StepParams<T, C>* ps, const int4* tiles, int nblocks, bool planar, bool uniform,
                              int march, bool h_half, int row, cudaStream_t s);
// Planar members in two buffers: H and E of a step in one launch of at most kSweepMembers members.
template <class T, class C>
SweepParams<T, C> sweep_params(const StepParams<T, C>& p);
template <class T, class C>
cudaError_t launch_batch_sweep(const SweepParams<T, C>* m, int n, const int4* tiles, int nblocks, bool uniform, int R,
                               int row, cudaStream_t s);
// The blocks' tiles for it; returns the rows a warp (R) that they are for.
template <class T, class C>
int sweep_tiles(const SweepParams<T, C>* m, int n, std::vector<int4>& tiles);
// blocks one member occupies in a batched update launch; march = cells each thread walks
// along x (planar: rows 8 apart; 3-D: planes), one of 1, 2, 4, 8
int batch_blocks(int Nx, int Ny, int Nz, bool planar, int march);
// block -> {member, block within the member} for a prefix `first` of n members
cudaError_t launch_block_map(const int* first, int n, int nblocks, int2* map, cudaStream_t s);
// The fields-independent part of steps k .. k+steps-1 of every member (step k runs at ts[sim] + k;
// launch_tick advances ts): row q of the members' tables, of srcv and of slots ([row][sim]).
template <class C>
cudaError_t launch_prologue_batch(const PrologueParams* pps, const int* ts, int k, int steps, int nsims, int max_entries,
                                  double* srcv, unsigned long long* slots, cudaStream_t s);
// The point sources of step k of the members without own_source, before its H updates (amplitudes
// v[sim]).
cudaError_t launch_source_batch(const PrologueParams* pps, const int* ts, int k, int nsims, const double* v, cudaStream_t s);
cudaError_t launch_tick(int* ts, int n, int steps, cudaStream_t s);
template <class T>
cudaError_t launch_dft_batch(const DftParams* ds, const int2* map, int nplanes, int nblocks, const int* ts, int k,
                             cudaStream_t s);
cudaError_t launch_dft_flux(const double* acc, int nfreq, long long ncell, double* part, double dA, double* out,
                            cudaStream_t s);

}  // namespace lx
