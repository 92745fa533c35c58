// lx_kernels.cu -- sm_103a kernels of the Yee time step.
//
// One step = prologue (TF/SF incident tables, point source, monitor reset; handles stepped alone
//             form the tables of several steps in one launch)
//          -> H kernel (curl E + TF/SF + CPML psi_H + H update, fused)
//          -> E kernel (curl H + TF/SF + CPML psi_E + E update + max|E|^2, fused)
// This is the order of every reference driver (e.g. three_dim_pml.cc:158-276): point source,
// E-curl, TF/SF on the curl, H update with psi, H-curl, TF/SF, E update with psi, |E|^2 max.
//
// The reference materialises each curl in a full-grid array and patches it in a separate
// pass (vfield.cc:196-275, maxwell.cc:512-812).  Here the curl of a cell lives in registers:
// each thread forms the neighbour differences of its cell, adds the TF/SF increment if the
// cell lies on a total-field-box plane (one table load), runs the psi recursion only when
// the cell lies in a CPML slab, and writes the updated component.  Cells outside the slabs
// and off the planes do 4 FP64 operations per component (3 differences + 1 FMA), which is
// the bound on GB300, whose FP64 pipe (~0.6 T lane-ops/s) limits before HBM does; they are all
// FMAs with three register operands, the pipe's fastest instruction (Fp in lx_device.cuh).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "lx_device.cuh"
#include "lx_internal.h"
#include "lx_kernels.h"

namespace lx {

// ------------------------------------------------------------------ prologue

// The entry before its plane's sign (curl - v or curl + v), in the table's type C.
template <class C>
__device__ C incident_value(const PrologueParams& p, const PatchSet& ps, int plane, int e, int t) {
  // table entry e of `plane` -> in-plane indices -> wave positions
  double pos[3];
  int rem = e;
#pragma unroll
  for (int b = 2; b >= 0; --b) {
    if (b == ps.axis) {
      pos[b] = ps.pos_n[plane];
      continue;
    }
    const int nb = ps.n[b];
    const int ib = rem % nb;
    rem /= nb;
    pos[b] = (double)(ps.lo[b] + ib) + ps.off[b];
  }
  // ((x*dx*kx + y*dy*ky + z*dz*kz) + init*dx) - t*c*dt   (maxwell.cc:289 and siblings;
  // the planar lines have no y term, maxwell.cc:206)
  double X;
  if (p.planar)
    X = __dadd_rn(__dmul_rn(__dmul_rn(pos[0], p.dx), p.kx), __dmul_rn(__dmul_rn(pos[2], p.dz), p.kz));
  else
    X = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(pos[0], p.dx), p.kx), __dmul_rn(__dmul_rn(pos[1], p.dy), p.ky)),
                  __dmul_rn(__dmul_rn(pos[2], p.dz), p.kz));
  const double tt = ps.hcurl ? (double)t : (double)t - 0.5;
  X = __dsub_rn(__dadd_rn(X, __dmul_rn(p.init, p.dx)), __dmul_rn(__dmul_rn(tt, p.c), p.dt));
  // exp(-X^2/sigma) times the set's constant factor: one exp and two multiplies per entry
  // (the reference divides by sigma, d, c and mu0 in turn; the products differ from its
  // quotients in the last bit only).  Float tables take the exponential in FP32: the position
  // arithmetic above, where x - c*t cancels, stays FP64, and the entry is stored as a float
  // either way.  The FP64 exp made the batched prologue of 256 lens simulations 23.6 us of an
  // 858 us step.
  const double a = -__dmul_rn(__dmul_rn(X, X), p.inv_sigma);
  if constexpr (sizeof(C) == 4) return (float)((double)expf((float)a) * ps.factor);
  else return __dmul_rn(exp(a), ps.factor);
}

// The point source's value at step t (three_dim_pml.cc:163; the pulse is an extension).
__device__ __forceinline__ double source_value(const PrologueParams& p, const int t) {
  if (p.src_kind == 0) {
    // amp_source*sin(omega_source*t*dt), int members (maxwell.h:203,206; three_dim_pml.cc:163)
    const int wt = (int)((unsigned)p.src_omega_i * (unsigned)t);
    return (double)p.src_amp_i * sin((double)wt * p.dt);
  }
  const double u = (t - p.src_t0) / p.src_tw;
  return p.src_amp * exp(-(u * u)) * sin(p.src_omega * t * p.dt);
}
template <class T>
__device__ __forceinline__ void source_apply(T* f, int kind, double v) {
  if constexpr (sizeof(T) == 2) {
    if (kind == 0) *f = __double2half(v);
    else *f = __float2half_rn(__half2float(*f) + (float)v);
  } else {
    if (kind == 0) *f = (T)v;
    else *f += (T)v;
  }
}

// The TF/SF tables of step t.
template <class C>
__device__ __forceinline__ void tables_body(const PrologueParams& p, const int t, C* tab_out, const int gid,
                                            const int gstride) {
  // Work items: one per entry, except that a set whose planes are normal to an axis k has no
  // component along shares its values between the two planes (the normal position is
  // multiplied by 0 in X), so one item writes both.  The sets' work ranges are staged in
  // shared memory once per block, so an item finds its set without a walk through the
  // parameter block in global memory.
  __shared__ int w_end[12];
  __shared__ unsigned char w_shared[12];
  if (threadIdx.x < 12) {  // one thread per set: the loads run in parallel
    const int s = threadIdx.x;
    const double kn[3] = {p.kx, p.ky, p.kz};
    const bool on = p.tab_total > 0 && s < p.nsets && p.sets[s].active;
    const bool sh = on && kn[p.sets[s].axis] == 0.0;
    w_end[s] = on ? (sh ? 1 : 2) * p.sets[s].plane_len : 0;
    w_shared[s] = sh;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int s = 1; s < 12; ++s) w_end[s] += w_end[s - 1];
  __syncthreads();
  const int work = w_end[11];
  for (int e = gid; e < work; e += gstride) {
    int s = 0;
    while (e >= w_end[s]) ++s;
    const PatchSet& ps = p.sets[s];
    const int rem = e - (s ? w_end[s - 1] : 0);
    const int plane = rem >= ps.plane_len ? 1 : 0;
    const int q = rem - plane * ps.plane_len;
    const C v = incident_value<C>(p, ps, plane, q, t);
    tab_out[ps.tab + plane * ps.plane_len + q] = ps.sign[plane] < 0 ? -v : v;
    if (w_shared[s]) tab_out[ps.tab + ps.plane_len + q] = ps.sign[1] < 0 ? -v : v;
  }
}

// Steps ahead of a handle stepped alone: blockIdx.y is the step of the sequence.  The launch's own
// latency (positions, exponentials and set walk in a few dependent chains, 6-7 us however small
// the tables) is paid once for up to kAhead steps instead of before every H update.
template <class C>
__global__ void prologue_ahead_kernel(const PrologueParams p, const StepCtl* ctl, C* tab, double* srcv,
                                      unsigned long long* ring) {
  const int q = blockIdx.y, t = (ctl ? ctl->t : p.t) + q;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid == 0) {
    ring[q] = 0ull;
    if (p.src_kind >= 0) srcv[q] = source_value(p, t);
  }
  tables_body<C>(p, t, tab + (long long)q * p.tab_total, gid, gridDim.x * blockDim.x);
}

template <class T>
__global__ void source_kernel(T* field, long long idx, int kind, const double* v) {
  step_behind();
  source_apply<T>(field + idx, kind, *v);
}

__global__ void finish_kernel(const unsigned long long* ring, unsigned mask, unsigned long long* series, int at, int cap,
                              StepCtl* ctl, int steps, int rows) {
  const int q = threadIdx.x;
  const int base = ctl ? ctl->series : at;
  const int n = base + __popc(mask & ((1u << q) - 1u));
  if (((mask >> q) & 1u) && n < cap) series[n] = ring[q];
  __syncwarp();
  if (q == 0 && ctl) {
    ctl->t += steps;
    ctl->row = min(ctl->row + steps, rows);
    ctl->series = min(base + __popc(mask), cap);
  }
}

__global__ void set_ctl_kernel(StepCtl* ctl, const StepCtl v) { *ctl = v; }

// Batched: blockIdx.y selects the simulation, blockIdx.z the step of the sequence.  A simulation's
// step counter lives on the device and advances once per chunk, so that a captured chunk can be
// replayed: step k of a chunk runs at ts[sim] + k.
template <class C>
__global__ void prologue_batch_kernel(const PrologueParams* __restrict__ pps, const int* __restrict__ ts, int k,
                                      double* srcv, unsigned long long* slots) {
  const PrologueParams& p = pps[blockIdx.y];
  const int q = blockIdx.z, t = ts[blockIdx.y] + k + q, gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid == 0) {
    slots[q * gridDim.y + blockIdx.y] = 0ull;
    if (p.src_kind >= 0) srcv[q * gridDim.y + blockIdx.y] = source_value(p, t);
  }
  tables_body<C>(p, t, (C*)p.tab + (long long)q * p.tab_total, gid, gridDim.x * blockDim.x);
}

__global__ void source_batch_kernel(const PrologueParams* __restrict__ pps, const int* __restrict__ ts, int k, int nsims,
                                    const double* __restrict__ v) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsims) return;
  const PrologueParams& p = pps[s];
  if (p.src_kind < 0 || p.own_source) return;
  void* const f = (((ts[s] + k) & 1) && p.src_field1) ? p.src_field1 : p.src_field;  // the state the step reads
  if (p.prec == 0) source_apply((double*)f + p.src_idx, p.src_kind, v[s]);
  else if (p.prec == 1) source_apply((float*)f + p.src_idx, p.src_kind, v[s]);
  else source_apply((__half*)f + p.src_idx, p.src_kind, v[s]);
}

__global__ void tick_kernel(int* ts, int n, int steps) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) ts[s] += steps;
}

// ------------------------------------------------------------------ 3-D kernels

// H half-step over cell (i,j,k) for Hx, Hy, Hz (three_dim_pml.cc:176-213, three_dim.cc:101-132).
// A cell's loads (h_load) are all issued before its update and stores (h_apply).  (Threads
// that own two cells and issue both cells' loads first were tried: the doubled registers
// halve the resident blocks and the kernels ran 12-15 % slower.)
template <class C>
struct HCell {
  long long c;
  bool ux, uy, uz;
  C ex, ey, ez, ez_j, ey_k, ex_k, ez_i, ey_i, ex_j, hx, hy, hz;
};

template <class T, class C, bool FAST = false>
__device__ __forceinline__ void h_load(const StepParams<T, C>& p, const int i, const int j, const int k, HCell<C>& v) {
  const long long c = (long long)i * p.si + (long long)j * p.sj + k;
  const bool ux = FAST || (j < p.Ny - 1 && k < p.Nz - 1), uy = FAST || (i < p.Nx - 1 && k < p.Nz - 1),
             uz = FAST || (i < p.Nx - 1 && j < p.Ny - 1);
  v.c = c;
  v.ux = ux;
  v.uy = uy;
  v.uz = uz;
  // Every load is issued before any store: the field arrays may alias as far as the compiler
  // knows, so interleaving would serialise one memory round trip per component.
  v.ex = ld<T, C>(p.E[0] + c);
  v.ey = ld<T, C>(p.E[1] + c);
  v.ez = ld<T, C>(p.E[2] + c);
  v.ez_j = ux ? ld<T, C>(p.E[2] + c + p.sj) : C(0);
  v.ey_k = ux ? ld<T, C>(p.E[1] + c + 1) : C(0);
  v.ex_k = uy ? ld<T, C>(p.E[0] + c + 1) : C(0);
  v.ez_i = uy ? ld<T, C>(p.E[2] + c + p.si) : C(0);
  v.ey_i = uz ? ld<T, C>(p.E[1] + c + p.si) : C(0);
  v.ex_j = uz ? ld<T, C>(p.E[0] + c + p.sj) : C(0);
  v.hx = ux ? ld<T, C>(p.H[0] + c) : C(0);
  v.hy = uy ? ld<T, C>(p.H[1] + c) : C(0);
  v.hz = uz ? ld<T, C>(p.H[2] + c) : C(0);
}

template <class T, class C, bool UNI, bool FAST = false>
__device__ __forceinline__ void h_apply(const StepParams<T, C>& p, const int i, const int j, const int k, bool tf,
                                        const HCell<C>& v) {
  const long long c = v.c;
  const bool ux = FAST || v.ux, uy = FAST || v.uy, uz = FAST || v.uz;
  if (FAST) tf = false;
  const C ex = v.ex, ey = v.ey, ez = v.ez, ez_j = v.ez_j, ey_k = v.ey_k, ex_k = v.ex_k, ez_i = v.ez_i, ey_i = v.ey_i,
          ex_j = v.ex_j, hx = v.hx, hy = v.hy, hz = v.hz;
  int sx = -1, sy = -1, sz = -1;
  if (!FAST && p.pml) {
    sx = slab_index(p.slab[0], i);
    sy = slab_index(p.slab[1], j);
    sz = slab_index(p.slab[2], k);
  }
  C nhx = hx, nhy = hy, nhz = hz;
  const Fp<C> fp(k);
  const C mdb = fp.neg(p.Dbs);
  // Hx: i < Nx, j < Ny-1, k < Nz-1; part 1 = dEz/dy (y profile), part 2 = dEy/dz (z profile)
  if (ux) {
    C d1 = fp.sub(ez_j, ez), d2 = fp.sub(ey_k, ey);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[1])); d2 = fp.mul(d2, fp.reg(p.rd[2])); }
    if (tf) {
      tfsf_apply<C>(p.setsH[0][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsH[0][1], p.tab, i, j, k, d2);
    }
    if (sy >= 0) d1 = pml_term<C>(fp, d1, p.psiH[0][0] + psi_index(1, p.slab[1], sy, i, j, k, p.Ny, p.Nzp), p.bH[1][j], p.cH[1][j], p.rkH[1][j]);
    if (sz >= 0) d2 = pml_term<C>(fp, d2, p.psiH[0][1] + psi_index(2, p.slab[2], sz, i, j, k, p.Ny, p.Nzp), p.bH[2][k], p.cH[2][k], p.rkH[2][k]);
    nhx = fmaC(mdb, fp.sub(d1, d2), hx);
  }
  // Hy: i < Nx-1, j < Ny, k < Nz-1; part 1 = dEx/dz (z), part 2 = dEz/dx (x)
  if (uy) {
    C d1 = fp.sub(ex_k, ex), d2 = fp.sub(ez_i, ez);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[2])); d2 = fp.mul(d2, fp.reg(p.rd[0])); }
    if (tf) {
      tfsf_apply<C>(p.setsH[1][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsH[1][1], p.tab, i, j, k, d2);
    }
    if (sz >= 0) d1 = pml_term<C>(fp, d1, p.psiH[1][0] + psi_index(2, p.slab[2], sz, i, j, k, p.Ny, p.Nzp), p.bH[2][k], p.cH[2][k], p.rkH[2][k]);
    if (sx >= 0) d2 = pml_term<C>(fp, d2, p.psiH[1][1] + psi_index(0, p.slab[0], sx, i, j, k, p.Ny, p.Nzp), p.bH[0][i], p.cH[0][i], p.rkH[0][i]);
    nhy = fmaC(mdb, fp.sub(d1, d2), hy);
  }
  // Hz: i < Nx-1, j < Ny-1, k < Nz; part 1 = dEy/dx (x), part 2 = dEx/dy (y)
  if (uz) {
    C d1 = fp.sub(ey_i, ey), d2 = fp.sub(ex_j, ex);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[0])); d2 = fp.mul(d2, fp.reg(p.rd[1])); }
    if (tf) {
      tfsf_apply<C>(p.setsH[2][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsH[2][1], p.tab, i, j, k, d2);
    }
    if (sx >= 0) d1 = pml_term<C>(fp, d1, p.psiH[2][0] + psi_index(0, p.slab[0], sx, i, j, k, p.Ny, p.Nzp), p.bH[0][i], p.cH[0][i], p.rkH[0][i]);
    if (sy >= 0) d2 = pml_term<C>(fp, d2, p.psiH[2][1] + psi_index(1, p.slab[1], sy, i, j, k, p.Ny, p.Nzp), p.bH[1][j], p.cH[1][j], p.rkH[1][j]);
    nhz = fmaC(mdb, fp.sub(d1, d2), hz);
  }
  if (ux) st<T, C>(p.H[0] + c, nhx);
  if (uy) st<T, C>(p.H[1] + c, nhy);
  if (uz) st<T, C>(p.H[2] + c, nhz);
}

template <class T, class C, bool UNI, bool FAST = false>
__device__ __forceinline__ void h_cell_3d(const StepParams<T, C>& p, const int i, const int j, const int k,
                                          const bool tf) {
  HCell<C> v;
  h_load<T, C, FAST>(p, i, j, k, v);
  h_apply<T, C, UNI, FAST>(p, i, j, k, tf, v);
}

// An array's element at a byte offset (an unsigned 32-bit one is added by the load instruction).
template <class T, class O>
__device__ __forceinline__ const T* at(const T* p, O o) {
  return reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + o);
}
template <class T, class O>
__device__ __forceinline__ T* at(T* p, O o) {
  return reinterpret_cast<T*>(reinterpret_cast<char*>(p) + o);
}

// Paths of a block: the slab of one axis (0, 1, 2), none, the general code, interior.
constexpr int kNoSlab = 3, kGeneral = 4, kInside = 5;

// Whether the slab paths also take blocks that meet TF/SF planes: FP16 storage, bound by
// instructions (201x187x259 193 -> 189 us a step).  FP32 is bound by memory and lost to the longer
// code more than it gained (512x512x128 598 -> 611).
template <class T>
constexpr bool kSlabTf = sizeof(T) == 2;

// The two psi terms of a cell in the slab of one axis AX: both half steps form the derivative
// along AX in part 1 of component AX+1 and part 0 of component AX+2, with one profile and one
// index for both.  Loaded with the cell's fields, ahead of every store (see h_load).
template <class C, class Off>
struct AxisPsi {
  bool on;
  Off q;         // in bytes
  C a, b;        // psi of component AX+1 part 1, AX+2 part 0
  C fb, fc, rk;  // profile b, c, 1/kappa
};

template <class T, class C, int AX, class Off>
__device__ __forceinline__ void axis_psi_load(const StepParams<T, C>& p, C* const (&psi)[3][2], const C* fb, const C* fc,
                                              const C* rk, int i, int j, int k, unsigned o, AxisPsi<C, Off>& w) {
  const int u = AX == 0 ? i : (AX == 1 ? j : k);
  const int s = u < p.free0[AX] ? u : u - p.free1[AX] + p.free0[AX];
  w.on = AX == 0 || u < p.free0[AX] || u >= p.free1[AX];
  if (w.on) {
    // the offset of the block's plane (or slab plane) is uniform, the rest 32 bits
    const unsigned n = p.slab[AX].n;
    const long long base = AX == 0 ? (long long)s * p.si : (AX == 1 ? (long long)i * n * p.Nzp : (long long)i * p.Ny * n);
    const unsigned q = AX == 0 ? o : (AX == 1 ? (unsigned)s * p.Nzp + k : (unsigned)j * n + s);
    w.q = (Off)(base + q) * (Off)sizeof(C);
    w.a = *at(psi[(AX + 1) % 3][1], w.q);
    w.b = *at(psi[(AX + 2) % 3][0], w.q);
    w.fb = __ldg(fb + u);
    w.fc = __ldg(fc + u);
    w.rk = __ldg(rk + u);
  }
}
// pml_term's arithmetic on a loaded psi.
template <class C, class Off>
__device__ __forceinline__ void axis_psi_term(const AxisPsi<C, Off>& w, C& psi, C& d) {
  psi = fmaC(w.fb, psi, w.fc * d);
  d = fmaC(d, w.rk, psi);
}

// H of a cell on planes 1 .. Nx-2 whose block meets the CPML slab of axis AX only
// (AX = 3: no slab, a block at the y or z walls): h_apply's arithmetic.  In h_apply each psi
// term's load waits behind the previous term's store (the arrays may alias as far as the compiler
// knows), and its conditions and 64-bit offsets double a cell's instructions.  Here every load is
// issued first and unconditionally (off these planes' walls a neighbour is memory of the same
// array, whatever it holds), and only the stores ask whether the cell updates.
template <class T, class C, bool UNI, int AX>
__device__ __forceinline__ void h_slab_3d(const StepParams<T, C>& p, const int i, const int j, const int k,
                                          const unsigned tf) {
  // FP32 keeps h_load's conditions: with the plain loads the kernel spills 12-36 bytes at its 32
  // registers, on the way of every block (512x512x128 H 265 us a launch against 269-282), which
  // FP16 storage, bound by instructions, makes up for (256^3 H 135 -> 124).
  constexpr bool kPlain = sizeof(T) == 2;
  HCell<C> v;
  const unsigned o = (unsigned)j * (unsigned)p.Nzp + (unsigned)k;
  if constexpr (kPlain) {
    const long long c = (long long)i * p.si + o;
    const bool jn = j < p.Ny - 1, kn = k < p.Nz - 1;
    v.c = c;
    v.ux = jn && kn;
    v.uy = kn;
    v.uz = jn;
    v.ex = ld<T, C>(p.E[0] + c);
    v.ey = ld<T, C>(p.E[1] + c);
    v.ez = ld<T, C>(p.E[2] + c);
    v.ez_j = ld<T, C>(p.E[2] + c + p.Nzp);
    v.ex_j = ld<T, C>(p.E[0] + c + p.Nzp);
    v.ey_k = ld<T, C>(p.E[1] + c + 1);
    v.ex_k = ld<T, C>(p.E[0] + c + 1);
    v.ez_i = ld<T, C>(p.E[2] + c + p.si);
    v.ey_i = ld<T, C>(p.E[1] + c + p.si);
    v.hx = ld<T, C>(p.H[0] + c);
    v.hy = ld<T, C>(p.H[1] + c);
    v.hz = ld<T, C>(p.H[2] + c);
  } else {
    h_load<T, C>(p, i, j, k, v);
  }
  const bool u[3] = {v.ux, v.uy, v.uz};
  constexpr int A = (AX + 1) % 3, B = (AX + 2) % 3;
  AxisPsi<C, long long> w;
  if constexpr (AX < 3) {
    if constexpr (kPlain) {
      axis_psi_load<T, C, AX>(p, p.psiH, p.bH[AX], p.cH[AX], p.rkH[AX], i, j, k, o, w);
    } else {
      const int n = AX == 0 ? i : (AX == 1 ? j : k);
      const int sl = slab_index(p.slab[AX], n);
      w.on = sl >= 0 && (u[A] || u[B]);
      w.a = w.b = w.fb = w.fc = w.rk = C(0);
      w.q = 0;
      if (w.on) {
        w.q = psi_index(AX, p.slab[AX], sl, i, j, k, p.Ny, p.Nzp) * (long long)sizeof(C);
        if (u[A]) w.a = *at(p.psiH[A][1], w.q);
        if (u[B]) w.b = *at(p.psiH[B][0], w.q);
        w.fb = __ldg(p.bH[AX] + n);
        w.fc = __ldg(p.cH[AX] + n);
        w.rk = __ldg(p.rkH[AX] + n);
      }
    }
  }
  // d[c][part]: Hx: dEz/dy, dEy/dz; Hy: dEx/dz, dEz/dx; Hz: dEy/dx, dEx/dy
  C d[3][2] = {{v.ez_j - v.ez, v.ey_k - v.ey}, {v.ex_k - v.ex, v.ez_i - v.ez}, {v.ey_i - v.ey, v.ex_j - v.ex}};
  if (!UNI) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      d[m][0] = mulC(d[m][0], p.rd[(m + 1) % 3]);
      d[m][1] = mulC(d[m][1], p.rd[(m + 2) % 3]);
    }
  }
  if (kSlabTf<T> && tf) {
    if (tf & 1u) {
      tfsf_axis<0, C>(p.setsH[1][1], p.tab, i, j, k, d[1][1]);
      tfsf_axis<0, C>(p.setsH[2][0], p.tab, i, j, k, d[2][0]);
    }
    if (tf & 2u) {
      tfsf_axis<1, C>(p.setsH[0][0], p.tab, i, j, k, d[0][0]);
      tfsf_axis<1, C>(p.setsH[2][1], p.tab, i, j, k, d[2][1]);
    }
    if (tf & 4u) {
      tfsf_axis<2, C>(p.setsH[0][1], p.tab, i, j, k, d[0][1]);
      tfsf_axis<2, C>(p.setsH[1][0], p.tab, i, j, k, d[1][0]);
    }
  }
  if constexpr (AX < 3) {
    if (w.on) {
      if (kPlain || u[A]) axis_psi_term(w, w.a, d[A][1]);
      if (kPlain || u[B]) axis_psi_term(w, w.b, d[B][0]);
      if (u[A]) *at(p.psiH[A][1], w.q) = w.a;
      if (u[B]) *at(p.psiH[B][0], w.q) = w.b;
    }
  }
  if (u[0]) st<T, C>(p.H[0] + v.c, fmaC(-p.Dbs, d[0][0] - d[0][1], v.hx));
  if (u[1]) st<T, C>(p.H[1] + v.c, fmaC(-p.Dbs, d[1][0] - d[1][1], v.hy));
  if (u[2]) st<T, C>(p.H[2] + v.c, fmaC(-p.Dbs, d[2][0] - d[2][1], v.hz));
}

// Whether a tile lies where every component updates and no slab reaches.
template <class T, class C>
__device__ __forceinline__ bool tile_in(const StepParams<T, C>& p, int i, int j0, int nj, int k0, int nk) {
  return i >= p.in0[0] && i < p.in1[0] && j0 >= p.in0[1] && j0 + nj <= p.in1[1] && k0 >= p.in0[2] && k0 + nk <= p.in1[2];
}

// The path of a block that is not interior: kGeneral when it meets the slabs of two axes, an x wall or
// (FP32) a TF/SF plane, else the axis of the one slab it meets, or kNoSlab.
template <class T, class C>
__device__ __forceinline__ int slab_path(const StepParams<T, C>& p, unsigned tf, int i, int j0, int nj, int k0, int nk) {
  if (i < 1 || i > p.Nx - 2) return kGeneral;
  const bool x = i < p.free0[0] || i >= p.free1[0];
  const bool y = j0 < p.free0[1] || min(j0 + nj, p.Ny) > p.free1[1];
  const bool z = k0 < p.free0[2] || min(k0 + nk, p.Nz) > p.free1[2];
  if (x + y + z > 1 || (!kSlabTf<T> && tf)) return kGeneral;
  return x ? 0 : (y ? 1 : (z ? 2 : kNoSlab));
}

// Resident blocks per SM asked of the compiler for the H kernel (a register cap): 8 for
// float compute (32 registers, 0-28 bytes spilled; FP16 storage 14 % faster than at 40
// registers), 5 for FP64 (its natural 48 registers; an explicit 1 lets the compiler take 54).
template <class C>
struct HMinBlocks {
  static constexpr int v = sizeof(C) == 4 ? 8 : 5;
};

// The z cells of a 3-D block.  Plain tiles are ZW consecutive cells (32, or 16 for float
// storage: a block is ZW z cells x 256/ZW y rows).  With zends (FP64 grids whose z CPML slabs
// are at most 16 cells wide; ZW = 32), tile 0 is the row's two ends, k in [0, 16) and
// [Nz-16, Nz), and tile m > 0 is [16 + 32(m-1), +32) up to Nz-16.  A 32-cell row's first and
// last tiles are half slab, and their warps run the z psi code with half the lanes idle; the
// end tile runs it once with all lanes busy, and sixteen doubles keep the other tiles on
// 128-byte lines.  Sixteen floats are half a line, so float storage takes 16-cell tiles
// instead: its slab tiles are whole slab, and half as many.  Each thread has one cell
// (valid = inside its tile's range).
struct ZTile {
  int k;
  bool valid;
  int lo0, n0, lo1, n1;  // the tile's cells: [lo0, lo0+n0) and [lo1, lo1+n1)
};

template <int ZW>
__device__ __forceinline__ ZTile z_tile(int Nz, bool ends) {
  ZTile z;
  const int lane = threadIdx.x;
  if (ZW != 32 || !ends) {
    z.lo0 = blockIdx.x * ZW;
    z.n0 = ZW;
    z.lo1 = z.n1 = 0;
    z.k = z.lo0 + lane;
    z.valid = z.k < Nz;
  } else if (blockIdx.x == 0) {
    z.lo0 = 0;
    z.n0 = 16;
    z.lo1 = Nz - 16;
    z.n1 = 16;
    z.k = lane < 16 ? lane : Nz - 32 + lane;
    z.valid = true;
  } else {
    z.lo0 = 16 + (blockIdx.x - 1) * 32;
    z.n0 = min(32, Nz - 16 - z.lo0);
    z.lo1 = z.n1 = 0;
    z.k = z.lo0 + lane;
    z.valid = lane < z.n0;
  }
  return z;
}

// Whether a 3-D block's tile (rows [j0, j0+nj)) meets a TF/SF plane.
__device__ __forceinline__ bool ztile_meets_planes(const int (&pl)[3][2], int i, int j0, int nj, const ZTile& z) {
  return tile_meets_planes(pl, i, 1, j0, nj, z.lo0, z.n0) || (z.n1 > 0 && tile_meets_planes(pl, i, 1, j0, nj, z.lo1, z.n1));
}
// The axes whose planes it meets, as bits.
__device__ __forceinline__ unsigned ztile_plane_axes(const int (&pl)[3][2], int i, int j0, int nj, const ZTile& z) {
  unsigned t = tile_plane_axes(pl, i, 1, j0, nj, z.lo0, z.n0);
  if (z.n1 > 0) t |= tile_plane_axes(pl, i, 1, j0, nj, z.lo1, z.n1);
  return t;
}

// One cell per thread; a block is ZW (z) x 256/ZW (y) cells of one x plane.  Blocks whose tile
// is interior take the cell code with every condition decided at compile time.
template <class T, class C, bool UNI, bool SLAB, int ZW>
__global__ void __launch_bounds__(256, HMinBlocks<C>::v) h_kernel_3d(const StepParams<T, C> p) {
  step_behind();
  step_open();
  constexpr int RY = 256 / ZW;
  const ZTile z = z_tile<ZW>(p.Nz, p.zends);
  const int k = z.k;
  const int j = blockIdx.y * RY + threadIdx.y;
  const int i = blockIdx.z;
  if (!z.valid || j >= p.Ny) return;
  std::conditional_t<SLAB && kSlabTf<T>, unsigned, bool> tf = 0;
  if constexpr (SLAB && kSlabTf<T>) tf = p.tfsf ? ztile_plane_axes(p.planesH, i, blockIdx.y * RY, RY, z) : 0u;
  else tf = p.tfsf && ztile_meets_planes(p.planesH, i, blockIdx.y * RY, RY, z);
  if (!tf && z.n1 == 0 && tile_is_interior(p.slab, p.pml, p.Nx, p.Ny, p.Nz, i, 1, blockIdx.y * RY, RY, z.lo0, z.n0))
    h_cell_3d<T, C, UNI, true>(p, i, j, k, false);
  else {
    const int path = SLAB ? slab_path(p, tf, i, blockIdx.y * RY, RY, z.lo0, z.n0) : kGeneral;
    if (path == 0) h_slab_3d<T, C, UNI, 0>(p, i, j, k, tf);
    else if (path == 1) h_slab_3d<T, C, UNI, 1>(p, i, j, k, tf);
    else if (path == 2) h_slab_3d<T, C, UNI, 2>(p, i, j, k, tf);
    else if (path == kNoSlab) h_slab_3d<T, C, UNI, kNoSlab>(p, i, j, k, tf);
    else h_cell_3d<T, C, UNI>(p, i, j, k, tf != 0);
  }
}

// E half-step over cell (i,j,k) for Ex, Ey, Ez (three_dim_pml.cc:218-276, three_dim.cc:134-189).
// Only cells where the reference's H-curl is computed (vfield.cc:241-269: the transverse
// index in [1, N-2]) change; on the PEC walls the reference adds Cb*0 and psi stays 0.
// Returns the bit pattern of this cell's |E|^2 when monitoring (0 otherwise).
template <class C>
struct ECell {
  long long c;
  bool ux, uy, uz, mon;
  C hx, hy, hz, hz_j, hy_k, hx_k, hz_i, hy_i, hx_j, ex, ey, ez, cbx, cby, cbz;
};

template <class T, class C, bool MON, bool FAST = false>
__device__ __forceinline__ void e_load(const StepParams<T, C>& p, const int i, const int j, const int k, ECell<C>& v) {
  const long long c = (long long)i * p.si + (long long)j * p.sj + k;
  const bool ii = (i >= 1 && i < p.Nx - 1), jj = (j >= 1 && j < p.Ny - 1), kk = (k >= 1 && k < p.Nz - 1);
  const bool ux = FAST || (i < p.Nx - 1 && jj && kk), uy = FAST || (ii && j < p.Ny - 1 && kk),
             uz = FAST || (ii && jj && k < p.Nz - 1);
  const bool mon = MON && (FAST || (i < p.Nx - 1 && j < p.Ny - 1 && k < p.Nz - 1));
  v.c = c;
  v.ux = ux;
  v.uy = uy;
  v.uz = uz;
  v.mon = mon;
  // all loads first (see h_load)
  v.hx = ld<T, C>(p.H[0] + c);
  v.hy = ld<T, C>(p.H[1] + c);
  v.hz = ld<T, C>(p.H[2] + c);
  v.hz_j = ux ? ld<T, C>(p.H[2] + c - p.sj) : C(0);
  v.hy_k = ux ? ld<T, C>(p.H[1] + c - 1) : C(0);
  v.hx_k = uy ? ld<T, C>(p.H[0] + c - 1) : C(0);
  v.hz_i = uy ? ld<T, C>(p.H[2] + c - p.si) : C(0);
  v.hy_i = uz ? ld<T, C>(p.H[1] + c - p.si) : C(0);
  v.hx_j = uz ? ld<T, C>(p.H[0] + c - p.sj) : C(0);
  v.ex = (ux || mon) ? ld<T, C>(p.E[0] + c) : C(0);
  v.ey = (uy || mon) ? ld<T, C>(p.E[1] + c) : C(0);
  v.ez = (uz || mon) ? ld<T, C>(p.E[2] + c) : C(0);
  v.cbx = ux ? p.Cbs[0][c] : C(0);
  v.cby = uy ? p.Cbs[1][c] : C(0);
  v.cbz = uz ? p.Cbs[2][c] : C(0);
}

template <class T, class C, bool UNI, bool MON, bool FAST = false>
__device__ __forceinline__ typename MaxBits<C>::type e_apply(const StepParams<T, C>& p, const int i, const int j,
                                                             const int k, bool tf, const ECell<C>& v,
                                                             const MaxScreen<C>& scr) {
  const long long c = v.c;
  const bool ux = FAST || v.ux, uy = FAST || v.uy, uz = FAST || v.uz, mon = MON && (FAST || v.mon);
  if (FAST) tf = false;
  const C hx = v.hx, hy = v.hy, hz = v.hz, hz_j = v.hz_j, hy_k = v.hy_k, hx_k = v.hx_k, hz_i = v.hz_i, hy_i = v.hy_i,
          hx_j = v.hx_j, ex = v.ex, ey = v.ey, ez = v.ez, cbx = v.cbx, cby = v.cby, cbz = v.cbz;
  int sx = -1, sy = -1, sz = -1;
  if (!FAST && p.pml) {
    sx = slab_index(p.slab[0], i);
    sy = slab_index(p.slab[1], j);
    sz = slab_index(p.slab[2], k);
  }
  C exn = ex, eyn = ey, ezn = ez;
  const Fp<C> fp(k);
  // Ex: i < Nx-1, j in [1,Ny-2], k in [1,Nz-2]; part 1 = dHz/dy (y), part 2 = dHy/dz (z)
  if (ux) {
    C d1 = fp.sub(hz, hz_j), d2 = fp.sub(hy, hy_k);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[1])); d2 = fp.mul(d2, fp.reg(p.rd[2])); }
    if (tf) {
      tfsf_apply<C>(p.setsE[0][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsE[0][1], p.tab, i, j, k, d2);
    }
    if (sy >= 0) d1 = pml_term<C>(fp, d1, p.psiE[0][0] + psi_index(1, p.slab[1], sy, i, j, k, p.Ny, p.Nzp), p.bE[1][j], p.cE[1][j], p.rkE[1][j]);
    if (sz >= 0) d2 = pml_term<C>(fp, d2, p.psiE[0][1] + psi_index(2, p.slab[2], sz, i, j, k, p.Ny, p.Nzp), p.bE[2][k], p.cE[2][k], p.rkE[2][k]);
    exn = fmaC(cbx, fp.sub(d1, d2), ex);
  }
  // Ey: i in [1,Nx-2], j < Ny-1, k in [1,Nz-2]; part 1 = dHx/dz (z), part 2 = dHz/dx (x)
  if (uy) {
    C d1 = fp.sub(hx, hx_k), d2 = fp.sub(hz, hz_i);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[2])); d2 = fp.mul(d2, fp.reg(p.rd[0])); }
    if (tf) {
      tfsf_apply<C>(p.setsE[1][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsE[1][1], p.tab, i, j, k, d2);
    }
    if (sz >= 0) d1 = pml_term<C>(fp, d1, p.psiE[1][0] + psi_index(2, p.slab[2], sz, i, j, k, p.Ny, p.Nzp), p.bE[2][k], p.cE[2][k], p.rkE[2][k]);
    if (sx >= 0) d2 = pml_term<C>(fp, d2, p.psiE[1][1] + psi_index(0, p.slab[0], sx, i, j, k, p.Ny, p.Nzp), p.bE[0][i], p.cE[0][i], p.rkE[0][i]);
    eyn = fmaC(cby, fp.sub(d1, d2), ey);
  }
  // Ez: i in [1,Nx-2], j in [1,Ny-2], k < Nz-1; part 1 = dHy/dx (x), part 2 = dHx/dy (y)
  if (uz) {
    C d1 = fp.sub(hy, hy_i), d2 = fp.sub(hx, hx_j);
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[0])); d2 = fp.mul(d2, fp.reg(p.rd[1])); }
    if (tf) {
      tfsf_apply<C>(p.setsE[2][0], p.tab, i, j, k, d1);
      tfsf_apply<C>(p.setsE[2][1], p.tab, i, j, k, d2);
    }
    if (sx >= 0) d1 = pml_term<C>(fp, d1, p.psiE[2][0] + psi_index(0, p.slab[0], sx, i, j, k, p.Ny, p.Nzp), p.bE[0][i], p.cE[0][i], p.rkE[0][i]);
    if (sy >= 0) d2 = pml_term<C>(fp, d2, p.psiE[2][1] + psi_index(1, p.slab[1], sy, i, j, k, p.Ny, p.Nzp), p.bE[1][j], p.cE[1][j], p.rkE[1][j]);
    ezn = fmaC(cbz, fp.sub(d1, d2), ez);
  }
  if (ux) st<T, C>(p.E[0] + c, exn);
  if (uy) st<T, C>(p.E[1] + c, eyn);
  if (uz) st<T, C>(p.E[2] + c, ezn);
  typename MaxBits<C>::type mbits = 0;
  if (mon && (p.etotal || scr.may(exn, eyn, ezn))) {
    // Etotal = Ez*Ez + Ey*Ey + Ex*Ex (three_dim_pml.cc:270), same association order
    const C e2 = fmaC(exn, exn, fmaC(eyn, eyn, fp.mul(ezn, ezn)));
    if (p.etotal) p.etotal[c] = e2;
    mbits = MaxBits<C>::of(e2);
  }
  return mbits;
}

template <class T, class C, bool UNI, bool MON, bool FAST = false>
__device__ __forceinline__ typename MaxBits<C>::type e_cell_3d(const StepParams<T, C>& p, const int i, const int j,
                                                               const int k, const bool tf) {
  ECell<C> v;
  const MaxScreen<C> scr(MON ? p.max_slot : nullptr);
  e_load<T, C, MON, FAST>(p, i, j, k, v);
  return e_apply<T, C, UNI, MON, FAST>(p, i, j, k, tf, v, scr);
}

// E of a cell on planes 1 .. Nx-2 whose block meets the CPML slab of axis AX only
// (see h_slab_3d): e_apply's arithmetic.  FP16 storage reads at 32-bit byte offsets and takes
// interior cells too (201x187x259 E 108 -> 104 us a launch, 256^3 monitored 191 -> 165; the same in
// h_slab_3d cost H 4-8 us of 92 there and 9 of 262 at 512x512x128 FP32); FP32 comes here with
// arrays that such offsets do not reach.
template <class T, class C, bool UNI, bool MON, int AX>
__device__ __forceinline__ typename MaxBits<C>::type e_slab_3d(const StepParams<T, C>& p, const int i, const int j,
                                                               const int k, const unsigned tf) {
  using Off = std::conditional_t<sizeof(T) == 2, unsigned, long long>;
  const unsigned o = (unsigned)j * (unsigned)p.Nzp + (unsigned)k;
  const Off c = (Off)i * (Off)p.si + o, b = c * (Off)sizeof(T), bi = b - (Off)p.si * (Off)sizeof(T),
            bj = b - p.Nzp * (Off)sizeof(T), bc = c * (Off)sizeof(C);
  const C hx = ld<T, C>(at(p.H[0], b)), hy = ld<T, C>(at(p.H[1], b)), hz = ld<T, C>(at(p.H[2], b));
  const C hz_j = ld<T, C>(at(p.H[2], bj)), hx_j = ld<T, C>(at(p.H[0], bj));
  const C hy_k = ld<T, C>(at(p.H[1], b) - 1), hx_k = ld<T, C>(at(p.H[0], b) - 1);
  const C hz_i = ld<T, C>(at(p.H[2], bi)), hy_i = ld<T, C>(at(p.H[1], bi));
  const C ex = ld<T, C>(at(p.E[0], b)), ey = ld<T, C>(at(p.E[1], b)), ez = ld<T, C>(at(p.E[2], b));
  const C cb[3] = {*at(p.Cbs[0], bc), *at(p.Cbs[1], bc), *at(p.Cbs[2], bc)};
  AxisPsi<C, Off> w;
  if constexpr (AX < 3) axis_psi_load<T, C, AX>(p, p.psiE, p.bE[AX], p.cE[AX], p.rkE[AX], i, j, k, o, w);
  constexpr bool in = AX == kInside;
  const bool jn = in || j < p.Ny - 1, kn = in || k < p.Nz - 1, jj = in || (j >= 1 && jn), kk = in || (k >= 1 && kn);
  const bool u[3] = {jj && kk, jn && kk, jj && kn};
  // d[c][part]: Ex: dHz/dy, dHy/dz; Ey: dHx/dz, dHz/dx; Ez: dHy/dx, dHx/dy
  C d[3][2] = {{hz - hz_j, hy - hy_k}, {hx - hx_k, hz - hz_i}, {hy - hy_i, hx - hx_j}};
  if (!UNI) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      d[m][0] = mulC(d[m][0], p.rd[(m + 1) % 3]);
      d[m][1] = mulC(d[m][1], p.rd[(m + 2) % 3]);
    }
  }
  if (kSlabTf<T> && !in && tf) {
    if (tf & 1u) {
      tfsf_axis<0, C>(p.setsE[1][1], p.tab, i, j, k, d[1][1]);
      tfsf_axis<0, C>(p.setsE[2][0], p.tab, i, j, k, d[2][0]);
    }
    if (tf & 2u) {
      tfsf_axis<1, C>(p.setsE[0][0], p.tab, i, j, k, d[0][0]);
      tfsf_axis<1, C>(p.setsE[2][1], p.tab, i, j, k, d[2][1]);
    }
    if (tf & 4u) {
      tfsf_axis<2, C>(p.setsE[0][1], p.tab, i, j, k, d[0][1]);
      tfsf_axis<2, C>(p.setsE[1][0], p.tab, i, j, k, d[1][0]);
    }
  }
  if constexpr (AX < 3) {
    constexpr int A = (AX + 1) % 3, B = (AX + 2) % 3;
    if (w.on) {
      axis_psi_term(w, w.a, d[A][1]);
      axis_psi_term(w, w.b, d[B][0]);
      if (u[A]) *at(p.psiE[A][1], w.q) = w.a;
      if (u[B]) *at(p.psiE[B][0], w.q) = w.b;
    }
  }
  const C exn = u[0] ? fmaC(cb[0], d[0][0] - d[0][1], ex) : ex;
  const C eyn = u[1] ? fmaC(cb[1], d[1][0] - d[1][1], ey) : ey;
  const C ezn = u[2] ? fmaC(cb[2], d[2][0] - d[2][1], ez) : ez;
  if (u[0]) st<T, C>(at(p.E[0], b), exn);
  if (u[1]) st<T, C>(at(p.E[1], b), eyn);
  if (u[2]) st<T, C>(at(p.E[2], b), ezn);
  if (!(MON && jn && kn)) return 0;
  const C e2 = fmaC(exn, exn, fmaC(eyn, eyn, ezn * ezn));
  if (p.etotal) p.etotal[c] = e2;
  return MaxBits<C>::of(e2);
}

template <class T, class C, bool UNI, bool MON, bool SLAB>
__device__ __forceinline__ typename MaxBits<C>::type e_in_3d(const StepParams<T, C>& p, const int i, const int j, const int k) {
  if constexpr (SLAB && sizeof(T) == 2) return e_slab_3d<T, C, UNI, MON, kInside>(p, i, j, k, 0u);
  else return e_cell_3d<T, C, UNI, MON, true>(p, i, j, k, false);
}

// Resident blocks per SM asked of the compiler for the 3-D E kernel.  FP16 storage with the slab
// paths' 32-bit offsets and FP32 run best at 40 registers (6 blocks; us an E launch of 201x187x259
// FP16 104 against 108 with 8, 256^3 145 and 147, monitored 165 and 172; the monitored forms spill
// 4-36 bytes), FP16 without CPML at 32 with 12-44 bytes spilled (256^3 0.3196 -> 0.3116 ms a step),
// and FP64 with its FMA forms at 6 blocks, although it spills 32-84 bytes there (256^3 with CPML and
// TF/SF 0.431 -> 0.415 ms against the compiler's own 60 registers).
template <class T, bool SLAB>
struct EMinBlocks {
  static constexpr int v = sizeof(T) == 2 && !SLAB ? 8 : 6;
};

template <class T, class C, bool UNI, bool MON, bool SLAB, int ZW>
__global__ void __launch_bounds__(256, EMinBlocks<T, SLAB>::v) e_kernel_3d(const StepParams<T, C> p) {
  step_behind();
  step_open();
  constexpr int RY = 256 / ZW;
  const ZTile z = z_tile<ZW>(p.Nz, p.zends);
  const int k = z.k;
  const int j = blockIdx.y * RY + threadIdx.y;
  const int i = blockIdx.z;
  std::conditional_t<SLAB && kSlabTf<T>, unsigned, bool> tf = 0;
  if constexpr (SLAB && kSlabTf<T>) tf = p.tfsf ? ztile_plane_axes(p.planesE, i, blockIdx.y * RY, RY, z) : 0u;
  else tf = p.tfsf && ztile_meets_planes(p.planesE, i, blockIdx.y * RY, RY, z);
  typename MaxBits<C>::type mbits = 0;
  if (z.valid && j < p.Ny) {
    if (!tf && z.n1 == 0 && tile_in(p, i, blockIdx.y * RY, RY, z.lo0, z.n0))
      mbits = e_in_3d<T, C, UNI, MON, SLAB>(p, i, j, k);
    else {
      const int path = SLAB ? slab_path(p, tf, i, blockIdx.y * RY, RY, z.lo0, z.n0) : kGeneral;
      if (path == 0) mbits = e_slab_3d<T, C, UNI, MON, 0>(p, i, j, k, tf);
      else if (path == 1) mbits = e_slab_3d<T, C, UNI, MON, 1>(p, i, j, k, tf);
      else if (path == 2) mbits = e_slab_3d<T, C, UNI, MON, 2>(p, i, j, k, tf);
      else if (path == kNoSlab) mbits = e_slab_3d<T, C, UNI, MON, kNoSlab>(p, i, j, k, tf);
      else mbits = e_cell_3d<T, C, UNI, MON>(p, i, j, k, tf != 0);
    }
  }
  if (MON && p.max_slot) block_max_atomic(mbits, p.max_slot);
}

// ------------------------------------------------------------------ 3-D cells, loads ahead

// The half steps of grids bound by latency or by instructions rather than by memory.  On a small
// grid a launch is one chain from its first load to its last store, and the general path, built
// for many warps at few registers, waits for a psi load behind every psi store; on a larger one
// with CPML its conditions and 64-bit offsets cost more than the update (100^3 FP32: 362
// instructions a warp in H with them, 78 % of the issue slots).  Here a cell issues every load it
// may need, psi of all three slabs and their profile values included, before anything waits.
// Fields, psi and coefficients are read at unsigned 32-bit byte offsets from their arrays, which
// the load instructions add themselves, and unconditionally: a neighbour beyond a wall is the cell
// itself, and only the stores ask whether the cell updates.  Blocks are small, to reach more SMs
// (128 threads; with 256 100^3 24.9 us a step against 23.8, 512x512x128 622 against 584).  H
// is capped at 48 registers (200^3 H 78.8 us against 82.4, E, at 56, 94.3 against 93.7).
template <class C>
struct SlabPsi {
  bool on;
  unsigned q;
  C a, b;        // psi of component AX+1 part 1, AX+2 part 0
  C fb, fc, rk;  // profile b, c, 1/kappa
};
template <int AX, class T, class C>
__device__ __forceinline__ void slab_psi_load(const StepParams<T, C>& p, C* const (&psi)[3][2], const C* fb, const C* fc,
                                              const C* rk, int i, int j, int k, SlabPsi<C>& w) {
  const int n = AX == 0 ? i : (AX == 1 ? j : k);
  const int s = p.pml ? slab_index(p.slab[AX], n) : -1;
  w.on = s >= 0;
  w.a = w.b = w.fb = w.fc = w.rk = C(0);
  w.q = 0;
  if (w.on) {
    const unsigned m = p.slab[AX].n;
    w.q = (AX == 0 ? ((unsigned)s * p.Ny + j) * p.Nzp + k
                   : (AX == 1 ? ((unsigned)i * m + s) * p.Nzp + k : ((unsigned)i * p.Ny + j) * m + s)) * (unsigned)sizeof(C);
    w.a = *at(psi[(AX + 1) % 3][1], w.q);
    w.b = *at(psi[(AX + 2) % 3][0], w.q);
    w.fb = __ldg(fb + n);
    w.fc = __ldg(fc + n);
    w.rk = __ldg(rk + n);
  }
}
template <int AX, class C>
__device__ __forceinline__ void slab_psi_apply(const Fp<C>& fp, SlabPsi<C>& w, C (&d)[3][2]) {
  constexpr int A = (AX + 1) % 3, B = (AX + 2) % 3;
  if (!w.on) return;
  w.a = fmaC(w.fb, w.a, fp.mul(w.fc, d[A][1]));
  d[A][1] = fmaC(d[A][1], w.rk, w.a);
  w.b = fmaC(w.fb, w.b, fp.mul(w.fc, d[B][0]));
  d[B][0] = fmaC(d[B][0], w.rk, w.b);
}
template <int AX, class C>
__device__ __forceinline__ void slab_psi_store(C* const (&psi)[3][2], const SlabPsi<C>& w, const bool (&u)[3]) {
  constexpr int A = (AX + 1) % 3, B = (AX + 2) % 3;
  if (w.on && u[A]) *at(psi[A][1], w.q) = w.a;
  if (w.on && u[B]) *at(psi[B][0], w.q) = w.b;
}
template <class C>
__device__ __forceinline__ void tfsf_all(const PlaneSet (&sets)[3][2], const C* tab, unsigned tf, int i, int j, int k,
                                         const bool (&u)[3], C (&d)[3][2]) {
  if (tf & 1u) {
    if (u[1]) tfsf_axis<0, C>(sets[1][1], tab, i, j, k, d[1][1]);
    if (u[2]) tfsf_axis<0, C>(sets[2][0], tab, i, j, k, d[2][0]);
  }
  if (tf & 2u) {
    if (u[0]) tfsf_axis<1, C>(sets[0][0], tab, i, j, k, d[0][0]);
    if (u[2]) tfsf_axis<1, C>(sets[2][1], tab, i, j, k, d[2][1]);
  }
  if (tf & 4u) {
    if (u[0]) tfsf_axis<2, C>(sets[0][1], tab, i, j, k, d[0][1]);
    if (u[1]) tfsf_axis<2, C>(sets[1][0], tab, i, j, k, d[1][0]);
  }
}

// A block is NT consecutive cells (y, z) of one x plane (PACK), or 32 z x NT/32 y cells of it.
template <class C>
struct SmallCells {
  static constexpr int v = sizeof(C) == 8 ? 64 : 128;
};
template <int NT, bool PACK>
__device__ __forceinline__ void small_cell(int Nz, int& i, int& j, int& k) {
  i = blockIdx.z;
  if (PACK) {
    const int c = blockIdx.x * NT + threadIdx.x;
    j = c / Nz;
    k = c - j * Nz;
  } else {
    j = blockIdx.y * (NT / 32) + (threadIdx.x >> 5);
    k = blockIdx.x * 32 + (threadIdx.x & 31);
  }
}
// Axes of the TF/SF planes that the block may touch.
template <int NT, bool PACK>
__device__ __forceinline__ unsigned small_plane_axes(const int (&planes)[3][2], int Nz) {
  if (!PACK) return tile_plane_axes(planes, blockIdx.z, 1, blockIdx.y * (NT / 32), NT / 32, blockIdx.x * 32, 32);
  const int c0 = blockIdx.x * NT, j0 = c0 / Nz, j1 = (c0 + NT - 1) / Nz;
  const bool row = j0 == j1;
  return tile_plane_axes(planes, blockIdx.z, 1, j0, j1 - j0 + 1, row ? c0 - j0 * Nz : 0, row ? NT : Nz);
}

template <class T, class C, bool UNI, bool PACK>
__global__ void __launch_bounds__(SmallCells<C>::v, sizeof(C) == 4 ? 10 : 1) h_small_3d(const StepParams<T, C> p) {
  step_behind();
  int i, j, k;
  small_cell<SmallCells<C>::v, PACK>(p.Nz, i, j, k);
  if (j >= p.Ny || (!PACK && k >= p.Nz)) return;
  const unsigned c = ((unsigned)i * p.Ny + j) * p.Nzp + k, b = c * (unsigned)sizeof(T);
  const bool in = i < p.Nx - 1, jn = j < p.Ny - 1, kn = k < p.Nz - 1;
  const bool u[3] = {jn && kn, in && kn, in && jn};
  const unsigned bi = b + (in ? (unsigned)p.si * (unsigned)sizeof(T) : 0u), bj = b + (jn ? p.Nzp * (unsigned)sizeof(T) : 0u),
                 bk = b + (kn ? (unsigned)sizeof(T) : 0u);
  HCell<C> v;
  v.ex = ld<T, C>(at(p.E[0], b));
  v.ey = ld<T, C>(at(p.E[1], b));
  v.ez = ld<T, C>(at(p.E[2], b));
  v.ez_j = ld<T, C>(at(p.E[2], bj));
  v.ey_k = ld<T, C>(at(p.E[1], bk));
  v.ex_k = ld<T, C>(at(p.E[0], bk));
  v.ez_i = ld<T, C>(at(p.E[2], bi));
  v.ey_i = ld<T, C>(at(p.E[1], bi));
  v.ex_j = ld<T, C>(at(p.E[0], bj));
  v.hx = ld<T, C>(at(p.H[0], b));
  v.hy = ld<T, C>(at(p.H[1], b));
  v.hz = ld<T, C>(at(p.H[2], b));
  SlabPsi<C> x, y, z;
  slab_psi_load<0>(p, p.psiH, p.bH[0], p.cH[0], p.rkH[0], i, j, k, x);
  slab_psi_load<1>(p, p.psiH, p.bH[1], p.cH[1], p.rkH[1], i, j, k, y);
  slab_psi_load<2>(p, p.psiH, p.bH[2], p.cH[2], p.rkH[2], i, j, k, z);
  const unsigned tf = p.tfsf ? small_plane_axes<SmallCells<C>::v, PACK>(p.planesH, p.Nz) : 0u;
  const Fp<C> fp(k);
  // d[c][part]: Hx: dEz/dy, dEy/dz; Hy: dEx/dz, dEz/dx; Hz: dEy/dx, dEx/dy
  C d[3][2] = {{fp.sub(v.ez_j, v.ez), fp.sub(v.ey_k, v.ey)},
               {fp.sub(v.ex_k, v.ex), fp.sub(v.ez_i, v.ez)},
               {fp.sub(v.ey_i, v.ey), fp.sub(v.ex_j, v.ex)}};
  if (!UNI) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      d[m][0] = fp.mul(d[m][0], fp.reg(p.rd[(m + 1) % 3]));
      d[m][1] = fp.mul(d[m][1], fp.reg(p.rd[(m + 2) % 3]));
    }
  }
  if (tf) tfsf_all<C>(p.setsH, p.tab, tf, i, j, k, u, d);
  slab_psi_apply<0>(fp, x, d);
  slab_psi_apply<1>(fp, y, d);
  slab_psi_apply<2>(fp, z, d);
  const C mdb = fp.neg(p.Dbs);
  if (u[0]) st<T, C>(at(p.H[0], b), fmaC(mdb, fp.sub(d[0][0], d[0][1]), v.hx));
  if (u[1]) st<T, C>(at(p.H[1], b), fmaC(mdb, fp.sub(d[1][0], d[1][1]), v.hy));
  if (u[2]) st<T, C>(at(p.H[2], b), fmaC(mdb, fp.sub(d[2][0], d[2][1]), v.hz));
  slab_psi_store<0>(p.psiH, x, u);
  slab_psi_store<1>(p.psiH, y, u);
  slab_psi_store<2>(p.psiH, z, u);
}

template <class T, class C, bool UNI, bool MON, bool PACK>
__global__ void __launch_bounds__(SmallCells<C>::v) e_small_3d(const StepParams<T, C> p) {
  step_behind();
  int i, j, k;
  small_cell<SmallCells<C>::v, PACK>(p.Nz, i, j, k);
  typename MaxBits<C>::type mbits = 0;
  if (j < p.Ny && (PACK || k < p.Nz)) {
    const unsigned c = ((unsigned)i * p.Ny + j) * p.Nzp + k, b = c * (unsigned)sizeof(T), cb = c * (unsigned)sizeof(C);
    const bool in = i < p.Nx - 1, jn = j < p.Ny - 1, kn = k < p.Nz - 1, ii = in && i >= 1, jj = jn && j >= 1,
               kk = kn && k >= 1;
    const bool u[3] = {in && jj && kk, ii && jn && kk, ii && jj && kn};
    const unsigned bi = b - (i >= 1 ? (unsigned)p.si * (unsigned)sizeof(T) : 0u),
                   bj = b - (j >= 1 ? p.Nzp * (unsigned)sizeof(T) : 0u), bk = b - (k >= 1 ? (unsigned)sizeof(T) : 0u);
    ECell<C> v;
    v.hx = ld<T, C>(at(p.H[0], b));
    v.hy = ld<T, C>(at(p.H[1], b));
    v.hz = ld<T, C>(at(p.H[2], b));
    v.hz_j = ld<T, C>(at(p.H[2], bj));
    v.hy_k = ld<T, C>(at(p.H[1], bk));
    v.hx_k = ld<T, C>(at(p.H[0], bk));
    v.hz_i = ld<T, C>(at(p.H[2], bi));
    v.hy_i = ld<T, C>(at(p.H[1], bi));
    v.hx_j = ld<T, C>(at(p.H[0], bj));
    v.ex = ld<T, C>(at(p.E[0], b));
    v.ey = ld<T, C>(at(p.E[1], b));
    v.ez = ld<T, C>(at(p.E[2], b));
    v.cbx = *at(p.Cbs[0], cb);
    v.cby = *at(p.Cbs[1], cb);
    v.cbz = *at(p.Cbs[2], cb);
    SlabPsi<C> x, y, z;
    slab_psi_load<0>(p, p.psiE, p.bE[0], p.cE[0], p.rkE[0], i, j, k, x);
    slab_psi_load<1>(p, p.psiE, p.bE[1], p.cE[1], p.rkE[1], i, j, k, y);
    slab_psi_load<2>(p, p.psiE, p.bE[2], p.cE[2], p.rkE[2], i, j, k, z);
    const unsigned tf = p.tfsf ? small_plane_axes<SmallCells<C>::v, PACK>(p.planesE, p.Nz) : 0u;
    const Fp<C> fp(k);
    // d[c][part]: Ex: dHz/dy, dHy/dz; Ey: dHx/dz, dHz/dx; Ez: dHy/dx, dHx/dy
    C d[3][2] = {{fp.sub(v.hz, v.hz_j), fp.sub(v.hy, v.hy_k)},
                 {fp.sub(v.hx, v.hx_k), fp.sub(v.hz, v.hz_i)},
                 {fp.sub(v.hy, v.hy_i), fp.sub(v.hx, v.hx_j)}};
    if (!UNI) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        d[m][0] = fp.mul(d[m][0], fp.reg(p.rd[(m + 1) % 3]));
        d[m][1] = fp.mul(d[m][1], fp.reg(p.rd[(m + 2) % 3]));
      }
    }
    if (tf) tfsf_all<C>(p.setsE, p.tab, tf, i, j, k, u, d);
    slab_psi_apply<0>(fp, x, d);
    slab_psi_apply<1>(fp, y, d);
    slab_psi_apply<2>(fp, z, d);
    const C exn = u[0] ? fmaC(v.cbx, fp.sub(d[0][0], d[0][1]), v.ex) : v.ex;
    const C eyn = u[1] ? fmaC(v.cby, fp.sub(d[1][0], d[1][1]), v.ey) : v.ey;
    const C ezn = u[2] ? fmaC(v.cbz, fp.sub(d[2][0], d[2][1]), v.ez) : v.ez;
    if (u[0]) st<T, C>(at(p.E[0], b), exn);
    if (u[1]) st<T, C>(at(p.E[1], b), eyn);
    if (u[2]) st<T, C>(at(p.E[2], b), ezn);
    slab_psi_store<0>(p.psiE, x, u);
    slab_psi_store<1>(p.psiE, y, u);
    slab_psi_store<2>(p.psiE, z, u);
    if (MON && in && jn && kn) {
      const C e2 = fmaC(exn, exn, fmaC(eyn, eyn, fp.mul(ezn, ezn)));
      if (p.etotal) p.etotal[c] = e2;
      mbits = MaxBits<C>::of(e2);
    }
  }
  if (MON && p.max_slot) block_max_atomic(mbits, p.max_slot);
}

// ------------------------------------------------------------------ planar kernels

// Planar H half-step (x-z plane, Ny = 1): Hx and Hz (two_dim_pml.cc:144-162, two_dim.cc:95-111).
// Loads (h2_load) are all issued before the update and stores (h2_apply).
template <class C>
struct HCell2 {
  long long c;
  bool ux, uz;
  C ey, ey_k, ey_i, hx, hz;
};

template <class T, class C, bool FAST = false>
__device__ __forceinline__ void h2_load(const StepParams<T, C>& p, const int i, const int k, HCell2<C>& v) {
  const long long c = (long long)i * p.si + k;
  const bool ux = FAST || k < p.Nz - 1, uz = FAST || i < p.Nx - 1;
  v.c = c;
  v.ux = ux;
  v.uz = uz;
  v.ey = ld<T, C>(p.E[1] + c);
  v.ey_k = ux ? ld<T, C>(p.E[1] + c + 1) : C(0);
  v.ey_i = uz ? ld<T, C>(p.E[1] + c + p.si) : C(0);
  v.hx = ux ? ld<T, C>(p.H[0] + c) : C(0);
  v.hz = uz ? ld<T, C>(p.H[2] + c) : C(0);
}

template <class T, class C, bool UNI, bool FAST = false>
__device__ __forceinline__ void h2_apply(const StepParams<T, C>& p, const int i, const int k, bool tf,
                                         const HCell2<C>& v) {
  const long long c = v.c;
  const bool ux = FAST || v.ux, uz = FAST || v.uz;
  if (FAST) tf = false;
  const C ey = v.ey, ey_k = v.ey_k, ey_i = v.ey_i, hx = v.hx, hz = v.hz;
  C nhx = hx, nhz = hz;
  const Fp<C> fp(k);
  const C db = fp.reg(p.Dbs);
  // Hx: k < Nz-1; Hx -= Db*(-curl2/kappa - psi2), curl2 = dEy/dz (z profile)
  if (ux) {
    C d2 = fp.sub(ey_k, ey);
    if (!UNI) d2 = fp.mul(d2, fp.reg(p.rd[2]));
    if (tf) tfsf_axis<2, C>(p.setsH[0][1], p.tab, i, 0, k, d2);
    if (!FAST && p.pml) {
      const int sz = slab_index(p.slab[2], k);
      if (sz >= 0) d2 = pml_term<C>(fp, d2, p.psiH[0][1] + (long long)i * p.slab[2].n + sz, p.bH[2][k], p.cH[2][k], p.rkH[2][k]);
    }
    nhx = fmaC(db, d2, hx);
  }
  // Hz: i < Nx-1; Hz -= Db*(curl1/kappa + psi1), curl1 = dEy/dx (x profile)
  if (uz) {
    C d1 = fp.sub(ey_i, ey);
    if (!UNI) d1 = fp.mul(d1, fp.reg(p.rd[0]));
    if (tf) tfsf_axis<0, C>(p.setsH[2][0], p.tab, i, 0, k, d1);
    if (!FAST && p.pml) {
      const int sx = slab_index(p.slab[0], i);
      if (sx >= 0) d1 = pml_term<C>(fp, d1, p.psiH[2][0] + (long long)sx * p.Nzp + k, p.bH[0][i], p.cH[0][i], p.rkH[0][i]);
    }
    nhz = fmaC(fp.neg(p.Dbs), d1, hz);
  }
  if (ux) st<T, C>(p.H[0] + c, nhx);
  if (uz) st<T, C>(p.H[2] + c, nhz);
}

template <class T, class C, bool UNI, bool FAST = false>
__device__ __forceinline__ void h_cell_2d(const StepParams<T, C>& p, const int i, const int k, const bool tf) {
  HCell2<C> v;
  h2_load<T, C, FAST>(p, i, k, v);
  h2_apply<T, C, UNI, FAST>(p, i, k, tf, v);
}

// One cell per thread; a block is 32 (z) x 8 (x) cells.
template <class T, class C, bool UNI>
__global__ void __launch_bounds__(256) h_kernel_2d(const StepParams<T, C> p) {
  step_behind();
  const int k = blockIdx.x * 32 + threadIdx.x;
  const int ib = blockIdx.y * 8, i = ib + threadIdx.y;
  if (k >= p.Nz || i >= p.Nx) return;
  const bool tf = p.tfsf && tile_meets_planes(p.planesH, ib, 8, 0, 1, blockIdx.x * 32, 32);
  if (!tf && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, ib, 8, blockIdx.x * 32, 32))
    h_cell_2d<T, C, UNI, true>(p, i, k, false);
  else
    h_cell_2d<T, C, UNI>(p, i, k, tf);
}

// Planar E half-step: Ey (two_dim_pml.cc:164-181, two_dim.cc:113-128).  The reference loop
// covers i < Nx-1, k < Nz-1, but its H-curl is only computed for i, k in [1, N-2]
// (vfield.cc:376-381), so the other cells add Cb*0 and are skipped here.
template <class C>
struct ECell2 {
  long long c;
  bool u;
  C ey, hx, hx_k, hz, hz_i, cb;
};

template <class T, class C, bool MON, bool FAST = false>
__device__ __forceinline__ void e2_load(const StepParams<T, C>& p, const int i, const int k, ECell2<C>& v) {
  const long long c = (long long)i * p.si + k;
  const bool u = FAST || (i >= 1 && i < p.Nx - 1 && k >= 1 && k < p.Nz - 1);
  v.c = c;
  v.u = u;
  v.ey = (u || MON) ? ld<T, C>(p.E[1] + c) : C(0);
  v.hx = u ? ld<T, C>(p.H[0] + c) : C(0);
  v.hx_k = u ? ld<T, C>(p.H[0] + c - 1) : C(0);
  v.hz = u ? ld<T, C>(p.H[2] + c) : C(0);
  v.hz_i = u ? ld<T, C>(p.H[2] + c - p.si) : C(0);
  v.cb = u ? p.Cbs[1][c] : C(0);
}

template <class T, class C, bool UNI, bool MON, bool FAST = false>
__device__ __forceinline__ typename MaxBits<C>::type e2_apply(const StepParams<T, C>& p, const int i, const int k,
                                                              bool tf, const ECell2<C>& v, const MaxScreen<C>& scr) {
  const long long c = v.c;
  const C ey = v.ey;
  C eyn = ey;
  const Fp<C> fp(k);
  if (FAST) tf = false;
  if (FAST || v.u) {
    C d1 = fp.sub(v.hx, v.hx_k);  // dHx/dz (z profile)
    C d2 = fp.sub(v.hz, v.hz_i);  // dHz/dx (x profile)
    if (!UNI) { d1 = fp.mul(d1, fp.reg(p.rd[2])); d2 = fp.mul(d2, fp.reg(p.rd[0])); }
    if (tf) {
      tfsf_axis<2, C>(p.setsE[1][0], p.tab, i, 0, k, d1);
      tfsf_axis<0, C>(p.setsE[1][1], p.tab, i, 0, k, d2);
    }
    if (!FAST && p.pml) {
      const int sz = slab_index(p.slab[2], k), sx = slab_index(p.slab[0], i);
      if (sz >= 0) d1 = pml_term<C>(fp, d1, p.psiE[1][0] + (long long)i * p.slab[2].n + sz, p.bE[2][k], p.cE[2][k], p.rkE[2][k]);
      if (sx >= 0) d2 = pml_term<C>(fp, d2, p.psiE[1][1] + (long long)sx * p.Nzp + k, p.bE[0][i], p.cE[0][i], p.rkE[0][i]);
    }
    eyn = fmaC(v.cb, fp.sub(d1, d2), ey);
    st<T, C>(p.E[1] + c, eyn);
  }
  // local_max = max(Ey*Ey) over the whole Ey array (two_dim_pml.cc:181)
  return MON && scr.may(eyn) ? MaxBits<C>::of(fp.mul(eyn, eyn)) : typename MaxBits<C>::type(0);
}

template <class T, class C, bool UNI, bool MON, bool FAST = false>
__device__ __forceinline__ typename MaxBits<C>::type e_cell_2d(const StepParams<T, C>& p, const int i, const int k,
                                                               const bool tf) {
  ECell2<C> v;
  const MaxScreen<C> scr(MON ? p.max_slot : nullptr);
  e2_load<T, C, MON, FAST>(p, i, k, v);
  return e2_apply<T, C, UNI, MON, FAST>(p, i, k, tf, v, scr);
}

template <class T, class C, bool UNI, bool MON>
__global__ void __launch_bounds__(256) e_kernel_2d(const StepParams<T, C> p) {
  step_behind();
  const int k = blockIdx.x * 32 + threadIdx.x;
  const int ib = blockIdx.y * 8, i = ib + threadIdx.y;
  const bool tf = p.tfsf && tile_meets_planes(p.planesE, ib, 8, 0, 1, blockIdx.x * 32, 32);
  const bool fast = !tf && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, ib, 8, blockIdx.x * 32, 32);
  typename MaxBits<C>::type mbits = 0;
  if (k < p.Nz && i < p.Nx) {
    if (fast) mbits = e_cell_2d<T, C, UNI, MON, true>(p, i, k, false);
    else mbits = e_cell_2d<T, C, UNI, MON>(p, i, k, tf);
  }
  if (MON && p.max_slot) block_max_atomic(mbits, p.max_slot);
}

// ------------------------------------------------------------------ single-sweep planar step

// Planar step in one sweep, for float compute.  The two-sweep kernels above move 40 bytes per
// FP32 cell and step (H sweep: Ey read, Hx and Hz read and written; E sweep: Hx, Hz and Cb read,
// Ey read and written); one sweep moves the compulsory 28 (Ey, Hx, Hz and Cb read once, Ey, Hx
// and Hz written once).  A warp owns 32 z columns and R consecutive x rows and walks the rows in
// order.  At row i it forms H(i): Hx from Ey(i,k+1) (a shuffle) and Hz from Ey(i+1,k), the next
// row's value, which it keeps for the next iteration.  Then it forms E(i) from H(i), the Hx of
// column k-1 (a shuffle) and the Hz of row i-1, kept from the previous iteration.  Two values
// belong to other warps and are recomputed from the old state with the same code as their
// owners': Hz(i0-1) before the first row, and lane 0's Hx(i,k0-1).  State n is read from one
// buffer and state n+1 written to the other, so no warp sees a neighbour's new values, and every
// cell of the run is written (the cells a half step does not update keep their old value).  H
// enters E as stored (FP16 storage rounds it first), so the step matches the two-sweep kernels
// bit for bit.

// One psi term of a planar cell with its old psi and profile values already loaded:
// psi = b*psi + c*d, d = d/kappa + psi (pml_term's arithmetic).
template <class C>
__device__ __forceinline__ void psi2_term(C b, C c, C rk, C& psi, C& d) {
  psi = fmaC(b, psi, c * d);
  d = fmaC(d, rk, psi);
}

// What one row of a run reads, issued as a block ahead of the row before it: with the loads of
// row i+1 in flight while row i is formed and stored, and none of a row's psi loads behind
// another psi term's store, a row costs one memory round trip.  (Loading each psi term where it
// is used cost a warp at the grid's edge six round trips a row: 2048^2 FP32 with CPML and TF/SF
// 69.7 us a step against 40.0 without either.)
template <class C>
struct Row2 {
  C ey_i;         // Ey of the next row
  C hx, hz, cb;
  C ey_k;         // lane 31: Ey of column k0+32
  C hxh, eyh;     // lane 0: Hx and Ey of column k0-1
  C phx, pez;     // psi of the z slab: Hx and Ey z parts
  C phxh;         // lane 0: psi of Hx at column k0-1
  C phz, pex;     // psi of the x slab: Hz and Ey x parts
};

// One warp's rows [i0, i1) of the 32 columns from k0; returns the bit pattern of its largest
// Ey^2 (the max over the whole Ey array, two_dim_pml.cc:181).
template <class T, class C, bool UNI, bool FAST, bool PML>
__device__ __forceinline__ typename MaxBits<C>::type step2_rows(const SweepParams<T, C>& p, const int i0, const int i1,
                                                                const int k0, const bool tfH, const bool tfE,
                                                                const C* tab) {
  const int lane = threadIdx.x;
  const int k = k0 + lane;
  const int Nx = p.Nx, Nz = p.Nz;
  const T *eyi = p.ey, *hxi = p.hx, *hzi = p.hz;
  const bool kin = FAST || k < Nz;
  const bool ux = FAST || k < Nz - 1;
  const bool ke = FAST || (k >= 1 && k < Nz - 1);
  const bool halo = lane == 0 && k0 >= 1;
  const long long si = p.si;
  // the z slab: psi index and profile values of this column, and (lane 0) of column k0-1
  const int zn = p.slab[2].n;
  const bool pml = !FAST && PML && p.pml;
  const int sz = pml ? slab_index(p.slab[2], k) : -1;
  const int szh = pml && halo ? slab_index(p.slab[2], k0 - 1) : -1;
  C bHz = C(0), cHz = C(0), rHz = C(0), bEz = C(0), cEz = C(0), rEz = C(0), bHh = C(0), cHh = C(0), rHh = C(0);
  if (sz >= 0 && ux) { bHz = __ldg(p.bHz + k); cHz = __ldg(p.cHz + k); rHz = __ldg(p.rHz + k); }
  if (sz >= 0 && kin) { bEz = __ldg(p.bEz + k); cEz = __ldg(p.cEz + k); rEz = __ldg(p.rEz + k); }
  if (szh >= 0) { bHh = __ldg(p.bHz + k0 - 1); cHh = __ldg(p.cHz + k0 - 1); rHh = __ldg(p.rHz + k0 - 1); }

  auto load = [&](int i, long long c, Row2<C>& r) {
    const bool nx = FAST || i + 1 < Nx;
    const bool ue = ke && (FAST || (i >= 1 && i < Nx - 1));
    r.ey_i = (kin && nx) ? ld<T, C>(eyi + c + si) : C(0);
    r.hx = kin ? ld<T, C>(hxi + c) : C(0);
    r.hz = kin ? ld<T, C>(hzi + c) : C(0);
    r.cb = (kin && ue) ? p.cb[c] : C(0);
    r.ey_k = r.hxh = r.eyh = C(0);
    if (lane == 31 && (FAST || k + 1 < Nz)) r.ey_k = ld<T, C>(eyi + c + 1);
    if (halo) {
      r.hxh = ld<T, C>(hxi + c - 1);
      r.eyh = ld<T, C>(eyi + c - 1);
    }
    if (!FAST) {
      r.phx = r.pez = r.phxh = r.phz = r.pex = C(0);
      if (pml) {
        const int sx = slab_index(p.slab[0], i);
        if (sz >= 0 && ux) r.phx = p.qhx[(long long)i * zn + sz];
        if (sz >= 0 && ue) r.pez = p.qez[(long long)i * zn + sz];
        if (szh >= 0) r.phxh = p.qhx[(long long)i * zn + szh];
        if (sx >= 0 && kin && nx) r.phz = p.qhz[(long long)sx * si + k];
        if (sx >= 0 && kin && ue) r.pex = p.qex[(long long)sx * si + k];
      }
    }
  };
  // new Hz of (i, k) from its x difference (two_dim_pml.cc:155-158)
  auto hz_value = [&](int i, int sx, C ey, C ey_i, C hz, C& psi) -> C {
    C d1 = ey_i - ey;
    if (!UNI) d1 = mulC(d1, p.rd[0]);
    if (!FAST && tfH) tfsf_axis<0, C>(p.setHz, tab, i, 0, k, d1);
    if (!FAST && sx >= 0) psi2_term(__ldg(p.bHx + i), __ldg(p.cHx + i), __ldg(p.rHx + i), psi, d1);
    return stored<T, C>(fmaC(-p.Dbs, d1, hz));
  };

  long long c = (long long)i0 * si + k;
  C ey = kin ? ld<T, C>(eyi + c) : C(0);
  Row2<C> cur;
  load(i0, c, cur);
  C hz_p = C(0);  // new Hz of the row above
  if (i0 >= 1) {
    const C eym = kin ? ld<T, C>(eyi + c - si) : C(0);
    const C hzm = kin ? ld<T, C>(hzi + c - si) : C(0);
    const int sx = pml ? slab_index(p.slab[0], i0 - 1) : -1;
    C psi = (!FAST && sx >= 0 && kin) ? p.qhz[(long long)sx * si + k] : C(0);  // its owner stores the new psi
    hz_p = hz_value(i0 - 1, sx, eym, ey, hzm, psi);
  }
  typename MaxBits<C>::type m = 0;
#pragma unroll 1
  for (int i = i0; i < i1; ++i, c += si) {
    Row2<C> nxt = cur;
    if (i + 1 < i1) load(i + 1, c + si, nxt);
    const bool nx = FAST || i + 1 < Nx;
    const bool ue = ke && (FAST || (i >= 1 && i < Nx - 1));
    const int sx = pml ? slab_index(p.slab[0], i) : -1;
    C ey_k = __shfl_down_sync(0xffffffffu, ey, 1);
    if (lane == 31) ey_k = cur.ey_k;
    // new Hx of (i, k) from its z difference (two_dim_pml.cc:149-152)
    C hxn = cur.hx;
    if (kin && ux) {
      C d2 = ey_k - ey;
      if (!UNI) d2 = mulC(d2, p.rd[2]);
      if (!FAST && tfH) tfsf_axis<2, C>(p.setHx, tab, i, 0, k, d2);
      if (!FAST && sz >= 0) psi2_term(bHz, cHz, rHz, cur.phx, d2);
      hxn = stored<T, C>(fmaC(p.Dbs, d2, cur.hx));
    }
    const C hzn = (kin && nx) ? hz_value(i, sx, ey, cur.ey_i, cur.hz, cur.phz) : cur.hz;
    C hx_k = __shfl_up_sync(0xffffffffu, hxn, 1);
    if (lane == 0) {
      hx_k = C(0);
      if (halo) {  // new Hx of column k0-1, recomputed; its owner stores the new psi
        C d2 = ey - cur.eyh;
        if (!UNI) d2 = mulC(d2, p.rd[2]);
        if (!FAST && tfH) tfsf_axis<2, C>(p.setHx, tab, i, 0, k0 - 1, d2);
        if (!FAST && szh >= 0) psi2_term(bHh, cHh, rHh, cur.phxh, d2);
        hx_k = stored<T, C>(fmaC(p.Dbs, d2, cur.hxh));
      }
    }
    // new Ey of (i, k), i and k in [1, N-2] (two_dim_pml.cc:164-176): e2_apply's arithmetic
    C eyw = ey;
    if (kin && ue) {
      C d1 = hxn - hx_k;  // dHx/dz (z profile)
      C d2 = hzn - hz_p;  // dHz/dx (x profile)
      if (!UNI) { d1 = mulC(d1, p.rd[2]); d2 = mulC(d2, p.rd[0]); }
      if (!FAST && tfE) {
        tfsf_axis<2, C>(p.setEz, tab, i, 0, k, d1);
        tfsf_axis<0, C>(p.setEx, tab, i, 0, k, d2);
      }
      if (!FAST) {
        if (sz >= 0) psi2_term(bEz, cEz, rEz, cur.pez, d1);
        if (sx >= 0) psi2_term(__ldg(p.bEx + i), __ldg(p.cEx + i), __ldg(p.rEx + i), cur.pex, d2);
      }
      eyw = fmaC(cur.cb, d1 - d2, ey);
    }
    if (kin) {
      st<T, C>(p.hx1 + c, hxn);
      st<T, C>(p.hz1 + c, hzn);
      st<T, C>(p.ey1 + c, eyw);
      if (!FAST) {
        if (sz >= 0 && ux) p.qhx1[(long long)i * zn + sz] = cur.phx;
        if (sz >= 0 && ue) p.qez1[(long long)i * zn + sz] = cur.pez;
        if (sx >= 0 && nx) p.qhz1[(long long)sx * si + k] = cur.phz;
        if (sx >= 0 && ue) p.qex1[(long long)sx * si + k] = cur.pex;
      }
      const typename MaxBits<C>::type b = MaxBits<C>::of(eyw * eyw);
      m = b > m ? b : m;
    }
    hz_p = hzn;
    ey = cur.ey_i;
    cur = nxt;
  }
  return m;
}

// A warp's run with its TF/SF and interior tests: H is formed on rows [i0-1, i1) and columns
// [k0-1, k0+32), E on rows [i0, i1) and columns [k0, k0+32).
template <class T, class C, bool UNI, bool PML>
__device__ __forceinline__ typename MaxBits<C>::type step2_warp(const SweepParams<T, C>& p, const int i0, const int i1,
                                                                const int k0, const C* tab) {
  const bool tfH = p.tfsf && tile_meets_planes(p.planesH, i0 - 1, i1 - i0 + 1, 0, 1, k0 - 1, 34);
  const bool tfE = p.tfsf && tile_meets_planes(p.planesE, i0, i1 - i0, 0, 1, k0, 32);
  if (!tfH && !tfE && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, i0 - 1, i1 - i0 + 2, k0 - 1, 34))
    return step2_rows<T, C, UNI, true, PML>(p, i0, i1, k0, false, false, tab);
  return step2_rows<T, C, UNI, false, PML>(p, i0, i1, k0, tfH, tfE, tab);
}

// Register cap of the single-sweep kernel: 5 blocks of 256 per SM (48 registers; the general path
// spills 64 bytes, FP16 72, and without CPML none).  4096^2 FP32 with CPML and TF/SF 112.7 us a step,
// with 6 blocks 122.5, with 4 118.9.
constexpr int kSweepMinBlocks = 5;

// One simulation: a block is 32 z columns x 8 warps of R rows.  Grids without CPML have their own
// form: with the psi code in it, and its spills, 100000x64 FP32 takes 66.6 us a step instead of 44.6,
// FP16 85.8 instead of 55.2, 512^2 FP32 5.4 instead of 3.9.
template <class T, class C, bool UNI, bool PML>
__global__ void __launch_bounds__(256, kSweepMinBlocks) step_kernel_2d(const SweepParams<T, C> p, const int R) {
  step_behind();
  step_open();
  const int k0 = blockIdx.x * 32;
  const int i0 = (blockIdx.y * 8 + threadIdx.y) * R;
  typename MaxBits<C>::type m = 0;
  if (i0 < p.Nx) m = step2_warp<T, C, UNI, PML>(p, i0, min(i0 + R, p.Nx), k0, p.tab);
  if (p.max_slot) block_max_atomic(m, p.max_slot);
}

// Members of a batch: a block is 32 z columns x 8 warps of R rows of one member, `row` the step's
// place in its sequence.  The members' blocks come by value in the launch's parameters, and a
// block finds its member, tile and path (interior: every warp's run) in one 16-byte entry.  At 4
// blocks per SM (64 registers: the pointers of a member that only the entry names take a pair
// each) 48 lenses of side 128-1024 take 142 us a step, at 5 with spills 158; parameters copied to
// shared memory took 168, and the half-step kernels h_batch_2d and e_batch_2d, which move 40
// bytes a cell where this moves 28, 166.
constexpr int kBatchSweepMinBlocks = 4;
template <class T, class C, bool UNI>
__global__ void __launch_bounds__(256, kBatchSweepMinBlocks) step_batch_2d(const __grid_constant__ SweepBatch<T, C> b,
                                                                       const int4* __restrict__ tiles, const int R,
                                                                       const int row) {
  const int4 tl = __ldg(tiles + blockIdx.x);
  const SweepParams<T, C>& g = b.m[tl.x];
  const int k0 = tl.w, i0 = tl.y + threadIdx.y * R;
  if (i0 >= g.Nx) return;
  const int i1 = min(i0 + R, g.Nx);
  const C* tab = g.tab + (long long)row * g.tab_stride;
  const typename MaxBits<C>::type v =
      warp_max(tl.z ? step2_rows<T, C, UNI, true, true>(g, i0, i1, k0, false, false, tab)
                    : step2_warp<T, C, UNI, true>(g, i0, i1, k0, tab));
  if (threadIdx.x == 0) {  // (a warp's maximum straight to the slot: a block's warps end at different times)
    unsigned long long* slot = g.max_slot + (long long)row * g.slot_stride;
    const unsigned long long bits = as_slot_bits(v);
    if (bits > *reinterpret_cast<volatile unsigned long long*>(slot)) atomicMax(slot, bits);
  }
}

// ------------------------------------------------------------------ batched update kernels

// The parameter block of a block's member, in shared memory, with the tables and the slot of step
// `row` of the sequence.  Read through a global pointer instead, the block is held in registers
// or loaded again behind every store.
template <class T, class C>
__device__ __forceinline__ void member_params(StepParams<T, C>& sp, const StepParams<T, C>* __restrict__ g, const int row) {
  static_assert(sizeof(StepParams<T, C>) % 4 == 0, "copied in words");
  const unsigned* src = reinterpret_cast<const unsigned*>(g);
  unsigned* dst = reinterpret_cast<unsigned*>(&sp);
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  for (int w = tid; w < (int)(sizeof(StepParams<T, C>) / 4); w += 256) dst[w] = __ldg(src + w);
  __syncthreads();
  if (tid == 0) {
    sp.tab += (long long)row * sp.tab_stride;
    sp.max_slot += (long long)row * sp.slot_stride;
  }
  __syncthreads();
}

__device__ __forceinline__ int find_member(const int* __restrict__ first, int n, int t) {
  int lo = 0, hi = n;  // first[lo] <= t < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Block map of a batched launch: member m owns blocks [first[m], first[m+1]).  Built on the
// device once per change of membership, so that a block of the update kernels finds its
// member and tile with one 16-byte load: {member, a, b, c} with a = first x plane (3-D) or
// first x row (planar), b = first y row (3-D), c = first z cell.
template <class T, class C>
__global__ void batch_tiles_kernel(const StepParams<T, C>* __restrict__ ps, const int* __restrict__ first, int n,
                                   int nblocks, int planar, int march, int4* __restrict__ tiles) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nblocks; t += gridDim.x * blockDim.x) {
    const int m = find_member(first, n, t);
    const int lt = t - first[m];
    const StepParams<T, C>& p = ps[m];
    const int nkb = (p.Nz + 31) / 32;
    if (planar) {
      tiles[t] = make_int4(m, (lt / nkb) * 8 * march, 0, (lt % nkb) * 32);
    } else {
      const int njb = (p.Ny + 7) / 8;
      tiles[t] = make_int4(m, (lt / (nkb * njb)) * march, ((lt / nkb) % njb) * 8, (lt % nkb) * 32);
    }
  }
}

// DFT planes of a batch: block -> {plane, block within the plane}.
__global__ void block_map_kernel(const int* __restrict__ first, int n, int nblocks, int2* __restrict__ map) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nblocks; t += gridDim.x * blockDim.x) {
    const int m = find_member(first, n, t);
    map[t] = make_int2(m, t - first[m]);
  }
}

// Resident blocks per SM asked of the compiler for the batched 3-D kernels: 5 for float
// compute (48 registers instead of 72, a few spilled; 21.5 -> 30.1 Gcell/s on 16 CPML
// cubes), 3 (no effective cap) for FP64.
template <class C>
struct B3MinBlocks {
  static constexpr int v = sizeof(C) == 4 ? 5 : 3;
};

// 3-D members: a block is 32 z x 8 y cells over M consecutive x planes.
template <class T, class C, bool UNI, int M>
__global__ void __launch_bounds__(256, B3MinBlocks<C>::v) h_batch_3d(const StepParams<T, C>* __restrict__ ps, const int4* __restrict__ tiles, int row) {
  __shared__ StepParams<T, C> p;
  const int4 tl = tiles[blockIdx.x];
  member_params(p, ps + tl.x, row);
  const int k = tl.w + threadIdx.x, j = tl.z + threadIdx.y, i0 = tl.y;
  if (k >= p.Nz || j >= p.Ny) return;
  const bool tf = p.tfsf && tile_meets_planes(p.planesH, i0, M, tl.z, 8, tl.w, 32);
  const int i1 = min(i0 + M, p.Nx);
  if (!tf && tile_is_interior(p.slab, p.pml, p.Nx, p.Ny, p.Nz, i0, M, tl.z, 8, tl.w, 32)) {
#pragma unroll 1
    for (int i = i0; i < i1; ++i) h_cell_3d<T, C, UNI, true>(p, i, j, k, false);
  } else {
#pragma unroll 1
    for (int i = i0; i < i1; ++i) h_cell_3d<T, C, UNI>(p, i, j, k, tf);
  }
}

template <class T, class C, bool UNI, int M>
__global__ void __launch_bounds__(256, B3MinBlocks<C>::v) e_batch_3d(const StepParams<T, C>* __restrict__ ps, const int4* __restrict__ tiles, int row) {
  __shared__ StepParams<T, C> p;
  const int4 tl = tiles[blockIdx.x];
  member_params(p, ps + tl.x, row);
  const int k = tl.w + threadIdx.x, j = tl.z + threadIdx.y, i0 = tl.y;
  const bool tf = p.tfsf && tile_meets_planes(p.planesE, i0, M, tl.z, 8, tl.w, 32);
  typename MaxBits<C>::type mbits = 0;
  if (k < p.Nz && j < p.Ny) {
    const int i1 = min(i0 + M, p.Nx);
    if (!tf && tile_is_interior(p.slab, p.pml, p.Nx, p.Ny, p.Nz, i0, M, tl.z, 8, tl.w, 32)) {
#pragma unroll 1
      for (int i = i0; i < i1; ++i) {
        const typename MaxBits<C>::type b = e_cell_3d<T, C, UNI, true, true>(p, i, j, k, false);
        mbits = b > mbits ? b : mbits;
      }
    } else {
#pragma unroll 1
      for (int i = i0; i < i1; ++i) {
        const typename MaxBits<C>::type b = e_cell_3d<T, C, UNI, true>(p, i, j, k, tf);
        mbits = b > mbits ? b : mbits;
      }
    }
  }
  if (p.max_slot) block_max_atomic(mbits, p.max_slot);
}

// planar members: a block is 32 z cells x 8*M x rows.  Rows are walked one after the
// other: issuing all rows' loads first doubles the registers, halves the resident blocks and
// ran 25 % slower.  Interior tiles issue the next row's loads before the current row's update
// and stores: two rows in flight per thread at the same 32 registers (each row's cells are
// written only by their own thread, and the rows are 8 apart); the 256-lens batch ran 103 ->
// 111 Gcell/s.  The same in the general tiles took 46-48 registers and ran 90.
template <class T, class C, bool UNI, int M>
__global__ void __launch_bounds__(256) h_batch_2d(const StepParams<T, C>* __restrict__ ps, const int4* __restrict__ tiles, int row) {
  __shared__ StepParams<T, C> p;
  const int4 tl = tiles[blockIdx.x];
  member_params(p, ps + tl.x, row);
  const int k = tl.w + threadIdx.x;
  if (k >= p.Nz) return;
  const bool tf = p.tfsf && tile_meets_planes(p.planesH, tl.y, 8 * M, 0, 1, tl.w, 32);
  const bool fast = !tf && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, tl.y, 8 * M, tl.w, 32);
  if (fast) {
    const int i0 = tl.y + threadIdx.y;
    HCell2<C> v[2];
    h2_load<T, C, true>(p, i0, k, v[0]);
#pragma unroll
    for (int r = 0; r < M; ++r) {
      if (r + 1 < M) h2_load<T, C, true>(p, i0 + 8 * (r + 1), k, v[(r + 1) & 1]);
      h2_apply<T, C, UNI, true>(p, i0 + 8 * r, k, false, v[r & 1]);
    }
    return;
  }
#pragma unroll 1
  for (int r = 0; r < M; ++r) {
    const int i = tl.y + threadIdx.y + 8 * r;
    if (i < p.Nx) h_cell_2d<T, C, UNI>(p, i, k, tf);
  }
}

// With float compute capped at 8 blocks per SM, 32 registers: left to itself the compiler took
// 40 for this kernel once the interior path prefetched, which leaves 6 blocks.  FP64 (doubles
// take register pairs) is left uncapped: at 32 registers it spilled 48 bytes.
template <class C>
struct E2BatchMinBlocks {
  static constexpr int v = sizeof(C) == 4 ? 8 : 1;
};
template <class T, class C, bool UNI, int M>
__global__ void __launch_bounds__(256, E2BatchMinBlocks<C>::v) e_batch_2d(const StepParams<T, C>* __restrict__ ps, const int4* __restrict__ tiles, int row) {
  __shared__ StepParams<T, C> p;
  const int4 tl = tiles[blockIdx.x];
  member_params(p, ps + tl.x, row);
  const int k = tl.w + threadIdx.x;
  const bool tf = p.tfsf && tile_meets_planes(p.planesE, tl.y, 8 * M, 0, 1, tl.w, 32);
  const bool fast = !tf && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, tl.y, 8 * M, tl.w, 32);
  typename MaxBits<C>::type mbits = 0;
  if (fast && k < p.Nz) {  // interior tile: the next row's loads first (see h_batch_2d)
    const int i0 = tl.y + threadIdx.y;
    ECell2<C> v[2];
    const MaxScreen<C> scr(p.max_slot);
    e2_load<T, C, true, true>(p, i0, k, v[0]);
#pragma unroll
    for (int r = 0; r < M; ++r) {
      if (r + 1 < M) e2_load<T, C, true, true>(p, i0 + 8 * (r + 1), k, v[(r + 1) & 1]);
      const typename MaxBits<C>::type b = e2_apply<T, C, UNI, true, true>(p, i0 + 8 * r, k, false, v[r & 1], scr);
      mbits = b > mbits ? b : mbits;
    }
  } else if (k < p.Nz) {
#pragma unroll 1
    for (int r = 0; r < M; ++r) {
      const int i = tl.y + threadIdx.y + 8 * r;
      typename MaxBits<C>::type b = 0;
      if (i < p.Nx) b = e_cell_2d<T, C, UNI, true>(p, i, k, tf);
      mbits = b > mbits ? b : mbits;
    }
  }
  if (p.max_slot) block_max_atomic(mbits, p.max_slot);
}

// ------------------------------------------------------------------ data movement

// The three kernels below walk an (n0, n1, n2) block of a padded (Nx, Ny, Nzp) array one
// warp per (i, j) row: the row index fits 32 bits (the launchers hold n0*n1 to 2^30), one division
// per row gives (i, j), and the lanes stride the row's k.  An element-wise 64-bit q -> (i, j, k)
// split costs two 64-bit divisions per element, which the GPU emulates on the FP64 pipe.
constexpr int kRowWarps = 8;  // warps (rows in flight) per 256-thread block

__device__ __forceinline__ double as_double(double v) { return v; }
__device__ __forceinline__ double as_double(float v) { return (double)v; }
__device__ __forceinline__ double as_double(__half v) { return (double)__half2float(v); }

// padded storage -> dense double array of extent (n0,n1,n2)
template <class T>
__global__ void __launch_bounds__(256) gather_kernel(const T* __restrict__ src, double* __restrict__ dst, int n0,
                                                     int n1, int n2, int Ny, int Nzp, double mul) {
  const int lane = threadIdx.x & 31;
  const int rows = n0 * n1;
  const bool scale = mul != 1.0;
  for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < rows; r += gridDim.x * kRowWarps) {
    const int i = r / n1, j = r - i * n1;
    const T* s = src + ((long long)i * Ny + j) * Nzp;
    double* d = dst + (long long)r * n2;
    // two loops, so that a plain copy issues no FP64 compare or multiply per element (the FP64
    // pipe is the narrowest on this GPU)
    if (scale)
      for (int k = lane; k < n2; k += 32) d[k] = as_double(s[k]) * mul;
    else
      for (int k = lane; k < n2; k += 32) d[k] = as_double(s[k]);
  }
}

// dense double array -> padded storage (optionally Cb-style transform)
// mode 0: dst = v; mode 1: dst = v * a (Cb -> Cb/dx); mode 2: Cb = dt/(eps0*(1+F*scale)) * a
template <class T>
__global__ void __launch_bounds__(256) scatter_kernel(const double* __restrict__ src, T* __restrict__ dst, int n0,
                                                      int n1, int n2, int Ny, int Nzp, int mode, double a, double dt,
                                                      double eps0, double scale) {
  const int lane = threadIdx.x & 31;
  const int rows = n0 * n1;
  for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < rows; r += gridDim.x * kRowWarps) {
    const int i = r / n1, j = r - i * n1;
    const double* s = src + (long long)r * n2;
    T* d = dst + ((long long)i * Ny + j) * Nzp;
    for (int k = lane; k < n2; k += 32) {
      double v = s[k];
      if (mode == 2) {
        // epsilon0*(1+F*1000000) then dt/that (three_dim_pml.cc:122-128), no contraction
        const double e = __dmul_rn(eps0, __dadd_rn(1.0, __dmul_rn(v, scale)));
        v = __ddiv_rn(dt, e);
      }
      if (mode >= 1) v = __dmul_rn(v, a);
      if constexpr (sizeof(T) == 2) d[k] = __double2half(v);
      else d[k] = (T)v;
    }
  }
}

// Cb = dt/(eps0*eps_r) * a over the box [lo, hi) clipped to the extent
template <class C>
__global__ void __launch_bounds__(256) eps_box_kernel(C* dst, int n0, int n1, int n2, int Ny, int Nzp, int lo0,
                                                      int lo1, int lo2, int hi0, int hi1, int hi2, double val) {
  const int a0 = max(lo0, 0), a1 = max(lo1, 0), a2 = max(lo2, 0);
  const int b0 = min(hi0, n0), b1 = min(hi1, n1), b2 = min(hi2, n2);
  if (a0 >= b0 || a1 >= b1 || a2 >= b2) return;
  const int w1 = b1 - a1;
  const int rows = (b0 - a0) * w1;
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < rows; r += gridDim.x * kRowWarps) {
    const int di = r / w1;
    C* d = dst + ((long long)(a0 + di) * Ny + a1 + (r - di * w1)) * Nzp;
    for (int k = a2 + lane; k < b2; k += 32) d[k] = (C)val;
  }
}

template <class T>
__global__ void probe_kernel(const ProbeParams pp, const T* f0, const T* f1, const T* f2, const T* f3, const T* f4,
                             const T* f5, double* out) {
  step_behind();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= pp.nprobes * 6) return;
  const int row = pp.ctl ? pp.ctl->row + pp.k : pp.row;
  if (row >= pp.cap) return;
  const int probe = q / 6, comp = q % 6;
  const T* f[6] = {f0, f1, f2, f3, f4, f5};
  const int i = pp.ijk[3 * probe], j = pp.ijk[3 * probe + 1], k = pp.ijk[3 * probe + 2];
  double v = 0.0;
  if (f[comp] && i >= 0 && j >= 0 && k >= 0 && i < pp.ext[comp][0] && j < pp.ext[comp][1] && k < pp.ext[comp][2]) {
    const T* src = f[comp] + ((long long)i * pp.Ny + j) * pp.Nzp + k;
    if constexpr (sizeof(T) == 2) v = (double)__half2float(*src);
    else v = (double)*src;
    if (comp >= 3 && pp.hmul != 1.0) v *= pp.hmul;
  }
  out[(long long)row * pp.nprobes * 6 + q] = v;
}

// Phase factors of one sample of a DFT plane: cos/sin of omega*(t+1)*dt for the E
// components (sampled after the E update) and of omega*(t+0.5)*dt for the H components,
// formed once per plane and sample (the accumulating blocks then only read them).
__device__ __forceinline__ void dft_phase_body(const DftParams& d, const int t) {
  for (int f = threadIdx.x; f < d.nfreq; f += blockDim.x) {
    const double pe = __dmul_rn(d.omega[f], __dmul_rn((double)(t + 1), d.dt));
    const double ph = __dmul_rn(d.omega[f], __dmul_rn((double)t + 0.5, d.dt));
    double se, ce, sh, ch;
    sincos(pe, &se, &ce);
    sincos(ph, &sh, &ch);
    d.phase[f] = ce;
    d.phase[kMaxDftFreq + f] = se;
    d.phase[2 * kMaxDftFreq + f] = ch;
    d.phase[3 * kMaxDftFreq + f] = sh;
  }
}

__global__ void dft_phase_kernel(const DftParams d) { dft_phase_body(d, d.t_at ? *d.t_at + d.k : d.t); }

// Batched: one block per plane of a sampling class.
__global__ void dft_phase_batch_kernel(const DftParams* __restrict__ ds, const int* __restrict__ ts, int k) {
  const DftParams& d = ds[blockIdx.x];
  dft_phase_body(d, ts[d.sim] + k);
}

// Running DFT of the four tangential components on one plane.  Each thread owns one
// (component, cell) and updates its nfreq complex accumulators (coalesced along the cell),
// four frequencies at a time with their loads issued before their stores.
template <class T>
__device__ __forceinline__ void dft_body(const DftParams& d, const T* f0, const T* f1, const T* f2, const T* f3,
                                         const int lb, const int fq0, const int fq1) {
  __shared__ double cs[2][kMaxDftFreq], sn[2][kMaxDftFreq];
  for (int f = fq0 + threadIdx.x; f < fq1; f += blockDim.x) {
    cs[0][f] = d.phase[f];
    sn[0][f] = d.phase[kMaxDftFreq + f];
    cs[1][f] = d.phase[2 * kMaxDftFreq + f];
    sn[1][f] = d.phase[3 * kMaxDftFreq + f];
  }
  __syncthreads();
  const long long ncell = (long long)d.na * d.nb;
  const long long q = lb * (long long)blockDim.x + threadIdx.x;
  if (q >= 4 * ncell) return;
  const int comp = (int)(q / ncell);
  const long long cell = q % ncell;
  const int a = (int)(cell / d.nb), b = (int)(cell % d.nb);
  int u[3];
  u[d.axis] = d.index;
  u[d.axis == 0 ? 1 : 0] = a;
  u[d.axis == 2 ? 1 : 2] = b;
  const T* f = comp == 0 ? f0 : comp == 1 ? f1 : comp == 2 ? f2 : f3;
  double v = 0.0;
  if (f && u[0] < d.ext[comp][0] && u[1] < d.ext[comp][1] && u[2] < d.ext[comp][2]) {
    const T* src = f + ((long long)u[0] * d.Ny + u[1]) * d.Nzp + u[2];
    if constexpr (sizeof(T) == 2) v = (double)__half2float(*src);
    else v = (double)*src;
  }
  if (comp >= 2 && d.hmul != 1.0) v = __dmul_rn(v, d.hmul);
  v = __dmul_rn(v, d.weight);
  const int w = comp < 2 ? 0 : 1;
  double2* acc = reinterpret_cast<double2*>(d.acc) + (long long)comp * ncell + cell;
  const long long stride = 4 * ncell;  // from one frequency to the next
  int fq = fq0;
  for (; fq + 4 <= fq1; fq += 4) {
    double2 x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = acc[(fq + r) * stride];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      x[r].x = fma(v, cs[w][fq + r], x[r].x);
      x[r].y = fma(-v, sn[w][fq + r], x[r].y);
      acc[(fq + r) * stride] = x[r];
    }
  }
  for (; fq < fq1; ++fq) {
    double2 x = acc[fq * stride];
    x.x = fma(v, cs[w][fq], x.x);
    x.y = fma(-v, sn[w][fq], x.y);
    acc[fq * stride] = x;
  }
}

// blockIdx.y: the frequencies [per * y, per * (y + 1)).
template <class T>
__global__ void dft_kernel(const DftParams d, const T* f0, const T* f1, const T* f2, const T* f3, const int per) {
  const int fq0 = blockIdx.y * per;
  dft_body<T>(d, f0, f1, f2, f3, blockIdx.x, fq0, min(fq0 + per, d.nfreq));
}

// Batched DFT planes: a flat launch over the planes sampled at this step; map gives each
// block its plane and its block within the plane.
template <class T>
__global__ void dft_batch_kernel(const DftParams* __restrict__ ds, const int2* __restrict__ map, const int* __restrict__ ts,
                                 int k) {
  const int2 bm = map[blockIdx.x];
  const DftParams& d = ds[bm.x];
  const int t = ts[d.sim] + k;
  if (t % d.every_ != 0) return;
  const void* const* f = (d.f1[0] || d.f1[1]) && ((t + 1) & 1) ? d.f1 : d.f;  // the state after step t
  dft_body<T>(d, (const T*)f[0], (const T*)f[1], (const T*)f[2], (const T*)f[3], bm.y, 0, d.nfreq);
}

// Net flux of a DFT plane per frequency: partial sums over fixed chunks of 1024 cells, then
// the chunks summed in order, so the result does not depend on scheduling.
__global__ void dft_flux_partial(const double* __restrict__ acc, int nfreq, long long ncell, double* __restrict__ part,
                                 int nchunk) {
  const int f = blockIdx.y, ch = blockIdx.x;
  const double2* a = reinterpret_cast<const double2*>(acc);
  double v = 0.0;
  const long long c0 = (long long)ch * 1024;
  for (long long c = c0 + threadIdx.x; c < c0 + 1024 && c < ncell; c += blockDim.x) {
    const double2 e1 = a[((long long)f * 4 + 0) * ncell + c], e2 = a[((long long)f * 4 + 1) * ncell + c];
    const double2 h1 = a[((long long)f * 4 + 2) * ncell + c], h2 = a[((long long)f * 4 + 3) * ncell + c];
    v += (e1.x * h2.x + e1.y * h2.y) - (e2.x * h1.x + e2.y * h1.y);
  }
  __shared__ double red[256];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(long long)f * nchunk + ch] = red[0];
}

__global__ void dft_flux_final(const double* __restrict__ part, int nfreq, int nchunk, double dA, double* __restrict__ out) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfreq) return;
  double v = 0.0;
  for (int c = 0; c < nchunk; ++c) v += part[(long long)f * nchunk + c];
  out[f] = v * dA;
}

// ------------------------------------------------------------------ launchers

// Blocks for a row-walking kernel: one warp per row, at most 16 blocks of 8 warps per SM.
static inline unsigned row_grid(long long rows) {
  const long long b = (rows + kRowWarps - 1) / kRowWarps;
  return (unsigned)(b < 152 * 16 ? b : 152 * 16);
}

static inline unsigned grid1d(long long n, int bs) {
  long long g = (n + bs - 1) / bs;
  if (g > 152LL * 64) g = 152LL * 64;
  return (unsigned)(g < 1 ? 1 : g);
}

template <class C>
cudaError_t launch_prologue_ahead(const PrologueParams& p, int steps, const StepCtl* ctl, C* tab, double* srcv,
                                  unsigned long long* ring, cudaStream_t s) {
  if (steps < 1 || steps > kAhead) return cudaErrorInvalidValue;
  const int bs = 256;
  prologue_ahead_kernel<C><<<dim3(grid1d(p.tab_total > 0 ? p.tab_total : 1, bs), steps), bs, 0, s>>>(p, ctl, tab, srcv, ring);
  return cudaGetLastError();
}

// Launches a kernel of a step; behind: after another step kernel, whose last blocks it may start
// beside (step_behind).
template <class... P, class... A>
static void start(void (*kernel)(P...), dim3 grid, dim3 block, bool behind, cudaStream_t s, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = behind ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, kernel, a...);  // the caller reads the error
}

template <class T>
cudaError_t launch_source(T* field, long long idx, int kind, const double* v, bool behind, cudaStream_t s) {
  start(source_kernel<T>, 1, 1, behind, s, field, idx, kind, v);
  return cudaGetLastError();
}

cudaError_t launch_finish(const unsigned long long* ring, unsigned mask, unsigned long long* series, int at, int cap,
                          StepCtl* ctl, int steps, int rows, cudaStream_t s) {
  finish_kernel<<<1, 32, 0, s>>>(ring, mask, series, at, cap, ctl, steps, rows);
  return cudaGetLastError();
}

cudaError_t launch_set_ctl(StepCtl* ctl, StepCtl v, cudaStream_t s) {
  set_ctl_kernel<<<1, 1, 0, s>>>(ctl, v);
  return cudaGetLastError();
}

// 16-cell z tiles for the 3-D E kernel with float storage (default); LUXUM_ZTILE=32 keeps the
// 32-cell tiles, read once per process.
static bool z16_tiles() {
  static const bool on = [] {
    const char* v = std::getenv("LUXUM_ZTILE");
    return !(v && std::strcmp(v, "32") == 0);
  }();
  return on;
}

template <class T, class C, bool UNI, bool SLAB>
static void launch_step_3d(const StepParams<T, C>& q, bool mon, bool h_half, bool behind, cudaStream_t s) {
  if constexpr (sizeof(T) < 8) {
    if (!h_half && z16_tiles()) {
      const dim3 block(16, 16), grid((q.Nz + 15) / 16, (q.Ny + 15) / 16, q.Nx);
      if (mon) start(e_kernel_3d<T, C, UNI, true, SLAB, 16>, grid, block, behind, s, q);
      else start(e_kernel_3d<T, C, UNI, false, SLAB, 16>, grid, block, behind, s, q);
      return;
    }
  }
  const dim3 block(32, 8), grid(q.zends ? 1 + (q.Nz - 32 + 31) / 32 : (q.Nz + 31) / 32, (q.Ny + 7) / 8, q.Nx);
  if (h_half) start(h_kernel_3d<T, C, UNI, SLAB, 32>, grid, block, behind, s, q);
  else if (mon) start(e_kernel_3d<T, C, UNI, true, SLAB, 32>, grid, block, behind, s, q);
  else start(e_kernel_3d<T, C, UNI, false, SLAB, 32>, grid, block, behind, s, q);
}

// Half steps that take h_small_3d / e_small_3d.  Us a step with them and without (a launch each):
// - FP64 while all blocks are resident (10 of 64 threads an SM at 90 registers): 20^3 with CPML 6.7
//   and 11.0, 34x30x36 9.0 and 12.4, 44^3 13.9 and 19.1; beyond, idle and diverged lanes of the
//   FP64 pipe cost more than the loads ahead give, 52^3 23.1 and 19.2.  Without CPML to half of
//   that: 34^3 9.2 and 10.2, 48^3 16.7 and 12.8.
// - FP32 with CPML, E: 100^3 24.0 and 30.4 (both halves), 128^3 launches of 24.6 and 27.3, 256^3
//   with CPML 6 150.6 and 152.8, with 25 169 and 187, 512x512x128 311 and 336 (monitored 636 and
//   674 a step).  H up to 5 M cells if tiled: 118^3 21.9 and 26, 160^3 with CPML 6 and 12 37.5 and
//   37.9, 38.3 and 40.0; 200^3 72.0 and 69.5, 75.1 and 77.1; 512x512x128 269 and 262: the general
//   kernel's 64 warps an SM hide more of the memory's latency than these 40.  Packed rows at any
//   size: 512x512x100 232 and 260, 800x800x40 249 and 320.
// - FP16 storage with CPML: H 128^3 with CPML 6 and 12 21.4 and 22.2, 21.7 and 23.7, 150^3 44 and
//   39; E 150^3 45.8 and 46.7 (with CPML 15 42.5 and 46.7), 200^3 113 and 77 (the slab paths there
//   have 64 warps an SM).  Not beside the launches of a batch's other lanes, which fill the waits of
//   either: 8 cubes of side 64-128 with CPML 5 and 10 208 and 185, 200 and 193.
// - Float without CPML: 64^3 5.7 and 6.4, 73^3 7.7 and 8.5, 80^3 9.5 and 9.2.
// 32-bit byte offsets: arrays below 2^31 bytes.
template <class T, class C>
static bool loads_ahead(const StepParams<T, C>& p, bool h_half, bool pack, bool lanes) {
  const long long cells = (long long)p.Nx * p.Ny * p.Nz;
  if (sizeof(C) == 8) return cells <= 152LL * SmallCells<C>::v * (p.pml ? 10 : 5);
  if ((long long)p.Nx * p.Ny * p.Nzp >= 1LL << 29 || p.Ny > 4 * 65535) return false;
  if (!p.pml) return cells <= 3LL << 17;
  if (sizeof(T) == 2) return !lanes && cells <= (h_half ? 1LL << 21 : 1LL << 22);
  return !h_half || pack || cells <= 5LL << 20;
}

// Float rows that fill less than 4/5 of their 32-cell tiles are packed (us a step, in tiles:
// 73^3 9.8 and 10.9 with CPML 8, 60x60x100 9.3 and 10.2, 512x512x100 519 and 541), longer ones keep
// the rows of a tile together (90^3 19.1, packed 21.3; 128^3 43.2 and 53.3 before the 32-bit
// offsets).  FP64 pays a pipe slot for each idle lane and is always packed (34^3 10.0, in tiles
// 14.2).
template <class T, class C, bool PACK>
static void launch_small_3d(const StepParams<T, C>& p, bool uniform, bool mon, bool h_half, bool behind, cudaStream_t s) {
  constexpr int NT = SmallCells<C>::v;
  const dim3 grid = PACK ? dim3((unsigned)(((long long)p.Ny * p.Nz + NT - 1) / NT), 1, p.Nx)
                         : dim3((p.Nz + 31) / 32, (p.Ny + NT / 32 - 1) / (NT / 32), p.Nx);
  if (h_half) {
    if (uniform) start(h_small_3d<T, C, true, PACK>, grid, NT, behind, s, p);
    else start(h_small_3d<T, C, false, PACK>, grid, NT, behind, s, p);
  } else if (mon) {
    if (uniform) start(e_small_3d<T, C, true, true, PACK>, grid, NT, behind, s, p);
    else start(e_small_3d<T, C, false, true, PACK>, grid, NT, behind, s, p);
  } else {
    if (uniform) start(e_small_3d<T, C, true, false, PACK>, grid, NT, behind, s, p);
    else start(e_small_3d<T, C, false, false, PACK>, grid, NT, behind, s, p);
  }
}

template <class T, class C>
cudaError_t launch_step(const StepParams<T, C>& p, bool planar, bool uniform, bool h_half, bool behind, bool lanes,
                        cudaStream_t s) {
  // single simulations: one cell per thread (their parameters sit in the constant bank, and
  // walking several cells raises register use past what pays off)
  dim3 block(32, 8);
  const bool mon = p.max_slot || p.etotal;
  if (planar) {
    dim3 grid((p.Nz + 31) / 32, (p.Nx + 7) / 8, 1);
    if (h_half) {
      if (uniform) start(h_kernel_2d<T, C, true>, grid, block, behind, s, p);
      else start(h_kernel_2d<T, C, false>, grid, block, behind, s, p);
    } else if (mon) {
      if (uniform) start(e_kernel_2d<T, C, true, true>, grid, block, behind, s, p);
      else start(e_kernel_2d<T, C, false, true>, grid, block, behind, s, p);
    } else {
      if (uniform) start(e_kernel_2d<T, C, true, false>, grid, block, behind, s, p);
      else start(e_kernel_2d<T, C, false, false>, grid, block, behind, s, p);
    }
  } else {
    // FP64 with z CPML slabs of at most 16 cells: the rows' two ends share one tile (ZTile).
    // The E kernel with float storage takes 16-cell z tiles (LUXUM_ZTILE=32 keeps 32): on the
    // 256^3 drop-in grid E 0.2035 -> 0.189 ms (FP32), 0.200 -> 0.187 (FP16 storage), from its
    // CPML and TF/SF tiles; the H kernel ran 0.015 ms slower with them, CPML or not.
    const bool pack = sizeof(C) == 8 || 5LL * p.Nz <= 4LL * ((p.Nz + 31) & ~31);
    if (loads_ahead<T, C>(p, h_half, pack, lanes)) {
      if (pack) launch_small_3d<T, C, true>(p, uniform, mon, h_half, behind, s);
      else if constexpr (sizeof(C) == 4) launch_small_3d<T, C, false>(p, uniform, mon, h_half, behind, s);
      return cudaGetLastError();
    }
    StepParams<T, C> q = p;
    q.zends = sizeof(T) == 8 && p.pml && p.slab[2].n > 0 && p.slab[2].lo <= 16 && p.Nz - p.slab[2].hi0 <= 16 &&
              p.Nz >= 48;
    // Float half steps beyond those give blocks in the slab of one axis their own path (h_slab_3d):
    // us a step of both with and without it, 512x512x128 FP32 (CPML 20) 592 and 654, 256^3 (CPML
    // 16, TF/SF) 299 and 324, in FP16 storage 268 and 299.  FP64 is bound by its pipe.
    bool slab = false;
    const bool reach = sizeof(T) != 2 || (long long)p.Nx * p.Ny * p.Nzp < (1LL << 30);  // e_slab_3d's offsets
    if constexpr (sizeof(C) == 4) slab = p.pml && reach;
    if constexpr (sizeof(C) == 4)
      if (slab) {
        if (uniform) launch_step_3d<T, C, true, true>(q, mon, h_half, behind, s);
        else launch_step_3d<T, C, false, true>(q, mon, h_half, behind, s);
        return cudaGetLastError();
      }
    if (uniform) launch_step_3d<T, C, true, false>(q, mon, h_half, behind, s);
    else launch_step_3d<T, C, false, false>(q, mon, h_half, behind, s);
  }
  return cudaGetLastError();
}

// Rows per warp of the planar sweep, by the rows each resident warp has to do (U).  Short runs
// spread a small grid over the SMs and even out the end of the launch; long ones form the row
// above a run's first less often.  With CPML 16 and TF/SF, us a step at 2, 4, 6, 8 rows: 1024^2
// (U 5.4) 20.0, 20.6, 22.6, 24.6; 2048^2 (21.6) 43.2, 41.1, 41.3, 42.6; 4096^2 (86) 127.2, 113.6,
// 111.6, 112.8.  Beside the launches of a batch's other lanes a launch has a quarter of the GPU, and
// its end is filled by theirs: us a step of 32 members, 2, 4, 5, 6, 8 rows, FP32 of side 724-760 (U
// 2.9) 146, 152, 162, 174, 197; of 800-850 (3.7) 190, 154, 145, 152, 169; of 900-1024 (4.9) 265, 217,
// 213, 205, 202; of 1024-1200 (6.6) 346, 287, 274, 270, 263; FP16 of 900-1024 255, 213, 208, 207, 214,
// 8 of 724-760 40, 36, 37, 41, 47.  (Four FP32 states of 800^2 and less stay in L2, where short runs
// cost little.)
static int sweep_rows(long long cols, int Nx, bool half, bool lanes) {
  const double U = (double)cols * Nx / (152.0 * 8 * kSweepMinBlocks);
  int R = U < 8 ? 2 : (U < 60 ? 4 : 6);
  if (lanes) R = U < 4.3 ? (half ? 4 : (U < 3.27 ? 2 : 5)) : (U < 6 ? 6 : 8);
  const int least = (int)(((long long)Nx + 8 * 65535 - 1) / (8 * 65535));  // the grid is at most 65535 blocks high
  return R < least ? least : R;
}

template <class T, class C>
SweepParams<T, C> sweep_params(const StepParams<T, C>& p) {
  SweepParams<T, C> q;
  std::memset(&q, 0, sizeof q);
  q.ey = p.E[1]; q.hx = p.H[0]; q.hz = p.H[2];
  q.ey1 = p.E1[1]; q.hx1 = p.H1[0]; q.hz1 = p.H1[2];
  q.cb = p.Cbs[1];
  q.qhx = p.psiH[0][1]; q.qhz = p.psiH[2][0]; q.qez = p.psiE[1][0]; q.qex = p.psiE[1][1];
  q.qhx1 = p.psiH1[0][1]; q.qhz1 = p.psiH1[2][0]; q.qez1 = p.psiE1[1][0]; q.qex1 = p.psiE1[1][1];
  q.bHx = p.bH[0]; q.cHx = p.cH[0]; q.rHx = p.rkH[0]; q.bHz = p.bH[2]; q.cHz = p.cH[2]; q.rHz = p.rkH[2];
  q.bEx = p.bE[0]; q.cEx = p.cE[0]; q.rEx = p.rkE[0]; q.bEz = p.bE[2]; q.cEz = p.cE[2]; q.rEz = p.rkE[2];
  q.tab = p.tab;
  q.max_slot = p.max_slot;
  q.Nx = p.Nx; q.Nz = p.Nz; q.si = p.Nzp;
  q.pml = p.pml; q.tfsf = p.tfsf;
  q.Dbs = p.Dbs;
  q.tab_stride = p.tab_stride; q.slot_stride = p.slot_stride;
  for (int a = 0; a < 3; ++a) {
    q.slab[a] = p.slab[a];
    q.rd[a] = p.rd[a];
    for (int e = 0; e < 2; ++e) {
      q.planesH[a][e] = p.planesH[a][e];
      q.planesE[a][e] = p.planesE[a][e];
    }
  }
  q.setHx = p.setsH[0][1]; q.setHz = p.setsH[2][0]; q.setEz = p.setsE[1][0]; q.setEx = p.setsE[1][1];
  return q;
}

template <class T, class C>
cudaError_t launch_step_sweep2(const StepParams<T, C>& p, bool uniform, bool behind, bool lanes, cudaStream_t s) {
  const long long cols = (p.Nz + 31) / 32;
  const int R = sweep_rows(cols, p.Nx, sizeof(T) == 2, lanes);
  const dim3 block(32, 8), grid((unsigned)cols, (unsigned)((p.Nx + 8 * R - 1) / (8 * R)));
  const SweepParams<T, C> q = sweep_params(p);
  if (q.pml) {
    if (uniform) start(step_kernel_2d<T, C, true, true>, grid, block, behind, s, q, R);
    else start(step_kernel_2d<T, C, false, true>, grid, block, behind, s, q, R);
  } else {
    if (uniform) start(step_kernel_2d<T, C, true, false>, grid, block, behind, s, q, R);
    else start(step_kernel_2d<T, C, false, false>, grid, block, behind, s, q, R);
  }
  return cudaGetLastError();
}

template <class T, class C>
cudaError_t launch_batch_sweep(const SweepParams<T, C>* m, int n, const int4* tiles, int nblocks, bool uniform, int R,
                               int row, cudaStream_t s) {
  if (n < 1 || n > kSweepMembers) return cudaErrorInvalidValue;
  SweepBatch<T, C> b;
  static_assert(sizeof(b) + 16 <= 32764, "a launch's parameter space");
  std::memcpy(b.m, m, n * sizeof(SweepParams<T, C>));
  const dim3 block(32, 8);
  if (uniform) step_batch_2d<T, C, true><<<nblocks, block, 0, s>>>(b, tiles, R, row);
  else step_batch_2d<T, C, false><<<nblocks, block, 0, s>>>(b, tiles, R, row);
  return cudaGetLastError();
}

// {member, first row, interior, first column} of each block of the members' sweeps.  Rows a warp
// (R): the fewest, up to 4, at which all blocks are resident at once, since short runs reach more
// SMs; beyond, by the rows each resident warp has to do (U), as in sweep_rows, long ones form the row
// above a run's first less often.  Us a step at 1, 2, 3, 4, 6, 8 rows, FP32: 4 lenses of side 64-128 (U
// 0.3) 4.9, 6.2, 7.5, 8.9, 11.6, 14.3; 16 (1.1) 10.0, 7.6, 8.1, 9.5, 11.6, 14.2; 8 of 128-256 (2.4) 16.5,
// 11.9, 9.6, 10.1, 12.6, 14.9; 16 of 128-256 (4.5) 31.5, 17.6, 14.9, 13.9, 14.8, 16.3; 16 of 256-512 (18)
// 56.7, 38.4, 33.1, 30.9, 30.3, 31.4; 16 of 400-700 (36) 108.7, 75.6, 65.9, 60.3, 57.7, 57.0; 48 of them
// (100) 306, 207, 176, 161, 150, 145.  FP16, bound by instructions rather than by memory, 4 and 6 rows: 8
// of 256-512 22.7 and 23.6, 8 of 400-700 30.9 and 32.3.
template <class T, class C>
int sweep_tiles(const SweepParams<T, C>* m, int n, std::vector<int4>& tiles) {
  constexpr double kResident = 152.0 * kBatchSweepMinBlocks;
  double U = 0;
  for (int q = 0; q < n; ++q) U += (double)((m[q].Nz + 31) / 32) * m[q].Nx / (8 * kResident);
  int R = U < 15 || sizeof(T) == 2 ? 4 : (U < 22 ? 6 : 8);
  for (int r = 3; r >= 1; --r) {
    double blocks = 0;
    for (int q = 0; q < n; ++q) blocks += (double)((m[q].Nz + 31) / 32) * ((m[q].Nx + 8 * r - 1) / (8 * r));
    if (blocks <= kResident) R = r;
  }
  tiles.clear();
  for (int q = 0; q < n; ++q) {
    const SweepParams<T, C>& p = m[q];
    for (int i = 0; i < p.Nx; i += 8 * R)
      for (int k = 0; k < p.Nz; k += 32) {
        // as step2_warp decides for each of the block's runs
        const int i1 = i + 8 * R;
        const bool tf = p.tfsf && (tile_meets_planes(p.planesH, i - 1, i1 - i + 1, 0, 1, k - 1, 34) ||
                                   tile_meets_planes(p.planesE, i, i1 - i, 0, 1, k, 32));
        const bool in = !tf && tile_is_interior_2d(p.slab, p.pml, p.Nx, p.Nz, i - 1, i1 - i + 2, k - 1, 34);
        tiles.push_back(make_int4(q, i, in ? 1 : 0, k));
      }
  }
  return R;
}

template <class T>
cudaError_t launch_gather(const T* src, double* dst, const int ext[3], int Ny, int Nzp, double mul, cudaStream_t s) {
  const long long rows = (long long)ext[0] * ext[1];
  if (rows == 0 || ext[2] == 0) return cudaSuccess;
  if (rows > (1LL << 30)) return cudaErrorInvalidValue;  // r + stride stays in int
  gather_kernel<T><<<row_grid(rows), 256, 0, s>>>(src, dst, ext[0], ext[1], ext[2], Ny, Nzp, mul);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_scatter(const double* src, T* dst, const int ext[3], int Ny, int Nzp, int mode, double a, double dt,
                           double eps0, double scale, cudaStream_t s) {
  const long long rows = (long long)ext[0] * ext[1];
  if (rows == 0 || ext[2] == 0) return cudaSuccess;
  if (rows > (1LL << 30)) return cudaErrorInvalidValue;  // r + stride stays in int
  scatter_kernel<T><<<row_grid(rows), 256, 0, s>>>(src, dst, ext[0], ext[1], ext[2], Ny, Nzp, mode, a, dt, eps0, scale);
  return cudaGetLastError();
}

template <class C>
cudaError_t launch_eps_box(C* dst, const int ext[3], int Ny, int Nzp, const int lo[3], const int hi[3], double val,
                           cudaStream_t s) {
  if ((long long)ext[0] * ext[1] > (1LL << 30)) return cudaErrorInvalidValue;
  eps_box_kernel<C><<<152 * 4, 256, 0, s>>>(dst, ext[0], ext[1], ext[2], Ny, Nzp, lo[0], lo[1], lo[2], hi[0], hi[1],
                                            hi[2], val);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_probes(const ProbeParams& pp, T* const f[6], double* out, bool behind, cudaStream_t s) {
  const int n = pp.nprobes * 6;
  start(probe_kernel<T>, (n + 127) / 128, 128, behind, s, pp, (const T*)f[0], (const T*)f[1], (const T*)f[2], (const T*)f[3],
        (const T*)f[4], (const T*)f[5], out);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dft(const DftParams& d, T* const f[4], cudaStream_t s) {
  const long long n = 4LL * d.na * d.nb;
  dft_phase_kernel<<<1, 128, 0, s>>>(d);
  // A thread walks its frequencies four at a time, one memory round trip each.  A small plane
  // (a planar grid's line: 17 blocks at side 1031) splits them over blocks instead: 32
  // frequencies 11.4 -> 4.9 us; a plane that fills the GPU reads its fields once.
  const long long nb = (n + 255) / 256;
  const int per = nb < 152 * 2 ? 4 : d.nfreq;
  dft_kernel<T><<<dim3((unsigned)nb, (unsigned)((d.nfreq + per - 1) / per)), 256, 0, s>>>(d, f[0], f[1], f[2], f[3], per);
  return cudaGetLastError();
}

template <class T, class C>
cudaError_t launch_batch_tiles(const StepParams<T, C>* ps, const int* first, int n, int nblocks, bool planar, int march,
                               int4* tiles, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  batch_tiles_kernel<T, C><<<grid1d(nblocks, 256), 256, 0, s>>>(ps, first, n, nblocks, planar ? 1 : 0, march, tiles);
  return cudaGetLastError();
}

template <class T, class C, int M>
static void batch_step_m(const StepParams<T, C>* ps, const int4* tiles, int nblocks, bool planar, bool uniform,
                         bool h_half, int row, cudaStream_t s) {
  dim3 block(32, 8);
  if (planar) {
    if (h_half) {
      if (uniform) h_batch_2d<T, C, true, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
      else h_batch_2d<T, C, false, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
    } else {
      if (uniform) e_batch_2d<T, C, true, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
      else e_batch_2d<T, C, false, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
    }
  } else {
    if (h_half) {
      if (uniform) h_batch_3d<T, C, true, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
      else h_batch_3d<T, C, false, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
    } else {
      if (uniform) e_batch_3d<T, C, true, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
      else e_batch_3d<T, C, false, M><<<nblocks, block, 0, s>>>(ps, tiles, row);
    }
  }
}

template <class T, class C>
cudaError_t launch_batch_step(const StepParams<T, C>* ps, const int4* tiles, int nblocks, bool planar, bool uniform,
                              int march, bool h_half, int row, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  switch (march) {
    case 1: batch_step_m<T, C, 1>(ps, tiles, nblocks, planar, uniform, h_half, row, s); break;
    case 2: batch_step_m<T, C, 2>(ps, tiles, nblocks, planar, uniform, h_half, row, s); break;
    case 4: batch_step_m<T, C, 4>(ps, tiles, nblocks, planar, uniform, h_half, row, s); break;
    case 8: batch_step_m<T, C, 8>(ps, tiles, nblocks, planar, uniform, h_half, row, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

int batch_blocks(int Nx, int Ny, int Nz, bool planar, int march) {
  if (planar) return ((Nz + 31) / 32) * ((Nx + 8 * march - 1) / (8 * march));
  return ((Nz + 31) / 32) * ((Ny + 7) / 8) * ((Nx + march - 1) / march);
}

cudaError_t launch_block_map(const int* first, int n, int nblocks, int2* map, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  block_map_kernel<<<grid1d(nblocks, 256), 256, 0, s>>>(first, n, nblocks, map);
  return cudaGetLastError();
}

template <class C>
cudaError_t launch_prologue_batch(const PrologueParams* pps, const int* ts, int k, int steps, int nsims, int max_entries,
                                  double* srcv, unsigned long long* slots, cudaStream_t s) {
  if (nsims <= 0 || steps <= 0) return cudaSuccess;
  long long gx = (max_entries + 255) / 256;
  if (gx < 1) gx = 1;
  if (gx > 1024) gx = 1024;
  prologue_batch_kernel<C><<<dim3((unsigned)gx, (unsigned)nsims, (unsigned)steps), 256, 0, s>>>(pps, ts, k, srcv, slots);
  return cudaGetLastError();
}

cudaError_t launch_source_batch(const PrologueParams* pps, const int* ts, int k, int nsims, const double* v, cudaStream_t s) {
  if (nsims <= 0) return cudaSuccess;
  source_batch_kernel<<<(nsims + 127) / 128, 128, 0, s>>>(pps, ts, k, nsims, v);
  return cudaGetLastError();
}

cudaError_t launch_tick(int* ts, int n, int steps, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  tick_kernel<<<(n + 255) / 256, 256, 0, s>>>(ts, n, steps);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dft_batch(const DftParams* ds, const int2* map, int nplanes, int nblocks, const int* ts, int k,
                             cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  dft_phase_batch_kernel<<<nplanes, 128, 0, s>>>(ds, ts, k);
  dft_batch_kernel<T><<<nblocks, 256, 0, s>>>(ds, map, ts, k);
  return cudaGetLastError();
}

cudaError_t launch_dft_flux(const double* acc, int nfreq, long long ncell, double* part, double dA, double* out,
                            cudaStream_t s) {
  const int nchunk = (int)((ncell + 1023) / 1024);
  dft_flux_partial<<<dim3(nchunk, nfreq), 256, 0, s>>>(acc, nfreq, ncell, part, nchunk);
  dft_flux_final<<<(nfreq + 63) / 64, 64, 0, s>>>(part, nfreq, nchunk, dA, out);
  return cudaGetLastError();
}

#define LX_INST(T, C)                                                                                                  \
  template cudaError_t launch_step<T, C>(const StepParams<T, C>&, bool, bool, bool, bool, bool, cudaStream_t);           \
  template cudaError_t launch_gather<T>(const T*, double*, const int[3], int, int, double, cudaStream_t);                     \
  template cudaError_t launch_scatter<T>(const double*, T*, const int[3], int, int, int, double, double, double,      \
                                         double, cudaStream_t);                                                        \
  template cudaError_t launch_source<T>(T*, long long, int, const double*, bool, cudaStream_t);                            \
  template cudaError_t launch_probes<T>(const ProbeParams&, T* const[6], double*, bool, cudaStream_t);                 \
  template cudaError_t launch_dft<T>(const DftParams&, T* const[4], cudaStream_t);                                 \
  template cudaError_t launch_batch_tiles<T, C>(const StepParams<T, C>*, const int*, int, int, bool, int, int4*,    \
                                                cudaStream_t);                                                     \
  template cudaError_t launch_batch_step<T, C>(const StepParams<T, C>*, const int4*, int, bool, bool, int, bool, int, \
                                               cudaStream_t);                                                          \
  template cudaError_t launch_dft_batch<T>(const DftParams*, const int2*, int, int, const int*, int, cudaStream_t);
LX_INST(double, double)
LX_INST(float, float)
LX_INST(__half, float)
template cudaError_t launch_step_sweep2<float, float>(const StepParams<float, float>&, bool, bool, bool, cudaStream_t);
template cudaError_t launch_step_sweep2<__half, float>(const StepParams<__half, float>&, bool, bool, bool, cudaStream_t);
template cudaError_t launch_prologue_ahead<double>(const PrologueParams&, int, const StepCtl*, double*, double*,
                                                   unsigned long long*, cudaStream_t);
template cudaError_t launch_prologue_ahead<float>(const PrologueParams&, int, const StepCtl*, float*, double*,
                                                  unsigned long long*, cudaStream_t);
template SweepParams<float, float> sweep_params<float, float>(const StepParams<float, float>&);
template SweepParams<__half, float> sweep_params<__half, float>(const StepParams<__half, float>&);
template cudaError_t launch_batch_sweep<float, float>(const SweepParams<float, float>*, int, const int4*, int, bool, int, int,
                                                      cudaStream_t);
template cudaError_t launch_batch_sweep<__half, float>(const SweepParams<__half, float>*, int, const int4*, int, bool, int,
                                                       int, cudaStream_t);
template int sweep_tiles<float, float>(const SweepParams<float, float>*, int, std::vector<int4>&);
template int sweep_tiles<__half, float>(const SweepParams<__half, float>*, int, std::vector<int4>&);
template cudaError_t launch_prologue_batch<double>(const PrologueParams*, const int*, int, int, int, int, double*,
                                                   unsigned long long*, cudaStream_t);
template cudaError_t launch_prologue_batch<float>(const PrologueParams*, const int*, int, int, int, int, double*,
                                                  unsigned long long*, cudaStream_t);
template cudaError_t launch_eps_box<double>(double*, const int[3], int, int, const int[3], const int[3], double,
                                            cudaStream_t);
template cudaError_t launch_eps_box<float>(float*, const int[3], int, int, const int[3], const int[3], double,
                                           cudaStream_t);

}  // namespace lx
