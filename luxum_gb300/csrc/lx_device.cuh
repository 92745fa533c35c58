// lx_device.cuh -- device helpers shared by the update kernels (lx_kernels.cu, lx_sweep3d.cu):
// storage access in the three precision forms, the CPML psi recursion, TF/SF increments and
// the max|E|^2 block reduction.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "lx_internal.h"

namespace lx {

// ------------------------------------------------------------------ storage access

// First statement of a step's kernels: their blocks may be on the SMs before the kernel ahead of
// them in the stream is complete, and go on when it is and its stores are visible.  Every thread
// passes here, so that a kernel is complete only after the one ahead of it.
__device__ __forceinline__ void step_behind() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// From here the next kernel's blocks may take the places that this one's leave (without it, from
// when the last of this one's blocks ends).
__device__ __forceinline__ void step_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class T, class C>
__device__ __forceinline__ C ld(const T* p) {
  return static_cast<C>(*p);
}
template <>
__device__ __forceinline__ float ld<__half, float>(const __half* p) {
  return __half2float(*p);
}
template <class T, class C>
__device__ __forceinline__ void st(T* p, C v) {
  *p = static_cast<T>(v);
}
template <>
__device__ __forceinline__ void st<__half, float>(__half* p, float v) {
  *p = __float2half_rn(v);
}

__device__ __forceinline__ double fmaC(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaC(float a, float b, float c) { return fmaf(a, b, c); }
// A rounded product that is never contracted into a neighbouring add: the 1/d factors of
// non-uniform spacing.  Contraction decisions differ between kernels, and the single-sweep
// and two-sweep planar kernels must give the same bits (the oracle does not contract).
__device__ __forceinline__ double mulC(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mulC(float a, float b) { return __fmul_rn(a, b); }

// Differences and products of the update arithmetic.  On this GPU an FP64 add or multiply, or an
// FMA with an operand from the constant bank or an immediate, holds an SM's FP64 pipe 18.6 cycles
// a warp, an FMA with three register operands 15.7 (a loop of independent chains), and that pipe
// bounds the FP64 kernels.  So their differences are fma(b, -1, a) and their products
// fma(a, b, -0), the same bits as a - b and a * b for every input, signed zeros included, with
// -1, -0 and the scalar coefficients in registers: 256^3 with CPML and TF/SF 917 -> 814 us a
// step, 4096^2 planar 278 -> 249.  The compiler would turn an FMA with a known 1 or 0 back into
// an add or a multiply and read a kernel parameter from the constant bank, so the values are tied
// to a cell index: u >> 31 is 0 for u >= 0 (in asm, since a block's interior test tells the
// compiler as much).
template <class C>
struct Fp {
  __device__ __forceinline__ explicit Fp(int) {}
  __device__ __forceinline__ C sub(C a, C b) const { return a - b; }
  __device__ __forceinline__ C mul(C a, C b) const { return mulC(a, b); }
  __device__ __forceinline__ C reg(C a) const { return a; }
  __device__ __forceinline__ C neg(C a) const { return -a; }
};
template <>
struct Fp<double> {
  int z;
  double m1, m0;
  __device__ __forceinline__ explicit Fp(int u) {
    asm("shr.s32 %0, %1, 31;" : "=r"(z) : "r"(u));
    m1 = reg(-1.0);
    m0 = reg(-0.0);
  }
  __device__ __forceinline__ double sub(double a, double b) const { return fma(b, m1, a); }
  __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, m0); }
  __device__ __forceinline__ double reg(double a) const {
    return __hiloint2double(__double2hiint(a) | z, __double2loint(a));
  }
  // a sign flip of a kernel parameter by the compiler is an FP64 add
  __device__ __forceinline__ double neg(double a) const {
    return __hiloint2double((__double2hiint(a) ^ 0x80000000) | z, __double2loint(a));
  }
};

// ------------------------------------------------------------------ TF/SF

// Adds the increments of the planes of `ps` that cell (i,j,k) lies on to d (reference:
// curl = curl +/- exp(...) * dir / d..., one line of plane_wave_execute per plane).
template <class C>
__device__ __forceinline__ void tfsf_apply(const PlaneSet& ps, const C* tab, int i, int j, int k, C& d) {
  if (!ps.active) return;
  const int a = ps.axis;
  const int n = a == 0 ? i : (a == 1 ? j : k);
  const bool h0 = (n == ps.plane[0]);
  const bool h1 = (n == ps.plane[1]);
  if (!(h0 || h1)) return;
  // in-plane ranges and table offset (the normal axis has lo = hi = 0 and stride 0 in the
  // checks below, so it is excluded by selecting 0 for it)
  const int ui = a == 0 ? 0 : i - ps.lo[0], uj = a == 1 ? 0 : j - ps.lo[1], uk = a == 2 ? 0 : k - ps.lo[2];
  const int wi = a == 0 ? 0 : ps.hi[0] - ps.lo[0], wj = a == 1 ? 0 : ps.hi[1] - ps.lo[1], wk = a == 2 ? 0 : ps.hi[2] - ps.lo[2];
  if (ui < 0 || uj < 0 || uk < 0 || ui > wi || uj > wj || uk > wk) return;
  const int off = ui * ps.stride[0] + uj * ps.stride[1] + uk * ps.stride[2];
  if (h0) d = d + __ldg(tab + ps.tab + off);
  if (h1) d = d + __ldg(tab + ps.tab + ps.plane_len + off);
}

// The same for a set whose planes are normal to axis A (the sets of one curl part are).
template <int A, class C>
__device__ __forceinline__ void tfsf_axis(const PlaneSet& ps, const C* tab, int i, int j, int k, C& d) {
  const int n = A == 0 ? i : (A == 1 ? j : k);
  const bool h0 = n == ps.plane[0], h1 = n == ps.plane[1];
  if (!ps.active || !(h0 || h1)) return;
  constexpr int U = A == 0 ? 1 : 0, V = A == 2 ? 1 : 2;  // the in-plane axes
  const int u = (A == 0 ? j : i) - ps.lo[U], v = (A == 2 ? j : k) - ps.lo[V];
  if (u < 0 || v < 0 || u > ps.hi[U] - ps.lo[U] || v > ps.hi[V] - ps.lo[V]) return;
  const C* e = tab + ps.tab + u * ps.stride[U] + v * ps.stride[V];
  if (h0) d = d + __ldg(e);
  if (h1) d = d + __ldg(e + ps.plane_len);
}

// psi = b*psi + c*curl; returns curl/kappa + psi (reference: three_dim_pml.cc:186-188).
template <class C>
__device__ __forceinline__ C pml_term(const Fp<C>& fp, C d, C* psi, C b, C cc, C rk) {
  C ps = fmaC(b, *psi, fp.mul(cc, d));
  *psi = ps;
  return fmaC(d, rk, ps);
}

__device__ __forceinline__ long long psi_index(int axis, const Slab& s, int si_, int i, int j, int k, int Ny,
                                               int Nzp) {
  if (axis == 0) return ((long long)si_ * Ny + j) * Nzp + k;
  if (axis == 1) return ((long long)i * s.n + si_) * Nzp + k;
  return ((long long)i * Ny + j) * s.n + si_;
}

// ------------------------------------------------------------------ monitor

// max|E|^2 is reduced on bit patterns: squares are non-negative, so their IEEE patterns
// order like their values, and NaN/inf sort above every finite value (blow-up detection).
// FP32 members reduce 32-bit float patterns and widen only the block's winner to the
// double pattern the monitor slot holds.
template <class C>
struct MaxBits;
template <>
struct MaxBits<double> {
  using type = unsigned long long;
  static __device__ __forceinline__ type of(double v) { return (unsigned long long)__double_as_longlong(v); }
};
template <>
struct MaxBits<float> {
  using type = unsigned;
  static __device__ __forceinline__ type of(float v) { return __float_as_uint(v); }
};

// Whether a cell's |E|^2 could raise the slot, from an upper bound in float: the slot's value when
// the cell was loaded is a lower bound of the maximum (it only grows while a launch runs), and a
// cell below it is left out without its exact square.  Exact squares cost three instructions of
// the FP64 pipe, which bounds these kernels (256^3 with CPML and TF/SF, monitored: E 509 us a
// launch against 415 unmonitored); the bound takes about twenty of the idle integer and float
// pipes.  The float of |v| is its high word one unit up, clamped to [2^-126, inf]: never below
// |v|, inf for anything a float cannot hold and for NaN.  (e_small_3d forms the squares of every
// cell: its launches are not bound by that pipe.)
template <class C>
struct MaxScreen {
  __device__ __forceinline__ explicit MaxScreen(const unsigned long long*) {}
  __device__ __forceinline__ bool may(C, C, C) const { return true; }
  __device__ __forceinline__ bool may(C) const { return true; }
};
template <>
struct MaxScreen<double> {
  float thr = 0.f;
  __device__ __forceinline__ explicit MaxScreen(const unsigned long long* slot) {
    if (!slot) return;
    const int hi = reinterpret_cast<const int*>(slot)[1];
    // the slot's value rounded down to a float, less 2^-19 for the rounding of the sum of squares
    if (hi >= 0x38100000) thr = __int_as_float(min(hi - 0x38000000, 0x0fefffff) << 3) * 0.999998f;
  }
  static __device__ __forceinline__ float up(double v) {
    const int h = max(__double2hiint(v) & 0x7fffffff, 0x38100000) + 1 - 0x38000000;
    return __int_as_float(min(h, 0x0ff00000) << 3);
  }
  __device__ __forceinline__ bool may(double x, double y, double z) const {
    const float a = up(x), b = up(y), c = up(z);
    return !(fmaf(a, a, fmaf(b, b, c * c)) < thr);
  }
  __device__ __forceinline__ bool may(double x) const {
    const float a = up(x);
    return !(a * a < thr);
  }
};

__device__ __forceinline__ unsigned long long as_slot_bits(unsigned long long v) { return v; }
__device__ __forceinline__ unsigned long long as_slot_bits(unsigned v) {
  return (unsigned long long)__double_as_longlong((double)__uint_as_float(v));
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}
__device__ __forceinline__ unsigned warp_max(unsigned v) { return __reduce_max_sync(0xffffffffu, v); }

// Block maximum of the bit patterns, then one atomicMax on the 64-bit slot per block.
template <class B>
__device__ __forceinline__ void block_max_atomic(B v, unsigned long long* slot) {
  __shared__ B red[32];
  v = warp_max(v);
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int nw = (blockDim.x * blockDim.y + 31) / 32;
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  if (tid < 32) {
    v = warp_max(tid < nw ? red[tid] : B(0));
    if (tid == 0 && v) atomicMax(slot, as_slot_bits(v));
  }
}

// A computed value as a later load of the stored value returns it.
template <class T, class C>
__device__ __forceinline__ C stored(C v) {
  return static_cast<C>(static_cast<T>(v));
}
template <>
__device__ __forceinline__ float stored<__half, float>(float v) {
  return __half2float(__float2half_rn(v));
}

}  // namespace lx
