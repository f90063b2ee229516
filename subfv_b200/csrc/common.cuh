// Shared device helpers for the subface finite-volume kernels (sm_100a).
//
// The plain-FP64 kernels are compiled with --fmad=false and evaluate every
// expression in the same order as the reference Fortran, so a kernel and the CPU
// restatement of the same routine produce the same bits.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>

namespace subfv {

constexpr double kGamma = 7.0 / 5.0;

// Error bits a kernel records in the step status word (it never traps).
enum StatusBits : unsigned {
  kErrMeshCheck = 1u << 0,   // check_mesh failed (mesh_geometry_module.F90:403-408)
  kErrNonFinite = 1u << 1,   // a non-finite state, volume or time step
  kErrNegDensity = 1u << 2,  // negative specific volume / density
  kErrBadOmega = 1u << 3,    // positivity limiter gave omega <= 1e-6 (ns_euler_module.F90:595)
  kErrGmres = 1u << 4,       // GMRES did not converge (warning)
  kErrIndex = 1u << 5,       // an index outside its array (checked builds)
};

// x / D for D = 3 or 6, bit-identical to the IEEE quotient (round to nearest), by a
// multiply with the rounded reciprocal R = RN(1/D) and one remainder correction
// (Markstein's correction step for division with a fused multiply-add):
//   q0 = RN(x R),  e = x - D q0 (exact, one FMA),  q = RN(q0 + e R) (one FMA).
// Why it is exact for D = 3 * 2^k: R = (1/D)(1 - 2^-54), so x R is within half an ulp of
// x/D and q0 within one ulp; then x - D q0 is a small multiple of ulp(q0), exactly
// representable. q0 + e R = x/D - (e/D) 2^-54 differs from x/D by less than
// ulp(x/D) 2^-54, while x/D is at least ulp(x/D)/6 away from every rounding midpoint
// (x is a multiple of 2 or 4 ulp(x/D), and 2K - 3(2M + 1) is odd), so both round to the
// same double. Zero (its sign), subnormal or huge x, infinities and NaN take the plain
// division (a zero is its own quotient). The kernels that use it stay bit-identical to the CPU restatement, which
// divides; subfv_probe_div_const checks it against CUDA's division.
template <int D>
__host__ __device__ inline double div_const(double x) {
  static_assert(D == 3 || D == 6, "exact only for 3 * 2^k, checked for 3 and 6");
  constexpr double R = 1.0 / D;
  const double ax = fabs(x);
  if (ax == 0.0) return x;
  if (!(ax >= 0x1p-960 && ax <= 0x1p960)) return x / D;
  const double q0 = x * R;
  const double e = fma(-q0, (double)D, x);
  return fma(e, R, q0);
}
__host__ __device__ inline double div3(double x) { return div_const<3>(x); }
__host__ __device__ inline double div6(double x) { return div_const<6>(x); }

// a / b and sqrt(x), bit-identical to the operators, at one cost whatever the values. The
// device's FP64 division leaves its fast path for a zero numerator, and its square root
// for a zero: 420 and 238 cycles a warp against 125 and 95 (FP32: 269 and 137 against 60
// and 58), for every lane of a warp in which one lane is zero. In these schemes zeros are
// the rule: the third velocity component and normal component of a slab, the pressure and
// velocity jumps of a uniform state, one side's pressure excess at every face. So a zero
// numerator is divided as 1 and its quotient, a zero of the quotient's sign, is selected
// afterwards (129 and 114 cycles in all cases, FP32 69). The empty asm keeps the compiler
// from seeing that the selected quotient does not need the substitute. b zero or NaN: the
// operator itself.
__device__ inline double qdiv(double a, double b) {
  const bool z = a == 0.0 && fabs(b) > 0.0;
  double n = z ? 1.0 : a;
  asm("" : "+d"(n));
  const double q = n / b;
  return z ? __hiloint2double((__double2hiint(a) ^ __double2hiint(b)) & 0x80000000, 0) : q;
}
__device__ inline float qdiv(float a, float b) {
  const bool z = a == 0.0f && fabsf(b) > 0.0f;
  float n = z ? 1.0f : a;
  asm("" : "+f"(n));
  const float q = n / b;
  return z ? __int_as_float((__float_as_int(a) ^ __float_as_int(b)) & 0x80000000) : q;
}
__device__ inline double qsqrt(double x) {
  double n = x == 0.0 ? 1.0 : x;
  asm("" : "+d"(n));
  const double s = sqrt(n);
  return x == 0.0 ? x : s;
}
__device__ inline float qsqrt(float x) {
  float n = x == 0.0f ? 1.0f : x;
  asm("" : "+f"(n));
  const float s = sqrtf(n);
  return x == 0.0f ? x : s;
}

// a / b, bit-identical to the IEEE quotient, from the correctly rounded reciprocal
// y = 1.0 / b, for denominators that several numerators share: a first quotient, one
// correction that makes it faithful, and Markstein's final correction, exact for a
// correctly rounded reciprocal and a faithful quotient (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990). a and b between 2^-400 and 2^400 in magnitude, so that no step under- or
// overflows; a zero numerator's quotient is a * y; anything else takes the division, which
// the empty volatile asm keeps from being computed ahead of the branch (a call out of line
// would make the kernels spill around it). 80-95 cycles a warp against qdiv's 129, and a
// third of its instructions.
__device__ inline bool exponent_in_reach(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((1023u - 400u) << 20) < (800u << 20);
}
__device__ inline double div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  const double q = fma(fma(-b, q1, a), y, q1);
  const bool z = a == 0.0;
  if (!((z || exponent_in_reach(a)) && exponent_in_reach(y))) {
    double n = a;
    asm volatile("" : "+d"(n));
    return n / b;
  }
  return z ? q0 : q;
}
// FP32: the division itself is short
__device__ inline float div_by(float a, float b, float) { return qdiv(a, b); }

// gfortran's inline NORM2 of a 3-vector: scaled sum of squares, scale starting at 1.
__device__ inline double fnorm2_3(double a0, double a1, double a2) {
  // With every |a_i| <= 1 the scale stays 1, each a_i / scale is a_i exactly and a zero
  // term adds nothing, so the scaled sum below reduces to this one, bit for bit.
  if (fabs(a0) <= 1.0 && fabs(a1) <= 1.0 && fabs(a2) <= 1.0) return qsqrt(a0 * a0 + a1 * a1 + a2 * a2);
  double scale = 1.0, res = 0.0;
  const double a[3] = {a0, a1, a2};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (a[i] != 0.0) {
      double ax = fabs(a[i]);
      if (ax > scale) {
        double v = scale / ax;
        res = 1.0 + res * v * v;
        scale = ax;
      } else {
        double v = ax / scale;
        res += v * v;
      }
    }
  }
  return scale * sqrt(res);
}

// Lagrangian pressure (lagrange_module.F90:429-436); u = (tau, u, v, w, e).
__device__ inline double lag_pressure(double tau, double u1, double u2, double u3, double e) {
  double n = fnorm2_3(u1, u2, u3);
  return (kGamma - 1.0) / tau * (e - 0.5 * (n * n));
}

__host__ __device__ inline double dot3(double a0, double a1, double a2, double b0, double b1, double b2) {
  double s = 0.0;
  s = s + a0 * b0;
  s = s + a1 * b1;
  s = s + a2 * b2;
  return s;
}

// min over non-negative doubles through their bit patterns (order independent, exact)
__device__ inline void atomic_min_pos(double* addr, double v) {
  atomicMin(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

void set_error(const std::string& msg);

#define SUBFV_CUDA(call)                                                          \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) {                                                      \
      ::subfv::set_error(std::string(#call) + ": " + cudaGetErrorString(e_));     \
      return -1;                                                                  \
    }                                                                             \
  } while (0)

// Makes `dev` current for a scope: a kernel launch and an allocation go to the current device,
// where a copy goes by its pointers and stream.
struct OnDevice {
  int before = -1;
  explicit OnDevice(int dev) {
    int cur = dev;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev && cudaSetDevice(dev) == cudaSuccess) before = cur;
  }
  OnDevice(const OnDevice&) = delete;
  ~OnDevice() {
    if (before >= 0) cudaSetDevice(before);
  }
};

// Device-side scalars of a time loop; one struct per in-flight problem.
struct LagScalars {
  double dtmin;               // running CFL minimum of the current step
  double dt;                  // time step of the current step
  double t, t_max, cfl;
  unsigned long long steps;   // steps taken
  int done;                   // t >= t_max: later steps are no-ops
  int skip;                   // this step was a no-op
};

// Cell record on the device: tau (or rho), the three velocities / momenta, energy, mass,
// pressure, pad. The pressure is recomputed whenever the state changes, with the same
// function the reference calls, so reading it is bit-identical to recomputing it.
constexpr int kRec = 8;
constexpr int kRhs = 6;  // rhs record: five residuals and a pad

inline int grid_for(long long n, int block) { return (int)((n + block - 1) / block); }

}  // namespace subfv
