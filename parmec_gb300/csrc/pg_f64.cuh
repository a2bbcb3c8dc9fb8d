// pg_f64.cuh -- FP64 sums and products in the form GB300 issues fastest.
//
// An FP64 instruction of a warp holds its scheduler's pipe for 64 clocks, but
// an SM starts DADD, DMUL and a DFMA with a constant operand only every 19
// clocks, against 16 for a DFMA whose three operands are registers (measured:
// 76 and 64 clocks per scheduler with four or more warps an SM, whatever the
// mix).  So a + b is taken as fma(a, 1, b) and a * b as fma(a, b, -0), with
// the 1 and the -0 in registers: the same values, roundings and signs of zero
// (a*1 is exact; a product plus -0 is the product, a zero keeping its sign).
// The compiler must not see that they are constants; they come out of a
// shuffle.  f64 carries them along with its value; they are the same two
// registers everywhere once the functions are inlined.
#pragma once

namespace pg {

#ifdef __CUDACC__

struct f64
{
  double v, one, nz;
  __device__ __forceinline__ f64() {}
  __device__ __forceinline__ f64(double x, double o, double z) : v(x), one(o), nz(z) {}
  __device__ __forceinline__ operator double() const { return v; }
  __device__ __forceinline__ f64 operator-() const { return f64(-v, one, nz); }
  template <class B> __device__ __forceinline__ f64 &operator+=(B b);
  template <class B> __device__ __forceinline__ f64 &operator-=(B b);
  template <class B> __device__ __forceinline__ f64 &operator*=(B b);
};

#define PG_F64_OP(op, expr) \
  __device__ __forceinline__ f64 operator op(f64 a, f64 b) { const double x = a.v, y = b.v, one = a.one, nz = a.nz; (void)one; (void)nz; return f64(expr, a.one, a.nz); } \
  __device__ __forceinline__ f64 operator op(f64 a, double y) { const double x = a.v, one = a.one, nz = a.nz; (void)one; (void)nz; return f64(expr, a.one, a.nz); } \
  __device__ __forceinline__ f64 operator op(double x, f64 b) { const double y = b.v, one = b.one, nz = b.nz; (void)one; (void)nz; return f64(expr, b.one, b.nz); }
PG_F64_OP(+, __fma_rn(x, one, y))
PG_F64_OP(-, __fma_rn(x, one, -y))
PG_F64_OP(*, __fma_rn(x, y, nz))
PG_F64_OP(/, x / y)
#undef PG_F64_OP

template <class B> __device__ __forceinline__ f64 &f64::operator+=(B b) { *this = *this + b; return *this; }
template <class B> __device__ __forceinline__ f64 &f64::operator-=(B b) { *this = *this - b; return *this; }
template <class B> __device__ __forceinline__ f64 &f64::operator*=(B b) { *this = *this * b; return *this; }

// makes the numbers of a kernel: double, or f64 with the two registers.  Every
// lane of the warp constructs it.
template <class R> struct Num;
template <> struct Num<double>
{
  __device__ __forceinline__ double operator()(double x) const { return x; }
};
template <> struct Num<f64>
{
  double one, nz;
  __device__ __forceinline__ Num()
  {
    // zero (the neighbour's thread index is below 1,024), but to the compiler a
    // value of its own in every lane, which keeps it out of the uniform registers
    const unsigned z = __shfl_xor_sync(0xffffffffu, threadIdx.x, 1) >> 20;
    one = __hiloint2double(0x3ff00000 | z, z);
    nz = __hiloint2double(0x80000000 | z, z);
  }
  __device__ __forceinline__ f64 operator()(double x) const { return f64(x, one, nz); }
};

// x as a number like a
__device__ __forceinline__ f64 like(f64 a, double x) { return f64(x, a.one, a.nz); }
__device__ __forceinline__ double like(double, double x) { return x; }

#else
inline double like(double, double x) { return x; }
#endif

} // namespace pg
