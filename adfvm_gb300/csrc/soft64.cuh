// FP64 products, reciprocals and reciprocal square roots on the integer pipes.
//
// GB300 issues one FP64 warp instruction in 64 cycles of an SM sub-partition, and the FP64 face
// kernels keep that pipe 88-90 % busy while 95 % of the issue slots stay empty. An FP64 product
// written with integer instructions (the schoolbook product of two 53-bit significands and IEEE
// 754 rounding, about 35 instructions) takes about 50 cycles of a sub-partition's issue and runs
// beside the FP64 pipe: with two or more warps a sub-partition, eight FMAs and eight such
// products took the time of the eight FMAs alone (152 against 152 cycles an SM and warp).
//
// soft_mul gives the bits of the hardware product (round to nearest even) of finite operands
// whose product stays below 2^1022, but for zeros, which lose their sign, and results below
// 2^-1021, which become zero. A caller passes inputs below 2^64 only (soft_seen, which also sees
// infinities and NaN): no product of the face flux or its VJP then reaches 2^1000. Where an input
// is larger, or the argument of a reciprocal or square root is out of the ordinary (soft_flag), it
// evaluates its item again with the hardware operations.
//
// sd is a double whose arithmetic evaluates through these: a sum, a difference or an FMA is the
// hardware's, and a product that no sum takes up (the ones the compiler would issue as DMUL) is
// soft_mul. A product is kept as its two factors (sd_prod) until its use decides which it is.
#pragma once
#include "face.cuh"

#ifdef __CUDACC__
namespace afvm {

// inputs at or above 2^64 (high word, sign shifted out)
constexpr unsigned SOFT_LIMIT = (1023u + 64u) << 21;
__device__ __forceinline__ void soft_seen(unsigned& most, double x) {
    most = max(most, (unsigned)__double2hiint(x) << 1);
}

constexpr int SOFT_MAX_THREADS = 128;
// the thread's flag: an argument outside the window of soft_rcp or soft_rsqrt
__device__ __forceinline__ int& soft_flag() {
    static __shared__ int flag[SOFT_MAX_THREADS];
    return flag[threadIdx.x];
}

__device__ __forceinline__ double soft_mul(double a, double b) {
    const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
    const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
    const unsigned am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
    const unsigned ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
    // the 106-bit product H : M : L : Z of the significands
    const unsigned long long ll = (unsigned long long)al * bl;
    const unsigned long long hh0 = (unsigned long long)am * bm;
    const unsigned long long mid = (unsigned long long)am * bl + (unsigned long long)al * bm;
    unsigned L, M, H;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;\n\t}"
        : "=r"(L), "=r"(M), "=r"(H)
        : "r"((unsigned)mid), "r"((unsigned)(ll >> 32)), "r"((unsigned)hh0), "r"((unsigned)(mid >> 32)),
          "r"((unsigned)(hh0 >> 32)));
    const unsigned Z = (unsigned)ll;
    const unsigned s = H >> 9;                 // the product of the significands is 2 or more
    const unsigned k = 12 - s;
    unsigned hi = __funnelshift_l(M, H, k), lo = __funnelshift_l(L, M, k);
    // round to nearest even: the dropped bits (their tail as one sticky bit) plus just under a
    // half, or exactly a half where lo is odd, carry out when the result is to be raised
    const unsigned rem = (L << k) | min(Z, 1u);
    const unsigned half = (lo & 1u) + 0x7fffffffu;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %0, 0;\n\taddc.u32 %1, %1, 0;\n\t}"
        : "+r"(lo), "+r"(hi)
        : "r"(rem), "r"(half));
    // exponents added (hi carries the leading 1 of the significand), the sign last
    const unsigned e = ea + eb;
    hi += e - 0x40000000u + (s << 20);
    hi ^= (ah ^ bh) & 0x80000000u;
    const bool z = min(ea, eb) == 0u || e < 0x40000000u;
    return __hiloint2double(z ? 0 : (int)hi, z ? 0 : (int)lo);
}

// y = 1/m of a significand m in [1, 2) as y0 - y0 (w - w^2) with the FP32 approximation y0 and
// w = m y0 - 1 (|w| < 2^-21, exact in 64-bit wrap-around arithmetic); the dropped terms are
// below 2^-62. Rounded once, to nearest; within 0.502 units in the last place. |x| in
// [2^-WIN, 2^WIN].
template <unsigned WIN>
__device__ __forceinline__ double soft_rcp(double x) {
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned ex = (xh >> 20) & 0x7ffu;
    if (ex - (1023u - WIN) > 2 * WIN) soft_flag() = 1;
    const unsigned mh = (xh & 0xfffffu) | 0x100000u;
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(0x3f800000u | ((xh & 0xfffffu) << 3) | (xl >> 29))));
    // rf in [0.5, 1] as Y 2^-24 (its bit pattern is linear over that range)
    const unsigned Y = __float_as_uint(rf) - 0x3e800000u;
    // W = (m y0 - 1) 2^76, m = (mh : xl) 2^-52
    unsigned long long W = (unsigned long long)xl * Y + ((unsigned long long)(mh * Y) << 32);
    const int Wh = (int)(W >> 32);                                    // w 2^44
    const long long S = (long long)W - (((long long)Wh * Wh) >> 12);   // (w - w^2) 2^76
    const long long D = (long long)(int)(S >> 32) * (int)Y + __umulhi((unsigned)S, Y);   // y0 (w - w^2) 2^68
    const long long y = ((long long)Y << 39) - (D >> 5) + 512;        // y 2^63, half a unit added
    const unsigned long long r = ((unsigned long long)y >> 10) + ((unsigned long long)(2044u - ex) << 52);
    return __hiloint2double((int)((unsigned)(r >> 32) | (xh & 0x80000000u)), (int)(unsigned)r);
}

// y = m^(-1/2) of m in [1, 4) as y0 - y0 (w/2 - 3 w^2/8), w = m y0^2 - 1 (|w| < 2^-21, formed
// to 2^-67); the dropped terms are below 2^-62. Rounded once, to nearest; within 0.502 units in
// the last place. x in [2^-64, 2^65).
__device__ __forceinline__ double soft_rsqrt(double x) {
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned ex = xh >> 20;                  // with the sign: a negative x is outside
    if (ex - (1023u - 64u) > 128u) soft_flag() = 1;
    const unsigned odd = (ex & 1u) ^ 1u;           // exponent ex - 1023 is odd
    float rf;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(rf)
        : "f"(__uint_as_float(((127u + odd) << 23) | ((xh & 0xfffffu) << 3) | (xl >> 29))));
    const unsigned Y = __float_as_uint(rf) - 0x3e800000u;
    const unsigned mh = __funnelshift_l(xl, (xh & 0xfffffu) | 0x100000u, odd), ml = xl << odd;
    const unsigned long long Q = (unsigned long long)Y * Y;          // y0^2 2^48
    const unsigned Qh = (unsigned)(Q >> 32), Ql = (unsigned)Q;
    // W = (m y0^2 - 1) 2^68, m = (mh : ml) 2^-52 (the bits below are dropped)
    unsigned long long W = (unsigned long long)mh * Ql + (((unsigned long long)ml * Ql) >> 32);
    W = (unsigned long long)ml * Qh + W;
    W += (unsigned long long)(mh * Qh) << 32;
    const int Wh = (int)((long long)W >> 24);                                  // w 2^44
    const long long S = ((long long)W - ((3LL * Wh * Wh) >> 22)) << 8;         // (w/2 - 3 w^2/8) 2^77
    const long long D = (long long)(int)(S >> 32) * (int)Y + __umulhi((unsigned)S, Y);   // y0 (...) 2^69
    const long long y = ((long long)Y << 39) - (D >> 6) + 512;                 // y 2^63
    const unsigned e = 1022u - 1u - ((int)(ex - 1023u - odd) >> 1);
    const unsigned long long r = ((unsigned long long)y >> 10) + ((unsigned long long)e << 52);
    return __longlong_as_double((long long)r);
}

struct sd;
// a product not yet evaluated
struct sd_prod {
    double a, b;
    __device__ __forceinline__ double value() const { return soft_mul(a, b); }
};

// first: the value is the -0 that starts a sum (acc0), whose first product is the sum. The flag
// is a constant wherever the code is straight: it is decided at compile time, and settled()
// ends it where branches meet.
struct sd {
    double v;
    bool first;
    sd() = default;
    __device__ __forceinline__ sd(double x) : v(x), first(false) {}
    __device__ __forceinline__ sd(const sd_prod& p) : v(p.value()), first(false) {}
    __device__ __forceinline__ sd& operator+=(const sd& x) { v = v + x.v; first = false; return *this; }
    __device__ __forceinline__ sd& operator+=(const sd_prod& p);
};

template <>
AFVM_HD sd acc0<sd>() {
    sd x;
    x.v = -0.0;
    x.first = true;
    return x;
}
__device__ __forceinline__ void settled(sd& x) { x.first = false; }

#define SD __device__ __forceinline__
SD sd& sd::operator+=(const sd_prod& p) {
    v = first ? p.value() : fma(p.a, p.b, v);
    first = false;
    return *this;
}
SD sd_prod operator*(const sd& x, const sd& y) { return {x.v, y.v}; }
SD sd_prod operator*(const sd_prod& x, const sd& y) { return {x.value(), y.v}; }
SD sd_prod operator*(const sd& x, const sd_prod& y) { return {x.v, y.value()}; }
SD sd_prod operator*(const sd_prod& x, const sd_prod& y) { return {x.value(), y.value()}; }
SD sd operator+(const sd& x, const sd& y) { return sd(x.v + y.v); }
SD sd operator+(const sd_prod& x, const sd& y) { return sd(fma(x.a, x.b, y.v)); }
SD sd operator+(const sd& x, const sd_prod& y) { return sd(fma(y.a, y.b, x.v)); }
SD sd operator+(const sd_prod& x, const sd_prod& y) { return sd(fma(y.a, y.b, x.value())); }
SD sd operator-(const sd& x, const sd& y) { return sd(x.v - y.v); }
SD sd operator-(const sd_prod& x, const sd& y) { return sd(fma(x.a, x.b, -y.v)); }
SD sd operator-(const sd& x, const sd_prod& y) { return sd(fma(-y.a, y.b, x.v)); }
SD sd operator-(const sd_prod& x, const sd_prod& y) { return sd(fma(-y.a, y.b, x.value())); }
SD sd operator-(const sd& x) { return sd(-x.v); }
SD sd_prod operator-(const sd_prod& x) { return {-x.a, x.b}; }
SD sd fabs(const sd& x) { return sd(::fabs(x.v)); }
SD sd fmax(const sd& x, const sd& y) { return sd(::fmax(x.v, y.v)); }
SD bool operator>=(const sd& x, const sd& y) { return x.v >= y.v; }
SD bool operator>(const sd& x, const sd& y) { return x.v > y.v; }
// the helpers of physics.cuh
SD sd mul_sgn(const sd& x, const sd& y) { return sd(mul_sgn<double>(x.v, y.v)); }
SD bool lt_twice(const sd& a, const sd& b) { return lt_twice<double>(a.v, b.v); }
SD sd twice_pos(const sd& x) { return sd(twice_pos<double>(x.v)); }
SD bool pos_(const sd& x) { return pos_<double>(x.v); }
SD sd rcp(const sd& x) { return sd(soft_rcp<64>(x.v)); }
SD sd rcp_eps(const sd& x) { return sd(soft_rcp<120>(x.v)); }
SD sd rsqrt_(const sd& x) { return sd(soft_rsqrt(x.v)); }
SD sd sqrt_(const sd& x) { return pos_(x) ? sd(x * rsqrt_(x)) : sd(0.0); }
SD sd fabs(const sd_prod& x) { return fabs(sd(x)); }
SD sd rcp(const sd_prod& x) { return rcp(sd(x)); }
SD sd rsqrt_(const sd_prod& x) { return rsqrt_(sd(x)); }
SD sd sqrt_(const sd_prod& x) { return sqrt_(sd(x)); }
#undef SD

// sd computes with the double constants
template <>
struct PhysOf<sd> {
    using type = PhysR<double>;
};
template <>
AFVM_HD const PhysR<double>& consts<sd>(const Phys& P) { return P.d; }

// the double of a value, for stores
__device__ __forceinline__ double raw(double x) { return x; }
__device__ __forceinline__ float raw(float x) { return x; }
__device__ __forceinline__ double raw(const sd& x) { return x.v; }

}  // namespace afvm
#endif
