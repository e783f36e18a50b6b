// The sums behind the solvers' dot products, from a thread's products to a warp's total: no narrower and
// no less precise than FP64, on the FP32 and integer pipes. Plain arithmetic that host code compiles too.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SKT_HD __host__ __device__ __forceinline__
#else
#define SKT_HD inline
#endif

namespace skt {

// single operations, never contracted or reordered (a host build needs -ffp-contract=off)
SKT_HD float rn_add(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
SKT_HD float rn_mul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
SKT_HD unsigned float_bits(float v) {
    unsigned u;
    memcpy(&u, &v, 4);
    return u;
}
SKT_HD float bits_float(unsigned u) {
    float v;
    memcpy(&v, &u, 4);
    return v;
}
SKT_HD int rn_int(float v) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(v);
#else
    return int(lrintf(v));
#endif
}
// s + e = a + b exactly, s rounded (two-sum)
SKT_HD void two_sum(float a, float b, float& s, float& e) {
    s = rn_add(a, b);
    const float v = rn_add(s, -a);
    e = rn_add(rn_add(a, -rn_add(s, -v)), rn_add(b, -v));
}

// A thread's sum, h + l + t + far: three floats of falling size (some 70 bits), and in FP64 what lies
// outside their exponents' range.
struct Sum {
    float h = 0.0f, l = 0.0f, t = 0.0f;
    double far = 0.0;
    // += a * b: the product and its rounding error are exact, and so are the two sums they go into (the
    // compensated dot product in three-fold precision of Ogita, Rump and Oishi). A product whose error
    // would leave FP32's range, below 2^-99 or from 2^101, goes to FP64. A warp's 512 products against exact
    // arithmetic, error over the terms' magnitudes: random terms 2.1e-18 on average and 1.1e-17 at most (FP64
    // products and tree 7.0e-18 and 3.7e-17), z.r over six decades 4.1e-17 and 9.5e-17 (6.4e-17 and 3.0e-16).
    // 22 FP32 instructions a product and the range's test, where FP64's product and its two conversions hold a
    // pipe of two lanes an SM for 48 cycles a warp (k_update at 251x118x275 43 us so, 66 with FP64 products).
    SKT_HD void add_prod(float a, float b) {
        const float p = rn_mul(a, b);
        if (near(p) || zero(p, a, b)) add(p, fmaf(a, b, -p));
        else far = fma(double(a), double(b), far);
    }
    // N products with one test of the largest: below 2^-90 (where what the small ones lose, 2^-149 each, could
    // reach 2^-56 of it) or from 2^101 all of them go to FP64
    template <int N>
    SKT_HD void add_prods(const float (&a)[N], const float (&b)[N]) {
        float p[N], most = 0.0f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            p[i] = rn_mul(a[i], b[i]);
            most = fmaxf(most, fabsf(p[i]));
        }
        if (most >= 0x1p-90f && most < 0x1p101f) {
#pragma unroll
            for (int i = 0; i < N; ++i) add(p[i], fmaf(a[i], b[i], -p[i]));
            return;
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (!zero(p[i], a[i], b[i])) far = fma(double(a[i]), double(b[i]), far);
    }
    // N products with no test: each loses up to 2^-149 where it is small, and one too large makes the sum not
    // finite, so a grid's total stands where total_holds, and is taken again by add_far elsewhere
    template <int N>
    SKT_HD void add_near(const float (&a)[N], const float (&b)[N]) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float p = rn_mul(a[i], b[i]);
            add(p, fmaf(a[i], b[i], -p));
        }
    }
    // 2^31 terms lose 2^-118 at most, 2^-58 of such a total
    static SKT_HD bool total_holds(double total) { return fabs(total) >= 0x1p-60 && fabs(total) < 0x1p120; }
    template <int N>
    SKT_HD void add_far(const float (&a)[N], const float (&b)[N]) {
#pragma unroll
        for (int i = 0; i < N; ++i) far = fma(double(a[i]), double(b[i]), far);
    }
    static SKT_HD bool near(float p) { return (float_bits(p) >> 23 & 0xffu) - 28u < 200u; }
    static SKT_HD bool zero(float p, float a, float b) { return p == 0.0f && (a == 0.0f || b == 0.0f); }  // not 0 * inf, not an underflow
    // a product p with its rounding error e
    SKT_HD void add(float p, float e) {
        float x, y, z;
        two_sum(h, p, h, x);
        two_sum(l, e, l, y);
        two_sum(l, x, l, z);
        t = rn_add(t, rn_add(y, z));
    }
};
// a running sum s with its compensation c (the sum is s - c) as a Sum
SKT_HD Sum sum_of(float s, float c) {
    Sum v;
    v.h = s;
    v.l = -c;
    return v;
}

// A warp's total of h + l + t in whole numbers: a lane's value is cut at 2^(E-25), 2^(E-48) and 2^(E-71),
// E the exponent above every lane's h, and each cut is summed by one integer reduction, in no order and
// without rounding. What a lane loses lies below 2^-70 of the largest value of the warp.
struct WarpSum {
    int a, b, c;  // in units of 2^(e-151), 2^(e-174), 2^(e-197)
    unsigned e;   // E + 126 (the largest exponent field, at least 48), 255: some lane's value is not finite
};

// A value as a whole number v of some 62 bits in units of 2^u: the form in which lanes are summed
struct Fixed {
    int64_t v;
    int u;  // -2048 to 2046; kNotFinite: the value is not finite
};
constexpr int kNotFinite = 2047;
SKT_HD int leading_zeros(uint64_t v) {  // of a number other than 0
#ifdef __CUDA_ARCH__
    return __clzll(int64_t(v));
#else
    return __builtin_clzll(v);
#endif
}
SKT_HD int room(int64_t v) { return leading_zeros(uint64_t(v < 0 ? ~v : v) | 1u) - 2; }  // bits to spare below 2^62
// a warp's total to 2^-61 of itself
SKT_HD Fixed fixed_of(const WarpSum& w) {
    const int64_t t = int64_t(w.a) * (1 << 23) + w.b;
    const int r = room(t), k = r < 23 ? r : 23;
    return Fixed{t * (int64_t(1) << k) + (w.c >> (23 - k)), w.e == 255u ? kNotFinite : int(w.e) - 174 - k};
}
// a double, exactly
SKT_HD Fixed fixed_of(double d) {
    uint64_t bits;
    memcpy(&bits, &d, 8);
    const int ex = int(bits >> 52) & 0x7ff;
    const int64_t m = int64_t((bits & 0xfffffffffffffull) | (ex ? 1ull << 52 : 0ull)) << 9;
    return Fixed{(bits >> 63) ? -m : m, ex == 0x7ff ? kNotFinite : (ex ? ex : 1) - 1084};
}
// v in units of 2^u, u at least the value's own; its three parts of 21, 21 and the leading bits are summed
// over the lanes on their own
SKT_HD void split(const Fixed& f, int u, int& hi, int& mid, int& lo) {
    const int64_t v = f.v >> (u - f.u < 63 ? u - f.u : 63);
    lo = int(v) & 0x1fffff;
    mid = int(v >> 21) & 0x1fffff;
    hi = int(v >> 42);
}
// the parts' sums over 2^K lanes together again
template <int K>
SKT_HD Fixed joined(int hi, int mid, int lo, int u) {
    const int64_t v = int64_t(hi) * (int64_t(1) << (42 - K)) + (int64_t(mid) << (21 - K)) + (lo >> K);
    const int k = room(v);
    return Fixed{v * (int64_t(1) << k), u == kNotFinite ? u : v == 0 ? -2048 : u + K - k};
}
SKT_HD double value(const Fixed& f) {
    uint64_t bits = 0x7ff8000000000000ull;
    double d;
    if (f.u != kNotFinite) bits = uint64_t(f.u + 1023 > 1 ? f.u + 1023 : 1) << 52;  // (no sum of FP32 products is smaller)
    memcpy(&d, &bits, 8);
    return double(f.v) * d;
}

// The sum unchanged, with l below an ulp of h and t below one of l, and h = 0 only for a sum of 0. T: there
// is a third part.
template <bool T>
SKT_HD void normalise(Sum& v) {
    if (T) {
        two_sum(v.l, v.t, v.l, v.t);
        two_sum(v.h, v.l, v.h, v.l);
        two_sum(v.l, v.t, v.l, v.t);
    }
    two_sum(v.h, v.l, v.h, v.l);
}
// the three cuts of a normalised lane (a, b and c above)
template <bool T>
SKT_HD void cut(const Sum& v, unsigned e, int& a, int& b, int& c) {
    const float sa = bits_float((278u - e) << 23), sb = bits_float((301u - e) << 23);
    const float ua = bits_float((e - 24u) << 23), ub = bits_float((e - 47u) << 23);
    a = rn_int(rn_mul(v.h, sa));
    const float r = fmaf(-float(a), ua, v.h);
    const int b1 = rn_int(rn_mul(r, sb)), b2 = rn_int(rn_mul(v.l, sb));
    b = b1 + b2;
    float rest = rn_add(fmaf(-float(b1), ub, r), fmaf(-float(b2), ub, v.l));
    if (T) rest = rn_add(rest, v.t);
    c = rn_int(rn_mul(rn_mul(rest, sb), 8388608.0f));
}

// 1 / b to some 21 bits
SKT_HD float rough_inverse(float b) {
#ifdef __CUDA_ARCH__
    return __fdividef(1.0f, b);
#else
    return (1.0f / b) * (1.0f + 0x1p-20f);
#endif
}
// a / b rounded to float: a quotient of some 20 bits, its remainder in FP64 and the remainder's quotient; where
// the last one's error could change the rounded sum, and outside the range of the first, FP64's division (561
// cycles of latency against some 250)
SKT_HD float quotient(double a, double b) {
    const float af = float(a), bf = float(b);
    const float big = fmaxf(fabsf(af), fabsf(bf)), small = fminf(fabsf(af), fabsf(bf));
    if (small > 0x1p-60f && big < 0x1p60f) {
        const float inv = rough_inverse(bf), q = rn_mul(af, inv);
        const float c = rn_mul(float(fma(-b, double(q), a)), inv);
        const float x = fmaf(c, 1.0f - 0x1p-16f, q), y = fmaf(c, 1.0f + 0x1p-16f, q);
        if (x == y) return x;
    }
    return float(a / b);
}

}  // namespace skt
