// Scales and digits of the split-precision operands (see split_tc.cuh), for
// the compiled kernels and, as source text, for the runtime-compiled ones.
#pragma once

namespace slgpu {

#define SLGPU_TEXT(...) #__VA_ARGS__
#define SLGPU_DEVICE_SOURCE(name, ...) \
    __VA_ARGS__                        \
    static const char* const name = SLGPU_TEXT(__VA_ARGS__);

// split_scale: scale of a row or column from the high word h of the largest
// magnitude in it: *q, 2^-8 of the value Q that 2^(B S) units stand for (R and
// Q of split_tc.cuh; Q itself can be above the largest double), and the factor
// that turns a value into those units.
//   B = 8: |x| < the double of high word h + 1, so |x| / Q < 0.498 and its S
//   balanced digits represent it (the largest such number is 0.49804); or,
//   where the digits then hold every value exactly (`exact`), four times the
//   power of two above |x|: whole numbers and dyadic fractions stay what they
//   are, and so do their sums of products;
//   B = 7: the power of two above |x|.
// Magnitudes below 2^-900 take a power of two and a factor below the
// overflow: *pre, by which values are multiplied first (1 otherwise).  High
// words 0 and 1 share a scale, so that the smallest doubles have digits.
// Infinities and NaN (h from 0x7ff00000): the scale is NaN, so that the results
// are.
//
// split_exact: whether B = 8 and the scale by powers of two hold x exactly, h
// as above: at most 21 significant bits (the low word is zero), the last of
// them not below the unit 2^(46 - B S) of the power of two above h.
//
// split_pow2: 2^k, a normal double.
//
// split_digits: the S digits of x in units of 1 / f, byte k the digit
// S - 1 - k.
// B = 8, each plus 128: 1.5 2^52 + rint(x f) holds the integer in its low
// bits, and adding 128 to every digit makes them all non-negative.
// B = 7, two's complement: the 7-bit fields of |x| f truncated, with x's sign.
//
// split_flip: what turns the bytes of a word of digits into signed ones.
//
// split_words: word k4 of each slice, digit s of four values.
SLGPU_DEVICE_SOURCE(
    kSplitDigitSource,
    __device__ __forceinline__ bool split_exact(double x, int h) {
        const int hx = __double2hiint(x) & 0x7fffffff;
        return __double2loint(x) == 0 && (hx == 0 || (h >> 20) - (hx >> 20) <= 25);
    }

    __device__ __forceinline__ double split_pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }

    template <int B, int S> __device__ __forceinline__ double split_scale(int h, bool exact, double* q, double* pre) {
        *pre = 1.0;
        h = max(h, 1);
        if (h >= 0x7ff00000) {
            *q = __longlong_as_double(0x7ff8000000000000ll);
            return 0.0;
        }
        const bool tiny = h < ((1023 - 900) << 20);
        if (tiny || exact || B == 7) {
            const int ex = (h < 0x100000 ? -1010 - __clz(h) : (h >> 20) - 1022) + (B == 7 ? 0 : 2);
            const int up = tiny ? 512 : 0;
            *pre = tiny ? 0x1p512 : 1.0;
            *q = split_pow2(ex - 8 + up) * (tiny ? 0x1p-512 : 1.0);
            return split_pow2(B * S - ex - up);
        }
        const double top = h >= 0x7fefffff ? __longlong_as_double(0x7fefffffffffffffll) : __hiloint2double(h + 1, 0);
        *q = top * (0x1p-8 / 0.498);
        return 0.498 * split_pow2(B * S) / top;
    }

    template <int B, int S> __device__ __forceinline__ unsigned long long split_digits(double x, double f) {
        if constexpr (B == 8) {
            constexpr unsigned long long kBias = 0x8080808080808080ull >> (8 * (8 - S));
            return (unsigned long long)__double_as_longlong(fma(x, f, 0x1.8p52)) + kBias;
        } else {
            const unsigned long long mag = __double2ull_rz(fabs(x) * f);
            unsigned long long u = 0;
            _Pragma("unroll")
            for (int k = 0; k < S; k++) {
                const int d = (int)((mag >> (7 * k)) & 127);
                u |= (unsigned long long)(unsigned char)(signed char)(x < 0 ? -d : d) << (8 * k);
            }
            return u;
        }
    }

    template <int B> __host__ __device__ constexpr unsigned int split_flip() { return B == 8 ? 0x80808080u : 0u; }

    template <int B, int S>
    __device__ __forceinline__ void split_words(const unsigned long long (&u)[4], unsigned int (&w)[S][4], int k4) {
        _Pragma("unroll")
        for (int s = 0; s < S; s++) {
            const int b = S - 1 - s;
            const unsigned int sel = (unsigned int)((b & 3) | ((b & 3) + 4) << 4);
            unsigned int v[4];
            _Pragma("unroll")
            for (int k = 0; k < 4; k++) v[k] = b < 4 ? (unsigned int)u[k] : (unsigned int)(u[k] >> 32);
            w[s][k4] = __byte_perm(__byte_perm(v[0], v[1], sel), __byte_perm(v[2], v[3], sel), 0x5410) ^ split_flip<B>();
        }
    })

}  // namespace slgpu
