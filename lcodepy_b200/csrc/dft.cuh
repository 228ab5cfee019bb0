// Small discrete Fourier transforms in registers: the radix steps of the
// field solver's fast transforms.  Forward sign, exp(-2 pi i j k / R); an
// inverse transform swaps the real and imaginary parts going in and coming
// out.
#pragma once

#include <cuda_runtime.h>

namespace lcb {

// cos(2 pi M / R) and sin(2 pi M / R), lowest terms; the halves, quarters and
// eighths are handled by mul_root itself.
template <int M, int R> struct Root;
#define LCB_ROOT(M, R, C, S)                             \
    template <> struct Root<M, R> {                      \
        static constexpr double c = C, s = S;            \
    };
LCB_ROOT(1, 3, -0.5, 0.866025403784438646764)
LCB_ROOT(2, 3, -0.5, -0.866025403784438646764)
LCB_ROOT(1, 5, 0.309016994374947424102, 0.951056516295153572116)
LCB_ROOT(2, 5, -0.809016994374947424102, 0.587785252292473129169)
LCB_ROOT(3, 5, -0.809016994374947424102, -0.587785252292473129169)
LCB_ROOT(4, 5, 0.309016994374947424102, -0.951056516295153572116)
LCB_ROOT(1, 6, 0.5, 0.866025403784438646764)
LCB_ROOT(5, 6, 0.5, -0.866025403784438646764)
LCB_ROOT(1, 7, 0.623489801858733530525, 0.781831482468029808708)
LCB_ROOT(2, 7, -0.222520933956314404289, 0.974927912181823607018)
LCB_ROOT(3, 7, -0.900968867902419126236, 0.433883739117558120476)
LCB_ROOT(4, 7, -0.900968867902419126236, -0.433883739117558120476)
LCB_ROOT(5, 7, -0.222520933956314404289, -0.974927912181823607018)
LCB_ROOT(6, 7, 0.623489801858733530525, -0.781831482468029808708)
LCB_ROOT(1, 9, 0.766044443118978035202, 0.642787609686539326323)
LCB_ROOT(2, 9, 0.173648177666930348852, 0.984807753012208059367)
LCB_ROOT(4, 9, -0.939692620785908384054, 0.342020143325668733044)
LCB_ROOT(5, 9, -0.939692620785908384054, -0.342020143325668733044)
LCB_ROOT(7, 9, 0.173648177666930348852, -0.984807753012208059367)
LCB_ROOT(8, 9, 0.766044443118978035202, -0.642787609686539326323)
LCB_ROOT(1, 10, 0.809016994374947424102, 0.587785252292473129169)
LCB_ROOT(3, 10, -0.309016994374947424102, 0.951056516295153572116)
LCB_ROOT(7, 10, -0.309016994374947424102, -0.951056516295153572116)
LCB_ROOT(9, 10, 0.809016994374947424102, -0.587785252292473129169)
LCB_ROOT(1, 11, 0.841253532831181168862, 0.540640817455597582108)
LCB_ROOT(2, 11, 0.415415013001886425529, 0.909631995354518371412)
LCB_ROOT(3, 11, -0.142314838273285140444, 0.989821441880932732376)
LCB_ROOT(4, 11, -0.654860733945285064057, 0.755749574354258283774)
LCB_ROOT(5, 11, -0.95949297361449738989, 0.281732556841429697711)
LCB_ROOT(6, 11, -0.95949297361449738989, -0.281732556841429697711)
LCB_ROOT(7, 11, -0.654860733945285064057, -0.755749574354258283774)
LCB_ROOT(8, 11, -0.142314838273285140444, -0.989821441880932732376)
LCB_ROOT(9, 11, 0.415415013001886425529, -0.909631995354518371412)
LCB_ROOT(10, 11, 0.841253532831181168862, -0.540640817455597582108)
LCB_ROOT(1, 12, 0.866025403784438646764, 0.5)
LCB_ROOT(5, 12, -0.866025403784438646764, 0.5)
LCB_ROOT(7, 12, -0.866025403784438646764, -0.5)
LCB_ROOT(11, 12, 0.866025403784438646764, -0.5)
LCB_ROOT(1, 13, 0.8854560256532098959, 0.464723172043768545656)
LCB_ROOT(2, 13, 0.568064746731155802512, 0.82298386589365639458)
LCB_ROOT(3, 13, 0.120536680255323053349, 0.992708874098053992801)
LCB_ROOT(4, 13, -0.35460488704253562597, 0.93501624268541482344)
LCB_ROOT(5, 13, -0.748510748171101098635, 0.663122658240795202377)
LCB_ROOT(6, 13, -0.970941817426052027157, 0.239315664287557767149)
LCB_ROOT(7, 13, -0.970941817426052027157, -0.239315664287557767149)
LCB_ROOT(8, 13, -0.748510748171101098635, -0.663122658240795202377)
LCB_ROOT(9, 13, -0.35460488704253562597, -0.93501624268541482344)
LCB_ROOT(10, 13, 0.120536680255323053349, -0.992708874098053992801)
LCB_ROOT(11, 13, 0.568064746731155802512, -0.82298386589365639458)
LCB_ROOT(12, 13, 0.8854560256532098959, -0.464723172043768545656)
LCB_ROOT(1, 16, 0.923879532511286756128, 0.382683432365089771728)
LCB_ROOT(3, 16, 0.382683432365089771728, 0.923879532511286756128)
LCB_ROOT(5, 16, -0.382683432365089771728, 0.923879532511286756128)
LCB_ROOT(7, 16, -0.923879532511286756128, 0.382683432365089771728)
LCB_ROOT(9, 16, -0.923879532511286756128, -0.382683432365089771728)
LCB_ROOT(11, 16, -0.382683432365089771728, -0.923879532511286756128)
LCB_ROOT(13, 16, 0.382683432365089771728, -0.923879532511286756128)
LCB_ROOT(15, 16, 0.923879532511286756128, -0.382683432365089771728)
#undef LCB_ROOT

__host__ __device__ constexpr int root_gcd(int a, int b) { return b == 0 ? a : root_gcd(b, a % b); }

// a exp(-2 pi i M / R)
template <int M0, int R>
__device__ __forceinline__ double2 mul_root(double2 a)
{
    constexpr int M = M0 % R;
    constexpr double h = 0.70710678118654752440;
    if constexpr (M == 0) return a;
    else if constexpr (4 * M == R) return make_double2(a.y, -a.x);
    else if constexpr (2 * M == R) return make_double2(-a.x, -a.y);
    else if constexpr (4 * M == 3 * R) return make_double2(-a.y, a.x);
    else if constexpr (8 * M == R) return make_double2(h * (a.x + a.y), h * (a.y - a.x));
    else if constexpr (8 * M == 3 * R) return make_double2(h * (a.y - a.x), -h * (a.x + a.y));
    else if constexpr (8 * M == 5 * R) return make_double2(-h * (a.x + a.y), h * (a.x - a.y));
    else if constexpr (8 * M == 7 * R) return make_double2(h * (a.x - a.y), h * (a.x + a.y));
    else {
        constexpr int G = root_gcd(M, R);
        constexpr double c = Root<M / G, R / G>::c, s = Root<M / G, R / G>::s;
        return make_double2(fma(a.x, c, a.y * s), fma(a.y, c, -(a.x * s)));
    }
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a w
__device__ __forceinline__ double2 cmul(double2 a, double2 w)
{
    return make_double2(fma(a.x, w.x, -(a.y * w.y)), fma(a.x, w.y, a.y * w.x));
}
__device__ __forceinline__ double2 cswap(double2 a) { return make_double2(a.y, a.x); }

template <int R> struct Dft;

template <> struct Dft<2> {
    __device__ __forceinline__ static void run(double2 *v)
    {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <> struct Dft<4> {
    __device__ __forceinline__ static void run(double2 *v)
    {
        const double2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
        const double2 t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
        v[0] = cadd(t0, t2);
        v[1] = make_double2(t1.x + t3.y, t1.y - t3.x);
        v[2] = csub(t0, t2);
        v[3] = make_double2(t1.x - t3.y, t1.y + t3.x);
    }
};

// Odd prime R from the sums and differences of the mirrored inputs.
template <int R, int K, int J>
__device__ __forceinline__ void odd_term(const double2 *a, const double2 *b, double2 &s, double2 &d)
{
    if constexpr (J <= (R - 1) / 2) {
        constexpr int M = (J * K) % R;
        constexpr double c = Root<M, R>::c, q = Root<M, R>::s;
        s = make_double2(fma(a[J].x, c, s.x), fma(a[J].y, c, s.y));
        d = make_double2(fma(b[J].x, q, d.x), fma(b[J].y, q, d.y));
        odd_term<R, K, J + 1>(a, b, s, d);
    }
}

template <int R, int K>
__device__ __forceinline__ void odd_out(const double2 *a, const double2 *b, double2 v0, double2 *v)
{
    if constexpr (K <= (R - 1) / 2) {
        double2 s = v0, d = make_double2(0.0, 0.0);
        odd_term<R, K, 1>(a, b, s, d);
        v[K] = make_double2(s.x + d.y, s.y - d.x);
        v[R - K] = make_double2(s.x - d.y, s.y + d.x);
        odd_out<R, K + 1>(a, b, v0, v);
    }
}

template <int R> struct DftOdd {
    __device__ __forceinline__ static void run(double2 *v)
    {
        constexpr int H = (R - 1) / 2;
        double2 a[H + 1], b[H + 1], t = v[0];
        const double2 v0 = v[0];
#pragma unroll
        for (int j = 1; j <= H; j++) {
            a[j] = cadd(v[j], v[R - j]);
            b[j] = csub(v[j], v[R - j]);
            t = cadd(t, a[j]);
        }
        v[0] = t;
        odd_out<R, 1>(a, b, v0, v);
    }
};
template <> struct Dft<3> : DftOdd<3> {};
template <> struct Dft<5> : DftOdd<5> {};
template <> struct Dft<7> : DftOdd<7> {};
template <> struct Dft<11> : DftOdd<11> {};
template <> struct Dft<13> : DftOdd<13> {};

// R = A B: B transforms of length A over the inputs n + B m, the twiddles,
// A transforms of length B.
template <int R, int A, int N2, int K1>
__device__ __forceinline__ void twiddle_row(double2 *u)
{
    if constexpr (K1 < A) {
        u[K1] = mul_root<N2 * K1, R>(u[K1]);
        twiddle_row<R, A, N2, K1 + 1>(u);
    }
}

template <int R, int A, int N2>
__device__ __forceinline__ void first_half(const double2 *v, double2 *w)
{
    constexpr int B = R / A;
    if constexpr (N2 < B) {
        double2 u[A];
#pragma unroll
        for (int m = 0; m < A; m++) u[m] = v[N2 + B * m];
        Dft<A>::run(u);
        twiddle_row<R, A, N2, 1>(u);
#pragma unroll
        for (int k = 0; k < A; k++) w[k * B + N2] = u[k];
        first_half<R, A, N2 + 1>(v, w);
    }
}

template <int A, int B> struct DftProduct {
    __device__ __forceinline__ static void run(double2 *v)
    {
        double2 w[A * B];
        first_half<A * B, A, 0>(v, w);
#pragma unroll
        for (int k = 0; k < A; k++) {
            Dft<B>::run(w + k * B);
#pragma unroll
            for (int m = 0; m < B; m++) v[k + A * m] = w[k * B + m];
        }
    }
};
template <> struct Dft<6> : DftProduct<3, 2> {};
template <> struct Dft<8> : DftProduct<4, 2> {};
template <> struct Dft<9> : DftProduct<3, 3> {};
template <> struct Dft<10> : DftProduct<5, 2> {};
template <> struct Dft<12> : DftProduct<4, 3> {};
template <> struct Dft<16> : DftProduct<4, 4> {};

}  // namespace lcb
