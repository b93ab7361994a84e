// Register-resident forward DFT butterflies of radix 1 to 10, 12, 14 to 16, 18, 20, 21, 24, 25, 27, 28, 30 and 32.
//
// All butterflies compute X_p = sum_q v_q * exp(-2*pi*i*p*q/R) in place on an array
// of R complex values held in registers. Inverse transforms are obtained by the
// caller through conjugation (IDFT(x) = conj(DFT(conj(x)))), so only the forward
// sign is compiled. Radix 3/5/7 use the symmetric (cos on sums, sin on
// differences) form; radix 8 and 16 are split-radix products of radix 2 and 4.
//
// The functions are __host__ __device__ so the host test library can check them
// against a direct DFT without a GPU.
#pragma once

#if defined(__CUDACC__)
#define SFB_HD __host__ __device__ __forceinline__
#else
#define SFB_HD inline
#endif

#include <cstdint>
#if defined(__CUDACC__)
#include <cuda_runtime.h>
#else
struct float2 { float x, y; };
struct double2 { double x, y; };
#endif

namespace sfb {

template <class T> struct cvec;
template <> struct cvec<float> { using type = float2; };
template <> struct cvec<double> { using type = double2; };
template <class T> using cplx = typename cvec<T>::type;

template <class C> SFB_HD C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <class C> SFB_HD C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <class C> SFB_HD C cmul(C a, C b) {
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <class C, class T> SFB_HD C cscale(C a, T s) { C r; r.x = a.x * s; r.y = a.y * s; return r; }
template <class C> SFB_HD C cconj(C a) { C r; r.x = a.x; r.y = -a.y; return r; }
// multiply by -i
template <class C> SFB_HD C cmul_mi(C a) { C r; r.x = a.y; r.y = -a.x; return r; }
template <class C> SFB_HD C cmake(decltype(C::x) x, decltype(C::x) y) { C r; r.x = x; r.y = y; return r; }

// Exact decimal expansions of cos/sin at rational multiples of pi.
#define SFB_K3S 0.866025403784438646764
#define SFB_K5C1 0.309016994374947424102
#define SFB_K5C2 -0.809016994374947424102
#define SFB_K5S1 0.951056516295153572116
#define SFB_K5S2 0.587785252292473129169
#define SFB_K7C1 0.623489801858733530525
#define SFB_K7C2 -0.222520933956314404289
#define SFB_K7C3 -0.900968867902419126236
#define SFB_K7S1 0.781831482468029808708
#define SFB_K7S2 0.974927912181823607018
#define SFB_K7S3 0.433883739117558120476
#define SFB_K9C1 0.766044443118978035202
#define SFB_K9S1 0.642787609686539326323
#define SFB_K9C2 0.173648177666930348852
#define SFB_K9S2 0.984807753012208059367
#define SFB_K9C4 -0.939692620785908384054
#define SFB_K9S4 0.342020143325668733044
#define SFB_K8 0.707106781186547524401
#define SFB_K32C1 0.980785280403230449126
#define SFB_K32S1 0.195090322016128267848
#define SFB_K32C3 0.831469612302545237079
#define SFB_K32S3 0.555570233019602224743
#define SFB_K25C1 0.968583161128631119490
#define SFB_K25S1 0.248689887164854788242
#define SFB_K25C2 0.876306680043863587308
#define SFB_K25S2 0.481753674101715274987
#define SFB_K25C3 0.728968627421411523147
#define SFB_K25S3 0.684547105928688673732
#define SFB_K25C4 0.535826794978996618271
#define SFB_K25S4 0.844327925502015078549
#define SFB_K25C6 0.0627905195293133760762
#define SFB_K25S6 0.998026728428271561952
#define SFB_K25C8 -0.425779291565072648863
#define SFB_K25S8 0.904827052466019527714
#define SFB_K25C9 -0.637423989748689710177
#define SFB_K25S9 0.770513242775789230803
#define SFB_K25C12 -0.992114701314477831050
#define SFB_K25S12 0.125333233564304245373
#define SFB_K25C16 -0.637423989748689710177
#define SFB_K25S16 -0.770513242775789230803
#define SFB_K27C1 0.973044870579823838833
#define SFB_K27S1 0.230615870742440178450
#define SFB_K27C2 0.893632640323412248193
#define SFB_K27S2 0.448799180200462172785
#define SFB_K27C4 0.597158591702786164852
#define SFB_K27S4 0.802123192755043785083
#define SFB_K27C5 0.396079766039156823696
#define SFB_K27S5 0.918216106880274014759
#define SFB_K27C7 -0.0581448289104758285387
#define SFB_K27S7 0.998308158271268208048
#define SFB_K27C8 -0.286803232711090253103
#define SFB_K27S8 0.957989512315488874437
#define SFB_K27C10 -0.686241637868733585730
#define SFB_K27S10 0.727373641573048695987
#define SFB_K27C14 -0.993238357741942988548
#define SFB_K27S14 -0.116092914125230229676
#define SFB_K27C16 -0.835487811412936419654
#define SFB_K27S16 -0.549508978070806035263
#define SFB_K16C 0.923879532511286756128
#define SFB_K16S 0.382683432365089771728

template <class C> SFB_HD void bfly2(C& a, C& b) {
    const C t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

template <class C> SFB_HD void bfly4(C& v0, C& v1, C& v2, C& v3) {
    const C t0 = cadd(v0, v2), t1 = csub(v0, v2);
    const C t2 = cadd(v1, v3), t3 = cmul_mi(csub(v1, v3));
    v0 = cadd(t0, t2);
    v2 = csub(t0, t2);
    v1 = cadd(t1, t3);
    v3 = csub(t1, t3);
}

template <class T, class C> SFB_HD void bfly3(C* v) {
    const T k3s = T(SFB_K3S);
    const C s = cadd(v[1], v[2]);
    const C d = csub(v[1], v[2]);
    const C m = cmake<C>(v[0].x - T(0.5) * s.x, v[0].y - T(0.5) * s.y);
    v[0] = cadd(v[0], s);
    // X1 = m - i*k3s*d, X2 = m + i*k3s*d
    v[1] = cmake<C>(m.x + k3s * d.y, m.y - k3s * d.x);
    v[2] = cmake<C>(m.x - k3s * d.y, m.y + k3s * d.x);
}

template <class T, class C> SFB_HD void bfly5(C* v) {
    const T c1 = T(SFB_K5C1), c2 = T(SFB_K5C2), s1 = T(SFB_K5S1), s2 = T(SFB_K5S2);
    const C a1 = cadd(v[1], v[4]), d1 = csub(v[1], v[4]);
    const C a2 = cadd(v[2], v[3]), d2 = csub(v[2], v[3]);
    const C x0 = v[0];
    const C A1 = cmake<C>(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
    const C A2 = cmake<C>(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
    const C B1 = cmake<C>(s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y);
    const C B2 = cmake<C>(s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y);
    v[0] = cmake<C>(x0.x + a1.x + a2.x, x0.y + a1.y + a2.y);
    v[1] = cmake<C>(A1.x + B1.y, A1.y - B1.x);
    v[4] = cmake<C>(A1.x - B1.y, A1.y + B1.x);
    v[2] = cmake<C>(A2.x + B2.y, A2.y - B2.x);
    v[3] = cmake<C>(A2.x - B2.y, A2.y + B2.x);
}

template <class T, class C> SFB_HD void bfly7(C* v) {
    const T c1 = T(SFB_K7C1), c2 = T(SFB_K7C2), c3 = T(SFB_K7C3);
    const T s1 = T(SFB_K7S1), s2 = T(SFB_K7S2), s3 = T(SFB_K7S3);
    const C a1 = cadd(v[1], v[6]), d1 = csub(v[1], v[6]);
    const C a2 = cadd(v[2], v[5]), d2 = csub(v[2], v[5]);
    const C a3 = cadd(v[3], v[4]), d3 = csub(v[3], v[4]);
    const C x0 = v[0];
    // p*q mod 7 table: p=1 -> (1,2,3); p=2 -> (2,4,6); p=3 -> (3,6,2)
    const C A1 = cmake<C>(x0.x + c1 * a1.x + c2 * a2.x + c3 * a3.x,
                          x0.y + c1 * a1.y + c2 * a2.y + c3 * a3.y);
    const C A2 = cmake<C>(x0.x + c2 * a1.x + c3 * a2.x + c1 * a3.x,
                          x0.y + c2 * a1.y + c3 * a2.y + c1 * a3.y);
    const C A3 = cmake<C>(x0.x + c3 * a1.x + c1 * a2.x + c2 * a3.x,
                          x0.y + c3 * a1.y + c1 * a2.y + c2 * a3.y);
    const C B1 = cmake<C>(s1 * d1.x + s2 * d2.x + s3 * d3.x, s1 * d1.y + s2 * d2.y + s3 * d3.y);
    const C B2 = cmake<C>(s2 * d1.x - s3 * d2.x - s1 * d3.x, s2 * d1.y - s3 * d2.y - s1 * d3.y);
    const C B3 = cmake<C>(s3 * d1.x - s1 * d2.x + s2 * d3.x, s3 * d1.y - s1 * d2.y + s2 * d3.y);
    v[0] = cmake<C>(x0.x + a1.x + a2.x + a3.x, x0.y + a1.y + a2.y + a3.y);
    v[1] = cmake<C>(A1.x + B1.y, A1.y - B1.x);
    v[6] = cmake<C>(A1.x - B1.y, A1.y + B1.x);
    v[2] = cmake<C>(A2.x + B2.y, A2.y - B2.x);
    v[5] = cmake<C>(A2.x - B2.y, A2.y + B2.x);
    v[3] = cmake<C>(A3.x + B3.y, A3.y - B3.x);
    v[4] = cmake<C>(A3.x - B3.y, A3.y + B3.x);
}

template <class T, class C> SFB_HD void bfly8(C* v) {
    const T k = T(SFB_K8);
    // DIT: DFT4 of evens and odds, then combine with W8^k.
    bfly4(v[0], v[2], v[4], v[6]);
    bfly4(v[1], v[3], v[5], v[7]);
    // odds: O1 *= W8 = (k, -k), O2 *= -i, O3 *= W8^3 = (-k, -k)
    const C o1 = cmake<C>(k * (v[3].x + v[3].y), k * (v[3].y - v[3].x));
    const C o2 = cmul_mi(v[5]);
    const C o3 = cmake<C>(k * (v[7].y - v[7].x), -k * (v[7].x + v[7].y));
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    const C o0 = v[1];
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
}

template <class T, class C> SFB_HD void bfly16(C* v) {
    const T c = T(SFB_K16C), s = T(SFB_K16S), k = T(SFB_K8);
    // n = n2 + 4*n1: DFT4 over n1 for each n2 (in place: v[n2 + 4*k1] = Y[n2][k1])
    bfly4(v[0], v[4], v[8], v[12]);
    bfly4(v[1], v[5], v[9], v[13]);
    bfly4(v[2], v[6], v[10], v[14]);
    bfly4(v[3], v[7], v[11], v[15]);
    // twiddles W16^(n2*k1): W1=(c,-s) W2=(k,-k) W3=(s,-c) W4=-i W6=(-k,-k) W9=(-c,s)
    v[5] = cmul(v[5], cmake<C>(c, -s));
    v[9] = cmul(v[9], cmake<C>(k, -k));
    v[13] = cmul(v[13], cmake<C>(s, -c));
    v[6] = cmul(v[6], cmake<C>(k, -k));
    v[10] = cmul_mi(v[10]);
    v[14] = cmul(v[14], cmake<C>(-k, -k));
    v[7] = cmul(v[7], cmake<C>(s, -c));
    v[11] = cmul(v[11], cmake<C>(-k, -k));
    v[15] = cmul(v[15], cmake<C>(-c, s));
    // DFT4 over n2 for each k1: X[k1 + 4*k2] from Y[.][k1] at v[4*k1 + n2]
    bfly4(v[0], v[1], v[2], v[3]);
    bfly4(v[4], v[5], v[6], v[7]);
    bfly4(v[8], v[9], v[10], v[11]);
    bfly4(v[12], v[13], v[14], v[15]);
    // now v[4*k1 + k2] = X[k1 + 4*k2]: transpose 4x4 in registers
    C t;
    t = v[1]; v[1] = v[4]; v[4] = t;
    t = v[2]; v[2] = v[8]; v[8] = t;
    t = v[3]; v[3] = v[12]; v[12] = t;
    t = v[6]; v[6] = v[9]; v[9] = t;
    t = v[7]; v[7] = v[13]; v[13] = t;
    t = v[11]; v[11] = v[14]; v[14] = t;
}

// Radix 15 as a prime-factor (Good-Thomas) DFT, 15 = 3 * 5 with coprime factors: no
// internal twiddles. Input n = (5*n1 + 3*n2) mod 15 feeds five-point DFTs over n2, then
// three-point DFTs over n1; output (k1, k2) is X[(10*k1 + 6*k2) mod 15], since
// W15^(n k) = W3^(n1 k1) * W5^(n2 k2) for those index maps.
template <class T, class C> SFB_HD void bfly15(C* v) {
    C a[3][5];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
        for (int n2 = 0; n2 < 5; ++n2) a[n1][n2] = v[(5 * n1 + 3 * n2) % 15];
        bfly5<T>(a[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 5; ++k2) {
        C b[3] = {a[0][k2], a[1][k2], a[2][k2]};
        bfly3<T>(b);
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) v[(10 * k1 + 6 * k2) % 15] = b[k1];
    }
}

// Radix A * B with coprime A and B as a prime-factor (Good-Thomas) DFT, as radix 15 above: input
// n = (B*n1 + A*n2) mod AB, B-point DFTs over n2, A-point DFTs over n1, output k = (B*b*k1 + A*a*k2)
// mod AB with b = B^-1 mod A and a = A^-1 mod B.
template <int R, class T, class C> SFB_HD void dft(C* v);

SFB_HD constexpr int inverse_mod(int a, int m) {
    for (int x = 1; x < m; ++x)
        if (a * x % m == 1) return x;
    return 1;
}

template <int A, int B, class T, class C> SFB_HD void bfly_pfa(C* v) {
    constexpr int R = A * B, kA = B * inverse_mod(B % A, A), kB = A * inverse_mod(A % B, B);
    C a[A][B];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) a[n1][n2] = v[(B * n1 + A * n2) % R];
        dft<B, T>(a[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
        C b[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) b[n1] = a[n1][k2];
        dft<A, T>(b);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) v[(kA * k1 + kB * k2) % R] = b[k1];
    }
}

// Radix 9 as 3 x 3: n = n2 + 3*n1, three-point DFTs over n1, twiddles W9^(n2*k1), three-point
// DFTs over n2; X[k1 + 3*k2].
template <class T, class C> SFB_HD void bfly9(C* v) {
    C a[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < 3; ++n1) a[n2][n1] = v[n2 + 3 * n1];
        bfly3<T>(a[n2]);
    }
    const C w1 = cmake<C>(T(SFB_K9C1), T(-SFB_K9S1)), w2 = cmake<C>(T(SFB_K9C2), T(-SFB_K9S2)),
            w4 = cmake<C>(T(SFB_K9C4), T(-SFB_K9S4));
    a[1][1] = cmul(a[1][1], w1);
    a[1][2] = cmul(a[1][2], w2);
    a[2][1] = cmul(a[2][1], w2);
    a[2][2] = cmul(a[2][2], w4);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
        C b[3] = {a[0][k1], a[1][k1], a[2][k1]};
        bfly3<T>(b);
#pragma unroll
        for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = b[k2];
    }
}

// Radix A * B in two steps: n = n2 + B*n1, A-point DFTs over n1, the constant twiddles W_AB^(n2*k1), B-point
// DFTs over n2; X[k1 + A*k2]. `w` holds (cos, sin) of 2 pi m / AB at index m.
template <int A, int B, class T, class C, class W> SFB_HD void bfly_two(C* v, W w) {
    C a[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) a[n2][n1] = v[n2 + B * n1];
        dft<A, T>(a[n2]);
#pragma unroll
        for (int k1 = 1; k1 < A; ++k1)
            if (n2 > 0) a[n2][k1] = w(n2 * k1, a[n2][k1]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        C b[B];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) b[n2] = a[n2][k1];
        dft<B, T>(b);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = b[k2];
    }
}

template <class T> struct Twiddle25 {
    template <class C> SFB_HD C operator()(int m, C a) const {
        switch (m) {
            case 1: return cmul(a, cmake<C>(T(SFB_K25C1), T(-SFB_K25S1)));
            case 2: return cmul(a, cmake<C>(T(SFB_K25C2), T(-SFB_K25S2)));
            case 3: return cmul(a, cmake<C>(T(SFB_K25C3), T(-SFB_K25S3)));
            case 4: return cmul(a, cmake<C>(T(SFB_K25C4), T(-SFB_K25S4)));
            case 6: return cmul(a, cmake<C>(T(SFB_K25C6), T(-SFB_K25S6)));
            case 8: return cmul(a, cmake<C>(T(SFB_K25C8), T(-SFB_K25S8)));
            case 9: return cmul(a, cmake<C>(T(SFB_K25C9), T(-SFB_K25S9)));
            case 12: return cmul(a, cmake<C>(T(SFB_K25C12), T(-SFB_K25S12)));
            default: return cmul(a, cmake<C>(T(SFB_K25C16), T(-SFB_K25S16)));
        }
    }
};

template <class T> struct Twiddle27 {
    template <class C> SFB_HD C operator()(int m, C a) const {
        switch (m) {
            case 1: return cmul(a, cmake<C>(T(SFB_K27C1), T(-SFB_K27S1)));
            case 2: return cmul(a, cmake<C>(T(SFB_K27C2), T(-SFB_K27S2)));
            case 3: return cmul(a, cmake<C>(T(SFB_K9C1), T(-SFB_K9S1)));
            case 4: return cmul(a, cmake<C>(T(SFB_K27C4), T(-SFB_K27S4)));
            case 5: return cmul(a, cmake<C>(T(SFB_K27C5), T(-SFB_K27S5)));
            case 6: return cmul(a, cmake<C>(T(SFB_K9C2), T(-SFB_K9S2)));
            case 7: return cmul(a, cmake<C>(T(SFB_K27C7), T(-SFB_K27S7)));
            case 8: return cmul(a, cmake<C>(T(SFB_K27C8), T(-SFB_K27S8)));
            case 10: return cmul(a, cmake<C>(T(SFB_K27C10), T(-SFB_K27S10)));
            case 12: return cmul(a, cmake<C>(T(SFB_K9C4), T(-SFB_K9S4)));
            case 14: return cmul(a, cmake<C>(T(SFB_K27C14), T(-SFB_K27S14)));
            default: return cmul(a, cmake<C>(T(SFB_K27C16), T(-SFB_K27S16)));
        }
    }
};

template <class T> struct Twiddle32 {
    template <class C> SFB_HD C operator()(int m, C a) const {
        const T k = T(SFB_K8);
        switch (m) {
            case 1: return cmul(a, cmake<C>(T(SFB_K32C1), T(-SFB_K32S1)));
            case 2: return cmul(a, cmake<C>(T(SFB_K16C), T(-SFB_K16S)));
            case 3: return cmul(a, cmake<C>(T(SFB_K32C3), T(-SFB_K32S3)));
            case 4: return cmake<C>(k * (a.x + a.y), k * (a.y - a.x));
            case 5: return cmul(a, cmake<C>(T(SFB_K32S3), T(-SFB_K32C3)));
            case 6: return cmul(a, cmake<C>(T(SFB_K16S), T(-SFB_K16C)));
            case 7: return cmul(a, cmake<C>(T(SFB_K32S1), T(-SFB_K32C1)));
            case 8: return cmul_mi(a);
            case 9: return cmul(a, cmake<C>(T(-SFB_K32S1), T(-SFB_K32C1)));
            case 10: return cmul(a, cmake<C>(T(-SFB_K16S), T(-SFB_K16C)));
            case 12: return cmake<C>(k * (a.y - a.x), -k * (a.x + a.y));
            case 14: return cmul(a, cmake<C>(T(-SFB_K16C), T(-SFB_K16S)));
            case 15: return cmul(a, cmake<C>(T(-SFB_K32C1), T(-SFB_K32S1)));
            case 18: return cmul(a, cmake<C>(T(-SFB_K16C), T(SFB_K16S)));
            default: return cmul(a, cmake<C>(T(-SFB_K32S3), T(SFB_K32C3)));  // 21
        }
    }
};

// u[r] *= w^r for r = 1..R-1, the powers formed by a balanced product tree
// (w^r = w^h * w^(r-h), h the largest power of two <= r): at most log2(R)+1 roundings deep.
template <int R, class C> SFB_HD void twiddle_powers(C* u, C w) {
    C p[R > 1 ? R : 1];
    p[0] = w;  // p[k] holds w^(k+1)
#pragma unroll
    for (int r = 2; r < R; ++r) {
        int h = 1;
        while (h * 2 <= r) h *= 2;
        p[r - 1] = (h == r) ? cmul(p[h / 2 - 1], p[h / 2 - 1]) : cmul(p[h - 1], p[r - h - 1]);
    }
#pragma unroll
    for (int r = 1; r < R; ++r) u[r] = cmul(u[r], p[r - 1]);
}

// Radix 15 twiddles u[r] *= w^r with few live registers: the powers of the balanced tree
// (w^r = w^h * w^(r-h), at most 4 roundings deep) are formed right before their use, so only
// w, w^2, w^4, w^8 and w^12 stay live instead of all fourteen.
template <class C> SFB_HD void twiddle_powers15(C* u, C w) {
    const C w2 = cmul(w, w);
    const C w4 = cmul(w2, w2);
    const C w8 = cmul(w4, w4);
    u[1] = cmul(u[1], w);
    u[2] = cmul(u[2], w2);
    u[3] = cmul(u[3], cmul(w2, w));
    u[4] = cmul(u[4], w4);
    u[5] = cmul(u[5], cmul(w4, w));
    const C w6 = cmul(w4, w2);
    u[6] = cmul(u[6], w6);
    u[7] = cmul(u[7], cmul(w6, w));
    u[8] = cmul(u[8], w8);
    u[9] = cmul(u[9], cmul(w8, w));
    const C w10 = cmul(w8, w2);
    u[10] = cmul(u[10], w10);
    u[11] = cmul(u[11], cmul(w10, w));
    const C w12 = cmul(w8, w4);
    u[12] = cmul(u[12], w12);
    u[13] = cmul(u[13], cmul(w12, w));
    u[14] = cmul(u[14], cmul(w12, w2));
}

template <int R, class T, class C> SFB_HD void dft(C* v) {
    if constexpr (R == 1) {
        (void)v;
    } else if constexpr (R == 2) {
        bfly2(v[0], v[1]);
    } else if constexpr (R == 3) {
        bfly3<T>(v);
    } else if constexpr (R == 4) {
        bfly4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 5) {
        bfly5<T>(v);
    } else if constexpr (R == 7) {
        bfly7<T>(v);
    } else if constexpr (R == 8) {
        bfly8<T>(v);
    } else if constexpr (R == 6) {
        bfly_pfa<2, 3, T>(v);
    } else if constexpr (R == 9) {
        bfly9<T>(v);
    } else if constexpr (R == 10) {
        bfly_pfa<2, 5, T>(v);
    } else if constexpr (R == 12) {
        bfly_pfa<3, 4, T>(v);
    } else if constexpr (R == 14) {
        bfly_pfa<2, 7, T>(v);
    } else if constexpr (R == 15) {
        bfly15<T>(v);
    } else if constexpr (R == 16) {
        bfly16<T>(v);
    } else if constexpr (R == 18) {
        bfly_pfa<2, 9, T>(v);
    } else if constexpr (R == 20) {
        bfly_pfa<4, 5, T>(v);
    } else if constexpr (R == 21) {
        bfly_pfa<3, 7, T>(v);
    } else if constexpr (R == 24) {
        bfly_pfa<3, 8, T>(v);
    } else if constexpr (R == 25) {
        bfly_two<5, 5, T>(v, Twiddle25<T>());
    } else if constexpr (R == 27) {
        bfly_two<9, 3, T>(v, Twiddle27<T>());
    } else if constexpr (R == 28) {
        bfly_pfa<4, 7, T>(v);
    } else if constexpr (R == 30) {
        bfly_pfa<2, 15, T>(v);
    } else {
        static_assert(R == 32, "no butterfly of this radix");
        bfly_two<8, 4, T>(v, Twiddle32<T>());
    }
}

// Real transforms of length 2N over a complex FFT Z of length N.
// X[k] = 1/2 [(Z[k] + conj Z[N-k]) - i W_2N^k (Z[k] - conj Z[N-k])] * scale; a = Z[k], c = Z[N-k]
template <class C, class T> SFB_HD C real_post_pair(C a, C c, C w, T half) {
    const C e = cmake<C>(a.x + c.x, a.y - c.y);
    const C d = cmake<C>(a.x - c.x, a.y + c.y);
    const T p = w.x * d.x - w.y * d.y, q = w.x * d.y + w.y * d.x;  // w * D
    return cmake<C>((e.x + q) * half, (e.y - p) * half);
}

// Z[k] = (X[k] + conj X[N-k]) + i conj(W_2N^k) (X[k] - conj X[N-k]); a = X[k], c = X[N-k]
template <class C, class T = decltype(C::x)> SFB_HD C real_pre_pair(C a, C c, C w) {
    const C e = cmake<C>(a.x + c.x, a.y - c.y);
    const C d = cmake<C>(a.x - c.x, a.y + c.y);
    const T p = w.x * d.x + w.y * d.y, q = w.x * d.y - w.y * d.x;  // conj(w) * D
    return cmake<C>(e.x - q, e.y + p);
}

// Both bins of a pair: a = Z[k], c = Z[N-k] become X[k], X[N-k] (w = W_2N^k; W_2N^(N-k) = -conj w, so the
// second bin is made of the same sum, difference and product).
template <class C, class T> SFB_HD void real_post_both(C& a, C& c, C w, T half) {
    const C e = cmake<C>((a.x + c.x) * half, (a.y - c.y) * half);
    const C d = cmake<C>((a.x - c.x) * half, (a.y + c.y) * half);
    const C p = cmul(w, d);
    a = cmake<C>(e.x + p.y, e.y - p.x);
    c = cmake<C>(e.x - p.y, -e.y - p.x);
}

// The reverse: a = X[k], c = X[N-k] become Z[k], Z[N-k].
template <class C> SFB_HD void real_pre_both(C& a, C& c, C w) {
    const C e = cmake<C>(a.x + c.x, a.y - c.y);
    const C d = cmake<C>(a.x - c.x, a.y + c.y);
    const C q = cmul(cconj(w), d);
    a = cmake<C>(e.x - q.y, e.y + q.x);
    c = cmake<C>(e.x + q.y, q.x - e.y);
}

}  // namespace sfb
