// Butterflies of the mixed-radix line passes (mix_dft_impl.cuh): radices 2 to
// 16, 18, 20, 24, 25 and 32, forward or inverse, on complex values in registers
// (which of them a kernel class uses: mix_radix_ok).  Primes by their symmetric
// sums (sum and difference of x_j and x_{R-j}, one real product per pair),
// composites of coprime factors by the prime-factor index maps (no twiddles
// between the two), 9 and 25 as squares of 3 and 5; 2, 3, 4, 8, 16 and 32 are
// the register DFTs' own (cplx.cuh).
#pragma once
#include "cplx.cuh"

namespace flb {

// a * s + c, component by component
template <typename C, typename S> __device__ __forceinline__ C caxpy(C a, S s, C c) { return mkc(fma(a.x, s, c.x), fma(a.y, s, c.y)); }
#if FLB_PAIRED_FP32 && defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
__device__ __forceinline__ float2 caxpy(float2 a, float s, float2 c) { return __ffma2_rn(a, make_float2(s, s), c); }
#endif

// cos(2 pi k / R) and sin(2 pi k / R), k < R
template <int R> struct RadixCS;
template <> struct RadixCS<5> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[5] = {
            1.000000000000000000000, 0.309016994374947424076, -0.809016994374947424104, -0.809016994374947424104,
            0.309016994374947424076
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[5] = {
            0.000000000000000000000, 0.951056516295153572111, 0.587785252292473129135, -0.587785252292473129135,
            -0.951056516295153572111
        };
        return t[k];
    }
};
template <> struct RadixCS<7> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[7] = {
            1.000000000000000000000, 0.623489801858733530527, -0.222520933956314404342, -0.900968867902419126320,
            -0.900968867902419126320, -0.222520933956314404342, 0.623489801858733530527
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[7] = {
            0.000000000000000000000, 0.781831482468029808730, 0.974927912181823606982, 0.433883739117558120293,
            -0.433883739117558120293, -0.974927912181823606982, -0.781831482468029808730
        };
        return t[k];
    }
};
template <> struct RadixCS<9> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[9] = {
            1.000000000000000000000, 0.766044443118978035190, 0.173648177666930348805, -0.500000000000000000163,
            -0.939692620785908384103, -0.939692620785908384103, -0.500000000000000000163, 0.173648177666930348805,
            0.766044443118978035190
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[9] = {
            0.000000000000000000000, 0.642787609686539326327, 0.984807753012208059401, 0.866025403784438646678,
            0.342020143325668732966, -0.342020143325668732966, -0.866025403784438646678, -0.984807753012208059401,
            -0.642787609686539326327
        };
        return t[k];
    }
};
template <> struct RadixCS<11> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[11] = {
            1.000000000000000000000, 0.841253532831181168863, 0.415415013001886425489, -0.142314838273285140460,
            -0.654860733945285064127, -0.959492973614497389901, -0.959492973614497389901, -0.654860733945285064127,
            -0.142314838273285140460, 0.415415013001886425489, 0.841253532831181168863
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[11] = {
            0.000000000000000000000, 0.540640817455597582101, 0.909631995354518371418, 0.989821441880932732359,
            0.755749574354258283704, 0.281732556841429697652, -0.281732556841429697652, -0.755749574354258283704,
            -0.989821441880932732359, -0.909631995354518371418, -0.540640817455597582101
        };
        return t[k];
    }
};
template <> struct RadixCS<13> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[13] = {
            1.000000000000000000000, 0.885456025653209895872, 0.568064746731155802487, 0.120536680255323053250,
            -0.354604887042535626003, -0.748510748171101098684, -0.970941817426052027193, -0.970941817426052027193,
            -0.748510748171101098684, -0.354604887042535626003, 0.120536680255323053250, 0.568064746731155802487,
            0.885456025653209895872
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[13] = {
            0.000000000000000000000, 0.464723172043768545663, 0.822983865893656394580, 0.992708874098053992835,
            0.935016242685414823450, 0.663122658240795202322, 0.239315664287557766952, -0.239315664287557766952,
            -0.663122658240795202322, -0.935016242685414823450, -0.992708874098053992835, -0.822983865893656394580,
            -0.464723172043768545663
        };
        return t[k];
    }
};
template <> struct RadixCS<25> {
    __host__ __device__ static constexpr double c(int k) {
        constexpr double t[25] = {
            1.000000000000000000000, 0.968583161128631119476, 0.876306680043863587301, 0.728968627421411523120,
            0.535826794978996618279, 0.309016994374947424076, 0.062790519529313376009, -0.187381314585724630546,
            -0.425779291565072648802, -0.637423989748689710192, -0.809016994374947424104, -0.929776485888251403612,
            -0.992114701314477831072, -0.992114701314477831072, -0.929776485888251403612, -0.809016994374947424104,
            -0.637423989748689710192, -0.425779291565072648802, -0.187381314585724630546, 0.062790519529313376009,
            0.309016994374947424076, 0.535826794978996618279, 0.728968627421411523120, 0.876306680043863587301,
            0.968583161128631119476
        };
        return t[k];
    }
    __host__ __device__ static constexpr double s(int k) {
        constexpr double t[25] = {
            0.000000000000000000000, 0.248689887164854788230, 0.481753674101715274988, 0.684547105928688673783,
            0.844327925502015078508, 0.951056516295153572111, 0.998026728428271561950, 0.982287250728688681085,
            0.904827052466019527712, 0.770513242775789230815, 0.587785252292473129135, 0.368124552684677959280,
            0.125333233564304245231, -0.125333233564304245231, -0.368124552684677959280, -0.587785252292473129135,
            -0.770513242775789230815, -0.904827052466019527712, -0.982287250728688681085, -0.998026728428271561950,
            -0.951056516295153572111, -0.844327925502015078508, -0.684547105928688673783, -0.481753674101715274988,
            -0.248689887164854788230
        };
        return t[k];
    }
};

// odd prime R: X_k = x_0 + sum_j cos(2 pi j k / R) (x_j + x_{R-j})
//                   -/+ i sum_j sin(2 pi j k / R) (x_j - x_{R-j})
template <int R, bool INV, typename C> __device__ __forceinline__ void dft_prime(C* v) {
    using S = decltype(v[0].x);
    constexpr int H = (R - 1) / 2;
    C a[H], d[H];
    const C x0 = v[0];
    C t = x0;
#pragma unroll
    for (int j = 0; j < H; ++j) {
        a[j] = cadd(v[j + 1], v[R - 1 - j]);
        d[j] = csub(v[j + 1], v[R - 1 - j]);
        t = cadd(t, a[j]);
    }
    v[0] = t;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        C p = x0, q = cscale(d[0], (S)RadixCS<R>::s(k));
#pragma unroll
        for (int j = 0; j < H; ++j) p = caxpy(a[j], (S)RadixCS<R>::c(((j + 1) * k) % R), p);
#pragma unroll
        for (int j = 1; j < H; ++j) q = caxpy(d[j], (S)RadixCS<R>::s(((j + 1) * k) % R), q);
        v[k] = INV ? cadd_i(p, q) : csub_i(p, q);
        v[R - k] = INV ? csub_i(p, q) : cadd_i(p, q);
    }
}

template <int R, bool INV, typename C> __device__ __forceinline__ void dft_any(C* v);

__host__ __device__ constexpr int radix_inv(int a, int m) {
    for (int i = 1; i < m; ++i)
        if ((a * i) % m == 1) return i;
    return 0;
}

// R = A B with coprime factors: x_n, n = (B n1 + A n2) mod R, through A-point
// transforms over n1 and B-point ones over n2; X_k at k = k1 (mod A), k2 (mod B)
template <int A, int B, bool INV, typename C> __device__ __forceinline__ void dft_coprime(C* v) {
    constexpr int R = A * B, EA = B * radix_inv(B % A, A), EB = A * radix_inv(A % B, B);
    C t[R];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
        C u[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) u[n1] = v[(B * n1 + A * n2) % R];
        dft_any<A, INV>(u);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) t[k1 * B + n2] = u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        dft_any<B, INV>(t + k1 * B);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) v[(EA * k1 + EB * k2) % R] = t[k1 * B + k2];
    }
}

// R = A A: x_{n1 + A n2} through A-point transforms over n2, W_R^{n1 k2}, A-point ones over n1
template <int A, bool INV, typename C> __device__ __forceinline__ void dft_square(C* v) {
    using S = decltype(v[0].x);
    C t[A * A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
        C u[A];
#pragma unroll
        for (int n2 = 0; n2 < A; ++n2) u[n2] = v[n1 + A * n2];
        dft_any<A, INV>(u);
        t[n1] = u[0];
#pragma unroll
        for (int k2 = 1; k2 < A; ++k2) {
            const S c = (S)RadixCS<A * A>::c(n1 * k2), s = (S)RadixCS<A * A>::s(n1 * k2);
            t[k2 * A + n1] = n1 == 0 ? u[k2] : cmul(u[k2], mkc(c, INV ? s : -s));
        }
    }
#pragma unroll
    for (int k2 = 0; k2 < A; ++k2) {
        dft_any<A, INV>(t + k2 * A);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) v[k2 + A * k1] = t[k2 * A + k1];
    }
}

template <int R, bool INV, typename C> __device__ __forceinline__ void dft_any(C* v) {
    if constexpr (R == 2) dft2<INV>(v);
    else if constexpr (R == 3) dft3<INV>(v);
    else if constexpr (R == 4) dft4<INV>(v);
    else if constexpr (R == 8) dft8<INV>(v);
    else if constexpr (R == 16) dft16<INV>(v);
    else if constexpr (R == 9) dft_square<3, INV>(v);
    else if constexpr (R == 25) dft_square<5, INV>(v);
    else if constexpr (R == 32) dft32<INV>(v);
    else if constexpr (R == 6) dft_coprime<2, 3, INV>(v);
    else if constexpr (R == 10) dft_coprime<2, 5, INV>(v);
    else if constexpr (R == 12) dft_coprime<4, 3, INV>(v);
    else if constexpr (R == 14) dft_coprime<2, 7, INV>(v);
    else if constexpr (R == 15) dft_coprime<3, 5, INV>(v);
    else if constexpr (R == 18) dft_coprime<2, 9, INV>(v);
    else if constexpr (R == 20) dft_coprime<4, 5, INV>(v);
    else if constexpr (R == 24) dft_coprime<8, 3, INV>(v);
    else dft_prime<R, INV>(v);
}

}  // namespace flb
