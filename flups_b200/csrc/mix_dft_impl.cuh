#pragma once
// Mixed-radix line passes: lengths 2^a 3^b 5^c 7^d 11^e 13^f in two to four
// stages of radices up to 16 (13 in FP64), or, for complex columns that would
// take three, in two of radices up to 32 (20 in FP64), for the lines the
// register DFTs (fast_dft_impl.cuh) do not take.
//
// A line sits in shared memory once.  A forward transform decimates in
// frequency: stage s reads the R values of a butterfly, transforms them in
// registers, multiplies by the twiddles and writes them back to the places it
// read, so a stage needs one barrier and no second buffer.  The first stage
// reads its values straight from global memory and the last hands its
// spectrum values, k = q + (M / R) j for j < R, straight to the store; an
// inverse transform runs the same stages backwards (decimation in time).
// The spectrum never has to be put in order: a fused pass multiplies the last
// stage's values by the Green's function and starts the inverse from the same
// registers.
//
// Digits: after stage s, element (k_1, ..., k_s, m) of the line is at
// k_1 s1 + k_2 nn_2 + ... + m, s1 = nn_1 or the next odd number, so that lanes
// whose k_1 differs meet distinct banks; butterflies are numbered with k_1
// fastest.
//
// Two real lines travel as z = a + i b.  Their spectra need Z_k and Z_{M-k},
// which are butterflies q and M/R - q of the last stage: one thread takes
// both, so parting the two costs no exchange.
//
// Column passes: lanes along x over TX lines, row passes: lanes along the
// line.  blockDim = (TX, P) or (P, TX): P threads share a line.
#include "cplx.cuh"
#include "mix_dft.h"
#include "radix.cuh"
#include "smem_attr.cuh"

namespace flb {

// Two classes of kernels.  MULTI: two to four stages of radices up to 16,
// three 256-thread CTAs per SM in FP32 (80 registers), two in FP64 (128).
// TWO: exactly two stages, radices up to 32 in FP32 (128 registers, 512
// threads per SM) and 20 in FP64 (168 registers, 384 threads), for lengths
// that MULTI runs in three: a stage less is a round trip through shared memory,
// a twiddle product per value and a barrier less (400-point fused columns of
// a 200^3 grid, FP32: 10 x 8 x 5 186 us, 20 x 20 156 us; FP64 302 -> 254 us).
template <typename T, int CLS> struct MixOcc {
    static constexpr int threads = mix_threads(sizeof(T) == 8, CLS);
    static constexpr int blocks = CLS == MIX_TWO ? (sizeof(T) == 8 ? 3 : 2) : (sizeof(T) == 8 ? 2 : 3);
};

// x / d for x d < 2^32, mul = ceil(2^32 / d)
__device__ __forceinline__ int mix_div(int x, int d, unsigned mul) { return d == 1 ? x : (int)__umulhi((unsigned)x, mul); }

template <int V> struct MixInt { static constexpr int v = V; };

// f(0), ..., f(N - 1) with compile-time arguments
template <int N, int I = 0, typename F> __device__ __forceinline__ void mix_each(F&& f) {
    if constexpr (I < N) {
        f(MixInt<I>{});
        mix_each<N, I + 1>(f);
    }
}

// f with the radix as a compile-time constant: the radices of a class (F64:
// of its FP64 kernels); SMALL: of a last stage that holds two or three
// butterflies
template <int CLS, bool F64, bool SMALL, int R = 32, typename F> __device__ __forceinline__ void mix_radix(int r, F&& f) {
    if constexpr (R >= 2) {
        if constexpr (mix_radix_ok(CLS, F64, SMALL, R)) {
            if (r == R) {
                f(MixInt<R>{});
                return;
            }
        }
        mix_radix<CLS, F64, SMALL, R - 1>(r, f);
    }
}

__device__ __forceinline__ int mix_fold(int i, int M) { return (M > 0 && 2 * i > M) ? M - i : i; }

// the outer index in mirror pairs (0, 1, M-1, 2, ...) when the Green's
// function is folded along it: its slab is read again while still in L2
__device__ __forceinline__ int mix_mirror(int by, int n, int fold) {
    if (fold != n || by == 0) return by;
    const int m = (by + 1) >> 1;
    return (by & 1) ? m : n - m;
}

template <typename T, bool ROWS, int CLS>
struct MixLine {
    using C = typename CT<T>::C;
    static constexpr bool F64 = sizeof(T) == 8;
    C* sm;           // element 0 of this thread's line
    int es;          // elements between neighbouring elements of the line
    int p, P;        // this thread of the line's P
    const MixPlan& pl;
    const C* tw;

    __device__ __forceinline__ C* at(int e) const { return ROWS ? sm + e : sm + e * es; }
    __device__ __forceinline__ int step(int n) const { return ROWS ? n : n * es; }
    // place of the block with digits (k_1, ..., k_{s-1}) packed in q, k_1 fastest (s: stage, from 0)
    __device__ __forceinline__ int block(int s, int q) const {
        if (CLS == MIX_TWO || s == 1) return q * pl.s1;
        int k = mix_div(q, pl.st[0].R, pl.st[1].qmul);
        int off = (q - k * pl.st[0].R) * pl.s1;
        if (s == 2) return off + k * pl.st[1].nn;
        const int k3 = mix_div(q, pl.st[2].Q, pl.st[2].qmul);
        return off + (k - k3 * pl.st[1].R) * pl.st[1].nn + k3 * pl.st[2].nn;
    }
    // forward first stage: ld(v, m, nn) fills v[n] = x[m + n nn]
    template <typename LD> __device__ __forceinline__ void first(LD&& ld) const {
        mix_radix<CLS, F64, false>(pl.st[0].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int nn = pl.st[0].nn, d = step(pl.s1);
            for (int m = p; m < nn; m += P) {
                C v[R];
                ld(v, m, nn, rc);
                dft_any<R, false>(v);
                const C* w = tw + pl.st[0].tw + m;
                C* dst = at(m);
                dst[0] = v[0];
#pragma unroll
                for (int k = 1; k < R; ++k) dst[k * d] = cmul(v[k], __ldg(w + (k - 1) * nn));
            }
        });
    }
    // forward middle stage
    __device__ __forceinline__ void middle(int s) const {
        mix_radix<CLS, F64, false>(pl.st[s].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int nn = pl.st[s].nn, Q = pl.st[s].Q, d = step(nn);
            for (int b = p; b < nn * Q; b += P) {
                const int m = mix_div(b, Q, pl.st[s].qmul);
                C* x = at(block(s, b - m * Q) + m);
                C v[R];
#pragma unroll
                for (int n = 0; n < R; ++n) v[n] = x[n * d];
                dft_any<R, false>(v);
                const C* w = tw + pl.st[s].tw + m;
                x[0] = v[0];
#pragma unroll
                for (int k = 1; k < R; ++k) x[k * d] = cmul(v[k], __ldg(w + (k - 1) * nn));
            }
        });
    }
    // inverse middle stage
    __device__ __forceinline__ void middle_inv(int s) const {
        mix_radix<CLS, F64, false>(pl.st[s].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int nn = pl.st[s].nn, Q = pl.st[s].Q, d = step(nn);
            for (int b = p; b < nn * Q; b += P) {
                const int m = mix_div(b, Q, pl.st[s].qmul);
                C* x = at(block(s, b - m * Q) + m);
                const C* w = tw + pl.st[s].tw + m;
                C v[R];
                v[0] = x[0];
#pragma unroll
                for (int k = 1; k < R; ++k) v[k] = cmulc(x[k * d], __ldg(w + (k - 1) * nn));
                dft_any<R, true>(v);
#pragma unroll
                for (int n = 0; n < R; ++n) x[n * d] = v[n];
            }
        });
    }
    // inverse last stage: st(v, m, nn) stores v[n] = x[m + n nn]
    template <typename ST> __device__ __forceinline__ void first_inv(ST&& sto) const {
        mix_radix<CLS, F64, false>(pl.st[0].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int nn = pl.st[0].nn, d = step(pl.s1);
            for (int m = p; m < nn; m += P) {
                const C* src = at(m);
                const C* w = tw + pl.st[0].tw + m;
                C v[R];
                v[0] = src[0];
#pragma unroll
                for (int k = 1; k < R; ++k) v[k] = cmulc(src[k * d], __ldg(w + (k - 1) * nn));
                dft_any<R, true>(v);
                sto(v, m, nn, rc);
            }
        });
    }
    __device__ __forceinline__ void forward_middles() const {
        if constexpr (CLS == MIX_TWO) return;
        for (int s = 1; s + 1 < pl.ns; ++s) {
            middle(s);
            __syncthreads();
        }
    }
    __device__ __forceinline__ void inverse_middles() const {
        if constexpr (CLS == MIX_TWO) return;
        for (int s = pl.ns - 2; s > 0; --s) {
            middle_inv(s);
            __syncthreads();
        }
    }
};

// line positions of a thread: one, or the two of a pair.  Lines are paired
// within a plane b and by their index a alone, so a pass over part of the
// planes (slabs) or with another tile pairs the same lines: rows 2i and
// 2i + 1, columns x and x + 8 of 16 (each half of a pair then loads whole
// runs).  Lines outside the array point at position 0 and are neither loaded
// nor stored.
template <bool PAIR, bool ROWS>
struct MixPos {
    static constexpr int H = PAIR ? 2 : 1;
    int ia[H], ib;
    bool ok[H];
    __device__ __forceinline__ MixPos(const MixArgs& a, int c, int TX, bool mirror) {
        const int units = mix_units(a.na, PAIR, ROWS);
        int u = blockIdx.x * TX + c;  // line or pair
        if constexpr (ROWS) {
            ib = u / units;
            u -= ib * units;
        } else {
            ib = mirror ? mix_mirror(blockIdx.y, a.nb, a.f_b) : (int)blockIdx.y;
        }
        const bool in = ib < a.nb && u < units;
        if (!in) ib = 0;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            ia[h] = !PAIR ? u : (ROWS ? 2 * u + h : 16 * (u >> 3) + (u & 7) + 8 * h);
            ok[h] = in && ia[h] < a.na;
            if (!ok[h]) ia[h] = 0;
        }
    }
    template <typename E> __device__ __forceinline__ const E* src(const MixArgs& a, int h) const {
        return reinterpret_cast<const E*>(a.in) + blockIdx.z * a.in_sc + ia[h] * a.in_sa + ib * a.in_sb;
    }
    template <typename E> __device__ __forceinline__ E* dst(const MixArgs& a, int h) const {
        return reinterpret_cast<E*>(a.out) + blockIdx.z * a.out_sc + ia[h] * a.out_sa + ib * a.out_sb;
    }
    template <typename T> __device__ __forceinline__ const T* green(const MixArgs& a, int h) const {
        return reinterpret_cast<const T*>(a.green) + (int64_t)mix_fold(ia[h], a.f_a) * a.g_sa + (int64_t)mix_fold(ib, a.f_b) * a.g_sb;
    }
};

template <typename T, int OP, bool ROWS, int CLS>
__global__ void __launch_bounds__(MixOcc<T, CLS>::threads, MixOcc<T, CLS>::blocks) mix_kernel(const __grid_constant__ MixArgs a) {
    using C = typename CT<T>::C;
    constexpr bool PAIR = mix_pairs(OP);
    extern __shared__ __align__(16) unsigned char smraw[];
    const int c = ROWS ? threadIdx.y : threadIdx.x;  // line of the tile
    const int TX = ROWS ? blockDim.y : blockDim.x;
    const MixLine<T, ROWS, CLS> L{reinterpret_cast<C*>(smraw) + (ROWS ? c * a.pl.len : c), TX, (int)(ROWS ? threadIdx.x : threadIdx.y),
                             (int)(ROWS ? blockDim.x : blockDim.y), a.pl, reinterpret_cast<const C*>(a.tw)};
    const int M = a.pl.M, ns = a.pl.ns;
    const MixPos<PAIR, ROWS> W(a, c, TX, OP == MX_FUSED);
    pass_begin();
    const auto& ok = W.ok;
    const int isl = (int)a.in_sl, osl = (int)a.out_sl;
    const C zero = mkc((T)0, (T)0);

    // ---------------------------------------------------------- to the frequency side
    if constexpr (OP == MX_C2C_F || OP == MX_FUSED) {
        const C* in = W.template src<C>(a, 0);
        const int n_src = ok[0] ? a.n_src : 0;
        L.first([&](auto& v, int m, int nn, auto rc) {
            constexpr int R = decltype(rc)::v;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int j = m + n * nn;
                v[n] = j < n_src ? in[j * isl] : zero;
            }
        });
        __syncthreads();
        L.forward_middles();
    }
    if constexpr (OP == MX_R2C) {
        auto load = [&](auto tag) {
            using E = decltype(tag);
            const E* in0 = W.template src<E>(a, 0);
            const E* in1 = W.template src<E>(a, 1);
            const int n0 = ok[0] ? a.n_src : 0, n1 = ok[1] ? a.n_src : 0;
            L.first([&](auto& v, int m, int nn, auto rc) {
                constexpr int R = decltype(rc)::v;
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int j = m + n * nn;
                    v[n] = mkc(j < n0 ? (T)in0[j * isl] : (T)0, j < n1 ? (T)in1[j * isl] : (T)0);
                }
            });
        };
        if (sizeof(T) == 8 || a.in64) load(double{});
        else load(T{});
        __syncthreads();
        L.forward_middles();
    }

    // ---------------------------------------------------------- at the frequency side
    const int nq = a.pl.st[ns - 1].Q;  // butterflies of the last stage: k = q + nq j
    if constexpr (OP == MX_C2C_F) {
        C* out = W.template dst<C>(a, 0);
        const int n_store = ok[0] ? (a.n_store < M ? a.n_store : M) : 0;
        mix_radix<CLS, sizeof(T) == 8, false>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; q < nq; q += L.P) {
                const C* x = L.at(L.block(ns - 1, q));
                C v[R];
#pragma unroll
                for (int n = 0; n < R; ++n) v[n] = x[n * d];
                dft_any<R, false>(v);
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    if (k < n_store) out[k * osl] = v[j];
                }
                if (q == 0 && a.period >= 0 && ok[0]) out[a.period * osl] = v[0];
            }
        });
        return;
    }
    if constexpr (OP == MX_C2C_I) {
        const C* in = W.template src<C>(a, 0);
        const int n_src = ok[0] ? a.n_src : 0;
        mix_radix<CLS, sizeof(T) == 8, false>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; q < nq; q += L.P) {
                C v[R];
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    v[j] = k < n_src ? in[k * isl] : zero;
                }
                dft_any<R, true>(v);
                C* x = L.at(L.block(ns - 1, q));
#pragma unroll
                for (int n = 0; n < R; ++n) x[n * d] = v[n];
            }
        });
    }
    if constexpr (OP == MX_FUSED) {
        const T* g = W.template green<T>(a, 0);
        const int gl = (int)a.g_sl;
        mix_radix<CLS, sizeof(T) == 8, false>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; q < nq; q += L.P) {
                T gv[R];
#pragma unroll
                for (int j = 0; j < R; ++j) gv[j] = __ldg(g + mix_fold(q + nq * j, a.f_l) * gl);
                C* x = L.at(L.block(ns - 1, q));
                C v[R];
#pragma unroll
                for (int n = 0; n < R; ++n) v[n] = x[n * d];
                dft_any<R, false>(v);
#pragma unroll
                for (int j = 0; j < R; ++j) v[j] = cscale(v[j], gv[j]);
                dft_any<R, true>(v);
#pragma unroll
                for (int n = 0; n < R; ++n) x[n * d] = v[n];
            }
        });
    }
    if constexpr (OP == MX_R2C) {
        C* out0 = W.template dst<C>(a, 0);
        C* out1 = W.template dst<C>(a, 1);
        mix_radix<CLS, sizeof(T) == 8, true>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; 2 * q <= nq; q += L.P) {
                const bool self = q == 0 || 2 * q == nq;  // k and M - k in one butterfly
                C v[R], w[R];
                const C* x = L.at(L.block(ns - 1, q));
#pragma unroll
                for (int n = 0; n < R; ++n) v[n] = x[n * d];
                const C* y = L.at(L.block(ns - 1, q == 0 ? 0 : nq - q));
#pragma unroll
                for (int n = 0; n < R; ++n) w[n] = y[n * d];
                dft_any<R, false>(v);
                dft_any<R, false>(w);
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    const bool up = 2 * k > M;
                    if (self && up) continue;
                    const C zk = v[j];
                    C zm = w[R - 1 - j];
                    if (q == 0) zm = w[(R - j) % R];
                    // A = (Z_k + conj Z_{M-k}) / 2, B = (Z_k - conj Z_{M-k}) / 2i
                    C A = mkc((T)0.5 * (zk.x + zm.x), (T)0.5 * (zk.y - zm.y));
                    C B = mkc((T)0.5 * (zk.y + zm.y), (T)0.5 * (zm.x - zk.x));
                    if (up) {
                        A = cconj(A);
                        B = cconj(B);
                    }
                    const int kk = (up ? M - k : k) * osl;
                    if (ok[0]) out0[kk] = A;
                    if (ok[1]) out1[kk] = B;
                    if (j == 0 && q == 0 && a.period >= 0) {
                        if (ok[0]) out0[a.period * osl] = A;
                        if (ok[1]) out1[a.period * osl] = B;
                    }
                }
            }
        });
        return;
    }
    if constexpr (OP == MX_C2R) {
        const C* in0 = W.template src<C>(a, 0);
        const C* in1 = W.template src<C>(a, 1);
        mix_radix<CLS, sizeof(T) == 8, true>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; 2 * q <= nq; q += L.P) {
                C v[R], w[R];
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    const bool up = 2 * k > M;
                    const int kk = (up ? M - k : k) * isl;
                    C A = ok[0] ? in0[kk] : zero;
                    C B = ok[1] ? in1[kk] : zero;
                    // Im A_0 and Im A_{M/2} do not enter a real result
                    if (k == 0 || 2 * k == M) A.y = B.y = (T)0;
                    if (up) {
                        A.y = -A.y;
                        B.y = -B.y;
                    }
                    v[j] = mkc(A.x - B.y, A.y + B.x);          // Z_k = A_k + i B_k
                    w[R - 1 - j] = mkc(A.x + B.y, B.x - A.y);  // Z_{M-k} = conj A_k + i conj B_k
                }
                dft_any<R, true>(v);
                C* x = L.at(L.block(ns - 1, q));
#pragma unroll
                for (int n = 0; n < R; ++n) x[n * d] = v[n];
                if (q != 0 && 2 * q != nq) {
                    dft_any<R, true>(w);
                    C* y = L.at(L.block(ns - 1, nq - q));
#pragma unroll
                    for (int n = 0; n < R; ++n) y[n * d] = w[n];
                }
            }
        });
    }

    // ---------------------------------------------------------- back to the spatial side
    __syncthreads();
    L.inverse_middles();
    if constexpr (OP == MX_C2C_I || OP == MX_FUSED) {
        C* out = W.template dst<C>(a, 0);
        const int n_store = ok[0] ? (a.n_store < M ? a.n_store : M) : 0;
        L.first_inv([&](auto& v, int m, int nn, auto rc) {
            constexpr int R = decltype(rc)::v;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int j = m + n * nn;
                if (j < n_store) out[j * osl] = v[n];
            }
            if (m == 0 && a.period >= 0 && ok[0]) out[a.period * osl] = v[0];
        });
    }
    if constexpr (OP == MX_C2R) {
        auto store = [&](auto tag) {
            using E = decltype(tag);
            E* out0 = W.template dst<E>(a, 0);
            E* out1 = W.template dst<E>(a, 1);
            const int ns0 = a.n_store < M ? a.n_store : M;
            const int n0 = ok[0] ? ns0 : 0, n1 = ok[1] ? ns0 : 0;
            L.first_inv([&](auto& v, int m, int nn, auto rc) {
                constexpr int R = decltype(rc)::v;
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int j = m + n * nn;
                    if (j < n0) out0[j * osl] = (E)v[n].x;
                    if (j < n1) out1[j * osl] = (E)v[n].y;
                }
                if (m == 0 && a.period >= 0) {
                    if (ok[0]) out0[a.period * osl] = (E)v[0].x;
                    if (ok[1]) out1[a.period * osl] = (E)v[0].y;
                }
            });
        };
        if (sizeof(T) == 8 || a.out64) store(double{});
        else store(T{});
    }
}

// ---------------------------------------------------------------- real transforms
// DCT / DST I-IV and the fused passes of a real last direction, by FFTW's
// definitions.  N: the kind's size.
//   II   v_n = x_{t(n)}, t = 2n for 2n < N, else 2(N - n) - 1; with A the
//        N-point spectrum of v, U_k = 2 W_4N^k A_k = Y_k - i Y_{N-k};
//   III  its inverse: A_k = W_4N^{-k} (x_k - i x_{N-k}), x_N = 0; y_{t(n)} = v_n;
//   I    the line's even (odd) extension of M = 2(N -/+ 1) points, whose
//        spectrum is real (imaginary);
//   IV   t_j = (x_{2j} + i x_{N-1-2j}) W_8N^{4j+1}, T its N/2-point spectrum,
//        2 W_4N^{2k} T_k = Y_{2k} - i Y_{N-1-2k}.
// DST-II(x)_k = DCT-II((-1)^j x_j)_{N-1-k}, DST-III(x)_k = (-1)^k DCT-III(x_{N-1-j})_k,
// DST-IV(x)_k = (-1)^k DCT-IV(x_{N-1-j})_k.  Between type III and type II of
// a fused pass the two signs cancel.
template <typename T, int OP, bool ROWS, int CLS>
__global__ void __launch_bounds__(MixOcc<T, CLS>::threads, MixOcc<T, CLS>::blocks) mix_real_kernel(const __grid_constant__ MixArgs a) {
    using C = typename CT<T>::C;
    constexpr bool PAIR = mix_pairs(OP);
    constexpr bool GREEN = OP >= MX_FUSED_R;
    constexpr bool TYPE1 = OP == MX_T1 || OP == MX_FUSED_11, TYPE4 = OP == MX_T4 || OP == MX_FUSED_44;
    constexpr bool FROM2 = OP == MX_T2 || OP == MX_FUSED_23;  // line values enter by t(n)
    constexpr bool TO3 = OP == MX_T3 || OP == MX_FUSED_23;    // line values leave by t(n)
    extern __shared__ __align__(16) unsigned char smraw[];
    const int c = ROWS ? threadIdx.y : threadIdx.x;
    const int TX = ROWS ? blockDim.y : blockDim.x;
    const MixLine<T, ROWS, CLS> L{reinterpret_cast<C*>(smraw) + (ROWS ? c * a.pl.len : c), TX, (int)(ROWS ? threadIdx.x : threadIdx.y),
                             (int)(ROWS ? blockDim.x : blockDim.y), a.pl, reinterpret_cast<const C*>(a.tw)};
    const MixPos<PAIR, ROWS> W(a, c, TX, GREEN);
    pass_begin();
    constexpr int H = MixPos<PAIR, ROWS>::H;
    const int M = a.pl.M, ns = a.pl.ns, R_last = a.pl.st[ns - 1].R, nq = a.pl.st[ns - 1].Q;
    const int isl = (int)a.in_sl, osl = (int)a.out_sl;
    const int cs = blockIdx.z % a.lda, N = a.N[cs];
    const bool odd = OP != MX_FUSED_R && a.dst[cs];
    const int ioff = a.fi[cs] - a.fieldstart, ooff = a.fo[cs] - a.store_off;  // line element of transform element 0
    const C* tw4 = reinterpret_cast<const C*>(a.tw4);
    const C* tw8 = reinterpret_cast<const C*>(a.tw8);
    const T zero = (T)0;
    const T* g[2] = {nullptr, nullptr};
    const int gl = (int)a.g_sl, goff = a.go[cs];
    if constexpr (GREEN) {
        g[0] = W.template green<T>(a, 0);
        g[1] = W.template green<T>(a, H - 1);
    }
    auto t_of = [&](int n) { return 2 * n < N ? 2 * n : 2 * (N - n) - 1; };

    // in: f(get) with get(h, t) = transform input t of line h (zero outside the source); out: f(put)
    auto with_input = [&](auto&& f) {
        auto go = [&](auto tag) {
            using E = decltype(tag);
            const E* p0 = W.template src<E>(a, 0);
            const E* p1 = W.template src<E>(a, H - 1);
            const int n0 = W.ok[0] ? a.n_src : 0, n1 = W.ok[H - 1] ? a.n_src : 0;
            f([&](int h, int t) {
                const int j = t + ioff;
                return j >= 0 && j < (h ? n1 : n0) ? (T)(h ? p1 : p0)[j * isl] : zero;
            });
        };
        if (sizeof(T) == 8 || a.in64) go(double{});
        else go(T{});
    };
    auto with_output = [&](auto&& f) {
        auto go = [&](auto tag) {
            using E = decltype(tag);
            E* p0 = W.template dst<E>(a, 0);
            E* p1 = W.template dst<E>(a, H - 1);
            const int n0 = W.ok[0] ? a.n_store : 0, n1 = W.ok[H - 1] ? a.n_store : 0;
            f([&](int h, int t, T y) {
                const int i = t + ooff;
                if (i >= 0 && i < (h ? n1 : n0)) (h ? p1 : p0)[i * osl] = (E)y;
            });
            // outputs outside the transform: zero, or the periodic copy (stored by its owner below)
            if (L.p == 0) {
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const int n = h ? n1 : n0;
                    E* p = h ? p1 : p0;
                    if (a.z0[cs] >= 0 && a.z0[cs] < n) p[a.z0[cs] * osl] = (E)0;
                    if (a.z1[cs] >= 0 && a.z1[cs] < n) p[a.z1[cs] * osl] = (E)0;
                }
            }
        };
        if (sizeof(T) == 8 || a.out64) go(double{});
        else go(T{});
    };
    // Green's value of line h at spectral element i of the line
    auto gval = [&](int h, int i) { return __ldg(g[h] + i * gl); };

    // ---------------------------------------------------------- line values in, to the frequency side
    if constexpr (OP != MX_T3 && OP != MX_FUSED_32) {
        with_input([&](auto&& get) {
            L.first([&](auto& v, int m, int nn, auto rc) {
                constexpr int R = decltype(rc)::v;
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int e = m + n * nn;
                    if constexpr (FROM2) {
                        const int t = t_of(e);
                        const T s = odd && (t & 1) ? (T)-1 : (T)1;
                        v[n] = mkc(s * get(0, t), s * get(1, t));
                    } else if constexpr (TYPE1) {
                        int t = e;
                        T s = (T)1;
                        if (odd) {
                            t = e <= N ? e - 1 : M - e - 1;
                            s = e == 0 || e == N + 1 ? zero : (e <= N ? (T)1 : (T)-1);
                            if (e == 0 || e == N + 1) t = 0;
                        } else if (e >= N) {
                            t = M - e;
                        }
                        v[n] = mkc(s * get(0, t), s * get(1, t));
                    } else if constexpr (TYPE4) {
                        const T x = get(0, 2 * e), y = get(0, N - 1 - 2 * e);
                        v[n] = cmul(odd ? mkc(y, x) : mkc(x, y), __ldg(tw8 + e));
                    } else {
                        v[n] = mkc(get(0, e), get(1, e));
                    }
                }
            });
        });
        __syncthreads();
        L.forward_middles();
    }

    // k and M - k of a pair: f(v, w, q, self, rc) between the forward and / or inverse butterflies of class q and nq - q
    auto mirrored = [&](auto fwd, auto inv, auto&& f) {
        mix_radix<CLS, sizeof(T) == 8, true>(R_last, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; 2 * q <= nq; q += L.P) {
                const bool self = q == 0 || 2 * q == nq;
                C v[R], w[R];
                C* x = L.at(L.block(ns - 1, q));
                C* y = L.at(L.block(ns - 1, q == 0 ? 0 : nq - q));
                if constexpr (decltype(fwd)::v) {
#pragma unroll
                    for (int n = 0; n < R; ++n) v[n] = x[n * d];
#pragma unroll
                    for (int n = 0; n < R; ++n) w[n] = y[n * d];
                    dft_any<R, false>(v);
                    dft_any<R, false>(w);
                }
                f(v, w, q, self, rc);
                if constexpr (decltype(inv)::v) {
                    dft_any<R, true>(v);
#pragma unroll
                    for (int n = 0; n < R; ++n) x[n * d] = v[n];
                    if (!self) {
                        dft_any<R, true>(w);
#pragma unroll
                        for (int n = 0; n < R; ++n) y[n * d] = w[n];
                    }
                }
            }
        });
    };
    // A_k, B_k of the two lines from Z_k = v[j] and Z_{M-k}
    auto part = [&](const auto& v, const auto& w, int q, auto jc, auto rc, C& A, C& B) {
        constexpr int R = decltype(rc)::v, j = decltype(jc)::v;
        const C zk = v[j];
        C zm = w[R - 1 - j];
        if (q == 0) zm = w[(R - j) % R];
        A = mkc((T)0.5 * (zk.x + zm.x), (T)0.5 * (zk.y - zm.y));
        B = mkc((T)0.5 * (zk.y + zm.y), (T)0.5 * (zm.x - zk.x));
    };
    using Yes = MixInt<1>;
    using No = MixInt<0>;

    // ---------------------------------------------------------- at the frequency side
    // the spectrum of line values at k as (Y_k, -Y_{N-k}) of type II, stored
    auto store2 = [&](auto&& put) {
        mirrored(Yes{}, No{}, [&](auto& v, auto& w, int q, bool self, auto rc) {
            constexpr int R = decltype(rc)::v;
            mix_each<R>([&](auto jc) {
                constexpr int j = decltype(jc)::v;
                const int k = q + nq * j;
                if (self && 2 * k > M) return;
                C A[2];
                part(v, w, q, jc, rc, A[0], A[1]);
                const C t = __ldg(tw4 + k);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const C u = cmul(t, A[h]);
                    put(h, odd ? N - 1 - k : k, (T)2 * u.x);
                    if (k > 0 && 2 * k != N) put(h, odd ? k - 1 : N - k, (T)-2 * u.y);
                }
            });
        });
    };
    // type III inputs to Z_k, first inverse stage
    auto load3 = [&](auto&& get) {
        mirrored(No{}, Yes{}, [&](auto& v, auto& w, int q, bool self, auto rc) {
            constexpr int R = decltype(rc)::v;
            mix_each<R>([&](auto jc) {
                constexpr int j = decltype(jc)::v;
                const int k = q + nq * j;
                const C t = __ldg(tw4 + k);
                C A[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const T x = get(h, odd ? N - 1 - k : k);
                    const T y = k > 0 ? get(h, odd ? k - 1 : N - k) : zero;
                    A[h] = cmulc(mkc(x, -y), t);
                }
                v[j] = mkc(A[0].x - A[1].y, A[0].y + A[1].x);
                w[R - 1 - j] = mkc(A[0].x + A[1].y, A[1].x - A[0].y);
            });
        });
    };
    if constexpr (OP == MX_T2) {
        with_output([&](auto&& put) { store2(put); });
        return;
    }
    if constexpr (OP == MX_T1) {
        with_output([&](auto&& put) {
            mix_radix<CLS, sizeof(T) == 8, false>(R_last, [&](auto rc) {
                constexpr int R = decltype(rc)::v;
                const int d = L.step(1);
                for (int q = L.p; q < nq; q += L.P) {
                    const C* x = L.at(L.block(ns - 1, q));
                    C v[R];
#pragma unroll
                    for (int n = 0; n < R; ++n) v[n] = x[n * d];
                    dft_any<R, false>(v);
#pragma unroll
                    for (int j = 0; j < R; ++j) {
                        const int k = q + nq * j;
                        if (odd ? (k < 1 || k > N) : k >= N) continue;
                        put(0, odd ? k - 1 : k, odd ? -v[j].y : v[j].x);
                        put(1, odd ? k - 1 : k, odd ? v[j].x : v[j].y);
                    }
                }
            });
        });
        return;
    }
    if constexpr (OP == MX_T4) {
        with_output([&](auto&& put) {
            mix_radix<CLS, sizeof(T) == 8, false>(R_last, [&](auto rc) {
                constexpr int R = decltype(rc)::v;
                const int d = L.step(1);
                for (int q = L.p; q < nq; q += L.P) {
                    const C* x = L.at(L.block(ns - 1, q));
                    C v[R];
#pragma unroll
                    for (int n = 0; n < R; ++n) v[n] = x[n * d];
                    dft_any<R, false>(v);
#pragma unroll
                    for (int j = 0; j < R; ++j) {
                        const int k = q + nq * j;
                        const C u = cmul(v[j], __ldg(tw4 + 2 * k));
                        put(0, 2 * k, (T)2 * u.x);
                        put(0, N - 1 - 2 * k, odd ? (T)2 * u.y : (T)-2 * u.y);
                    }
                }
            });
        });
        return;
    }
    if constexpr (OP == MX_T3 || OP == MX_FUSED_32) with_input([&](auto&& get) { load3(get); });
    if constexpr (OP == MX_FUSED_R || OP == MX_FUSED_23) {
        mirrored(Yes{}, Yes{}, [&](auto& v, auto& w, int q, bool self, auto rc) {
            constexpr int R = decltype(rc)::v;
            mix_each<R>([&](auto jc) {
                constexpr int j = decltype(jc)::v;
                const int k = q + nq * j;
                C A[2];
                part(v, w, q, jc, rc, A[0], A[1]);
                if constexpr (OP == MX_FUSED_R) {
                    const int kk = 2 * k > M ? M - k : k;
#pragma unroll
                    for (int h = 0; h < 2; ++h) A[h] = cscale(A[h], gval(h, kk));
                } else {
                    const C t = __ldg(tw4 + k);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // (Y_k, -Y_{N-k}) times the Green's values of their places
                        C u = cmul(t, A[h]);
                        u.x *= (T)2 * gval(h, goff + (odd ? N - 1 - k : k));
                        u.y = k > 0 ? u.y * ((T)2 * gval(h, goff + (odd ? k - 1 : N - k))) : zero;
                        A[h] = cmulc(u, t);
                    }
                }
                v[j] = mkc(A[0].x - A[1].y, A[0].y + A[1].x);
                if (!self) w[R - 1 - j] = mkc(A[0].x + A[1].y, A[1].x - A[0].y);
            });
        });
    }
    if constexpr (OP == MX_FUSED_11 || OP == MX_FUSED_44) {
        mix_radix<CLS, sizeof(T) == 8, false>(R_last, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L.step(1);
            for (int q = L.p; q < nq; q += L.P) {
                C* x = L.at(L.block(ns - 1, q));
                C v[R];
#pragma unroll
                for (int n = 0; n < R; ++n) v[n] = x[n * d];
                dft_any<R, false>(v);
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    if constexpr (OP == MX_FUSED_11) {
                        const int kk = 2 * k > M ? M - k : k;
                        if (!odd) {
                            v[j] = mkc(v[j].x * gval(0, goff + kk), v[j].y * gval(1, goff + kk));
                        } else if (kk == 0 || kk == N + 1) {
                            v[j] = mkc(zero, zero);
                        } else {
                            // Z = S_b - i S_a
                            v[j] = mkc(v[j].x * gval(1, goff + kk - 1), v[j].y * gval(0, goff + kk - 1));
                        }
                    } else {
                        C u = cmul(v[j], __ldg(tw4 + 2 * k));
                        u = mkc((T)2 * u.x * gval(0, goff + 2 * k), (T)2 * u.y * gval(0, goff + N - 1 - 2 * k));
                        // conj(t_k) of the second transform, which then runs backwards
                        v[j] = cmulc(odd ? mkc(u.y, -u.x) : u, __ldg(tw8 + k));
                    }
                }
                dft_any<R, true>(v);
#pragma unroll
                for (int n = 0; n < R; ++n) x[n * d] = v[n];
            }
        });
    }

    // ---------------------------------------------------------- back to the line values
    __syncthreads();
    L.inverse_middles();
    if constexpr (OP == MX_FUSED_32) {
        mix_radix<CLS, sizeof(T) == 8, false>(a.pl.st[0].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int nn = a.pl.st[0].nn, d = L.step(a.pl.s1);
            for (int m = L.p; m < nn; m += L.P) {
                C* x = L.at(m);
                const C* tw = L.tw + a.pl.st[0].tw + m;
                C v[R];
                v[0] = x[0];
#pragma unroll
                for (int k = 1; k < R; ++k) v[k] = cmulc(x[k * d], __ldg(tw + (k - 1) * nn));
                dft_any<R, true>(v);
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int t = t_of(m + n * nn) + goff;
                    v[n] = mkc(v[n].x * gval(0, t), v[n].y * gval(1, t));
                }
                dft_any<R, false>(v);
                x[0] = v[0];
#pragma unroll
                for (int k = 1; k < R; ++k) x[k * d] = cmul(v[k], __ldg(tw + (k - 1) * nn));
            }
        });
        __syncthreads();
        L.forward_middles();
        with_output([&](auto&& put) { store2(put); });
        return;
    }
    with_output([&](auto&& put) {
        L.first_inv([&](auto& v, int m, int nn, auto rc) {
            constexpr int R = decltype(rc)::v;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int e = m + n * nn;
                if constexpr (TO3) {
                    const int t = t_of(e);
                    const T s = odd && (t & 1) ? (T)-1 : (T)1;
                    put(0, t, s * v[n].x);
                    put(1, t, s * v[n].y);
                } else if constexpr (OP == MX_FUSED_11) {
                    if (odd ? (e >= 1 && e <= N) : e < N) {
                        put(0, odd ? e - 1 : e, v[n].x);
                        put(1, odd ? e - 1 : e, v[n].y);
                    }
                } else if constexpr (OP == MX_FUSED_44) {
                    const C s = cmulc(v[n], __ldg(tw4 + 2 * e));
                    put(0, 2 * e, (T)2 * s.x);
                    put(0, N - 1 - 2 * e, odd ? (T)-2 * s.y : (T)2 * s.y);
                } else {  // MX_FUSED_R
                    put(0, e, v[n].x);
                    put(1, e, v[n].y);
                    if (e == 0 && a.period >= 0) {
                        put(0, a.period, v[n].x);
                        put(1, a.period, v[n].y);
                    }
                }
            }
        });
    });
}

// ---------------------------------------------------------------- ROT
// The fused pass of a ROT solve: the three components of a line position in
// one CTA, one after the other through the stages, together in the last one,
// where a thread holds the same wave numbers of all three and forms
//   u_g = G (w_{g+2} K_{g+1,g+2} - w_{g+1} K_{g+2,g+1})  (indices mod 3)
// between the two transforms, in FP64 with FP64 symbols whatever the working
// precision (one rounding of the result, as in the general pass; the FP32 pass
// at 200^3 takes 721 us for it, 663 with an FP32 curl, the general pass 4750:
// 13 conversions between the precisions per wave number).  IMAG: every symbol
// is imaginary (no walls), so the factor i is taken out (FP32 772 us without
// that, FP64 1188 against 1315).
// Along the line the symbols change with k; those of the other two directions
// are constants of the thread.
template <typename T, bool ROWS, int CLS, bool IMAG>
__global__ void __launch_bounds__(MixOcc<T, CLS>::threads, MixOcc<T, CLS>::blocks) mix_rot_kernel(const __grid_constant__ MixArgs a) {
    using C = typename CT<T>::C;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int c = ROWS ? threadIdx.y : threadIdx.x;
    const int TX = ROWS ? blockDim.y : blockDim.x;
    const int plane = TX * a.pl.len;  // elements of one component's lines
    const MixLine<T, ROWS, CLS> L0{reinterpret_cast<C*>(smraw) + (ROWS ? c * a.pl.len : c), TX, (int)(ROWS ? threadIdx.x : threadIdx.y),
                              (int)(ROWS ? blockDim.x : blockDim.y), a.pl, reinterpret_cast<const C*>(a.tw)};
    auto line = [&](int g) { return MixLine<T, ROWS, CLS>{L0.sm + g * plane, L0.es, L0.p, L0.P, L0.pl, L0.tw}; };
    const MixPos<false, ROWS> W(a, c, TX, true);
    pass_begin();
    const int ns = a.pl.ns, nq = a.pl.st[ns - 1].Q;
    const int isl = (int)a.in_sl, osl = (int)a.out_sl;
    const C zero = mkc((T)0, (T)0);
    {
        const int n_src = W.ok[0] ? a.n_src : 0;
        for (int g = 0; g < 3; ++g) {
            const C* in = W.template src<C>(a, 0) + g * a.in_sc;
            line(g).first([&](auto& v, int m, int nn, auto rc) {
                constexpr int R = decltype(rc)::v;
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int j = m + n * nn;
                    v[n] = j < n_src ? in[j * isl] : zero;
                }
            });
        }
    }
    __syncthreads();
    for (int s = 1; s + 1 < ns; ++s) {
        for (int g = 0; g < 3; ++g) line(g).middle(s);
        __syncthreads();
    }
    {
        const T* g = W.template green<T>(a, 0);
        const int gl = (int)a.g_sl;
        const double2* K = reinterpret_cast<const double2*>(a.ksym);
        // a table K_{d,c} is real or imaginary throughout (kim): one value of each
        auto symbol = [](const double2* p) {
            const double2 z = __ldg(p);
            return z.x + z.y;
        };
        // K_{d,c}: kc[d][0] for c = d + 1, kc[d][1] for c = d + 2 (mod 3)
        double kc[3][2];
        const double2* kl[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int i = d == a.ax_a ? W.ia[0] : W.ib;
#pragma unroll
            for (int e = 0; e < 2; ++e) kc[d][e] = d == a.ax_l ? 0.0 : symbol(K + (3 * d + (d + 1 + e) % 3) * a.kstr + i);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) kl[e] = K + (3 * a.ax_l + (a.ax_l + 1 + e) % 3) * a.kstr;
        mix_radix<CLS, sizeof(T) == 8, true>(a.pl.st[ns - 1].R, [&](auto rc) {
            constexpr int R = decltype(rc)::v;
            const int d = L0.step(1);
            for (int q = L0.p; q < nq; q += L0.P) {
                C* x = L0.at(L0.block(ns - 1, q));
                C v[3][R];
#pragma unroll
                for (int h = 0; h < 3; ++h) {
#pragma unroll
                    for (int n = 0; n < R; ++n) v[h][n] = x[h * plane + n * d];
                    dft_any<R, false>(v[h]);
                }
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int k = q + nq * j;
                    const double gv = (double)__ldg(g + mix_fold(k, a.f_l) * gl);
                    const double ka = symbol(kl[0] + k), kb = symbol(kl[1] + k);
                    C u[3];
#pragma unroll
                    for (int h = 0; h < 3; ++h) {
                        const int p = (h + 1) % 3, q2 = (h + 2) % 3;
                        const double kp = p == a.ax_l ? ka : kc[p][0];    // K_{h+1, h+2}
                        const double kq = q2 == a.ax_l ? kb : kc[q2][1];  // K_{h+2, h+1}
                        C wq = v[q2][j], wp = v[p][j];
                        if constexpr (!IMAG) {
                            if ((a.kim >> (3 * p + q2)) & 1) wq = cmul_pi(wq);
                            if ((a.kim >> (3 * q2 + p)) & 1) wp = cmul_pi(wp);
                        }
                        double2 r = make_double2((double)wq.x * kp - (double)wp.x * kq, (double)wq.y * kp - (double)wp.y * kq);
                        if constexpr (IMAG) r = cmul_pi(r);
                        u[h] = mkc((T)(r.x * gv), (T)(r.y * gv));
                    }
#pragma unroll
                    for (int h = 0; h < 3; ++h) v[h][j] = u[h];
                }
#pragma unroll
                for (int h = 0; h < 3; ++h) {
                    dft_any<R, true>(v[h]);
#pragma unroll
                    for (int n = 0; n < R; ++n) x[h * plane + n * d] = v[h][n];
                }
            }
        });
    }
    __syncthreads();
    for (int s = ns - 2; s > 0; --s) {
        for (int g = 0; g < 3; ++g) line(g).middle_inv(s);
        __syncthreads();
    }
    const int n_store = W.ok[0] ? (a.n_store < a.pl.M ? a.n_store : a.pl.M) : 0;
    for (int g = 0; g < 3; ++g) {
        C* out = W.template dst<C>(a, 0) + g * a.out_sc;
        line(g).first_inv([&](auto& v, int m, int nn, auto rc) {
            constexpr int R = decltype(rc)::v;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int j = m + n * nn;
                if (j < n_store) out[j * osl] = v[n];
            }
            if (m == 0 && a.period >= 0 && W.ok[0]) out[a.period * osl] = v[0];
        });
    }
}

template <typename T, int OP, bool ROWS, int CLS, typename K>
inline cudaError_t launch_mix_kernel(K kernel, std::atomic<unsigned long long>& attr, const MixArgs& a, int ncomp, cudaStream_t s) {
    if (cudaError_t e = smem_attr_once(attr, kernel, 227 * 1024); e != cudaSuccess) return e;
    const int64_t units = (int64_t)mix_units(a.na, mix_pairs(OP), ROWS) * (ROWS ? a.nb : 1);
    const size_t smem = (size_t)a.tx * a.pl.len * mix_planes(OP) * sizeof(typename CT<T>::C);
    if (a.tx < 1 || a.P < 1 || a.tx * a.P > MixOcc<T, CLS>::threads || smem > 227 * 1024) return cudaErrorInvalidValue;
    const unsigned gx = (unsigned)((units + a.tx - 1) / a.tx);
    return launch_pass(kernel, ROWS ? dim3(gx, 1, ncomp) : dim3(gx, a.nb, ncomp), ROWS ? dim3(a.P, a.tx) : dim3(a.tx, a.P), smem, s, a,
                       a.chain);
}

template <typename T, int OP, bool ROWS, int CLS>
inline cudaError_t launch_mix_t(const MixArgs& a, int ncomp, cudaStream_t s) {
    static std::atomic<unsigned long long> attr{0};
    if constexpr (OP == MX_ROT) {
        static std::atomic<unsigned long long> attr_im{0};
        // the six tables of the curl (d != c) all imaginary: no walls
        if ((a.kim & 0b011101110) == 0b011101110) return launch_mix_kernel<T, OP, ROWS, CLS>(mix_rot_kernel<T, ROWS, CLS, true>, attr_im, a, ncomp, s);
        return launch_mix_kernel<T, OP, ROWS, CLS>(mix_rot_kernel<T, ROWS, CLS, false>, attr, a, ncomp, s);
    } else if constexpr (OP >= MX_T2) {
        return launch_mix_kernel<T, OP, ROWS, CLS>(mix_real_kernel<T, OP, ROWS, CLS>, attr, a, ncomp, s);
    } else {
        return launch_mix_kernel<T, OP, ROWS, CLS>(mix_kernel<T, OP, ROWS, CLS>, attr, a, ncomp, s);
    }
}

template <typename T, int OP, bool ROWS>
cudaError_t launch_mix_op(const MixArgs& a, int ncomp, cudaStream_t s) {
    if constexpr (mix_two(OP, ROWS)) {
        if (a.pl.cls == MIX_TWO) return launch_mix_t<T, OP, ROWS, MIX_TWO>(a, ncomp, s);
    }
    if (a.pl.cls != MIX_MULTI) return cudaErrorInvalidValue;
    return launch_mix_t<T, OP, ROWS, MIX_MULTI>(a, ncomp, s);
}

}  // namespace flb
