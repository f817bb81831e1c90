// Mixed-radix line passes for the transform lengths the register DFTs do not
// take: arguments, factorisation and launcher (kernels in mix_dft_impl.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace flb {

// What one pass does with its lines.  "Pairs" carry two real lines a, b in one
// complex transform z = a + i b and part them at the frequency side.
enum MixOp : int {
    MX_C2C_F = 0,  // forward complex DFT
    MX_C2C_I = 1,  // inverse complex DFT
    MX_R2C = 2,    // pairs of real lines -> half spectra
    MX_C2R = 3,    // half spectra -> pairs of real lines
    MX_FUSED = 4,  // forward complex DFT, Green's multiply, inverse DFT, in place
    // r2r kinds (FFTW size N); pairs but for type 4
    MX_T2 = 5,     // DCT-II / DST-II, M = N
    MX_T3 = 6,     // DCT-III / DST-III, M = N
    MX_T1 = 7,     // DCT-I (M = 2 (N - 1)) / DST-I (M = 2 (N + 1))
    MX_T4 = 8,     // DCT-IV / DST-IV of even N, M = N / 2
    // a real last direction: transform, Green's multiply, inverse transform, in place
    MX_FUSED_R = 9,    // r2c, c2r
    MX_FUSED_23 = 10,  // type II, type III
    MX_FUSED_32 = 11,  // type III, type II
    MX_FUSED_11 = 12,  // type I twice
    MX_FUSED_44 = 13,  // type IV twice
    MX_ROT = 14,       // forward complex DFT of three components, curl and Green's multiply, inverse DFT, in place
};
// two real lines per complex transform
constexpr bool mix_pairs(int op) { return op == MX_R2C || op == MX_C2R || (op >= MX_T2 && op <= MX_FUSED_11 && op != MX_T4); }
// lines of a tile's line position held together
constexpr int mix_planes(int op) { return op == MX_ROT ? 3 : 1; }
// the last stage takes the butterflies of k and M - k together
constexpr bool mix_mirrors(int op) {
    return op == MX_R2C || op == MX_C2R || op == MX_T2 || op == MX_T3 || op == MX_FUSED_R || op == MX_FUSED_23 || op == MX_FUSED_32;
}

// lines or pairs of lines among na neighbouring positions (MixPos pairs them)
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int mix_units(int na, bool pair, bool rows) {
    if (!pair) return na;
    return rows ? (na + 1) / 2 : 8 * (na / 16) + (na % 16 < 8 ? na % 16 : 8);
}

constexpr int kMixStages = 4;
// kernel classes: two to four stages of smaller radices, or two of larger ones
enum MixClass : int { MIX_MULTI = 0, MIX_TWO = 1 };
constexpr int mix_threads(int f64, int cls) { return cls == MIX_TWO && f64 ? 128 : 256; }
// the operations compiled in class TWO: column passes of the complex kinds and
// r2c / c2r.  Row passes lose by it (288-point real rows of a 145 x 121 x 101
// grid, FP32, 20 us in three stages, 26 in two: few threads share a line there),
// and so do the r2r and fused real ones, whose last stage holds two butterflies
// and their twiddles (180-point fused z of a 250 x 150 x 180 box, FP64, 60 ->
// 92 us).
constexpr bool mix_two(int op, bool rows) { return !rows && op <= MX_FUSED; }
// radices of a class.  small: of a last stage that takes two or three
// butterflies in one thread.  The limits are those that keep the butterflies
// in the class's registers.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr bool mix_radix_ok(int cls, bool f64, bool small, int r) {
    if (cls == MIX_TWO) {
        if (small) return r >= 4 && r <= (f64 ? 10 : 12);
        return (r >= 8 && r <= 16) || r == 18 || r == 20 || (!f64 && (r == 24 || r == 25 || r == 32));
    }
    if (small) return (r >= 2 && r <= 8) || r == 11 || r == 13;
    return r >= 2 && r != 14 && r <= (f64 ? 13 : 16);
}

// Stage s of the decimation in frequency: radix R on sub-blocks of R * nn
// points (nn points are left of each after it); Q = product of the radices
// before it, so a line has Q * nn butterflies.
struct MixStage {
    int R, nn, Q;
    unsigned qmul;  // ceil(2^32 / Q): x / Q = umulhi(x, qmul) for x Q < 2^32 (Q = 1: not used)
    int tw;         // first entry of the stage's twiddles W_{R nn}^{k m} at (k - 1) nn + m, 0 < k < R, m < nn
};

struct MixPlan {
    int M, ns, cls;         // line length, number of stages, kernel class
    int s1;                 // distance in shared memory between the first digit's blocks
    int len;                // elements a line takes in shared memory
    int ntw;                // complex entries of the stage twiddles
    MixStage st[kMixStages];
};

struct MixArgs {
    int chain;                             // launched behind the solve's previous pass (launch_pass)
    const void* in;
    void* out;
    MixPlan pl;
    const void* tw;                        // stage twiddles, working precision
    int na, nb;                            // line positions: a (lanes of the column passes), b
    int n_src, n_store;                    // source / stored extent of a line
    int64_t in_sl, in_sa, in_sb, in_sc;    // element strides: along the line, a, b, component
    int64_t out_sl, out_sa, out_sb, out_sc;
    int in64, out64;                       // a real side holds doubles
    int period;                            // output index that receives a copy of output 0, or -1
    // r2r kinds: pre / post twiddles W_4N^k (type IV: W_8N^{4j+1} in tw8), the place of the source in the padded
    // line and of the stored part in the output line, and per component: FFTW's size, the odd (DST) kind, first
    // input and output element of the transform in its line, first spectral element of a fused pass, output
    // elements (of the stored part) set to zero, or -1
    const void *tw4, *tw8;
    int fieldstart, store_off, lda;
    int N[3], dst[3], fi[3], fo[3], go[3], z0[3], z1[3];
    int tx, P;                             // tile: lines per CTA (pairs count once), threads per line
    // Green's multiply
    const void* green;
    int64_t g_sa, g_sb, g_sl;
    int f_a, f_b, f_l;                     // fold lengths (0 = none)
    // FP64 curl symbols K_{d,c}(i) at (3 d + c) kstr + i, imaginary where bit 3 d + c of kim is set, else real;
    // the directions of a, b and the line
    const void* ksym;
    int kstr, kim, ax_a, ax_b, ax_l;
};

// Factorisation of M for a pass of operation `op`; false when M has a prime
// factor above 13, or does not split into two to four of the radices.
bool mix_plan(int M, int op, bool rows, int f64, MixPlan& p);
// W_{R nn}^{k m} of entry e of the stage twiddles: exponent and root order
void mix_twiddle_exponent(const MixPlan& p, int e, int* q, int* n);
// lines per CTA and threads per line (a.tx, a.P) for the pass's extents
void mix_tile(MixArgs& a, int f64, int op, bool rows, int64_t ncomp);
// rows: lines along the lanes' direction (x); ncomp: grid z
cudaError_t launch_mix(int f64, int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s);
// one operation in one precision and direction (mix_unit.cu)
template <typename T, int OP, bool ROWS> cudaError_t launch_mix_op(const MixArgs& a, int ncomp, cudaStream_t s);
// whether one line position of the pass fits in shared memory
bool mix_fits(const MixPlan& p, int op, int f64);

}  // namespace flb
