// Mixed-radix line passes: factorisation, tiles and dispatch (kernels in
// mix_dft_impl.cuh, instantiated in mix_*.cu so that the units compile in
// parallel).
#include <algorithm>

#include "mix_dft_impl.cuh"

namespace flb {

namespace {

constexpr int kRadices[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16};

// radices of a last stage that takes two or three butterflies in one thread
bool small_radix(int r) { return r <= 8 || r == 11 || r == 13; }

// search over ordered factorisations: fewest stages first (each one is a
// round trip through shared memory), then the smallest sum of the radices
// (butterfly work), then the larger radix first
struct Search {
    int op, f64;
    int best[kMixStages], nbest = 0, cost = 1 << 30;
    int cur[kMixStages];
    void go(int m, int n, int sum) {
        if (m == 1) {
            if (n < 2) return;
            if ((mix_mirrors(op) || op == MX_ROT) && !small_radix(cur[n - 1])) return;
            int up = 0;  // steps up: the order with the larger radices first wins
            for (int i = 1; i < n; ++i) up += cur[i] > cur[i - 1];
            const int c = n * 10000 + sum * 100 + up;
            if (c < cost) {
                cost = c;
                nbest = n;
                std::copy(cur, cur + n, best);
            }
            return;
        }
        if (n == kMixStages) return;
        for (int r : kRadices) {
            if (m % r != 0 || r > max_radix()) continue;
            cur[n] = r;
            go(m / r, n + 1, sum + r);
        }
    }
    // FP64 butterflies of 15 and 16 values do not fit the 128 registers of two CTAs per SM
    int max_radix() const { return f64 ? 13 : 16; }
};

}  // namespace

bool mix_plan(int M, int op, int f64, MixPlan& p) {
    if (M < 4 || M > 16384) return false;
    Search s{op, f64};
    s.go(M, 0, 0);
    if (s.nbest == 0) return false;
    p = MixPlan{};
    p.M = M;
    p.ns = s.nbest;
    int Q = 1, left = M;
    for (int i = 0; i < s.nbest; ++i) {
        MixStage& st = p.st[i];
        st.R = s.best[i];
        st.Q = Q;
        st.qmul = Q > 1 ? (unsigned)((0x100000000ull + Q - 1) / Q) : 0;
        left /= st.R;
        st.nn = left;
        st.tw = p.ntw;
        if (i + 1 < s.nbest) p.ntw += (st.R - 1) * left;
        Q *= st.R;
    }
    p.s1 = p.st[0].nn | 1;
    p.len = p.st[0].R * p.s1;
    return true;
}

void mix_twiddle_exponent(const MixPlan& p, int e, int* q, int* n) {
    int s = 0;
    while (s + 2 < p.ns && e >= p.st[s + 1].tw) ++s;
    const MixStage& st = p.st[s];
    const int w = e - st.tw, k = w / st.nn + 1, m = w % st.nn;
    *q = k * m;
    *n = st.R * st.nn;
}

// lines per CTA and threads per line.  Shared memory for three resident CTAs
// where the line allows it, 256 threads at most; the number of threads per line
// wastes the fewest butterfly slots over the stages.
void mix_tile(MixArgs& a, int f64, int op, bool rows, int64_t ncomp) {
    const bool pair = mix_pairs(op);
    const size_t line = (size_t)a.pl.len * mix_planes(op) * (f64 ? 16 : 8);
    const int64_t lines = (int64_t)mix_units(a.na, pair, rows) * (rows ? a.nb : 1);
    const int64_t outer = (rows ? 1 : (int64_t)a.nb) * ncomp;
    const size_t target = 72 * 1024;
    int maxp = 1, minnb = 1 << 30;
    for (int s = 0; s < a.pl.ns; ++s) {
        const int nb = a.pl.M / a.pl.st[s].R;
        maxp = std::max(maxp, nb);
        minnb = std::min(minnb, nb);
    }
    auto waste = [&](int P, int tx) {
        // butterfly slots offered over those needed
        double need = 0, have = 0;
        for (int s = 0; s < a.pl.ns; ++s) {
            const int nb = a.pl.M / a.pl.st[s].R;
            need += nb * (double)a.pl.st[s].R;
            have += (double)((nb + P - 1) / P) * P * a.pl.st[s].R;
        }
        const int th = P * tx, up = (th + 31) / 32 * 32;
        return have / need * up / th;
    };
    a.tx = 1;
    a.P = std::min(maxp, 32);
    double cost = 1e30;
    auto consider = [&](int tx, int P) {
        const double c = waste(P, tx) * (1.0 + 24.0 / (P * tx));
        if (c < cost) {
            cost = c;
            a.tx = tx;
            a.P = P;
        }
    };
    if (rows) {
        for (int P = std::min(16, maxp); P <= std::min(maxp, kMixThreads); ++P) {
            for (int tx = std::max(1, kMixThreads / P); tx >= 1; --tx) {
                if (tx > 1 && (size_t)tx * line > target) continue;
                if (tx > 1 && (lines + tx - 1) / tx * outer < 296) continue;  // two CTAs per SM before larger tiles
                consider(tx, P);
            }
        }
        return;
    }
    int tx = f64 ? 4 : 8;
    while (tx > 2 && ((size_t)tx * line > target || (lines + tx - 1) / tx * outer < 296)) tx /= 2;
    if ((size_t)tx * line > 227 * 1024) tx = 1;
    for (int P = std::max(1, std::min(maxp, 32 / tx)); P <= std::min(maxp, kMixThreads / tx); ++P) {
        consider(tx, P);
    }
}

bool mix_fits(const MixPlan& p, int op, int f64) { return (size_t)p.len * mix_planes(op) * (f64 ? 16 : 8) <= 227 * 1024; }

cudaError_t launch_mix(int f64, int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    switch (op) {
        case MX_C2C_F:
        case MX_C2C_I: return f64 ? launch_mix_c2c_f64(op, rows, a, ncomp, s) : launch_mix_c2c_f32(op, rows, a, ncomp, s);
        case MX_R2C:
        case MX_C2R: return f64 ? launch_mix_real_f64(op, rows, a, ncomp, s) : launch_mix_real_f32(op, rows, a, ncomp, s);
        case MX_T1:
        case MX_T2:
        case MX_T3:
        case MX_T4: return f64 ? launch_mix_r2r_f64(op, rows, a, ncomp, s) : launch_mix_r2r_f32(op, rows, a, ncomp, s);
        case MX_FUSED_R:
        case MX_FUSED_23:
        case MX_FUSED_32:
        case MX_FUSED_11:
        case MX_FUSED_44:
            return f64 ? launch_mix_fused_real_f64(op, rows, a, ncomp, s) : launch_mix_fused_real_f32(op, rows, a, ncomp, s);
        case MX_ROT: return launch_mix_rot(f64, rows, a, ncomp, s);
        case MX_FUSED: return launch_mix_fused(f64, rows, a, ncomp, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace flb
