// Mixed-radix line passes: factorisation, tiles and dispatch (kernels in
// mix_dft_impl.cuh, one module per operation, precision and direction:
// mix_unit.cu).
#include <algorithm>

#include "mix_dft.h"

namespace flb {

namespace {

// the last stage takes the butterflies of k and M - k, or of three components, together
bool small_last(int op) { return mix_mirrors(op) || op == MX_ROT; }

// search over ordered factorisations: fewest stages first (each one is a
// round trip through shared memory), then the smallest sum of the radices
// (butterfly work), then the order with the larger radices first
struct Search {
    int op, cls;
    bool f64;
    int best[kMixStages], nbest = 0, cost = 1 << 30;
    int cur[kMixStages];
    void go(int m, int n, int sum) {
        if (m == 1) {
            if (n < 2 || (small_last(op) && !mix_radix_ok(cls, f64, true, cur[n - 1]))) return;
            int up = 0;
            for (int i = 1; i < n; ++i) up += cur[i] > cur[i - 1];
            const int c = n * 10000 + sum * 100 + up;
            if (c < cost) {
                cost = c;
                nbest = n;
                std::copy(cur, cur + n, best);
            }
            return;
        }
        if (n == (cls == MIX_TWO ? 2 : kMixStages)) return;
        for (int r = 2; r <= 32; ++r) {
            // (a small last radix need not be one of the others)
            if (m % r != 0 || !(mix_radix_ok(cls, f64, false, r) || (m == r && small_last(op)))) continue;
            cur[n] = r;
            go(m / r, n + 1, sum + r);
        }
    }
};

int host_block(const MixPlan& p, int s, int q) {
    int off = q % p.st[0].R * p.s1, k = q / p.st[0].R;
    for (int i = 1; i < s; ++i) {
        off += k % p.st[i].R * p.st[i].nn;
        k /= p.st[i].R;
    }
    return off;
}

// shared-memory cycles of a row tile's accesses after the first stage: lanes
// along a line, `lanes` of them per cycle when their banks differ
int row_cycles(const MixPlan& p, int lanes) {
    int total = 0;
    for (int s = 1; s < p.ns; ++s) {
        const int nb = p.st[s].nn * p.st[s].Q;
        for (int b0 = 0; b0 < nb; b0 += lanes) {
            int hits[16] = {0}, worst = 0;
            for (int b = b0; b < std::min(nb, b0 + lanes); ++b) {
                const int m = b / p.st[s].Q;
                worst = std::max(worst, ++hits[(host_block(p, s, b - m * p.st[s].Q) + m) % lanes]);
            }
            total += worst * p.st[s].R;
        }
    }
    return total;
}

}  // namespace

bool mix_plan(int M, int op, bool rows, int f64, MixPlan& p) {
    if (M < 4 || M > 16384) return false;
    Search s{op, MIX_MULTI, f64 != 0};
    s.go(M, 0, 0);
    if (s.nbest != 2 && mix_two(op, rows)) {
        Search t{op, MIX_TWO, f64 != 0};
        t.go(M, 0, 0);
        if (t.nbest) s = t;
    }
    if (s.nbest == 0) return false;
    p = MixPlan{};
    p.M = M;
    p.ns = s.nbest;
    p.cls = s.cls;
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
    // columns: an odd distance puts the rows met by a half-warp on distinct
    // banks; rows: the distance of the fewest shared-memory cycles
    p.s1 = p.st[0].nn | 1;
    if (rows) {
        const int lanes = f64 ? 8 : 16;
        int best = 1 << 30, at = p.s1;
        for (int d = 0; d < lanes; ++d) {
            p.s1 = p.st[0].nn + d;
            const int c = row_cycles(p, lanes);
            if (c < best) {
                best = c;
                at = p.s1;
            }
        }
        p.s1 = at;
    }
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

// lines per CTA and threads per line: the tile of the least cost, a product of
//  - butterfly slots offered over those needed, whole warps counted, and a
//    CTA's fixed work,
//  - the column tile's lanes past the last line and its run of x: 128 bytes 1,
//    64 bytes 1.15, 32 bytes 1.35 (400-point fused columns at 200^3, FP32: 156
//    us with 16 columns, 170 with 8; FP64: 302 with 8, 354 with 4),
//  - resident threads: a CTA's warps go round the four schedulers, each with a
//    quarter of the registers, so a fifth warp costs as much as four more (at
//    200^3 FP32, real rows of 400 points: 8 x 16 threads 63 us, 10 x 16 77 us),
//  - row tiles whose lanes straddle two lines in a bank group,
//  - too few CTAs for the 148 SMs.
void mix_tile(MixArgs& a, int f64, int op, bool rows, int64_t ncomp) {
    const size_t line = (size_t)a.pl.len * mix_planes(op) * (f64 ? 16 : 8);
    const int64_t lines = (int64_t)mix_units(a.na, mix_pairs(op), rows) * (rows ? a.nb : 1);
    const int64_t outer = (rows ? 1 : (int64_t)a.nb) * ncomp;
    const int maxth = mix_threads(f64, a.pl.cls);
    int maxp = 1;
    for (int s = 0; s < a.pl.ns; ++s) maxp = std::max(maxp, a.pl.M / a.pl.st[s].R);
    // registers per thread of the kernel, and the resident threads per SM that hide its latencies
    const int regs = a.pl.cls == MIX_TWO ? (f64 ? 168 : 128) : (f64 ? 128 : 80), want = 65536 / regs / 128 * 128;
    double best = 1e30;
    a.tx = 1;
    a.P = std::min(maxp, 32);
    auto consider = [&](int tx, int P) {
        const size_t smem = tx * line;
        if (smem > 227 * 1024) return;
        double need = 0, have = 0;
        for (int s = 0; s < a.pl.ns; ++s) {
            const int nb = a.pl.M / a.pl.st[s].R;
            need += (double)nb * a.pl.st[s].R;
            have += (double)((nb + P - 1) / P) * P * a.pl.st[s].R;
        }
        const int th = P * tx;
        double c = have / need * ((th + 31) / 32 * 32) / th * (1.0 + 10.0 / th + std::max(0, th - 160) * 0.001);
        if (!rows) {
            const int run = tx * (f64 ? 16 : 8);
            c *= run >= 128 ? 1.0 : (run >= 96 ? 1.03 : (run >= 64 ? 1.15 : (run >= 32 ? 1.35 : 1.8)));
        } else if (P % (f64 ? 8 : 16) != 0) {
            c *= 1.12;  // a bank group of lanes straddles two lines
        }
        // a CTA's warps go round the four schedulers, each with a quarter of the registers
        const int quarter = (th + 127) / 128;
        const int ctas_sm = std::min((int)(227 * 1024 / (smem + 1024)), 16384 / (regs * 32 * quarter));
        const int resident = std::max(1, ctas_sm) * th;
        if (resident < want) c *= 1.0 + 0.5 * ((double)want / resident - 1.0);
        const double ctas = (double)((lines + tx - 1) / tx) * outer;
        if (!rows) c *= (double)((lines + tx - 1) / tx) * tx / lines;  // lanes past the last column
        if (ctas < 148) c *= 1.3 * 148 / ctas;
        else if (ctas < 296) c *= 1.0 + 0.3 * (296 - ctas) / 148;
        if (c < best) {
            best = c;
            a.tx = tx;
            a.P = P;
        }
    };
    if (rows) {
        for (int P = std::min(16, maxp); P <= std::min(maxp, maxth); ++P)
            for (int tx = std::max(1, maxth / P); tx >= 1; --tx) consider(tx, P);
        return;
    }
    for (int run : {16, 12, 8, 6, 4, 2, 1}) {
        const int tx = f64 ? (run == 1 ? 0 : run / 2) : run;
        if (tx == 0) continue;
        for (int P = 1; P <= std::min(maxp, maxth / tx); ++P) consider(tx, P);
    }
}

bool mix_fits(const MixPlan& p, int op, int f64) { return (size_t)p.len * mix_planes(op) * (f64 ? 16 : 8) <= 227 * 1024; }

template <int OP>
static cudaError_t launch_op(int f64, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    if (f64) return rows ? launch_mix_op<double, OP, true>(a, ncomp, s) : launch_mix_op<double, OP, false>(a, ncomp, s);
    return rows ? launch_mix_op<float, OP, true>(a, ncomp, s) : launch_mix_op<float, OP, false>(a, ncomp, s);
}

cudaError_t launch_mix(int f64, int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    switch (op) {
        case MX_C2C_F: return launch_op<MX_C2C_F>(f64, rows, a, ncomp, s);
        case MX_C2C_I: return launch_op<MX_C2C_I>(f64, rows, a, ncomp, s);
        case MX_R2C: return launch_op<MX_R2C>(f64, rows, a, ncomp, s);
        case MX_C2R: return launch_op<MX_C2R>(f64, rows, a, ncomp, s);
        case MX_FUSED: return launch_op<MX_FUSED>(f64, rows, a, ncomp, s);
        case MX_T2: return launch_op<MX_T2>(f64, rows, a, ncomp, s);
        case MX_T3: return launch_op<MX_T3>(f64, rows, a, ncomp, s);
        case MX_T1: return launch_op<MX_T1>(f64, rows, a, ncomp, s);
        case MX_T4: return launch_op<MX_T4>(f64, rows, a, ncomp, s);
        case MX_FUSED_R: return launch_op<MX_FUSED_R>(f64, rows, a, ncomp, s);
        case MX_FUSED_23: return launch_op<MX_FUSED_23>(f64, rows, a, ncomp, s);
        case MX_FUSED_32: return launch_op<MX_FUSED_32>(f64, rows, a, ncomp, s);
        case MX_FUSED_11: return launch_op<MX_FUSED_11>(f64, rows, a, ncomp, s);
        case MX_FUSED_44: return launch_op<MX_FUSED_44>(f64, rows, a, ncomp, s);
        // one launch per field: the three components of a line position are the CTA's
        case MX_ROT: return ncomp == 3 ? launch_op<MX_ROT>(f64, rows, a, 1, s) : cudaErrorInvalidValue;
    }
    return cudaErrorInvalidValue;
}

}  // namespace flb
