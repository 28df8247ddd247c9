// The general scan under a soft address with its token chain reduced to scalars.
//
// Within a chunk of C tokens every score is a linear recurrence of dot products that are known at its start: with
// u_n(j) = <K_n, q_j>, e_n(j) = <K_n, k_j> and s_n = |K_n|^2 of the row as it stands, a write of token t with weight w does
//     u_n(j) += w (<k_t, q_j> - u_n(j)),  e_n(j) += w (<k_t, k_j> - e_n(j)),
//     s_n     = (1-w)^2 s_n + 2 w (1-w) e_n(t) + w^2 |k_t|^2,
// so a token costs a thread per row a handful of operations, one sum over the rows and one barrier; the rows themselves are
// touched once per chunk.  [the recurrence: gqa25/slotkern_kv.py:84-120]
// Scores, softmax, occupancies and these recurrences run in double, the rows are float32: every rounding error of a score
// comes back in every row at every later token.
// Warp roles: row warps (a thread per row: dots, chain, row update) and helper warps (the next chunk's tokens and their
// C x C products, the key snapshots, the values one chunk behind).
// Bound: the chain -- exp, a sum over 32 lanes, a barrier, a reciprocal, a reciprocal square root per token, all in double.
#pragma once
#include "slotscan_common.cuh"

namespace slotscan {

constexpr int DC_HELP = 256;                 // helper threads
constexpr int DC_NMAX = 256;                 // rows

__host__ __device__ inline int dc_kpad(int DK) { return (DK + 3) & ~3; }
// bytes of one token buffer: q and k in double (row stride kp + 2), k in float, two C x C products, 1/|q|, gate, fr
__host__ __device__ inline size_t dc_tok_bytes(int C, int DK) {
    const int kp = dc_kpad(DK);
    return 8 * ((size_t)2 * C * (kp + 2) + 2 * C * C + C) + 4 * ((size_t)C * kp + 2 * C);
}
__host__ __device__ inline size_t dc_smem(int C, int N, int DK, int DV, bool values) {
    const int kp = dc_kpad(DK);
    const size_t n4 = (N + 3) & ~3;
    return 2 * dc_tok_bytes(C, DK) + 8 * 128 + 8 * (size_t)2 * C * 8 + 4 * ((size_t)N * (kp + 4) + (values ? n4 * DV : 0) + 2 * C * n4 + 16);
}

__device__ __forceinline__ void dc_bar_rows(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }
__device__ __forceinline__ void dc_bar_help() { asm volatile("bar.sync 2, %0;" ::"n"(DC_HELP) : "memory"); }
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
    return v;
}

// N rows of DK floats into rows of stride kpad + 4 (the padding zero), 16 bytes at a time and several in flight where the
// rows allow it
__device__ __forceinline__ void dense_load_rows(float* K, const float* src, int N, int DK, int tid, int nt) {
    const int kp = dc_kpad(DK), KS = kp + 4;
    if (DK % 4 == 0 && (reinterpret_cast<size_t>(src) & 15) == 0) {
        const int q = DK / 4, n = N * q;
#pragma unroll 8
        for (int i = tid; i < n; i += nt) { const int r = i / q, c = (i - r * q) * 4; st4(K + r * KS + c, __ldg(reinterpret_cast<const float4*>(src) + i)); }
        for (int r = tid; r < N; r += nt) st4(K + r * KS + kp, make_float4(0.f, 0.f, 0.f, 0.f));
    } else {
        for (int i = tid; i < N * KS; i += nt) { const int r = i / KS, d = i % KS; K[i] = d < DK ? src[(size_t)r * DK + d] : 0.f; }
    }
}

struct DenseChainArgs {
    slotscan_params p;
    const void *k, *q, *v;
    const float *gate, *fr, *temp;
    // forward: snapshots, log and final state out.  tables: kbuf / obuf in
    float *kbuf, *vbuf, *obuf;
    int* addr;
    float *kfin, *vfin, *ofin;
    // tables of the backward, [nbh][T][N] each, and lim [nbh][NB]: last candidate row at the block's first token
    float *as, *sf, *ki, *ot;
    int* lim;
    int bh0;
};

// TABLES = false: the whole scan of one sequence.  TABLES = true: one block of G tokens from its emitted snapshot, writing
// softmax address, score, 1/|K_n| and occupancy of every token and row for the backward.
template <typename Tin, int C, bool TABLES>
__global__ void __launch_bounds__(DC_NMAX + DC_HELP) dense_chain_kernel(const DenseChainArgs A) {
    extern __shared__ __align__(16) char dc_sm[];
    const slotscan_params& p = A.p;
    const int N = p.N, T = p.T, H = p.H, DK = p.DK, DV = p.DV, G = p.G, NB = (T + G - 1) / G;
    const int kp = dc_kpad(DK), KS = kp + 4, QS = kp + 2, N4 = (N + 3) & ~3;
    const size_t tokb = dc_tok_bytes(C, DK);
    double* ex = reinterpret_cast<double*>(dc_sm + 2 * tokb);        // [2][64] exchange of the row warps
    int2* s_arg = reinterpret_cast<int2*>(ex + 128);                 // [2][C][8] a row warp's largest address (float bits) and its row
    float* K = reinterpret_cast<float*>(s_arg + 2 * C * 8);          // [N][KS]
    float* wbuf = K + (size_t)N * KS;                                // [2][C][N4]
    float* V = wbuf + 2 * C * N4;                                    // [N4][DV] (forward)
    auto tq = [&](int b) { return reinterpret_cast<double*>(dc_sm + b * tokb); };            // [C][QS] q
    auto tk = [&](int b) { return tq(b) + C * QS; };                                         // [C][QS] k
    auto tB = [&](int b) { return tk(b) + C * QS; };                                         // [C][C] <k_t, q_j>
    auto tC = [&](int b) { return tB(b) + C * C; };                                          // [C][C] <k_t, k_j>
    auto tqi = [&](int b) { return tC(b) + C * C; };                                         // [C] 1 / max(|q|, 1e-6)
    auto tkf = [&](int b) { return reinterpret_cast<float*>(tqi(b) + C); };                  // [C][kp] k
    auto tg = [&](int b) { return tkf(b) + C * kp; };                                        // [C] gate
    auto tf = [&](int b) { return tg(b) + C; };                                              // [C] fr

    const int lb = TABLES ? (int)blockIdx.x / NB : (int)blockIdx.x, jb0 = TABLES ? (int)blockIdx.x % NB : 0;
    const int jb1 = TABLES ? jb0 + 1 : NB;
    const int bh = A.bh0 + lb, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, NT = blockDim.x, rows_t = NT - DC_HELP, warp = tid >> 5, RW = rows_t >> 5;
    const bool row = tid < rows_t;
    const int n = tid, ht = tid - rows_t;
    const bool live = row && n < N;
    const float eps = p.eps, tempf = A.temp[0];
    const double temp = (double)tempf;
    const Tin* kg = static_cast<const Tin*>(A.k);
    const Tin* qg = static_cast<const Tin*>(A.q);
    const Tin* vg = static_cast<const Tin*>(A.v);
    auto snap = [&](int jb) { return ((size_t)b * NB + jb) * H + h; };

    // helper: tokens [t0, t0 + cn) of the chunk into buffer bf, then their products
    auto prep = [&](int bf, int t0, int cn) {
        double *Q = tq(bf), *Kd = tk(bf);
        float* Kf = tkf(bf);
        for (int i = ht; i < C * kp; i += DC_HELP) {
            const int j = i / kp, d = i % kp;
            const bool in = j < cn && d < DK;
            const size_t at = (((size_t)b * T + t0 + j) * H + h) * DK + d;
            const float qv = in ? ld1(qg + at) : 0.f, kv = in ? ld1(kg + at) : 0.f;
            Q[j * QS + d] = (double)qv;
            Kd[j * QS + d] = (double)kv;
            Kf[j * kp + d] = kv;
        }
        if (ht < C) {
            const size_t ix = ((size_t)b * T + t0 + ht) * H + h;
            tg(bf)[ht] = ht < cn ? gate_eff(A.gate[ix], p.hard_gate) : 0.f;
            tf(bf)[ht] = ht < cn ? (p.fr_per_token ? A.fr[ix] : A.fr[0]) : 0.f;
        }
        dc_bar_help();
        if (ht < 2 * C * C + C) {
            const int m = ht < C * C ? 0 : (ht < 2 * C * C ? 1 : 2);
            const int e = ht - m * C * C, t = m == 2 ? e : e / C, j = m == 2 ? e : e % C;
            const double* x = (m == 2 ? Q : Kd) + t * QS;
            const double* y = (m == 1 ? Kd : Q) + j * QS;
            double s0 = 0.0, s1 = 0.0;
            for (int d = 0; d < kp; d += 2) {
                const double2 a = *reinterpret_cast<const double2*>(x + d), c = *reinterpret_cast<const double2*>(y + d);
                s0 = fma(a.x, c.x, s0);
                s1 = fma(a.y, c.y, s1);
            }
            const double s = s0 + s1;
            if (m == 0) tB(bf)[e] = s;
            else if (m == 1) tC(bf)[e] = s;
            else tqi(bf)[t] = 1.0 / fmax(sqrt(s), 1e-6);
        }
    };
    // helper: a thread keeps its column (DV <= 128 of 256 threads; `hper` threads share one), so that a token's value is loaded
    // once for all its rows, a chunk ahead; 4 rows at a time, two to an instruction
    const int hper = DC_HELP / DV, hd = row ? 0 : ht % DV, hg = row ? 0 : ht / DV;
    float xn[C];
    auto fetch_v = [&](int t0, int cn) {
#pragma unroll
        for (int j = 0; j < C; j++) xn[j] = j < cn ? ld1(vg + (((size_t)b * T + t0 + j) * H + h) * DV + hd) : 0.f;
    };
    // the values of a chunk whose tokens fetch_v has loaded, first token at place ph of block jb; and its addresses
    auto values = [&](int bf, int t0, int cn, int ph, int jb) {
        const float* wr = wbuf + bf * C * N4;
        if (A.addr != nullptr && ht < cn) {
            int2 m = s_arg[(bf * C + ht) * 8];
            for (int w = 1; w < RW; w++) { const int2 x = s_arg[(bf * C + ht) * 8 + w]; if ((unsigned)x.x > (unsigned)m.x) m = x; }
            A.addr[((size_t)b * T + t0 + ht) * H + h] = m.y;
        }
        if (hg >= hper) return;
        bool odd = false;                                    // a row a token does not write must not see it: only an infinite
#pragma unroll
        for (int j = 0; j < C; j++) odd |= !(fabsf(xn[j]) <= 3e38f);     // or NaN value would tell
        const f32x2 one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
        for (int n0 = hg * 4; n0 < N4; n0 += hper * 4) {
            float s[4];
#pragma unroll
            for (int i = 0; i < 4; i++) s[i] = V[(n0 + i) * DV + hd];
            if (ph == 0) {
                float* out = A.vbuf + (snap(jb) * N + n0) * DV + hd;
#pragma unroll
                for (int i = 0; i < 4; i++) if (n0 + i < N) out[(size_t)i * DV] = s[i];
            }
            if (!odd) {
                f32x2 s0 = pack2(s[0], s[1]), s1 = pack2(s[2], s[3]);
#pragma unroll
                for (int j = 0; j < C; j++) {                        // tokens past cn: weight 0
                    const f32x4 w = ld4x2(wr + j * N4 + n0);
                    const f32x2 x = pack2(xn[j], xn[j]);
                    s0 = fma2(w.a, x, mul2(fma2(w.a, minus, one), s0));
                    s1 = fma2(w.b, x, mul2(fma2(w.b, minus, one), s1));
                }
                const float2 p0 = unpack2(s0), p1 = unpack2(s1);
                s[0] = p0.x; s[1] = p0.y; s[2] = p1.x; s[3] = p1.y;
            } else {
#pragma unroll
                for (int j = 0; j < C; j++) {
                    const float4 w = ld4(wr + j * N4 + n0);
                    const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) s[i] = wv[i] != 0.f ? (1.f - wv[i]) * s[i] + wv[i] * xn[j] : s[i];
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) V[(n0 + i) * DV + hd] = s[i];
        }
    };

    // ---- initial state ----
    double o = 0.0;
    int fe = 0;                                              // first empty row; candidates: rows 0 .. min(fe, N - 1)
    if (TABLES) dense_load_rows(K, A.kbuf + snap(jb0) * N * DK, N, DK, tid, NT);
    else for (int i = tid; i < N * KS; i += NT) K[i] = 0.f;
    for (int i = tid; i < 2 * C * N4; i += NT) wbuf[i] = 0.f;
    if (!TABLES) for (int i = tid; i < N4 * DV; i += NT) V[i] = 0.f;
    if (TABLES && live) o = (double)A.obuf[snap(jb0) * N + n];
    if (!row) prep(0, jb0 * G, min(C, min(G, T - jb0 * G)));
    if (TABLES && row) {
        int* s_fe = reinterpret_cast<int*>(ex);
        const unsigned free_rows = __ballot_sync(FULL, !live || (float)o < eps);
        const unsigned unbounded = __ballot_sync(FULL, live && !(o >= 0.0 && o <= 1.0));
        if (lane == 0) { s_fe[warp] = free_rows ? warp * 32 + __ffs(free_rows) - 1 : BIGI; s_fe[8 + warp] = unbounded != 0u; }
    }
    bool wild = false;               // a gate outside [0, 1] so far (tables: one that shows in the block's occupancies, or later)
    __syncthreads();
    if (TABLES && row) {
        const int* s_fe = reinterpret_cast<const int*>(ex);
        fe = BIGI;
        for (int w = 0; w < RW; w++) { fe = min(fe, s_fe[w]); wild |= s_fe[8 + w] != 0; }
        fe = min(fe, N);
        if (tid == 0) A.lim[(size_t)lb * NB + jb0] = min(fe, N - 1);
    }
    __syncthreads();                                         // the exchange slots are used again below
    for (int i = tid; row && i < 128; i += rows_t) ex[i] = 0.0;     // row warps that are not there: no weight, no key
    if (row) dc_bar_rows(rows_t);
    if (!TABLES && !row) fetch_v(0, min(C, min(G, T)));

    int par = 0, c = 0, pt0 = 0, pcn = 0, pph = 0, pjb = 0;  // parity of the exchange, chunk, the chunk before
    for (int jb = jb0; jb < jb1; jb++) {
        const int tb = jb * G, bn = min(G, T - tb);
        for (int s0 = 0; s0 < bn; s0 += C, c++) {
            const int t0 = tb + s0, cn = min(C, bn - s0), bf = c & 1;
            float* wr = wbuf + bf * C * N4;
            float w[C];
            if (row) {
                if (!TABLES && s0 == 0 && live) A.obuf[snap(jb) * N + n] = (float)o;
                double u[C], e[C], ns = 0.0;
#pragma unroll
                for (int j = 0; j < C; j++) { u[j] = 0.0; e[j] = 0.0; w[j] = 0.f; }
                if (warp * 32 <= fe && live) {               // rows above the first empty one are zero
                    const double *Q = tq(bf), *Kd = tk(bf);
                    for (int d = 0; d < kp; d += 4) {
                        const float4 x4 = ld4(K + n * KS + d);
                        const double x[4] = {(double)x4.x, (double)x4.y, (double)x4.z, (double)x4.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) ns = fma(x[i], x[i], ns);
#pragma unroll
                        for (int j = 0; j < C; j++) {
                            const double2 q0 = *reinterpret_cast<const double2*>(Q + j * QS + d), q1 = *reinterpret_cast<const double2*>(Q + j * QS + d + 2);
                            const double2 k0 = *reinterpret_cast<const double2*>(Kd + j * QS + d), k1 = *reinterpret_cast<const double2*>(Kd + j * QS + d + 2);
                            u[j] = fma(x[0], q0.x, u[j]);
                            e[j] = fma(x[0], k0.x, e[j]);
                            u[j] = fma(x[1], q0.y, u[j]);
                            e[j] = fma(x[1], k0.y, e[j]);
                            u[j] = fma(x[2], q1.x, u[j]);
                            e[j] = fma(x[2], k1.x, e[j]);
                            u[j] = fma(x[3], q1.y, u[j]);
                            e[j] = fma(x[3], k1.y, e[j]);
                        }
                    }
                }
                const double *Bm = tB(bf), *Cm = tC(bf), *qi = tqi(bf);
#pragma unroll
                for (int j = 0; j < C; j++) {
                    if (j < cn) {                            // uniform
                        const float g = tg(bf)[j], frf = tf(bf)[j];
                        const double fr = (double)frf;
                        wild |= !(g >= 0.f && g <= 1.f);
                        const bool cand = live && n <= fe;
                        const double kinv = ns <= 1e-12 ? 1e6 : rsqrt(ns);     // NaN stays NaN
                        const double s = (u[j] * kinv * qi[j]) * temp;
                        const double z = s - fr * (p.occ_bin ? (o >= (double)eps ? 1.0 : 0.0) : o);
                        double* xs = ex + par * 64;          // [0..7] sums, [8..15] maxima, [16] e, [17] o of row fe
                        par ^= 1;
                        // the softmax's shift: a bound of every z where that cannot under- or overflow, the maximum else
                        // (after a wild gate the occupancies are not bounded by 1)
                        double shift = fabs(temp) + fmax(0.0, -fr);
                        const bool bounded = 2.0 * fabs(temp) + fabs(fr) < 600.0 && (p.occ_bin || !wild);
                        if (!bounded) {
                            double m = cand ? z : -INFINITY;
#pragma unroll
                            for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(FULL, m, off));
                            if (lane == 0) xs[8 + warp] = m;
                            dc_bar_rows(rows_t);
                            shift = xs[8];
                            for (int i = 1; i < RW; i++) shift = fmax(shift, xs[8 + i]);
                        }
                        const double E = cand ? exp(z - shift) : 0.0;
                        double sw = E;
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1) sw += __shfl_xor_sync(FULL, sw, off);
                        if (lane == 0) xs[warp] = sw;
                        if (n == fe && live) { xs[16] = E; xs[17] = o; }
                        dc_bar_rows(rows_t);
                        const double2 e0 = *reinterpret_cast<const double2*>(xs), e1 = *reinterpret_cast<const double2*>(xs + 2);
                        const double2 e2 = *reinterpret_cast<const double2*>(xs + 4), e3 = *reinterpret_cast<const double2*>(xs + 6);
                        const double se = ((e0.x + e0.y) + (e1.x + e1.y)) + ((e2.x + e2.y) + (e3.x + e3.y));
                        const double si = bounded ? rcp_normal(se) : 1.0 / se;
                        const float a = cand ? (float)(E * si) : 0.f;        // also where the sum is not finite
                        if (TABLES) {
                            if (live) {
                                const size_t at = ((size_t)lb * T + t0 + j) * N + n;
                                A.as[at] = a;
                                A.sf[at] = cand ? (float)s : 0.f;
                                A.ki[at] = (float)kinv;
                                A.ot[at] = (float)o;
                            }
                        }
                        const double wd0 = (double)g * (double)a;
                        if (fe < N) {                        // only the first empty row can become occupied
                            const float af = (float)(xs[16] * si);
                            const double wf = (double)g * (double)af, of = xs[17];
                            if ((af != 0.f ? (1.0 - wf) * of + wf : of) >= (double)eps) fe++;
                        }
                        if (!TABLES && A.addr != nullptr) {      // the argmax of the address, for the log
                            const unsigned ak = a > 0.f ? __float_as_uint(a) : 0u, mk = __reduce_max_sync(FULL, ak);
                            const unsigned who = __ballot_sync(FULL, ak == mk);
                            if (lane == 0) s_arg[(bf * C + j) * 8 + warp] = make_int2((int)mk, warp * 32 + __ffs((int)who) - 1);
                        }
                        if (a != 0.f) o = (1.0 - wd0) * o + wd0;
                        w[j] = g * a;
                        if (live) wr[j * N4 + n] = w[j];
                        if (w[j] != 0.f) {                   // a row that token j does not write never sees its key, finite or not
                            const double wd = (double)w[j], om = 1.0 - wd;
                            ns = fma(om * om, ns, fma(2.0 * wd * om, e[j], wd * wd * Cm[j * C + j]));
#pragma unroll
                            for (int i = j + 1; i < C; i++) {
                                u[i] = fma(wd, Bm[j * C + i] - u[i], u[i]);
                                e[i] = fma(wd, Cm[j * C + i] - e[i], e[i]);
                            }
                        }
                    } else if (live) {
                        wr[j * N4 + n] = 0.f;
                    }
                }
            } else {
                if (!TABLES && s0 == 0) {                    // the pre-write keys, every G tokens
                    float* out = A.kbuf + snap(jb) * N * DK;
                    if (DK % 4 == 0 && DC_HELP % (DK / 4) == 0 && (reinterpret_cast<size_t>(A.kbuf) & 15) == 0) {
                        const int q4 = DK / 4, cc = (ht % q4) * 4;
                        for (int r = ht / q4; r < N; r += DC_HELP / q4) st4(out + r * DK + cc, ld4(K + r * KS + cc));
                    } else {
                        for (int i = ht; i < N * DK; i += DC_HELP) out[i] = K[(i / DK) * KS + i % DK];
                    }
                }
                const bool more = s0 + C < bn;
                if (more || jb + 1 < jb1) {
                    const int nt0 = more ? t0 + C : tb + G;
                    prep(bf ^ 1, nt0, min(C, more ? bn - s0 - C : min(G, T - nt0)));
                }
                if (!TABLES && c > 0) {
                    values(bf ^ 1, pt0, pcn, pph, pjb);
                    fetch_v(t0, cn);
                }
            }
            pt0 = t0; pcn = cn; pph = s0; pjb = jb;
            __syncthreads();
            if (row) {                                       // the rows, one pass: K <- (prod) K + sum w_j (prod after j) k_j
                float cf[C];
                double cr = 1.0;
                bool any = false;
#pragma unroll
                for (int j = C - 1; j >= 0; j--) {
                    cf[j] = (float)((double)w[j] * cr);
                    cr *= 1.0 - (double)w[j];
                    any |= w[j] != 0.f;
                }
                if (__any_sync(FULL, any) && live) {
                    const float pr = (float)cr;
                    const float* Kf = tkf(bf);
                    for (int d = 0; d < kp; d += 4) {
                        float4 x = ld4(K + n * KS + d);
                        x.x *= pr; x.y *= pr; x.z *= pr; x.w *= pr;
#pragma unroll
                        for (int j = 0; j < C; j++) {
                            const float4 kv = ld4(Kf + j * kp + d);
                            if (cf[j] != 0.f) {              // a row that token j did not write never sees it
                                x.x = fmaf(cf[j], kv.x, x.x);
                                x.y = fmaf(cf[j], kv.y, x.y);
                                x.z = fmaf(cf[j], kv.z, x.z);
                                x.w = fmaf(cf[j], kv.w, x.w);
                            }
                        }
                        st4(K + n * KS + d, x);
                    }
                }
            }
            __syncthreads();
        }
    }
    if (TABLES) return;
    if (!row) values((c - 1) & 1, pt0, pcn, pph, pjb);
    __syncthreads();
    const size_t f0 = (size_t)bh * N;
    if (A.kfin != nullptr) for (int i = tid; i < N * DK; i += NT) A.kfin[f0 * DK + i] = K[(i / DK) * KS + i % DK];
    if (A.vfin != nullptr) for (int i = tid; i < N * DV; i += NT) A.vfin[f0 * DV + i] = V[i];
    if (A.ofin != nullptr && live) A.ofin[f0 + n] = (float)o;
}

// Softmax adjoint of every token, a warp per `chunk` tokens of one sequence, in reverse:
//     dw = D + (1 - o) dO,  dgate = sum a dw,  dz = a (g dw - sum a g dw)        [gqa25/slotkern_kvg.py:165-179, soft address]
// D is overwritten with dz temp / |K_n|, the weight of row n in the raw query gradient.  With the binary occupancy penalty
// dO is zero throughout and the tokens are independent (chunk = 32); with the penalty on o itself dO is a chain (chunk = T).
template <int R>
__global__ void __launch_bounds__(128) dense_dz_kernel(const slotscan_params p, int chunk, const float* __restrict__ gate,
                                                       const float* __restrict__ fr, const float* __restrict__ temp_p,
                                                       const float* __restrict__ as, const float* __restrict__ sf,
                                                       const float* __restrict__ ki, const float* __restrict__ ot,
                                                       float* __restrict__ D, int bh0, int nbh,
                                                       float* __restrict__ dgate, float* __restrict__ dfr,
                                                       float* __restrict__ part, size_t part_n) {
    const int N = p.N, T = p.T, H = p.H, NC = (T + chunk - 1) / chunk, lane = threadIdx.x & 31;
    const size_t wid = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (wid >= (size_t)nbh * NC) return;
    const int lb = (int)(wid / NC), ck = (int)(wid % NC), bh = bh0 + lb, b = bh / H, h = bh % H;
    const float temp = temp_p[0];
    float dO[R], ca[R], cs[R], ck_[R], co[R], cd[R];
    double f1a = 0.0, f2a = 0.0;
#pragma unroll
    for (int i = 0; i < R; i++) dO[i] = 0.f;
    auto fetch = [&](int t) {
        const size_t at = ((size_t)lb * T + t) * N + lane;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const bool in = lane + 32 * i < N;
            ca[i] = in ? as[at + 32 * i] : 0.f;
            cs[i] = in ? sf[at + 32 * i] : 0.f;
            ck_[i] = in ? ki[at + 32 * i] : 0.f;
            co[i] = in ? ot[at + 32 * i] : 0.f;
            cd[i] = in ? D[at + 32 * i] : 0.f;
        }
    };
    const int t0 = ck * chunk, t1 = min(T, t0 + chunk);
    fetch(t1 - 1);
    for (int t = t1 - 1; t >= t0; t--) {
        const size_t ix = ((size_t)b * T + t) * H + h;
        const float g = gate_eff(gate[ix], p.hard_gate), frt = p.fr_per_token ? fr[ix] : fr[0];
        float a[R], s[R], k[R], oc[R], dw[R], dg = 0.f;
#pragma unroll
        for (int i = 0; i < R; i++) {
            a[i] = ca[i]; s[i] = cs[i]; k[i] = ck_[i];
            dw[i] = fmaf(1.f - co[i], dO[i], cd[i]);
            oc[i] = p.occ_bin ? (co[i] >= p.eps ? 1.f : 0.f) : co[i];
            dg = fmaf(a[i], dw[i], dg);
        }
        if (t > t0) fetch(t - 1);
        dg = warp_sum(dg);
        float f1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const float z = a[i] * (g * dw[i] - g * dg);
            if (lane + 32 * i < N) D[((size_t)lb * T + t) * N + lane + 32 * i] = z * temp * k[i];
            f1 = fmaf(-oc[i], z, f1);
            f2a += (double)z * (double)s[i];
            if (!p.occ_bin) dO[i] = fmaf(1.f - g * a[i], dO[i], -frt * z);
        }
        if (p.fr_per_token) {
            f1 = warp_sum(f1);
            if (lane == 0) dfr[ix] = f1;
        } else {
            f1a += (double)f1;
        }
        if (lane == 0) dgate[ix] = dg;
    }
    f1a = warp_sum_d(f1a);
    f2a = warp_sum_d(f2a);
    if (lane == 0) {
        const size_t at = (size_t)bh * NC + ck;
        part[at] = (float)(f2a / (double)temp);
        part[part_n + at] = (float)f1a;
    }
}

// Query gradient of a block of G tokens: dqn_t = sum_n (dz temp / |K_n|) K_n(t), the rows replayed from the block's
// snapshot (16 tokens at a time, rows in shared memory), then back through the query's normalisation.
constexpr int DQ_T = 256, DQ_C = 16, DQ_R = 8;
__host__ __device__ inline size_t dense_dq_smem(int N, int DK) {
    const int kp = dc_kpad(DK), rg = DQ_T / (kp / 4);
    return 4 * ((size_t)N * (kp + 4) + 2 * (size_t)DQ_C * N + 2 * DQ_C * kp + (size_t)rg * DQ_C * kp);
}
template <typename Tin>
__global__ void __launch_bounds__(DQ_T) dense_dq_kernel(const slotscan_params p, const Tin* __restrict__ k,
                                                        const Tin* __restrict__ q, const float* __restrict__ gate,
                                                        const float* __restrict__ kbuf, const float* __restrict__ as,
                                                        const float* __restrict__ cz, int bh0, Tin* __restrict__ dq) {
    extern __shared__ __align__(16) char dc_sm[];
    const int N = p.N, T = p.T, H = p.H, DK = p.DK, G = p.G, NB = (T + G - 1) / G;
    const int kp = dc_kpad(DK), KS = kp + 4, CG = kp / 4, RG = DQ_T / CG;
    float* K = reinterpret_cast<float*>(dc_sm);              // [N][KS]
    float* ws = K + (size_t)N * KS;                          // [DQ_C][N] write weights
    float* zs = ws + DQ_C * N;                               // [DQ_C][N] dz temp / |K_n|
    float* kt = zs + DQ_C * N;                               // [DQ_C][kp]
    float* gq = kt + DQ_C * kp;                              // [DQ_C][kp] raw query gradient
    float* red = gq + DQ_C * kp;                             // [RG][DQ_C][kp]
    __shared__ float gs[DQ_C];
    const int lb = blockIdx.x / NB, jb = blockIdx.x % NB, bh = bh0 + lb, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cg = tid % CG, rg = tid / CG;
    const bool act = rg < RG;
    const size_t so = ((size_t)b * NB + jb) * H + h;
    dense_load_rows(K, kbuf + so * N * DK, N, DK, tid, DQ_T);
    const int tb = jb * G, te = min(T, tb + G);
    for (int t0 = tb; t0 < te; t0 += DQ_C) {
        const int cn = min(DQ_C, te - t0);
        if (tid < DQ_C) gs[tid] = tid < cn ? gate_eff(gate[((size_t)b * T + t0 + tid) * H + h], p.hard_gate) : 0.f;
        __syncthreads();
#pragma unroll 6
        for (int i = tid; i < DQ_C * N; i += DQ_T) {         // tokens t0 .. are rows of the tables: one run of memory
            const size_t at = ((size_t)lb * T + t0) * N + i;
            const bool in = i < cn * N;
            const float a = in ? as[at] : 0.f, z = in ? cz[at] : 0.f;
            ws[i] = gs[i / N] * a;
            zs[i] = z;
        }
        for (int i = tid; i < DQ_C * kp; i += DQ_T) {
            const int j = i / kp, d = i % kp;
            kt[i] = (j < cn && d < DK) ? ld1(k + (((size_t)b * T + t0 + j) * H + h) * DK + d) : 0.f;
        }
        __syncthreads();
        float4 acc[DQ_C];
#pragma unroll
        for (int j = 0; j < DQ_C; j++) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int n0 = rg; act && n0 < N; n0 += RG * DQ_R) {
            float4 x[DQ_R];
#pragma unroll
            for (int r = 0; r < DQ_R; r++) x[r] = n0 + r * RG < N ? ld4(K + (n0 + r * RG) * KS + cg * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < DQ_C; j++) {
                const float4 kv = ld4(kt + j * kp + cg * 4);
#pragma unroll
                for (int r = 0; r < DQ_R; r++) {
                    const int n = min(n0 + r * RG, N - 1);   // past the last row: x is zero and is not stored
                    const float w = ws[j * N + n], z = n0 + r * RG < N ? zs[j * N + n] : 0.f;
                    acc[j].x = fmaf(z, x[r].x, acc[j].x);
                    acc[j].y = fmaf(z, x[r].y, acc[j].y);
                    acc[j].z = fmaf(z, x[r].z, acc[j].z);
                    acc[j].w = fmaf(z, x[r].w, acc[j].w);
                    if (w != 0.f) {
                        x[r].x = fmaf(w, kv.x, (1.f - w) * x[r].x);
                        x[r].y = fmaf(w, kv.y, (1.f - w) * x[r].y);
                        x[r].z = fmaf(w, kv.z, (1.f - w) * x[r].z);
                        x[r].w = fmaf(w, kv.w, (1.f - w) * x[r].w);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < DQ_R; r++) if (n0 + r * RG < N) st4(K + (n0 + r * RG) * KS + cg * 4, x[r]);
        }
        if (act) {
#pragma unroll
            for (int j = 0; j < DQ_C; j++) st4(red + (rg * DQ_C + j) * kp + cg * 4, acc[j]);
        }
        __syncthreads();
        for (int i = tid; i < DQ_C * kp; i += DQ_T) {
            float v = 0.f;
            for (int r = 0; r < RG; r++) v += red[r * DQ_C * kp + i];
            gq[i] = v;
        }
        __syncthreads();
        for (int j = warp; j < cn; j += DQ_T / 32) {         // g_q = (dqn - qn <dqn, qn>) / |q|
            const size_t ix = ((size_t)b * T + t0 + j) * H + h;
            double qq = 0.0;
            float pr = 0.f, qv[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = lane + 32 * c;
                qv[c] = d < DK ? ld1(q + ix * DK + d) : 0.f;
                qq = fma((double)qv[c], (double)qv[c], qq);
            }
            qq = warp_sum_d(qq);
            const double qn = sqrt(qq);
            const float qi = (float)(1.0 / fmax(qn, 1e-6));
#pragma unroll
            for (int c = 0; c < 4; c++) { const int d = lane + 32 * c; if (d < DK) pr = fmaf(gq[j * kp + d], qv[c] * qi, pr); }
            pr = warp_sum(pr);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = lane + 32 * c;
                if (d < DK) {
                    const float x = gq[j * kp + d];
                    st1(dq + ix * DK + d, (float)qn < 1e-6f ? qi * x : qi * (x - qv[c] * qi * pr));
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace slotscan
