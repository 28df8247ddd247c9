// Forward address scan with the key rows in registers and a resolver thread per row: the same decisions, bit for bit, as
// addr_fwd_direct_kernel (every partial dot, sum, norm and score in the same order), in about three quarters of the time per token.
//
// What bounds the direct kernel past 64 rows is the instruction stream of its one resolver warp (six rows a lane at 192 rows)
// and the shared-memory traffic of the key rows (98 KB per token at 192 x 128).  Here
//   column warps    a quarter of the columns x 64 rows each; lane = row (two of them), the rows' quarters in registers, so a
//                   token costs the broadcast reads of its query and key slices and the multiply-adds;
//   resolver warps  one per 32 rows, lane = row: adds the four partials, repairs the one row that lacks the latest write,
//                   forms z and takes the argmax of its 32 rows into an entry in shared memory; after the token's barrier every
//                   warp of the CTA takes the largest of the entries for itself;
//   helper warps    2, every other token each: loads in registers three of its tokens ahead, then into a ring in shared
//                   memory with the token's constants; the log out.
// The roles run one token apart as in the direct kernel (see its schedule comment), one barrier per token.  Every warp issues an
// instruction about every five cycles, so what counts is the longest role's instructions per token.  One CTA fills an SM, as the direct
// kernel's 192 rows did; it is the last pass where that pays (slotscan_addr_fwd_inst.cuh: wide_second_pass), with at most a sequence per
// SM right behind the narrow kernel.  B200, against the full-size direct kernel, each on its own: 192 sequences x 1024 tokens, 192 rows
// x 128 all in use, bf16: 2.27 -> 1.62 ms (two CTAs' worth of rounds on 148 SMs; column warps of three slots: 2.02); 48 x 1000, ~60 rows
// x 64, float32: 0.81 -> 0.53; 24 x 8 carried-in tokens: 31 -> 17 us.
#pragma once
#include "slotscan_addr_fwd.cuh"

namespace slotscan {

constexpr int AW_SPG = 2;                                 // row slots (32 rows each) of a column warp
__host__ __device__ constexpr int aw_col(int RPL) { return 4 * RPL / AW_SPG; }           // column warps: 4 quarters x the slots
constexpr int AW_HELP = 2;                                // helper warps
constexpr int AW_RING = 32, AW_LEAD = 8, AW_PRE = 3;      // token ring; tokens staged ahead; loads in flight ahead of that, per helper
__host__ __device__ constexpr int aw_threads(int RPL) { return 32 * (aw_col(RPL) + RPL + AW_HELP); }

constexpr int AW_TOK = 16;                                // floats of a token's constants: temp * qinv, fr, g, -, <k_{t-1}, q_t>,
                                                          // <k_{t-1}, k_t>, -, -, and in double (1-g)^2, 2 g (1-g), g^2 |k|^2
struct AddrWideSmem { int part, tok, log, am, cmb, Qs, Ks, total; };    // offsets in floats
__host__ __device__ inline AddrWideSmem addr_wide_layout(int RPL, int DK) {
    AddrWideSmem L;
    L.part = 0;                                           // [2][RPL][4][32] float2
    L.tok = L.part + 2 * RPL * 4 * 32 * 2;                // [RING][AW_TOK]
    L.log = L.tok + AW_TOK * AW_RING;                     // [2][RING]: oold, kiold
    L.am = L.log + 2 * AW_RING;                           // [RING] address
    L.cmb = L.am + AW_RING;                               // [2][8] int4: key, row, occupancy, -; then [8] masks of free rows
    L.Qs = L.cmb + 2 * 8 * 4 + 8;
    L.Ks = L.Qs + AW_RING * DK;
    L.total = L.Ks + AW_RING * DK;
    return L;
}

// a partial dot from the four chains of each of F pieces of a quarter, the pieces paired as the direct kernel's shuffles pair
// the lanes that share a row
template <int F>
__device__ __forceinline__ float aw_sum(const f32x4 (&a)[F]) {
    if constexpr (F == 4) return (sum4(a[0]) + sum4(a[2])) + (sum4(a[1]) + sum4(a[3]));
    else if constexpr (F == 2) return sum4(a[0]) + sum4(a[1]);
    else return sum4(a[0]);
}
__device__ __forceinline__ f32x4 aw_mul(const f32x4& a, const f32x4& b) { return {mul2(a.a, b.a), mul2(a.b, b.b)}; }

template <int DK, int RPL, bool OCCB, bool CARRY, typename Tin>
__global__ void __launch_bounds__(aw_threads(RPL), 1) addr_fwd_wide_kernel(
    const slotscan_params p, const Tin* __restrict__ q, const Tin* __restrict__ k, const float* __restrict__ gate,
    const float* __restrict__ fr, const float* __restrict__ temp_p, int* __restrict__ am_out,
    float* __restrict__ oold_out, float* __restrict__ kiold_out, float* __restrict__ ofin, int* __restrict__ tfirst,
    const float* __restrict__ K0, const float* __restrict__ o0, const double* __restrict__ nsq0,
    double* __restrict__ nsqfin, const float* __restrict__ hand) {
    extern __shared__ __align__(16) float smem[];
    constexpr int CW = DK / 4, NF = CW / 4, SPG = AW_SPG;              // columns and float4 per quarter, slots per column warp
    constexpr int AW_COL = aw_col(RPL);
    constexpr int F8 = NF >= 4 ? 4 : 1, F16 = NF >= 2 ? 2 : 1;        // the direct kernel's splits below 8 and 16 rows
    constexpr int NT = aw_threads(RPL);
    const int N = p.N, H = p.H;
    const AddrWideSmem L = addr_wide_layout(RPL, DK);
    float2* part = reinterpret_cast<float2*>(smem + L.part);
    float* s_tok = smem + L.tok;
    float* s_oold = smem + L.log;
    float* s_kiold = smem + L.log + AW_RING;
    int* s_am = reinterpret_cast<int*>(smem + L.am);
    int4* s_cmb = reinterpret_cast<int4*>(smem + L.cmb);
    unsigned* s_free = reinterpret_cast<unsigned*>(s_cmb + 16);
    float* Qs = smem + L.Qs;
    float* Ks = smem + L.Ks;
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float temp = temp_p[0], eps = p.eps;
    const int mark = tfirst[(size_t)bh * N];
    if (mark >= 0) return;                                            // finished in an earlier pass (uniform per CTA)
    const AfResume rs(mark, am_out, (size_t)b * p.T * H + h, H);
    const int T = p.T - rs.t0;                                        // tokens are counted from rs.t0 on
    const size_t bT = (size_t)b * p.T + rs.t0;
    __syncthreads();
    // a carried-in state: squared norms as the direct kernel takes or sums them, the highest row it has touched
    int hw0 = rs.am;
    double* s_nsq = reinterpret_cast<double*>(smem + L.part);         // [N] before `part` is first written
    if (CARRY && !rs.on) {
        for (int n = warp; n < N; n += NT / 32) {
            double a = 0.0;
            if (nsq0 != nullptr) {
                a = nsq0[(size_t)bh * N + n];
            } else {
                for (int c = lane; c < DK; c += 32) {
                    const double xk = (double)K0[((size_t)bh * N + n) * DK + c];
                    a = fma(xk, xk, a);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(FULL, a, off);
            }
            if (lane == 0) s_nsq[n] = a;
        }
        __syncthreads();
        for (int n0 = 0; n0 < N; n0 += 32) {                          // same in every thread
            const int n = n0 + lane;
            const unsigned used = __ballot_sync(FULL, n < N && (s_nsq[n] > 0.0 || o0[(size_t)bh * N + n] != 0.f));
            if (used) hw0 = n0 + 31 - __clz(used);
        }
    }
    const int lim0 = CARRY || rs.on ? min(hw0 + 1, N - 1) : 0;        // candidate limit of token 0
    if (rs.on) {
        if (tid == 0) tfirst[(size_t)bh * N] = 0;                     // the others stand as the pass before left them
    } else {
        for (int i = tid; i < N; i += NT) tfirst[(size_t)bh * N + i] = (i <= hw0 + 1) ? 0 : T;
    }
    if (tid < 16) s_cmb[tid] = make_int4(0, 0, 0, 0);
#define AW_BARRIER() asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory")
    // the address of the token whose entries lie in buffer `buf` (lim: its last candidate row): the largest score, in the lowest
    // 32 rows that hold it; without one (NaN scores) row lim.  oa: that row's occupancy before the write.  Every lane alike.
    struct Addr { int am; float oa; bool any; };
    auto resolved = [&](int buf, int lim) {
        const int4 c = s_cmb[buf * 8 + (lane & 7)];
        const unsigned kmax = __reduce_max_sync(FULL, (unsigned)c.x);
        const unsigned who = __ballot_sync(FULL, (unsigned)c.x == kmax);
        const int src = kmax ? __ffs((int)who) - 1 : lim >> 5;
        Addr a;
        a.am = __shfl_sync(FULL, c.y, src);
        a.oa = __int_as_float(__shfl_sync(FULL, c.z, src));
        a.any = kmax != 0u;
        return a;
    };

    if (warp < AW_COL) {
        // ------------------------------------------------------------------ column warps
        const int cw = warp & 3, s_base = (warp >> 2) * SPG, c0 = cw * CW;
        f32x4 K[SPG][NF];
#pragma unroll
        for (int s = 0; s < SPG; s++) {
            const int n = (s_base + s) * 32 + lane;
#pragma unroll
            for (int i = 0; i < NF; i++) {
                K[s][i] = {0ull, 0ull};
                if (rs.on) { if (n <= rs.am) K[s][i] = ld4x2(hand + ((size_t)bh * N + n) * DK + c0 + 4 * i); }
                else if (CARRY && n < N) K[s][i] = ld4x2(K0 + ((size_t)bh * N + n) * DK + c0 + 4 * i);
            }
        }
        auto dots = [&](int limd, int sl, int buf) {
            const float* qr = Qs + sl * DK + c0;
            const float* kr = Ks + sl * DK + c0;
            float2* out = part + ((buf * RPL + s_base) * 4 + cw) * 32 + lane;
            auto few = [&](auto fc) {                                 // fewer than 16 rows: slot 0 only, in pieces
                constexpr int F = decltype(fc)::value, NFS = NF / F;
                f32x4 aS[F], aR[F];
#pragma unroll
                for (int f = 0; f < F; f++) {
#pragma unroll
                    for (int i = 0; i < NFS; i++) {
                        const f32x4 q4 = ld4x2(qr + 4 * (f * NFS + i)), k4 = ld4x2(kr + 4 * (f * NFS + i));
                        if (i == 0) { aS[f] = aw_mul(K[0][f * NFS], q4); aR[f] = aw_mul(K[0][f * NFS], k4); }
                        else { fma4(aS[f], K[0][f * NFS + i], q4); fma4(aR[f], K[0][f * NFS + i], k4); }
                    }
                }
                out[0] = make_float2(aw_sum<F>(aS), aw_sum<F>(aR));
            };
            auto many = [&](auto nc) {                                // the first NS slots of this warp
                constexpr int NS = decltype(nc)::value;
                float sS[NS];
#pragma unroll
                for (int pass = 0; pass < 2; pass++) {                // queries, then keys: half the sums in registers
                    const float* r = pass ? kr : qr;
                    f32x4 a[NS];
#pragma unroll
                    for (int i = 0; i < NF; i++) {
                        const f32x4 r4 = ld4x2(r + 4 * i);
#pragma unroll
                        for (int s = 0; s < NS; s++) {
                            if (i == 0) a[s] = aw_mul(K[s][0], r4);
                            else fma4(a[s], K[s][i], r4);
                        }
                    }
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        const float v = sum4(a[s]);
                        if (pass == 0) sS[s] = v;
                        else out[s * 4 * 32] = make_float2(sS[s], v);
                    }
                }
            };
            if (limd < 16) {
                if (s_base == 0) {
                    if (limd < 8) few(std::integral_constant<int, F8>());
                    else few(std::integral_constant<int, F16>());
                }
                return;
            }
            const int ns = limd / 32 + 1 - s_base;                    // slots of this warp that hold candidates
            if (ns <= 0) return;
            if (ns == 1) many(std::integral_constant<int, 1>());
            else many(std::integral_constant<int, SPG>());
        };
        __syncthreads();                                              // the prologue's tokens are staged (and s_nsq is read)
        dots(lim0, 0, 0);
        AW_BARRIER();
        int lim = lim0, a = rs.am;
        for (int t = 0; t < T; t++) {
            if (t >= 1) {
                a = resolved((t - 1) & 1, lim).am;
                lim = max(lim, min(a + 1, N - 1));
            }
            const int sa = a < 0 ? -1 : (a >> 5) - s_base;            // the write of token t - 1
            if (sa >= 0 && sa < SPG) {
                const int sl = (t - 1) & (AW_RING - 1);
                const float g = s_tok[AW_TOK * sl + 2];
                const f32x2 g2 = pack2(g, g), om2 = pack2(1.f - g, 1.f - g);
                const float* kr = Ks + sl * DK + c0;
#pragma unroll
                for (int s = 0; s < SPG; s++) {
                    if (s == sa && lane == (a & 31)) {
#pragma unroll
                        for (int i = 0; i < NF; i++) {
                            const f32x4 k4 = ld4x2(kr + 4 * i);
                            K[s][i].a = fma2(g2, k4.a, mul2(om2, K[s][i].a));      // blend, two columns at a time
                            K[s][i].b = fma2(g2, k4.b, mul2(om2, K[s][i].b));
                        }
                    }
                }
                __syncwarp();
            }
            if (t + 1 < T) dots(min(lim + 1, N - 1), (t + 1) & (AW_RING - 1), (t + 1) & 1);
            AW_BARRIER();
        }
    } else if (warp < AW_COL + RPL) {
        // ------------------------------------------------------------------ resolver warps
        const int rw = warp - AW_COL, n = rw * 32 + lane;
        const bool live = n < N;
        double nsq = 0.0;
        float kinv = 1e6f, o = 0.f;
        if (rs.on ? n <= rs.am : CARRY && live) {
            nsq = rs.on ? nsqfin[(size_t)bh * N + n] : s_nsq[n];
            kinv = fminf(rsqrtf((float)nsq), 1e6f);
            o = (rs.on ? ofin : o0)[(size_t)bh * N + n];
        }
        // lowest free row (N if none): every resolver warp knows it.  After a change: one mask per warp, in shared memory.
        auto publish = [&](bool is_free) {
            const unsigned m = __ballot_sync(FULL, is_free);
            if (lane == 0) s_free[rw] = m;
            asm volatile("bar.sync 2, %0;" ::"n"(32 * RPL) : "memory");
            int f = N;
#pragma unroll
            for (int w = RPL - 1; w >= 0; w--) { const unsigned x = s_free[w]; if (x) f = 32 * w + __ffs((int)x) - 1; }
            asm volatile("bar.sync 2, %0;" ::"n"(32 * RPL) : "memory");
            return f;
        };
        int lim = lim0;
        float R = 0.f, g_prev = 0.f;
        bool mine = false;                                            // the previous token wrote this row
        // what the address of token t - 1 changes: the candidates, and in its row norm, occupancy and the lowest free row
        int fe;
        auto settle = [&](int t) {
            const Addr a = resolved((t - 1) & 1, lim);
            const int ps = (t - 1) & (AW_RING - 1);
            if (tid == AW_COL * 32) s_am[ps] = a.am;
            if (a.am >= lim && lim < N - 1) {                         // a row not written before: one more candidate
                lim++;
                if (tid == AW_COL * 32) tfirst[(size_t)bh * N + lim] = rs.t0 + t;
            }
            mine = n == a.am;
            if (mine) {
                const double* dc = reinterpret_cast<const double*>(s_tok + AW_TOK * ps + 8);
                const double nn = fmax(fma(dc[0], nsq, fma(dc[1], (double)(a.any ? R : 0.f), dc[2])), 0.0);
                s_oold[ps] = o;
                s_kiold[ps] = kinv;
                nsq = nn;
                kinv = fminf(rsqrtf((float)nn), 1e6f);
                o = __fmaf_rn(1.f - g_prev, o, g_prev);
            }
            const bool is_free = __fmaf_rn(1.f - g_prev, a.oa, g_prev) < eps;
            if (a.am == fe && !is_free) fe = publish(live && o < eps);                       // the free row got taken
            else if (is_free && a.am < fe) fe = a.am;
        };
        __syncthreads();
        if (rs.on) { mine = n == rs.am; g_prev = s_tok[AW_TOK * (AW_RING - 1) + 2]; }
        fe = publish(live && o < eps);
        AW_BARRIER();
        for (int t = 0; t < T; t++) {
            const int buf = t & 1;
            const float* tk = s_tok + AW_TOK * (t & (AW_RING - 1));
            const float4 c4 = ld4(tk);                                // temp * qinv, fr, g
            const float2 x2 = *reinterpret_cast<const float2*>(tk + 4);
            float2 pr[4];
#pragma unroll
            for (int w = 0; w < 4; w++) pr[w] = part[((buf * RPL + rw) * 4 + w) * 32 + lane];
            if (t >= 1) settle(t);
            const bool act = 32 * rw <= lim;                          // uniform per warp
            float S = 0.f;
            R = 0.f;
#pragma unroll
            for (int w = 0; w < 4; w++) { S += pr[w].x; R += pr[w].y; }
            if (mine) {                                               // the one row whose latest write the dots have not seen
                S = blend(S, x2.x, g_prev, 1.f - g_prev);
                R = blend(R, x2.y, g_prev, 1.f - g_prev);
            }
            // product, product, difference, each rounded: as the direct kernel's expression comes out
            const float sc = __fmul_rn(c4.x, __fmul_rn(kinv, S));
            const float z = (OCCB ? __fsub_rn(sc, o >= eps ? c4.y : __fmul_rn(c4.y, 0.f)) : __fmaf_rn(-c4.y, o, sc)) + 0.f;
            const bool ok = n <= lim && (o >= eps || n == fe) && z > -INFINITY;
            const unsigned key = ok ? ord_key(z) : 0u;
            if (act) {
                const unsigned kmax = __reduce_max_sync(FULL, key);
                const unsigned who = __ballot_sync(FULL, ok && key == kmax);
                if (lane == (who ? __ffs((int)who) - 1 : lim & 31))   // the smallest row of the largest score
                    s_cmb[buf * 8 + rw] = make_int4((int)(who ? kmax : 0u), n, __float_as_int(o), 0);
            }
            g_prev = c4.z;
            AW_BARRIER();
        }
        settle(T);
        if (live) {
            ofin[(size_t)bh * N + n] = o;
            if (nsqfin != nullptr) nsqfin[(size_t)bh * N + n] = nsq;
        }
    } else {
        // ------------------------------------------------------------------ helper warps: the tokens of one parity each
        const int hp = warp - AW_COL - RPL;
        constexpr int EPL = DK / 32;                                  // elements of a token's row per lane: 2 or 4
        struct alignas(EPL * sizeof(Tin)) Vec { Tin v[EPL]; };
        struct Tok { Vec q, k; float g, f; };
        auto fetch = [&](Tok& d, int u) {                             // loads only: they stay in flight
            const size_t ix = (bT + min(u, T - 1)) * H + h;
            d.q = *reinterpret_cast<const Vec*>(q + ix * DK + lane * EPL);
            d.k = *reinterpret_cast<const Vec*>(k + ix * DK + lane * EPL);
            d.g = gate[ix];
            d.f = p.fr_per_token ? fr[ix] : fr[0];
        };
        auto commit = [&](const Tok& d, int u) {
            const int sl = u & (AW_RING - 1);
#pragma unroll
            for (int i = 0; i < EPL; i++) {
                Qs[sl * DK + lane * EPL + i] = (float)d.q.v[i];
                Ks[sl * DK + lane * EPL + i] = (float)d.k.v[i];
            }
            if (lane == 0) { s_tok[AW_TOK * sl + 2] = gate_eff(d.g, p.hard_gate); s_tok[AW_TOK * sl + 1] = d.f; }
            __syncwarp();
        };
        // the constants of token u, whose row and the row before it are in the ring; both half-warps alike
        auto token = [&](int u) {
            const int sl = u & (AW_RING - 1);
            float* tk = s_tok + AW_TOK * sl;
            af_token_consts<DK, float>(Qs + sl * DK, Ks + sl * DK, Ks + ((sl + AW_RING - 1) & (AW_RING - 1)) * DK, lane & 15, temp,
                                       tk, reinterpret_cast<double*>(tk + 8), tk + 4);
            __syncwarp();
        };
        auto flush = [&](int t0, int t1) {                            // log of tokens [t0, t1), at most 32
            const int t = t0 + lane;
            if (t < t1) {
                const int sl = t & (AW_RING - 1);
                const size_t ix = (bT + t) * H + h;
                am_out[ix] = s_am[sl];
                oold_out[ix] = s_oold[sl];
                kiold_out[ix] = s_kiold[sl];
            }
        };
        if (hp == 0) {                                                // "the key before token 0"
            if (rs.on) {
                Tok e;
                fetch(e, -1);
                commit(e, -1);
            } else {
#pragma unroll
                for (int i = 0; i < EPL; i++) Ks[(AW_RING - 1) * DK + lane * EPL + i] = 0.f;
            }
        }
        Tok d[AW_PRE];
        for (int u0 = hp; u0 < AW_LEAD; u0 += 2 * AW_HELP) {          // the first tokens, two in flight
            Tok e[2];
            fetch(e[0], u0);
            fetch(e[1], u0 + AW_HELP);
            commit(e[0], u0);
            commit(e[1], u0 + AW_HELP);
        }
#pragma unroll
        for (int j = 0; j < AW_PRE; j++) fetch(d[j], AW_LEAD + hp + AW_HELP * j);
        asm volatile("bar.sync 3, %0;" ::"n"(32 * AW_HELP) : "memory");       // both parities' rows are there
        for (int u = hp; u < AW_LEAD - 1; u += AW_HELP) token(u);
        __syncthreads();
        AW_BARRIER();
        // phase t, for the helper of parity (t + AW_LEAD) % 2: the row of token t + AW_LEAD; the other one: the constants of token
        // t + AW_LEAD - 1, whose row it staged a phase ago
        for (int t0 = 0; t0 < T; t0 += AW_PRE * AW_HELP) {
#pragma unroll
            for (int j = 0; j < AW_PRE; j++) {
#pragma unroll
                for (int e = 0; e < AW_HELP; e++) {
                    const int t = t0 + AW_HELP * j + e;
                    if (t < T) {
                        if (e == hp) {                                // AW_LEAD is even
                            if (t + AW_LEAD < T) {
                                commit(d[j], t + AW_LEAD);
                                fetch(d[j], t + AW_LEAD + AW_PRE * AW_HELP);
                            }
                            if ((t & 15) == 1 && t > 16) flush(t - 17, t - 1);        // tokens finished a phase ago
                        } else if (t + AW_LEAD - 1 < T) {
                            token(t + AW_LEAD - 1);
                        }
                        AW_BARRIER();
                    }
                }
            }
        }
    }
    __syncthreads();
    if (warp == AW_COL + RPL) {                                       // the log entries still in the ring
        const int done = T < 18 ? 0 : ((T - 2) / 16) * 16;            // last flush: at the last t = 1 (mod 16), t <= T - 1, t > 16
        for (int t0 = done; t0 < T; t0 += 32) {
            const int t = t0 + lane;
            if (t < T) {
                const int sl = t & (AW_RING - 1);
                const size_t ix = (bT + t) * H + h;
                am_out[ix] = s_am[sl];
                oold_out[ix] = s_oold[sl];
                kiold_out[ix] = s_kiold[sl];
            }
        }
    }
#undef AW_BARRIER
}

}  // namespace slotscan
