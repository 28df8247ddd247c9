// Forward address scan while at most 32 rows are in use, keys 64 or 128 wide: the same decisions, bit for bit, as
// addr_fwd_direct_kernel (every partial dot, sum, norm and score in the same order), in about half the time per token.
//
// A warp that runs a dependent stream issues an instruction about every five cycles, so what counts is the longest role's
// instructions per token.  Here
//   resolver warp   lane = row: z and the argmax, nothing else;
//   norm warp       lane = row: what a write by the token in work would make of the row's norm, its reciprocal and the occupancy,
//                   beside the token's argmax; the next token selects;
//   column warps    4: a quarter of the columns each; the rows' pieces in registers, a row split over 4, 2 or 1 lanes as the direct
//                   kernel splits it (below 8, 16 and 32 rows), so a token costs the reads of its vectors (each delivers 512
//                   bytes to the warp, broadcast or not), one blend and the multiply-adds of the lane's pieces;
//   loader warps    2: everything that is not per token: rows of the chunk after next, token constants, log.
// Resolver, norm and column warps run one token apart and meet at one barrier per token, as in the direct kernel; the loaders meet
// the resolver once per chunk of 8.
// B200, about 11 of 192 rows x 128 in use, this kernel against the direct one, each on its own: 48 sequences x 1024 tokens, bf16: 497 ->
// 251 us (487 cycles per token; 271 us beside the zero-fill); 12 x 256, float32: 126 -> 67; 3072 x 128 (96 rows), three CTAs to an SM:
// 632 -> 433 (80 registers; at 128 columns 32 bytes are spilled, where the pieces of the rows change lanes).
#pragma once
#include "slotscan_addr_fwd.cuh"
#include "slotscan_async.cuh"

namespace slotscan {

constexpr int AN_ROWS = 32;
constexpr int AN_L = 8;                                   // tokens staged at a time
constexpr int AN_RING = 32;                               // tokens staged
constexpr int AN_THREADS = 32 * 8;
constexpr int AN_PART = 4 * AN_ROWS;                      // partial sums of a token and type
constexpr int AN_TOK = 16;                                // a token's constants: temp * qinv, fr, <k_{t-1}, q_t>, <k_{t-1}, k_t> | g, g,
                                                          // 1-g, 1-g | (double) (1-g)^2, 2 g (1-g) | (double) g^2 |k|^2, g, 1-g
struct AddrNarrowSmem { int part, tok, hyp, am, oold, kiold, leave, Q, K, total; };    // offsets in floats
__host__ __device__ inline AddrNarrowSmem addr_narrow_layout(int DK) {
    AddrNarrowSmem L;
    L.part = 0;                                           // [2][q, k][32 / F rows][4 quarters][F lanes]
    L.tok = L.part + 2 * 2 * AN_PART;                     // [RING][AN_TOK]
    L.hyp = L.tok + AN_RING * AN_TOK;                     // [2][32] float2: reciprocal norm and occupancy after a write
    L.am = L.hyp + 2 * AN_ROWS * 2;                       // [RING] address; bit 31: the row was not written before; bit 30: no score
    L.oold = L.am + AN_RING;
    L.kiold = L.oold + AN_RING;
    L.leave = L.kiold + AN_RING;
    L.Q = L.leave + 4;                                    // [RING][DK]
    L.K = L.Q + AN_RING * DK;
    L.total = L.K + AN_RING * DK;
    return L;
}
__device__ __forceinline__ float redux_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// a row's dot product from its partial sums: the F lanes' parts as the direct kernel's shuffles add them, then the quarters
// (lanes past the rows that F lanes leave room for read some row's: not used)
template <int F>
__device__ __forceinline__ float an_sum(const float* p, int lane) {
    float q[4];
    p += (lane & (32 / F - 1)) * 4 * F;
    if constexpr (F == 1) {
        const float4 a = ld4(p);
        q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
    } else if constexpr (F == 2) {
        const float4 a = ld4(p), b = ld4(p + 4);
        q[0] = a.x + a.y; q[1] = a.z + a.w; q[2] = b.x + b.y; q[3] = b.z + b.w;
    } else {
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const float4 a = ld4(p + 4 * w);
            q[w] = (a.x + a.z) + (a.y + a.w);
        }
    }
    return ((q[0] + q[1]) + q[2]) + q[3];
}
// acc = g x + om acc in the lanes with row == a, two columns at a time, rounded as blend(); predicated, so that the warp does not
// part ways
__device__ __forceinline__ void blend_if(f32x4& acc, const f32x4& x, f32x2 g, f32x2 om, int row, int a) {
    asm("{\n.reg .pred p;\n.reg .b64 u, v;\nsetp.eq.s32 p, %6, %7;\n"
        "@p mul.rn.f32x2 u, %5, %0;\n@p mul.rn.f32x2 v, %5, %1;\n"
        "@p fma.rn.f32x2 %0, %4, %2, u;\n@p fma.rn.f32x2 %1, %4, %3, v;\n}"
        : "+l"(acc.a), "+l"(acc.b) : "l"(x.a), "l"(x.b), "l"(g), "l"(om), "r"(row), "r"(a));
}

// CTAS: CTAs that share an SM.  With two the length of a token's chain counts: no branch around a blend, and the lanes' sums go to
// the resolver as they are.  With three (80 registers) the instructions of all warps count: the column warps add them up.
template <int DK, int CTAS, bool OCCB, bool CARRY, typename Tin>
__global__ void __launch_bounds__(AN_THREADS, CTAS) addr_fwd_narrow_kernel(
    const slotscan_params p, const Tin* __restrict__ q, const Tin* __restrict__ k, const float* __restrict__ gate,
    const float* __restrict__ fr, const float* __restrict__ temp_p, int* __restrict__ am_out,
    float* __restrict__ oold_out, float* __restrict__ kiold_out, float* __restrict__ ofin, int* __restrict__ tfirst,
    const float* __restrict__ K0, const float* __restrict__ o0, const double* __restrict__ nsq0,
    double* __restrict__ nsqfin, float* __restrict__ hand) {
    // A sequence that needs a row above the 32 is left to the next pass (slotscan_addr_fwd.cuh: AfResume).
    extern __shared__ __align__(16) float smem[];
    constexpr int CW = DK / 4, NF = CW / 4;               // columns and float4 per quarter
    const int N = p.N, T = p.T, H = p.H, ncap = min(N, AN_ROWS);
    const AddrNarrowSmem L = addr_narrow_layout(DK);
    float* s_part = smem + L.part;
    float* s_tok = smem + L.tok;
    float2* s_hyp = reinterpret_cast<float2*>(smem + L.hyp);
    int* s_am = reinterpret_cast<int*>(smem + L.am);
    float* s_oold = smem + L.oold;
    float* s_kiold = smem + L.kiold;
    int* s_leave = reinterpret_cast<int*>(smem + L.leave);
    float* Qs = smem + L.Q;
    float* Ks = smem + L.K;
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float eps = p.eps;

    // ---- carried-in state: every warp looks at the norms and occupancies itself (lane = row) ----
    double nsq = 0.0;
    float o = 0.f;
    int lim = 0;                                          // the current token's last candidate row
    if (CARRY) {
        double* s_nsq = reinterpret_cast<double*>(s_part);            // [N], where none came with the state: the direct kernel's sums
        for (bool sums = nsq0 != nullptr;; sums = true) {             // (first without them: a row in use most often shows in its occupancy)
            int hw0 = -1;                                 // highest row that the state has touched
            for (int n0 = 0; n0 < N; n0 += 32) {
                const int n = n0 + lane;
                const double a = n >= N || !sums ? 0.0 : (nsq0 != nullptr ? nsq0[(size_t)bh * N + n] : s_nsq[n]);
                const float on = n < N ? o0[(size_t)bh * N + n] : 0.f;
                const unsigned used = __ballot_sync(FULL, a > 0.0 || on != 0.f);
                if (used) hw0 = n0 + 31 - __clz(used);
                if (n0 == 0) { nsq = a; o = on; }
            }
            lim = min(hw0 + 1, N - 1);
            if (lim >= ncap) {                            // uniform over the CTA
                if (tid == 0) tfirst[(size_t)bh * N] = af_mark(0);
                return;
            }
            if (sums) break;
            for (int n = warp; n < N; n += AN_THREADS / 32) {
                double a = 0.0;
                for (int c = lane; c < DK; c += 32) {
                    const double xk = (double)K0[((size_t)bh * N + n) * DK + c];
                    a = fma(xk, xk, a);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(FULL, a, off);
                if (lane == 0) s_nsq[n] = a;
            }
            __syncthreads();
        }
        __syncthreads();
    }
    const int lim0 = lim;
    // lanes that share a row, by the last row that a token's dots visit
    auto mode_of = [](int limd) { return limd < 8 ? 4 : (limd < 16 ? 2 : 1); };
    for (int i = tid; i < N; i += AN_THREADS) tfirst[(size_t)bh * N + i] = i <= lim0 ? 0 : T;
    for (int i = tid; i < DK; i += AN_THREADS) Ks[(AN_RING - 1) * DK + i] = 0.f;           // "the key before token 0"
    for (int i = tid; i < 2 * 2 * AN_PART; i += AN_THREADS) s_part[i] = 0.f;
    if (tid == 0) *s_leave = 0;
    __syncthreads();
#define AN_BAR(ID, N_) asm volatile("bar.sync " #ID ", %0;" ::"n"(N_) : "memory")
#define AN_PHASE_BARRIER() AN_BAR(1, 32 * 6)

    if (warp >= 6) {
        // ------------------------------------------------------------------ loader warps: half of a chunk each
        const float temp = temp_p[0];
        constexpr bool CONV = sizeof(Tin) != 4;           // float32 rows go to shared memory as they are
        constexpr int EU = 16 / (int)sizeof(Tin), UPR = DK / EU, RPW = 32 / UPR, NL = AN_L / 2 / RPW;   // elements per load, loads
        const int half = (warp - 6) * (AN_L / 2);                                                  // per row, rows per warp-wide load
        const int lr = half + lane / UPR, lc = (lane % UPR) * EU;
        uint4 rq[CONV ? NL : 1], rk[CONV ? NL : 1];
        float rg = 0.f;
        auto fetch = [&](int ck) {                        // loads only: they stay in flight
#pragma unroll
            for (int i = 0; i < NL; i++) {
                const int t = ck * AN_L + i * RPW + lr, sl = t & (AN_RING - 1);
                const size_t ix = (((size_t)b * T + min(t, T - 1)) * H + h) * DK + lc;
                if constexpr (CONV) {
                    rq[i] = *reinterpret_cast<const uint4*>(q + ix);
                    rk[i] = *reinterpret_cast<const uint4*>(k + ix);
                } else {
                    cp_async16(Qs + sl * DK + lc, q + ix);
                    cp_async16(Ks + sl * DK + lc, k + ix);
                }
            }
            if (lane < AN_L) {                            // gates, then penalties
                const size_t ix = ((size_t)b * T + min(ck * AN_L + half + (lane & 3), T - 1)) * H + h;
                rg = lane < 4 ? gate[ix] : (p.fr_per_token ? fr[ix] : fr[0]);
            }
        };
        auto commit = [&](int ck) {
            if constexpr (CONV) {
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const int sl = (ck * AN_L + i * RPW + lr) & (AN_RING - 1);
                    Pre8<__nv_bfloat16> x;
                    x.u = rq[i];
                    x.store(Qs + sl * DK + lc);
                    x.u = rk[i];
                    x.store(Ks + sl * DK + lc);
                }
            } else {
                cp_async_wait();
            }
            if (lane < AN_L) {
                float* tk = s_tok + AN_TOK * ((ck * AN_L + half + (lane & 3)) & (AN_RING - 1));
                if (lane < 4) {
                    const float g = gate_eff(rg, p.hard_gate);
                    st4(tk + 4, make_float4(g, g, 1.f - g, 1.f - g));
                    tk[14] = g;
                    tk[15] = 1.f - g;
                } else {
                    tk[1] = rg;
                }
            }
            __syncwarp();
        };
        auto consts = [&](int ck) {                       // two tokens at a time
#pragma unroll
            for (int i = 0; i < AN_L / 2; i += 2) {
                const int sl = (ck * AN_L + half + i + (lane >> 4)) & (AN_RING - 1);
                float* tk = s_tok + AN_TOK * sl;
                float4 tok4;
                double d[4];
                float x[2];
                tok4.z = tk[14];
                af_token_consts<DK, float>(Qs + sl * DK, Ks + sl * DK, Ks + ((sl + AN_RING - 1) & (AN_RING - 1)) * DK, lane & 15, temp,
                                           &tok4.x, d, x);
                if ((lane & 15) == 0) {
                    tk[0] = tok4.x;
                    tk[2] = x[0];
                    tk[3] = x[1];
                    double* td = reinterpret_cast<double*>(tk + 8);
                    td[0] = d[0]; td[1] = d[1]; td[2] = d[2];
                }
            }
            __syncwarp();
        };
        fetch(0);
        commit(0);
        if (AN_L < T) { fetch(1); commit(1); }
        __syncthreads();                                  // the first rows are staged
        consts(0);
        __syncthreads();                                  // and what the resolver's first token needs is there
        for (int c = 0; c * AN_L < T; c++) {
            const bool more = (c + 2) * AN_L < T;
            if (more) fetch(c + 2);
            if ((c + 1) * AN_L < T) consts(c + 1);
            // the log of 8 tokens: the resolver came here in the phase of token 8 c - 1, which the norm warp may still be in, and
            // there it writes the entries of token 8 c - 2
            if (c >= 1) {
                const int t = (c - 1) * AN_L - 2 + (lane & 7);
                if (t >= 0 && lane < 24 && half == 0) {
                    const size_t ix = ((size_t)b * T + t) * H + h;
                    const int sl = t & (AN_RING - 1);
                    if (lane < 8) am_out[ix] = s_am[sl] & 0x3fffffff;
                    else if (lane < 16) oold_out[ix] = s_oold[sl];
                    else kiold_out[ix] = s_kiold[sl];
                }
            }
            if (more) commit(c + 2);
            if (c * AN_L + AN_L - 1 >= T) break;
            AN_BAR(2, 96);                                // with the resolver, in the phase of the chunk's last token
            if (*s_leave && *s_leave <= c * AN_L + AN_L - 1) break;       // (it may be of the next chunk's tokens already)
        }
    } else if (warp >= 2) {
        // ------------------------------------------------------------------ column warps
        const int cw = warp - 2;
        const float* qcol = Qs + cw * CW;
        const float* kcol = Ks + cw * CW;
        int t = -1;                                       // phase: the write of token t - 1, the dots of token t + 1
        bool left = false, written = true;
        // A row's quarter over F lanes, lane = row + 32 / F * part; returns with the write of token t - 1 done where the dots of token
        // t + 1 visit too many rows for F (or at the end).  Where registers reach, a token's key is read once, for its dots, and
        // kept for its write two phases on.
        auto run = [&](auto fc, auto& K) {
            constexpr int F = decltype(fc)::value, R = 32 / F, NFS = NF / F;
            constexpr bool KEEP = F > 1;
            const int row = lane & (R - 1), c0 = (lane / R) * (CW / F);
            f32x4 ka[NFS], kb[KEEP ? NFS : 1];
            auto read = [&](auto& d, const float* cols, int u) {
                const float* r = cols + (u & (AN_RING - 1)) * DK + c0;
#pragma unroll
                for (int i = 0; i < NFS; i++) d[i] = ld4x2(r + 4 * i);
            };
            auto dots = [&](auto& kk, auto& qv) {         // of token t + 1
                read(kk, kcol, t + 1);
                f32x4 sq = {0ull, 0ull}, sk = sq;
#pragma unroll
                for (int i = 0; i < NFS; i++) {
                    if constexpr (KEEP) fma4(sq, K[i], qv[i]);
                    else fma4(sq, K[i], ld4x2(qcol + ((t + 1) & (AN_RING - 1)) * DK + c0 + 4 * i));
                }
#pragma unroll
                for (int i = 0; i < NFS; i++) fma4(sk, K[i], kk[i]);
                float x = sum4(sq), y = sum4(sk);
                float* d = s_part + ((t + 1) & 1) * 2 * AN_PART;
                if constexpr (CTAS >= 3) {
#pragma unroll
                    for (int off = 16; off >= R; off >>= 1) {
                        x += __shfl_xor_sync(FULL, x, off);
                        y += __shfl_xor_sync(FULL, y, off);
                    }
                    d += row * 4 + cw;
                    if (lane < R) { d[0] = x; d[AN_PART] = y; }
                } else {
                    d += (row * 4 + cw) * F + lane / R;
                    d[0] = x;
                    d[AN_PART] = y;
                }
            };
            auto phase = [&](auto& kk) {                  // kk: key t - 1, then key t + 1; true: leave
                f32x4 qv[KEEP ? NFS : 1];
                if constexpr (KEEP && CTAS >= 3) read(qv, qcol, t + 1);
                if (!written) {
                    const int sl = (t - 1) & (AN_RING - 1);
                    int a = s_am[sl];
                    const float4 gg = ld4(s_tok + AN_TOK * sl + 4);
                    if constexpr (!KEEP) read(kk, kcol, t - 1);
                    bool more = false;
                    if ((unsigned)a >= 0x40000000u) {
                        if (a < 0) {                      // a row not written before: one more candidate
                            if (++lim >= ncap) { left = true; return true; }
                            more = F > 1 && min(lim + 1, N - 1) >= R;
                        }
                        a &= 0x3fffffff;
                    }
                    const f32x2 g2 = pack2(gg.x, gg.y), om2 = pack2(gg.z, gg.w);
                    if constexpr (CTAS >= 3 || !KEEP) {
                        if (row == a) {
#pragma unroll
                            for (int i = 0; i < NFS; i++) {
                                K[i].a = fma2(g2, kk[i].a, mul2(om2, K[i].a)); // blend, two columns at a time
                                K[i].b = fma2(g2, kk[i].b, mul2(om2, K[i].b));
                            }
                        }
                        __syncwarp();
                    } else {
#pragma unroll
                        for (int i = 0; i < NFS; i++) blend_if(K[i], kk[i], g2, om2, row, a);
                    }
                    if (more) { written = true; return true; }
                }
                written = false;
                if constexpr (KEEP && CTAS < 3) read(qv, qcol, t + 1);        // (the address comes first: the chain waits for it)
                dots(kk, qv);
                AN_PHASE_BARRIER();
                return ++t >= T;
            };
            if (t < 0) {                                  // before the first token
                f32x4 qv[NFS];
                read(qv, qcol, 0);
                dots(ka, qv);
                __syncthreads();
                t = 0;                                    // token 0 has no write before it
                if (F > 1 && min(lim + 1, N - 1) >= R) return;
            } else if constexpr (KEEP) {
                read(ka, kcol, t);
            }
            if constexpr (KEEP) {
                while (true) {
                    if (phase(kb)) return;
                    if (phase(ka)) return;
                }
            } else {
                while (!phase(ka)) {}
            }
        };
        auto load_state = [&](int n, int c) { return ld4x2(K0 + ((size_t)bh * N + n) * DK + cw * CW + c); };
        const f32x4 zero = {0ull, 0ull};
        f32x4 K4[NF / 4], K2[NF / 2], K1[NF];
        __syncthreads();                                  // the first rows are staged
        // below 8 rows; then 16, then 32: the pieces change lanes
        const int m0 = mode_of(lim);
        if (m0 == 4) {
#pragma unroll
            for (int i = 0; i < NF / 4; i++) {
                K4[i] = zero;
                if (CARRY && (lane & 7) < N) K4[i] = load_state(lane & 7, (lane >> 3) * (CW / 4) + 4 * i);
            }
            run(std::integral_constant<int, 4>(), K4);
        }
        if (!left && t < T && m0 >= 2) {
#pragma unroll
            for (int i = 0; i < NF / 2; i++) {
                K2[i] = zero;
                if (m0 == 4) {
                    const int src = (lane & 7) + 8 * (2 * (lane >> 4) + i / (NF / 4));
                    const f32x2 x = __shfl_sync(FULL, K4[i % (NF / 4)].a, src), y = __shfl_sync(FULL, K4[i % (NF / 4)].b, src);
                    if (!(lane & 8)) K2[i] = {x, y};      // rows 8 to 15: empty
                } else if (CARRY && (lane & 15) < N) {
                    K2[i] = load_state(lane & 15, (lane >> 4) * (CW / 2) + 4 * i);
                }
            }
            run(std::integral_constant<int, 2>(), K2);
        }
        if (!left && t < T) {
#pragma unroll
            for (int i = 0; i < NF; i++) {
                K1[i] = zero;
                if (m0 >= 2) {
                    const int src = (lane & 15) + 16 * (i / (NF / 2));
                    const f32x2 x = __shfl_sync(FULL, K2[i % (NF / 2)].a, src), y = __shfl_sync(FULL, K2[i % (NF / 2)].b, src);
                    if (!(lane & 16)) K1[i] = {x, y};     // rows 16 to 31: empty
                } else if (CARRY && lane < N) {
                    K1[i] = load_state(lane, 4 * i);
                }
            }
            run(std::integral_constant<int, 1>(), K1);
        }
        if (left && hand != nullptr) {                    // lane = row, as in every token since row 16 (the write of token t - 1 is open)
            float* d = hand + ((size_t)bh * N + lane) * DK + cw * CW;
#pragma unroll
            for (int i = 0; i < NF; i++) *reinterpret_cast<f32x4*>(d + 4 * i) = K1[i];
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ norm warp
        __syncthreads();
        __syncthreads();
        float kinv = fminf(rsqrtf((float)nsq), 1e6f);
        double hn = 0.0;                                  // this lane's row after a write of the token in work
        float2 hy = make_float2(0.f, 0.f);
        float g1 = 0.f, om1 = 0.f;
        int t = 0;
        bool left = false;
        // the row after a write of token u with <K, k_u> = R
        auto would = [&](int u, double R, float g, float om) {
            const float* tk = s_tok + AN_TOK * (u & (AN_RING - 1));
            const double2 d01 = *reinterpret_cast<const double2*>(tk + 8);
            hn = fmax(fma(d01.x, nsq, fma(d01.y, R, *reinterpret_cast<const double*>(tk + 12))), 0.0);
            hy = make_float2(fminf(rsqrtf((float)hn), 1e6f), __fmaf_rn(om, o, g));
            s_hyp[(u & 1) * AN_ROWS + lane] = hy;
        };
        // the write of token t - 1, and its log
        auto settle = [&](bool mine) {
            float* lg = s_oold + ((t - 1) & (AN_RING - 1));
            if (mine) {
                lg[0] = o;
                lg[AN_RING] = kinv;
            }
            nsq = mine ? hn : nsq;
            kinv = mine ? hy.x : kinv;
            o = mine ? hy.y : o;
        };
        auto none = [&](bool meet) {                      // no score compared greater: token t - 1 again, as if the dot were zero
            would(t - 1, 0.0, g1, om1);
            if (meet) AN_BAR(3, 64);
        };
        auto run = [&](auto fc) {                         // while the token's dots come in F parts
            constexpr int F = decltype(fc)::value;
            while (t < T) {
                const float* tk = s_tok + AN_TOK * (t & (AN_RING - 1));
                int a1 = t > 0 ? s_am[(t - 1) & (AN_RING - 1)] : -1;
                const float2 gg = *reinterpret_cast<const float2*>(tk + 14);
                const float x1 = tk[3];
                float R = an_sum<CTAS >= 3 ? 1 : F>(s_part + ((t & 1) * 2 + 1) * AN_PART, lane);
                bool more = t == 0;                       // the next token's dots may come in fewer parts
                if ((unsigned)a1 >= 0x40000000u && t > 0) {
                    if (a1 < 0) {
                        more = true;
                        if (++lim >= ncap) { left = true; return; }           // before the meeting below: the resolver has left too
                    }
                    if (a1 & 0x40000000) none(true);
                    a1 &= 0x3fffffff;
                }
                const bool mine = lane == a1;
                settle(mine);
                const float Rm = blend(R, x1, g1, om1);   // the dot has not seen that write
                R = mine ? Rm : R;
                would(t, (double)R, gg.x, gg.y);
                g1 = gg.x; om1 = gg.y;
                AN_PHASE_BARRIER();
                t++;
                if (F > 1 && more && min(lim + 1, N - 1) >= 32 / F) return;
            }
        };
        if (mode_of(lim0) == 4) run(std::integral_constant<int, 4>());
        if (!left && t < T && mode_of(t ? min(lim + 1, N - 1) : lim0) == 2) run(std::integral_constant<int, 2>());
        if (!left && t < T) run(std::integral_constant<int, 1>());
        const int a1 = s_am[(t - 1) & (AN_RING - 1)];     // the last token, or the one before it leaves
        if (a1 & 0x40000000) none(!left);
        settle(lane == (a1 & 0x3fffffff));
        if (lane < ncap && (!left || hand != nullptr)) {
            ofin[(size_t)bh * N + lane] = o;
            if (nsqfin != nullptr) nsqfin[(size_t)bh * N + lane] = nsq;
        }
    } else {
        // ------------------------------------------------------------------ resolver warp
        __syncthreads();
        __syncthreads();
        float kinv = fminf(rsqrtf((float)nsq), 1e6f), g1 = 0.f, om1 = 0.f;
        if (lane > lim) o = NAN;                          // a row above lim is neither occupied (which eps <= 0 makes every row) nor free
        const unsigned below = (1u << lane) - 1u;
        int t = 0, a1 = -1;                               // the previous token's address
        bool left = false, none = false;
        auto run = [&](auto fc) {                         // while the token's dots come in F parts
            constexpr int F = decltype(fc)::value;
            while (t < T) {
                const int sl = t & (AN_RING - 1);
                const float* tk = s_tok + AN_TOK * sl;
                const float4 c4 = ld4(tk);
                const float2 gg = *reinterpret_cast<const float2*>(tk + 14);
                float S = an_sum<CTAS >= 3 ? 1 : F>(s_part + (t & 1) * 2 * AN_PART, lane);
                if (none) AN_BAR(3, 64);                  // the norm warp took the previous token again
                const float2 hy = s_hyp[((t - 1) & 1) * AN_ROWS + lane];
                const bool mine = lane == a1;             // the one row whose latest write the dots have not seen
                const float Sm = blend(S, c4.z, g1, om1);
                S = mine ? Sm : S;
                kinv = mine ? hy.x : kinv;
                o = mine ? hy.y : o;
                const bool occ = o >= eps, isfree = o < eps;
                const unsigned fm = __ballot_sync(FULL, isfree);
                // product, product, difference, each rounded: as the direct kernel's expression comes out
                const float sc = __fmul_rn(c4.x, __fmul_rn(kinv, S));
                // (a penalty that is infinite or NaN is NaN on a row that is not occupied too: times zero, not left out)
                const float z = __fmaf_rn(-c4.y, OCCB ? (occ ? 1.f : 0.f) : o, sc);
                // candidates: occupied rows and the lowest free one
                const float zc = occ || (isfree && !(fm & below)) ? z : -INFINITY;
                const float zm = redux_max(zc);
                a1 = __ffs((int)__ballot_sync(FULL, zc == zm)) - 1;           // the lowest row of the largest score
                none = !(zm > -INFINITY);                 // no candidate compares greater (NaN scores): row lim
                if (none) a1 = lim;
                const bool fresh = a1 >= lim && lim < N - 1;                  // a row not written before: one more candidate
                s_am[sl] = a1 | (fresh ? (int)0x80000000 : 0) | (none ? 0x40000000 : 0);
                g1 = gg.x; om1 = gg.y;
                if ((t & 7) == 7) AN_BAR(2, 96);
                AN_PHASE_BARRIER();
                t++;
                const bool more = F > 1 && min(lim + 1, N - 1) >= 32 / F;     // token t's dots, taken before this address was known
                if (fresh) {
                    lim++;
                    if (lane == lim) o = 0.f;             // never written: from here on a candidate
                    if (lane == 0) tfirst[(size_t)bh * N + lim] = t;
                    if (t < T && lim >= ncap) {           // the next token may address a row this CTA does not hold
                        if (lane == 0) { tfirst[(size_t)bh * N] = af_mark(hand != nullptr ? t : 0); *s_leave = t; }
                        __syncwarp();
                        if ((t | 7) < T) AN_BAR(2, 96);   // the loaders come to it
                        left = true;
                        return;
                    }
                }
                if (more) return;
            }
        };
        if (mode_of(lim0) == 4) run(std::integral_constant<int, 4>());
        if (!left && t < T && !(t == 0 && mode_of(lim0) == 1)) run(std::integral_constant<int, 2>());
        if (!left && t < T) run(std::integral_constant<int, 1>());
        if (!left && none) AN_BAR(3, 64);
    }
    __syncthreads();
    const int Tn = *s_leave ? *s_leave : T;               // tokens whose log is complete
    if (Tn == T) for (int i = ncap + tid; i < N; i += AN_THREADS) {                // rows this pass never held
        ofin[(size_t)bh * N + i] = 0.f;
        if (nsqfin != nullptr) nsqfin[(size_t)bh * N + i] = 0.0;
    }
    {   // log entries not written out yet (the loaders' last turn was in the chunk of the token in work)
        const int t = max((*s_leave ? Tn : T - 1) / AN_L * AN_L - 2, 0) + tid;
        if (t < Tn) {
            const size_t ix = ((size_t)b * T + t) * H + h;
            const int sl = t & (AN_RING - 1);
            am_out[ix] = s_am[sl] & 0x3fffffff;
            oold_out[ix] = s_oold[sl];
            kiold_out[ix] = s_kiold[sl];
        }
    }
#undef AN_BAR
#undef AN_PHASE_BARRIER
}

}  // namespace slotscan
