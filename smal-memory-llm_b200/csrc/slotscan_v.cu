// Keyless slot scan: the address logits come from outside, the state holds values only.
//   [reference gqa25/slotkern_v.py: definition ref_scan_v :242-261, Triton kernels _vfwd :25, _vrecompute :75,
//    _vadjoint :120, adjoint stated in the module docstring :14-19]
//
//   z = wa_t - fr o over ALL N rows (no free-row mask),  a_s = softmax(z),  a = onehot(argmax z) if hard else a_s,
//   g_h = [g > 0.5] if hard_gate else g,  w = g_h a,  V <- (1 - w) V + w v_t,  o <- (1 - w) o + w;
//   the pre-write V goes out every G tokens.  Backward (straight-through for the hard address and the hard gate):
//   dw = <v - V, dV'> + (1 - o) do',  dv = sum_n w dV',  dg = a . dw,  dz = a_s (g_h dw - a_s . g_h dw),  dwa = dz,
//   dfr -= o . dz,  dV = (1 - w) dV' + dbuf,  do = (1 - w) do' - fr dz.
//
// The address of a token depends on the occupancies alone, never on the values, and the values are linear in the known
// addresses.  Only the occupancy recurrence is a chain over the tokens; everything that is wide is split off from it:
//   forward   one warp per (sequence, head) runs the occupancies (rows in registers, 2 per lane at 64 rows) and hands the
//             write weights over in chunks of tokens; eight warps of the same CTA apply them to the values, a chunk behind
//   backward  the addresses again from the emitted occupancies, every block of G tokens at once (keyless_tables); the
//             value gradients block by block (row_adjoint_kernel); then the chain of the occupancy gradient alone, one
//             warp per (sequence, head) (keyless_bwd_chain)
// Bound: the occupancy chain, one double-precision exp, sum over the rows and division per token.  B = 8, T = 512, H = 8,
// 64 x 64, G = 4, forward + backward: 12.9 ms walking token by token in one CTA (2.35 + 10.4), 0.85 ms split (forward 0.39;
// backward: tables 0.02, value gradients 0.29, chain 0.12).
// The occupancies and the softmax run in double: with the penalty on o itself every rounding error of o comes back
// multiplied by fr at every later token.
// More than 256 rows (the reference's shape is 48 x 16) keep the kernels below that hold everything in one CTA and walk
// token by token.
#include <math.h>
#include <stdio.h>

#include <algorithm>

#include "slotscan_common.cuh"
#include "slotscan_launch.h"
#include "slotscan_rowadj.cuh"

namespace slotscan {

constexpr int KV_THREADS = 128, KV_WARPS = KV_THREADS / 32;


// One warp: address of a token from its logits and the occupancies.  z[n] (double scratch) is overwritten.
// Returns the argmax (first maximum); asoft / afwd receive the softmax and the address the forward uses.
template <typename TO>
__device__ __forceinline__ int keyless_address(const float* wa_t, const TO* o, int N, double fr, int hard, double* z,
                                               float* asoft, float* afwd) {
    const int lane = threadIdx.x & 31;
    double bz = -INFINITY;
    int bi = BIGI;
    for (int n = lane; n < N; n += 32) {
        const double zz = (double)wa_t[n] - fr * (double)o[n];
        z[n] = zz;
        if (zz > bz) { bz = zz; bi = n; }
    }
    double zmax = bz;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) zmax = fmax(zmax, __shfl_xor_sync(FULL, zmax, off));
    int am = (int)__reduce_min_sync(FULL, (unsigned)((bi != BIGI && bz == zmax) ? bi : BIGI));
    am = min(am, N - 1);
    double se = 0.0;
    for (int n = lane; n < N; n += 32) { const double e = exp(z[n] - zmax); z[n] = e; se += e; }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) se += __shfl_xor_sync(FULL, se, off);
    for (int n = lane; n < N; n += 32) {
        const float a = (float)(z[n] / se);
        asoft[n] = a;
        afwd[n] = hard ? (n == am ? 1.f : 0.f) : a;
    }
    __syncwarp();
    return am;
}

__host__ __device__ inline size_t keyless_fwd_smem_floats(int N, int DV) { return (size_t)N * DV + 8 * (size_t)N + DV + 32; }
__host__ __device__ inline size_t keyless_bwd_smem_floats(int N, int DV) { return (size_t)N * DV + 10 * (size_t)N + DV + 64; }
__host__ __device__ inline size_t keyless_state_floats(int N, int DV) { return (size_t)N * (DV + 1); }

template <typename Tin>
__global__ void __launch_bounds__(KV_THREADS) keyless_fwd_kernel(const slotscan_v_params p, const Tin* __restrict__ v,
                                                                 const float* __restrict__ wa,
                                                                 const float* __restrict__ gate,
                                                                 const float* __restrict__ fr_p, float* __restrict__ buf,
                                                                 float* __restrict__ obuf, int* __restrict__ addr) {
    extern __shared__ __align__(16) float ksm[];
    const int N = p.N, T = p.T, H = p.H, DV = p.DV, G = p.G;
    const int NB = (T + G - 1) / G, NE = (N + 1) & ~1;
    double* z = reinterpret_cast<double*>(ksm);             // [N]
    double* o = z + NE;                                     // [N]
    float* V = ksm + 4 * (size_t)NE;
    float* a = V + (size_t)N * DV;
    float* as = a + N;
    float* wt = as + N;                                     // this token's logits
    float* vt = wt + N;
    float* s_f = vt + DV;                                   // [0] g_h
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, warp = tid >> 5;
    const double fr = (double)fr_p[0];
    for (int i = tid; i < N * DV; i += KV_THREADS) V[i] = 0.f;
    for (int i = tid; i < N; i += KV_THREADS) o[i] = 0.0;
    __syncthreads();
    for (int t = 0; t < T; t++) {
        const size_t ix = ((size_t)b * T + t) * H + h;
        if (t % G == 0) {
            const size_t so = ((size_t)b * NB + t / G) * H + h;
            for (int i = tid; i < N * DV; i += KV_THREADS) buf[so * N * DV + i] = V[i];
            for (int i = tid; i < N; i += KV_THREADS) obuf[so * N + i] = (float)o[i];
        }
        for (int n = tid; n < N; n += KV_THREADS) wt[n] = wa[ix * N + n];
        for (int d = tid; d < DV; d += KV_THREADS) vt[d] = ld1(v + ix * DV + d);
        __syncthreads();
        if (warp == 0) {
            const int am = keyless_address(wt, o, N, fr, p.hard, z, as, a);
            const float g = gate_eff(gate[ix], p.hard_gate);
            for (int n = (tid & 31); n < N; n += 32) {
                const double w = (double)g * (double)a[n];
                if (a[n] != 0.f) o[n] = (1.0 - w) * o[n] + w;
            }
            if (tid == 0) {
                s_f[0] = g;
                if (addr != nullptr) addr[ix] = am;
            }
        }
        __syncthreads();
        const float g = s_f[0];
        for (int n = tid >> 5; n < N; n += KV_THREADS / 32) {      // a warp per row, lanes over the columns
            const float an = a[n];
            if (an == 0.f) continue;
            const float w = g * an;
            float* Vr = V + (size_t)n * DV;
            for (int d = tid & 31; d < DV; d += 32) Vr[d] = (1.f - w) * Vr[d] + w * vt[d];
        }
        __syncthreads();
    }
}

template <typename Tin>
__global__ void __launch_bounds__(KV_THREADS) keyless_bwd_kernel(const slotscan_v_params p, const Tin* __restrict__ v,
                                                                 const float* __restrict__ wa,
                                                                 const float* __restrict__ gate,
                                                                 const float* __restrict__ fr_p,
                                                                 const float* __restrict__ buf,
                                                                 const float* __restrict__ obuf,
                                                                 const float* __restrict__ dbuf, float* __restrict__ seg,
                                                                 Tin* __restrict__ dv, float* __restrict__ dwa,
                                                                 float* __restrict__ dgate, float* __restrict__ part) {
    extern __shared__ __align__(16) float ksm[];
    const int N = p.N, T = p.T, H = p.H, DV = p.DV, G = p.G;
    const int NB = (T + G - 1) / G, NE = (N + 1) & ~1;
    double* z = reinterpret_cast<double*>(ksm);             // [N]
    float* dV = ksm + 2 * (size_t)NE;
    float* dO = dV + (size_t)N * DV;
    float* a = dO + N;
    float* as = a + N;
    float* wt = as + N;
    float* dw = wt + N;
    float* dz = dw + N;
    float* vt = dz + N;
    float* s_f = vt + DV;                                   // [0] g_h
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double fr = (double)fr_p[0];
    const float frf = fr_p[0];
    const size_t SV = (size_t)N * DV, SS = keyless_state_floats(N, DV);
    float* myseg = seg + (size_t)bh * G * SS;               // slot j: state before token t0 + j (slot 0 unused: the snapshot)
    for (size_t i = tid; i < SV; i += KV_THREADS) dV[i] = 0.f;
    for (int i = tid; i < N; i += KV_THREADS) dO[i] = 0.f;
    float dfr_acc = 0.f;                                    // lane 0 of warp 0
    __syncthreads();
    for (int jb = NB - 1; jb >= 0; jb--) {
        const int t0 = jb * G, cn = min(G, T - t0);
        const size_t so = ((size_t)b * NB + jb) * H + h;
        auto stV = [&](int j) -> const float* { return j == 0 ? buf + so * SV : myseg + (size_t)j * SS; };
        auto stO = [&](int j) -> const float* { return j == 0 ? obuf + so * N : myseg + (size_t)j * SS + SV; };
        for (int j = 0; j + 1 < cn; j++) {                  // replay: slot j + 1 from slot j
            const size_t ix = ((size_t)b * T + t0 + j) * H + h;
            const float *Vp = stV(j), *op = stO(j);
            float* Vn = myseg + (size_t)(j + 1) * SS;
            float* on = Vn + SV;
            for (int n = tid; n < N; n += KV_THREADS) wt[n] = wa[ix * N + n];
            for (int d = tid; d < DV; d += KV_THREADS) vt[d] = ld1(v + ix * DV + d);
            __syncthreads();
            if (warp == 0) {
                keyless_address(wt, op, N, fr, p.hard, z, as, a);
                if (lane == 0) s_f[0] = gate_eff(gate[ix], p.hard_gate);
            }
            __syncthreads();
            const float g = s_f[0];
            for (int n = tid >> 5; n < N; n += KV_THREADS / 32) {  // a warp per row; the row's loads first (global memory)
                const bool hit = a[n] != 0.f;
                const float w = hit ? g * a[n] : 0.f;
                for (int d0 = 0; d0 < DV; d0 += 128) {         // 128 columns at a time, four loads per lane in flight
                    float vx[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) { const int d = d0 + (tid & 31) + 32 * c; vx[c] = d < DV ? Vp[(size_t)n * DV + d] : 0.f; }
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const int d = d0 + (tid & 31) + 32 * c;
                        if (d < DV) Vn[(size_t)n * DV + d] = hit ? (1.f - w) * vx[c] + w * vt[d] : vx[c];
                    }
                }
            }
            for (int n = tid; n < N; n += KV_THREADS) {
                float x = op[n];
                if (a[n] != 0.f) { const float w = g * a[n]; x = (1.f - w) * x + w; }
                on[n] = x;
            }
            __syncthreads();
        }
        for (int j = cn - 1; j >= 0; j--) {                 // the block in reverse
            const size_t ix = ((size_t)b * T + t0 + j) * H + h;
            const float *Vp = stV(j), *op = stO(j);
            for (int n = tid; n < N; n += KV_THREADS) wt[n] = wa[ix * N + n];
            for (int d = tid; d < DV; d += KV_THREADS) vt[d] = ld1(v + ix * DV + d);
            __syncthreads();
            for (int n = warp; n < N; n += KV_WARPS) {      // dw_n = <v - V_n, dV_n> + (1 - o_n) dO_n
                float a1 = 0.f;
                for (int d = lane; d < DV; d += 32) a1 = fmaf(vt[d] - Vp[(size_t)n * DV + d], dV[(size_t)n * DV + d], a1);
                a1 = warp_sum(a1);
                if (lane == 0) dw[n] = a1 + (1.f - op[n]) * dO[n];
            }
            __syncthreads();
            if (warp == 0) {
                keyless_address(wt, op, N, fr, p.hard, z, as, a);
                const float g = gate_eff(gate[ix], p.hard_gate);
                float dg = 0.f, sa = 0.f;
                for (int n = lane; n < N; n += 32) { dg = fmaf(a[n], dw[n], dg); sa = fmaf(as[n], g * dw[n], sa); }
                dg = warp_sum(dg);
                sa = warp_sum(sa);
                float f1 = 0.f;
                for (int n = lane; n < N; n += 32) {
                    const float zz = as[n] * (g * dw[n] - sa);
                    dz[n] = zz;
                    dwa[ix * N + n] = zz;
                    f1 = fmaf(-op[n], zz, f1);
                }
                f1 = warp_sum(f1);
                if (lane == 0) { dgate[ix] = dg; dfr_acc += f1; s_f[0] = g; }
            }
            __syncthreads();
            const float g = s_f[0];
            for (int d = tid; d < DV; d += KV_THREADS) {    // dv_t = sum_n w_n dV_n (before dV moves to the pre-write side)
                float acc = 0.f;
                for (int n = 0; n < N; n++)
                    if (a[n] != 0.f) acc = fmaf(g * a[n], dV[(size_t)n * DV + d], acc);
                st1(dv + ix * DV + d, acc);
            }
            __syncthreads();
            const bool emit = (j == 0);
            for (int n = tid >> 5; n < N; n += KV_THREADS / 32) {
                const float om = 1.f - g * a[n];
                for (int d = tid & 31; d < DV; d += 32) {
                    const size_t i = (size_t)n * DV + d;
                    float x = om * dV[i];
                    if (emit && dbuf != nullptr) x += dbuf[so * SV + i];
                    dV[i] = x;
                }
            }
            for (int n = tid; n < N; n += KV_THREADS) dO[n] = (1.f - g * a[n]) * dO[n] - frf * dz[n];
            __syncthreads();
        }
    }
    if (tid == 0) part[bh] = dfr_acc;
}

__global__ void __launch_bounds__(256) keyless_finish_kernel(const float* __restrict__ part, int n, float* dfr) {
    __shared__ float s_a[256];
    float a = 0.f;
    for (int i = threadIdx.x; i < n; i += 256) a += part[i];
    s_a[threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        a = 0.f;
        for (int i = 0; i < 256; i++) a += s_a[i];          // fixed order: bitwise repeatable
        dfr[0] = a;
    }
}

// ---- up to 256 rows: lane l of a warp holds rows l, l + 32, ... ----
constexpr int KL_CT = 16;                                   // tokens per chunk handed from the chain to the value warps
constexpr int KL_CW = 8;                                    // value warps

// e[i] = exp(z_n - max z), returns the sum over the rows; am: the first row of the largest z.  zmax over finite and
// infinite z alike; a NaN never wins, as in the token-by-token kernels.
template <int R>
__device__ __forceinline__ double kl_softmax(const float (&wa)[R], const double (&o)[R], int N, double fr, double (&e)[R],
                                             int& am, bool soft = true) {
    const int lane = threadIdx.x & 31;
    double bz = -INFINITY;
    int bi = BIGI;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int n = lane + 32 * i;
        e[i] = (double)wa[i] - fr * o[i];
        if (n < N && e[i] > bz) { bz = e[i]; bi = n; }
    }
    // largest z through its order-preserving 64-bit key: two integer warp maxima instead of five 64-bit shuffle rounds
    const long long zb = __double_as_longlong(bz + 0.0);    // -0 -> +0: equal values have one key
    const unsigned long long key = (unsigned long long)(zb ^ ((zb >> 63) | (long long)0x8000000000000000ull));
    const unsigned hi = (unsigned)(key >> 32), mhi = __reduce_max_sync(FULL, hi);
    const unsigned mlo = __reduce_max_sync(FULL, hi == mhi ? (unsigned)key : 0u);
    const bool mine = hi == mhi && (unsigned)key == mlo;
    const unsigned long long mk = ((unsigned long long)mhi << 32) | mlo;
    const double zmax = __longlong_as_double((mk >> 63) ? (long long)(mk ^ 0x8000000000000000ull) : (long long)~mk);
    am = min((int)__reduce_min_sync(FULL, (unsigned)((bi != BIGI && mine) ? bi : BIGI)), N - 1);
    if (!soft) return 1.0;                                  // the argmax is all that is asked for
    double se = 0.0;
#pragma unroll
    for (int i = 0; i < R; i++) {
        if (lane + 32 * i < N) { e[i] = exp(e[i] - zmax); se += e[i]; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) se += __shfl_xor_sync(FULL, se, off);
    return se;
}

// Warp 0: the chain.  Warp 1: what of a token's address does not depend on the occupancies -- exp(wa_n - max wa), a chunk
// ahead -- so that the chain is exp(-fr o_n), one sum, one reciprocal and the blend.  Warps 2..9: the values, a chunk
// behind.  The factors neither overflow nor vanish while |fr| <= 300 and the gates stay in [0, 1] (o in [0, 1]); anything
// else takes the shifted softmax of kl_softmax.  hard: the chain needs the largest wa_n - fr o_n only.
template <typename Tin, int R, int MINB>
__global__ void __launch_bounds__(32 * (2 + KL_CW), MINB) keyless_fwd_chain_kernel(
    const slotscan_v_params p, const Tin* __restrict__ v, const float* __restrict__ wa, const float* __restrict__ gate,
    const float* __restrict__ fr_p, float* __restrict__ buf, float* __restrict__ obuf, int* __restrict__ addr) {
    extern __shared__ __align__(16) float ksm[];
    constexpr int NR = 32 * R;
    const int N = p.N, T = p.T, H = p.H, DV = p.DV, G = p.G, NB = (T + G - 1) / G;
    const int N4 = (N + 3) & ~3, NG = N4 / 4;
    double* X = reinterpret_cast<double*>(ksm);             // [2][KL_CT][NR] exp(wa - max wa); hard: wa
    float* gs = reinterpret_cast<float*>(X + 2 * KL_CT * NR);        // [2][KL_CT] gates
    int* wild = reinterpret_cast<int*>(gs + 2 * KL_CT);     // [2] a gate of the chunk lies outside [0, 1]
    int* soft_chunk = wild + 2;                             // [2] the chunk's factors are in X
    float* wbuf = gs + 2 * KL_CT + 4;                       // [2][KL_CT][N4] write weights, 0 = row not written
    float* V = wbuf + 2 * KL_CT * N4;                       // [N4][DV]
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ct = tid - 64;
    const double fr = (double)fr_p[0];
    const int NC = (T + KL_CT - 1) / KL_CT;
    double o[R], e[R];
#pragma unroll
    for (int i = 0; i < R; i++) o[i] = 0.0;
    bool slow = !(fabs(fr) <= 300.0);
    int ph = 0, jb = 0;                                     // chain: token's place in its block, block
    for (int i = ct; i < N4 * DV && ct >= 0; i += 32 * KL_CW) V[i] = 0.f;
    // value threads: column and first group of four rows; with more columns than threads every thread walks all rows
    const int per = DV <= 32 * KL_CW ? 32 * KL_CW / DV : 1;
    const int dl = ct < 0 ? 0 : (DV <= 32 * KL_CW ? ct % DV : ct), gl = ct < 0 || DV > 32 * KL_CW ? 0 : ct / DV;
    const int gstep = per, NGt = gl < per ? NG : 0;                // threads past the last whole set of columns idle
    float xn[KL_CT];
    auto fetch_v = [&](int t0) {
#pragma unroll
        for (int j = 0; j < KL_CT; j++) xn[j] = t0 + j < T ? ld1(v + (((size_t)b * T + t0 + j) * H + h) * DV + dl) : 0.f;
    };
    if (ct >= 0 && DV <= 32 * KL_CW) fetch_v(0);
    for (int c = -1; c <= NC; c++) {
        if (warp == 0) {
            if (c >= 0 && c < NC) {
                float* wr = wbuf + (c & 1) * KL_CT * N4;
                const double* Xc = X + (c & 1) * KL_CT * NR + lane;
                double* Xw = X + (c & 1) * KL_CT * NR + lane;
                slow |= wild[c & 1] != 0;
                const int cn = min(KL_CT, T - c * KL_CT);
                for (int j = 0; j < cn; j++) {
                    const size_t ix = ((size_t)b * T + c * KL_CT + j) * H + h;
                    const float g = gs[(c & 1) * KL_CT + j];
                    if (ph == 0) {
                        const size_t so = ((size_t)b * NB + jb) * H + h;
#pragma unroll
                        for (int i = 0; i < R; i++) if (lane + 32 * i < N) obuf[so * N + lane + 32 * i] = (float)o[i];
                    }
                    if (++ph == G) { ph = 0; jb++; }
                    int am = 0;
                    double si;
                    if (slow || p.hard) {
                        float la[R];
#pragma unroll
                        for (int i = 0; i < R; i++) la[i] = lane + 32 * i < N ? (p.hard ? (float)Xc[j * NR + 32 * i] : wa[ix * N + lane + 32 * i]) : 0.f;
                        si = 1.0 / kl_softmax<R>(la, o, N, fr, e, am, !p.hard);
                    } else {
                        double se = 0.0;
#pragma unroll
                        for (int i = 0; i < R; i++) {
                            e[i] = Xc[j * NR + 32 * i] * exp(-fr * o[i]);          // rows past N: X = 0
                            se += e[i];
                        }
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1) se += __shfl_xor_sync(FULL, se, off);
                        si = rcp_normal(se);
                    }
#pragma unroll
                    for (int i = 0; i < R; i++) {
                        const int n = lane + 32 * i;
                        const float a = p.hard ? (n == am ? 1.f : 0.f) : (float)(e[i] * si);
                        const double w = (double)g * (double)a;
                        if (a != 0.f) o[i] = (1.0 - w) * o[i] + w;
                        if (n < N4) wr[j * N4 + n] = n < N ? g * a : 0.f;
                    }
                    if (p.hard || slow) {
                        if (lane == 0 && addr != nullptr) addr[ix] = am;
                    } else {                                         // the factors, for warp 1 to find the largest of
#pragma unroll
                        for (int i = 0; i < R; i++) Xw[j * NR + 32 * i] = e[i];
                    }
                }
                if (lane == 0) soft_chunk[c & 1] = !(p.hard || slow);
            }
        } else if (warp == 1) {
            if (c >= 1 && addr != nullptr && soft_chunk[(c - 1) & 1]) {      // the address of the chunk before, for the caller's log
                const int cn = min(KL_CT, T - (c - 1) * KL_CT);
                for (int j = 0; j < cn; j++) {
                    const double* E = X + ((c - 1) & 1) * KL_CT * NR + j * NR + lane;
                    double be = -1.0;
                    int bi = BIGI;
#pragma unroll
                    for (int i = 0; i < R; i++) if (lane + 32 * i < N && E[32 * i] > be) { be = E[32 * i]; bi = lane + 32 * i; }
                    const unsigned hi = (unsigned)(__double_as_longlong(be) >> 32) ^ 0x80000000u, lo = (unsigned)__double_as_longlong(be);
                    const unsigned mhi = __reduce_max_sync(FULL, hi), mlo = __reduce_max_sync(FULL, hi == mhi ? lo : 0u);
                    const int am = min((int)__reduce_min_sync(FULL, (unsigned)(hi == mhi && lo == mlo ? bi : BIGI)), N - 1);
                    if (lane == 0) addr[((size_t)b * T + (c - 1) * KL_CT + j) * H + h] = am;
                }
                __syncwarp();
            }
            if (c + 1 < NC) {
                const int bf = (c + 1) & 1, t0 = (c + 1) * KL_CT;
                double* Xc = X + bf * KL_CT * NR + lane;
                if (lane < KL_CT) {
                    const float g = t0 + lane < T ? gate_eff(gate[((size_t)b * T + t0 + lane) * H + h], p.hard_gate) : 0.f;
                    gs[bf * KL_CT + lane] = g;
                    const unsigned any = __ballot_sync(0xffffu, !(g >= 0.f && g <= 1.f));
                    if (lane == 0) wild[bf] = any != 0u;
                }
                for (int j = 0; j < KL_CT; j += 4) {                 // four tokens' loads in flight
                    float la[4][R];
#pragma unroll
                    for (int u = 0; u < 4; u++)
#pragma unroll
                        for (int i = 0; i < R; i++)
                            la[u][i] = (t0 + j + u < T && lane + 32 * i < N) ? wa[(((size_t)b * T + t0 + j + u) * H + h) * N + lane + 32 * i] : -INFINITY;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        float m = -INFINITY;
#pragma unroll
                        for (int i = 0; i < R; i++) m = fmaxf(m, la[u][i]);
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, off));
#pragma unroll
                        for (int i = 0; i < R; i++)
                            Xc[(j + u) * NR + 32 * i] = p.hard ? (double)la[u][i] : (lane + 32 * i < N ? exp((double)la[u][i] - (double)m) : 0.0);
                    }
                }
            }
        } else if (c > 0) {
            const int t0 = (c - 1) * KL_CT, cn = min(KL_CT, T - t0), ph0 = t0 % G, jb0 = t0 / G;
            const float* wr = wbuf + ((c - 1) & 1) * KL_CT * N4;
            // a thread keeps its column, so that a token's value is loaded once for all its rows, a chunk ahead of its use;
            // 4 rows at a time
            for (int d = dl; d < DV; d += 32 * KL_CW) {
                float xv[KL_CT];
                bool odd = p.hard != 0;                            // a row a token does not write must not see it: only an
#pragma unroll
                for (int j = 0; j < KL_CT; j++) {                  // infinite or NaN value would tell
                    xv[j] = DV <= 32 * KL_CW ? xn[j] : (j < cn ? ld1(v + (((size_t)b * T + t0 + j) * H + h) * DV + d) : 0.f);
                    odd |= !(fabsf(xv[j]) <= 3e38f);
                }
                if (DV <= 32 * KL_CW) fetch_v(t0 + KL_CT);
                for (int ng = gl; ng < NGt; ng += gstep) {
                    const int n0 = ng * 4;
                    float s[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) s[i] = V[(n0 + i) * DV + d];
                    int q = ph0, k = jb0;
#pragma unroll
                    for (int j = 0; j < KL_CT; j++) {
                        if (j < cn) {
                            if (q == 0) {                          // the pre-write state, every G tokens
                                float* out = buf + ((((size_t)b * NB + k) * H + h) * N + n0) * DV + d;
#pragma unroll
                                for (int i = 0; i < 4; i++) if (n0 + i < N) out[(size_t)i * DV] = s[i];
                            }
                            if (++q == G) { q = 0; k++; }
                            const float4 w = ld4(wr + j * N4 + n0);
                            const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const float t = fmaf(wv[i], xv[j], (1.f - wv[i]) * s[i]);
                                s[i] = odd && wv[i] == 0.f ? s[i] : t;
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) V[(n0 + i) * DV + d] = s[i];
                }
            }
        }
        __syncthreads();
    }
}

// The backward's tables: a warp per (sequence, block) runs the block's tokens from the emitted occupancies.
template <int R>
__global__ void __launch_bounds__(128) keyless_tables_kernel(const slotscan_v_params p, const float* __restrict__ wa,
                                                             const float* __restrict__ gate, const float* __restrict__ fr_p,
                                                             const float* __restrict__ obuf, int bh0, int nbh,
                                                             float* __restrict__ as, float* __restrict__ ot, int* __restrict__ am) {
    const int N = p.N, T = p.T, H = p.H, G = p.G, NB = (T + G - 1) / G, lane = threadIdx.x & 31;
    const size_t wid = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (wid >= (size_t)nbh * NB) return;
    const int lb = (int)(wid / NB), jb = (int)(wid % NB), bh = bh0 + lb, b = bh / H, h = bh % H;
    const int t0 = jb * G, t1 = min(T, t0 + G);
    const double fr = (double)fr_p[0];
    const size_t so = ((size_t)b * NB + jb) * H + h;
    double o[R], e[R];
    float cur[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int n = lane + 32 * i;
        o[i] = n < N ? (double)obuf[so * N + n] : 0.0;
        cur[i] = n < N ? wa[(((size_t)b * T + t0) * H + h) * N + n] : 0.f;
    }
    for (int t = t0; t < t1; t++) {
        const size_t ix = ((size_t)b * T + t) * H + h;
        float la[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int n = lane + 32 * i;
            la[i] = cur[i];
            cur[i] = (t + 1 < t1 && n < N) ? wa[(ix + H) * N + n] : 0.f;
        }
        int m;
        const double si = 1.0 / kl_softmax<R>(la, o, N, fr, e, m);
        const float g = gate_eff(gate[ix], p.hard_gate);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int n = lane + 32 * i;
            if (n < N) {
                const float s = (float)(e[i] * si), a = p.hard ? (n == m ? 1.f : 0.f) : s;
                as[((size_t)lb * T + t) * N + n] = s;
                ot[((size_t)lb * T + t) * N + n] = (float)o[i];
                const double w = (double)g * (double)a;
                if (a != 0.f) o[i] = (1.0 - w) * o[i] + w;
            }
        }
        if (lane == 0) am[(size_t)lb * T + t] = m;
    }
}

// The chain of the backward: the occupancy gradient, token by token in reverse.  D: <v_t - V_n(t), dV_n> per token and row.
template <int R>
__global__ void __launch_bounds__(32) keyless_bwd_chain_kernel(const slotscan_v_params p, const float* __restrict__ gate,
                                                               const float* __restrict__ fr_p, const float* __restrict__ as,
                                                               const float* __restrict__ ot, const int* __restrict__ am,
                                                               const float* __restrict__ D, int bh0,
                                                               float* __restrict__ dwa, float* __restrict__ dgate,
                                                               float* __restrict__ part) {
    constexpr int PF = R <= 2 ? 8 : (R == 4 ? 4 : 2);       // tokens in flight
    const int N = p.N, T = p.T, H = p.H, lane = threadIdx.x;
    const int lb = blockIdx.x, bh = bh0 + lb, b = bh / H, h = bh % H;
    const float fr = fr_p[0];
    const bool hard = p.hard != 0;
    const size_t tab = (size_t)lb * T * N + lane;
    as += tab; ot += tab; D += tab;
    dwa += ((size_t)b * T * H + h) * N + lane;
    gate += (size_t)b * T * H + h;
    dgate += (size_t)b * T * H + h;
    am += (size_t)lb * T;
    float dO[R], ca[PF][R], co[PF][R], cd[PF][R];
    double f1 = 0.0;
#pragma unroll
    for (int i = 0; i < R; i++) dO[i] = 0.f;
    auto fetch = [&](int u, int t) {
        const size_t at = (size_t)t * N;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const bool in = t >= 0 && lane + 32 * i < N;    // rows past N: all zero, they add nothing below
            ca[u][i] = in ? as[at + 32 * i] : 0.f;
            co[u][i] = in ? ot[at + 32 * i] : 0.f;
            cd[u][i] = in ? D[at + 32 * i] : 0.f;
        }
    };
#pragma unroll
    for (int u = 0; u < PF; u++) fetch(u, T - 1 - u);
    for (int tw = T - 1; tw >= 0; tw -= 32) {               // gates and addresses of 32 tokens, one per lane
        const float gl = tw - lane >= 0 ? gate_eff(gate[(size_t)(tw - lane) * H], p.hard_gate) : 0.f;
        const int ml = (hard && tw - lane >= 0) ? am[tw - lane] : 0;
        float dgl = 0.f;
        for (int tb = 0; tb < 32 && tb <= tw; tb += PF) {
#pragma unroll
            for (int u = 0; u < PF; u++) {
                const int t = tw - tb - u;
                const float g = __shfl_sync(FULL, gl, tb + u);
                const int m = hard ? __shfl_sync(FULL, ml, tb + u) : 0;
                float dw[R], a[R], dg = 0.f, sa = 0.f;
#pragma unroll
                for (int i = 0; i < R; i++) {
                    dw[i] = fmaf(1.f - co[u][i], dO[i], cd[u][i]);
                    a[i] = hard ? (lane + 32 * i == m ? 1.f : 0.f) : ca[u][i];
                    dg = fmaf(a[i], dw[i], dg);
                    sa = fmaf(ca[u][i], g * dw[i], sa);
                }
                dg = warp_sum(dg);
                sa = hard ? warp_sum(sa) : g * dg;
#pragma unroll
                for (int i = 0; i < R; i++) {
                    const float z = ca[u][i] * (g * dw[i] - sa);
                    if (t >= 0 && lane + 32 * i < N) dwa[(size_t)t * H * N + 32 * i] = z;
                    f1 -= (double)co[u][i] * (double)z;
                    dO[i] = fmaf(1.f - g * a[i], dO[i], -fr * z);
                }
                if (lane == tb + u) dgl = dg;
                fetch(u, t - PF);
            }
        }
        if (tw - lane >= 0) dgate[(size_t)(tw - lane) * H] = dgl;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) f1 += __shfl_xor_sync(FULL, f1, off);
    if (lane == 0) part[bh] = (float)f1;
}

// scratch of the split backward: the tables of `nbh` sequences at a time (as many as 2 GiB hold), then the sums
struct KeylessScratch { size_t as, ot, am, dp, part, bytes; int nbh, nsl; };
inline KeylessScratch keyless_scratch(const slotscan_v_params& p) {
    KeylessScratch s;
    const size_t BH = (size_t)p.B * p.H, tn = (size_t)p.T * p.N;
    s.nsl = row_adjoint_slices(p.N, p.DV);
    const size_t per = 4 * (tn * (2 + s.nsl) + p.T);
    s.nbh = (int)std::min(std::min(BH, (size_t)65535), std::max((size_t)1, ((size_t)2 << 30) / per));
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    s.as = 0;
    s.ot = up(4 * tn * s.nbh);
    s.dp = 2 * s.ot;
    s.am = s.dp + up(4 * tn * s.nbh * s.nsl);
    s.part = s.am + up(4 * (size_t)p.T * s.nbh);
    s.bytes = s.part + 4 * BH;
    return s;
}
inline size_t keyless_chain_smem(int N, int DV) {
    const size_t n4 = (N + 3) & ~3, nr = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
    return 8 * (2 * KL_CT * nr) + 4 * (2 * KL_CT + 4 + 2 * KL_CT * n4 + n4 * DV);
}
// the split kernels: rows in one warp's registers, and the forward's chunk of weights beside the values
inline bool keyless_split(const slotscan_v_params& p) {
    return p.N <= 256 && keyless_chain_smem(p.N, p.DV) <= 227 * 1024 && row_adjoint_slices(p.N, p.DV) <= 64;
}
#define KEYLESS_ROWS(N_, ...)                                \
    if ((N_) <= 32) { constexpr int R = 1; __VA_ARGS__; }           \
    else if ((N_) <= 64) { constexpr int R = 2; __VA_ARGS__; }      \
    else if ((N_) <= 128) { constexpr int R = 4; __VA_ARGS__; }     \
    else { constexpr int R = 8; __VA_ARGS__; }

template <typename Tin>
cudaError_t run_keyless_fwd(const slotscan_v_params& p, const Tin* v, const float* wa, const float* gate, const float* fr,
                            float* buf, float* obuf, int* addr, cudaStream_t st) {
    const size_t sm = keyless_chain_smem(p.N, p.DV);
    cudaError_t e = cudaSuccess;
    // one CTA per SM at most: registers for the value warps' loads ahead (0.43 ms where the form for two has 0.50)
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool alone = (long long)p.B * p.H <= sms;
    KEYLESS_ROWS(p.N, {
        auto kern = alone ? keyless_fwd_chain_kernel<Tin, R, 1> : keyless_fwd_chain_kernel<Tin, R, 2>;
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return e;
        kern<<<p.B * p.H, 32 * (2 + KL_CW), sm, st>>>(p, v, wa, gate, fr, buf, obuf, addr);
    });
    return cudaGetLastError();
}

template <typename Tin>
cudaError_t run_keyless_bwd(const slotscan_v_params& p, const Tin* v, const float* wa, const float* gate, const float* fr,
                            const float* buf, const float* obuf, const float* dbuf, char* scratch, Tin* dv, float* dwa,
                            float* dgate, cudaStream_t st) {
    const KeylessScratch s = keyless_scratch(p);
    float *as = (float*)(scratch + s.as), *ot = (float*)(scratch + s.ot), *dp = (float*)(scratch + s.dp);
    int* am = (int*)(scratch + s.am);
    float* part = (float*)(scratch + s.part);
    const int BH = p.B * p.H, NB = (p.T + p.G - 1) / p.G;
    cudaError_t e;
    for (int bh0 = 0; bh0 < BH; bh0 += s.nbh) {
        const int nbh = std::min(s.nbh, BH - bh0);
        const size_t warps = (size_t)nbh * NB, tn = (size_t)nbh * p.T * p.N;
        KEYLESS_ROWS(p.N, (keyless_tables_kernel<R><<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(p, wa, gate, fr, obuf, bh0, nbh,
                                                                                                as, ot, am)));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        RowAdjArgs A = {p.N, p.T, p.H, p.G, p.hard, p.hard_gate, as, am, nullptr, gate, dp, bh0, nbh, s.nsl,
                        {v, buf, dbuf, dv, p.DV}, {nullptr, nullptr, nullptr, nullptr, 0}};
        if ((e = run_row_adjoint(A, p.in_dtype, st)) != cudaSuccess) return e;
        if ((e = run_row_dsum(dp, tn, s.nsl, st)) != cudaSuccess) return e;
        KEYLESS_ROWS(p.N, (keyless_bwd_chain_kernel<R><<<nbh, 32, 0, st>>>(p, gate, fr, as, ot, am, dp, bh0, dwa, dgate, part)));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace slotscan

using namespace slotscan;

extern "C" int slotscan_v_check(const slotscan_v_params* p) {
    if (!p) return SLOTSCAN_E_NULL;
    if (p->B < 1 || p->T < 1 || p->H < 1 || p->N < 1 || p->G < 1 || p->DV < 1) return SLOTSCAN_E_SHAPE;
    if ((long long)p->B * p->H > 2147483647LL / 4) return SLOTSCAN_E_SHAPE;
    if (sizeof(float) * keyless_bwd_smem_floats(p->N, p->DV) > 227 * 1024) return SLOTSCAN_E_SHAPE;
    if (p->in_dtype != SLOTSCAN_F32 && p->in_dtype != SLOTSCAN_BF16) return SLOTSCAN_E_DTYPE;
    return SLOTSCAN_OK;
}

extern "C" int slotscan_v_fwd(const slotscan_v_params* p, const void* v, const float* wa, const float* gate,
                              const float* fr, float* buf, float* obuf, int32_t* addr, void* stream) {
    const int rc = slotscan_v_check(p);
    if (rc) return rc;
    if (!v || !wa || !gate || !fr || !buf || !obuf) return SLOTSCAN_E_NULL;
    cudaStream_t st = (cudaStream_t)stream;
    if (keyless_split(*p))
        return (int)(p->in_dtype == SLOTSCAN_F32
                         ? run_keyless_fwd<float>(*p, (const float*)v, wa, gate, fr, buf, obuf, addr, st)
                         : run_keyless_fwd<__nv_bfloat16>(*p, (const __nv_bfloat16*)v, wa, gate, fr, buf, obuf, addr, st));
    const size_t sm = sizeof(float) * keyless_fwd_smem_floats(p->N, p->DV);
    cudaError_t e;
    if (p->in_dtype == SLOTSCAN_F32) {
        auto kern = keyless_fwd_kernel<float>;
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return (int)e;
        kern<<<p->B * p->H, KV_THREADS, sm, st>>>(*p, (const float*)v, wa, gate, fr, buf, obuf, addr);
    } else {
        auto kern = keyless_fwd_kernel<__nv_bfloat16>;
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return (int)e;
        kern<<<p->B * p->H, KV_THREADS, sm, st>>>(*p, (const __nv_bfloat16*)v, wa, gate, fr, buf, obuf, addr);
    }
    return (int)cudaGetLastError();
}

extern "C" size_t slotscan_v_bwd_scratch_bytes(const slotscan_v_params* p) {
    if (slotscan_v_check(p)) return 0;
    if (keyless_split(*p)) return keyless_scratch(*p).bytes;
    size_t o = sizeof(float) * (size_t)p->B * p->H * p->G * keyless_state_floats(p->N, p->DV);
    o = (o + 255) & ~(size_t)255;
    return o + sizeof(float) * (size_t)p->B * p->H;
}

extern "C" int slotscan_v_bwd(const slotscan_v_params* p, const void* v, const float* wa, const float* gate,
                              const float* fr, const float* buf, const float* obuf, const float* dbuf, void* scratch,
                              size_t scratch_bytes, void* dv, float* dwa, float* dgate, float* dfr, void* stream) {
    const int rc = slotscan_v_check(p);
    if (rc) return rc;
    if (!v || !wa || !gate || !fr || !buf || !obuf || !scratch || !dv || !dwa || !dgate || !dfr) return SLOTSCAN_E_NULL;
    if (scratch_bytes < slotscan_v_bwd_scratch_bytes(p)) return SLOTSCAN_E_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    if (keyless_split(*p)) {
        const cudaError_t e = p->in_dtype == SLOTSCAN_F32
            ? run_keyless_bwd<float>(*p, (const float*)v, wa, gate, fr, buf, obuf, dbuf, (char*)scratch, (float*)dv, dwa, dgate, st)
            : run_keyless_bwd<__nv_bfloat16>(*p, (const __nv_bfloat16*)v, wa, gate, fr, buf, obuf, dbuf, (char*)scratch,
                                             (__nv_bfloat16*)dv, dwa, dgate, st);
        if (e != cudaSuccess) return (int)e;
        keyless_finish_kernel<<<1, 256, 0, st>>>((const float*)((char*)scratch + keyless_scratch(*p).part), p->B * p->H, dfr);
        return (int)cudaGetLastError();
    }
    const size_t sm = sizeof(float) * keyless_bwd_smem_floats(p->N, p->DV);
    const size_t seg_bytes = (sizeof(float) * (size_t)p->B * p->H * p->G * keyless_state_floats(p->N, p->DV) + 255) & ~(size_t)255;
    float* seg = (float*)scratch;
    float* part = (float*)((char*)scratch + seg_bytes);
    cudaError_t e;
    if (p->in_dtype == SLOTSCAN_F32) {
        auto kern = keyless_bwd_kernel<float>;
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return (int)e;
        kern<<<p->B * p->H, KV_THREADS, sm, st>>>(*p, (const float*)v, wa, gate, fr, buf, obuf, dbuf, seg, (float*)dv, dwa, dgate,
                                                  part);
    } else {
        auto kern = keyless_bwd_kernel<__nv_bfloat16>;
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return (int)e;
        kern<<<p->B * p->H, KV_THREADS, sm, st>>>(*p, (const __nv_bfloat16*)v, wa, gate, fr, buf, obuf, dbuf, seg,
                                                  (__nv_bfloat16*)dv, dwa, dgate, part);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    keyless_finish_kernel<<<1, 256, 0, st>>>(part, p->B * p->H, dfr);
    return (int)cudaGetLastError();
}
