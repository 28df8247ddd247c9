// Reverse scan of the row gradients for addresses that are known for every token (the keyless scan, and the keyed scan
// with a detached address): what is left is linear in the rows.
//
// Inside a block of G tokens the gradient of row n changes only by factors: with S_n the gradient after the block's last
// token, the gradient after token t is c_n(t) S_n, c_n(t) = prod_{t' > t} (1 - w_n(t')).  So per block, row and token
//     D[t,n]  = <x_t - X_n(t), dX_n(t)> = c_n(t) (<x_t, S_n> - y_n(t)),   y_n(t) = <X_n(t), S_n>,
//     y_n(0)  = <X_n(snapshot), S_n>,   y_n(t+1) = y_n(t) + w_n(t) (<x_t, S_n> - y_n(t)),
//     dx_t    = sum_n w_n(t) c_n(t) S_n,
// and no row is replayed token by token: G + 1 dot products of a row against the block's tokens and its snapshot, one
// weighted sum over the rows, one pass over the snapshots and over their gradients.  The dots and y run in double: D is a
// difference of two of them.
//
// Grid: (column slice of DS, sequence).  The CTA walks the blocks from the last to the first with S in registers (a
// thread per row), so the only chain is one step per block; the slices add their D's in a table each (row_dsum_kernel).
// Snapshot and gradient tiles arrive by cp.async, issued half a block ahead.
// Bound: the double-precision dots (N * DS * (G + 1) per block and slice) and, for few rows, the latency of one block's
// phases -- hence 16-wide slices (half the dot's chain, twice the CTAs) up to 64 rows.  64 sequences, 64 x 64, 128 blocks of
// 4 tokens: 0.29 ms (0.54 with loads that waited for one another before the weighted sum, 1.23 with 32-wide slices and 16
// tokens a step); 48 sequences, 192 x (64 + 64), 32 blocks of 16: 0.42 ms.
#include <algorithm>

#include "slotscan_async.cuh"
#include "slotscan_common.cuh"
#include "slotscan_launch.h"
#include "slotscan_rowadj.cuh"

namespace slotscan {

__device__ __forceinline__ void ra_cp4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// CT: tokens per step (a power of two >= min(G, 16)); DS: columns per slice
template <int CT, int DS>
struct RowAdjShape {
    static constexpr int FS = CT + 4, SS = DS + 4;         // row strides: 16-byte rows, conflict-free by quarter warps
    static size_t smem(int nt) { return 8 * (size_t)CT * DS + 4 * ((size_t)nt * (FS + 3 * SS) + (size_t)(nt / 32) * CT * DS + 2 * CT); }
};

// 168 registers for the 32-wide slices: 129 to 192 rows then run two CTAs to an SM where 255 would leave one, 65 to 96 three
// instead of two (97 to 128: two either way, by shared memory; past 192 one).  What that spills (at most 146 bytes a thread,
// at 16 tokens a step) costs less than the missing warps: 192 rows, 48 sequences x 4 slices, 0.60 -> 0.42 ms.  The 16-wide slices
// (two warps at most) keep all they ask for.
template <typename Tin, int CT, int DS, bool HARD>
__global__ void __maxnreg__(DS == 32 ? 168 : 255) row_adjoint_kernel(const RowAdjArgs A) {
    constexpr int FS = RowAdjShape<CT, DS>::FS, SS = RowAdjShape<CT, DS>::SS;
    constexpr int XP = (CT * DS + 31) / 32;                          // token elements per thread at 32 threads
    constexpr int NQ = DS / 4, PER = CT / 4 * NQ, NSUB = 32 / PER;   // weighted sum: lanes per row, rows side by side
    static_assert(CT % 4 == 0 && DS % 4 == 0 && 32 % PER == 0, "lane split");
    extern __shared__ __align__(16) double ra_sm[];
    const int NT = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = NT >> 5;
    double* xs = ra_sm;                                              // [CT][DS] tokens of the step
    float* fw = reinterpret_cast<float*>(xs + CT * DS);              // [NT][FS] w_n(t) c_n(t)
    float* Ss = fw + NT * FS;                                        // [NT][SS] S
    float* Xs = Ss + NT * SS;                                        // [NT][SS] snapshot tile
    float* Gs = Xs + NT * SS;                                        // [NT][SS] tile of the snapshot's gradient
    float* red = Gs + NT * SS;                                       // [nw][CT][DS]
    float* gs = red + nw * CT * DS;                                  // [CT] gates of the step
    int* ms = reinterpret_cast<int*>(gs + CT);                       // [CT] addresses of the step (HARD)
    const bool second = (int)blockIdx.x >= A.nsl0;
    const RowAdjTensor R = second ? A.t1 : A.t0;
    const int N = A.N, T = A.T, H = A.H, G = A.G, D = R.D, NB = (T + G - 1) / G;
    const int lb = blockIdx.y, bh = A.bh0 + lb, b = bh / H, h = bh % H;
    const int d0 = ((int)blockIdx.x - (second ? A.nsl0 : 0)) * DS, dn = min(DS, D - d0);
    const int n = tid;
    const bool live = n < N;
    const bool vec = dn % 4 == 0 && D % 4 == 0 && ((reinterpret_cast<size_t>(R.x0) | reinterpret_cast<size_t>(R.dbuf)) & 15) == 0;
    const Tin* x = static_cast<const Tin*>(R.x) + ((size_t)b * T * H + h) * D + d0;       // token t: + t * H * D
    Tin* dx = static_cast<Tin*>(R.dx) + ((size_t)b * T * H + h) * D + d0;
    const float* gate = A.gate + (size_t)b * T * H + h;
    const float* as = A.as + (size_t)lb * T * N + n;
    const int* am = A.am + (size_t)lb * T;
    float* dp = A.dp + ((size_t)blockIdx.x * A.nbh + lb) * T * N + n;

    for (int i = tid; i < NT * SS; i += NT) { Xs[i] = 0.f; Gs[i] = 0.f; }
    __syncthreads();
    auto tile = [&](float* dst, const float* src, int jb) {          // rows [0, N) x columns [d0, d0 + dn) of snapshot jb
        if (src == nullptr || jb < 0) return;
        const float* base = src + (((size_t)b * NB + jb) * H + h) * N * D + d0;
        if (vec) {
            const int q = dn >> 2;
            for (int i = tid; i < N * q; i += NT) { const int r = i / q, c = (i % q) * 4; cp_async16(dst + r * SS + c, base + (size_t)r * D + c); }
        } else {
            for (int i = tid; i < N * dn; i += NT) { const int r = i / dn, c = i % dn; ra_cp4(dst + r * SS + c, base + (size_t)r * D + c); }
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // the next step's operands, loads only: nothing here may wait for one of them
    Tin xp[XP];
    float ap[CT], gp = 0.f;
    int mp = 0;
    auto fetch = [&](int ts, int cn) {
#pragma unroll
        for (int i = 0; i < XP; i++) {
            const int e = tid + i * NT, j = e / DS, d = e % DS;
            if (e < CT * DS) xp[i] = (j < cn && d < dn) ? x[(size_t)(ts + j) * H * D + d] : Tin(0.f);
        }
        if (HARD) {
            if (tid < CT) mp = tid < cn ? am[ts + tid] : -1;
        } else {
#pragma unroll
            for (int j = 0; j < CT; j++) ap[j] = (j < cn && live) ? as[(size_t)(ts + j) * N] : 0.f;
        }
        if (tid < CT) gp = tid < cn ? gate[(size_t)(ts + tid) * H] : 0.f;
    };

    float S[DS];
#pragma unroll
    for (int c = 0; c < DS; c++) S[c] = 0.f;
    tile(Xs, R.x0, NB - 1);
    commit();
    fetch((NB - 1) * G, min(CT, T - (NB - 1) * G));
    for (int jb = NB - 1; jb >= 0; jb--) {
        const int t0 = jb * G, bn = min(G, T - t0);
        if (bn > CT) {                                               // more than one step: c after each step, kept in D's place
            double c = 1.0;
            for (int j = bn - 1; j >= 0; j--) {
                if (!live) break;
                if ((j + 1) % CT == 0 || j == bn - 1) dp[(size_t)(t0 + j) * N] = (float)c;
                const float g = gate_eff(gate[(size_t)(t0 + j) * H], A.hard_gate);
                c *= 1.0 - (double)(HARD ? (am[t0 + j] == n ? g : 0.f) : g * as[(size_t)(t0 + j) * N]);
            }
        }
        double y = 0.0;
        float ptot = 1.f;
        for (int s0 = 0; s0 < bn; s0 += CT) {
            const int cn = min(CT, bn - s0), ts = t0 + s0;
#pragma unroll
            for (int i = 0; i < XP; i++)
                if (tid + i * NT < CT * DS) xs[tid + i * NT] = (double)(float)xp[i];
            if (tid < CT) { gs[tid] = gate_eff(gp, A.hard_gate); if (HARD) ms[tid] = mp; }
            const float cend = (bn > CT && live) ? dp[(size_t)(ts + cn - 1) * N] : 1.f;
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (s0 == 0) { tile(Gs, R.dbuf, jb); commit(); }         // all have read the block before's tile
            float w[CT];                                             // tokens past cn: 0
#pragma unroll
            for (int j = 0; j < CT; j++) w[j] = j < cn ? (HARD ? (ms[j] == n ? gs[j] : 0.f) : gs[j] * ap[j]) : 0.f;
            double m[CT], y1 = 0.0;
#pragma unroll
            for (int j = 0; j < CT; j++) m[j] = 0.0;
#pragma unroll
            for (int c = 0; c < DS; c += 4) {
                const double sd[4] = {(double)S[c], (double)S[c + 1], (double)S[c + 2], (double)S[c + 3]};
                if (s0 == 0) {
                    const float4 q = ld4(Xs + tid * SS + c);
                    y = fma((double)q.x, sd[0], y);
                    y1 = fma((double)q.y, sd[1], y1);
                    y = fma((double)q.z, sd[2], y);
                    y1 = fma((double)q.w, sd[3], y1);
                }
#pragma unroll
                for (int j = 0; j < CT; j++) {                       // tokens past cn are zero
                    const double2 q0 = *reinterpret_cast<const double2*>(xs + j * DS + c);
                    const double2 q1 = *reinterpret_cast<const double2*>(xs + j * DS + c + 2);
                    m[j] = fma(q0.x, sd[0], m[j]);
                    m[j] = fma(q0.y, sd[1], m[j]);
                    m[j] = fma(q1.x, sd[2], m[j]);
                    m[j] = fma(q1.y, sd[3], m[j]);
                }
            }
            y += y1;
            float cj[CT];
            double c = (double)cend;
#pragma unroll
            for (int j = CT - 1; j >= 0; j--) {                      // weights past cn are zero
                cj[j] = (float)c;
                c *= 1.0 - (double)w[j];
            }
            if (s0 == 0) ptot = (float)c;
#pragma unroll
            for (int j = 0; j < CT; j++) {
                const double e = m[j] - y;
                if (live && j < cn) dp[(size_t)(ts + j) * N] = (float)((double)cj[j] * e);
                y = fma((double)w[j], e, y);
            }
#pragma unroll
            for (int j = 0; j < CT; j += 4)
                st4(fw + tid * FS + j, make_float4(w[j] * cj[j], w[j + 1] * cj[j + 1], w[j + 2] * cj[j + 2], w[j + 3] * cj[j + 3]));
            if (s0 == 0) {
#pragma unroll
                for (int d = 0; d < DS; d += 4) st4(Ss + tid * SS + d, make_float4(S[d], S[d + 1], S[d + 2], S[d + 3]));
            }
            // the next step's operands travel while the rows are summed
            if (s0 + CT < bn) fetch(ts + CT, min(CT, bn - s0 - CT));
            else if (jb > 0) fetch(t0 - G, min(CT, G));
            __syncthreads();
            if (s0 == 0) { tile(Xs, R.x0, jb - 1); commit(); }
            {   // dx: lane = 4 tokens x 4 columns, the warp's rows (and, with few tokens, NSUB of them) side by side
                const int sub = lane / PER, tq = (lane % PER) / NQ, dq = lane % NQ;
                float acc[4][4];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[i][k] = 0.f;
#pragma unroll 4
                for (int r = sub; r < 32; r += NSUB) {
                    const int rn = warp * 32 + r;
                    const float4 f = ld4(fw + rn * FS + tq * 4), s = ld4(Ss + rn * SS + dq * 4);
                    const bool hit = f.x != 0.f || f.y != 0.f || f.z != 0.f || f.w != 0.f;   // row not written: stays out
                    const float fv[4] = {f.x, f.y, f.z, f.w};
                    const float sv[4] = {hit ? s.x : 0.f, hit ? s.y : 0.f, hit ? s.z : 0.f, hit ? s.w : 0.f};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int k = 0; k < 4; k++) acc[i][k] = fmaf(fv[i], sv[k], acc[i][k]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {
#pragma unroll
                        for (int off = 16; off >= PER; off >>= 1) acc[i][k] += __shfl_xor_sync(FULL, acc[i][k], off);
                    }
                if (sub == 0) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        st4(red + (warp * CT + tq * 4 + i) * DS + dq * 4, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
                }
            }
            if (s0 + CT >= bn) {                                     // the gradient tile, not the snapshot tile behind it
                if (s0 == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            for (int e = tid; e < cn * DS; e += NT) {
                const int j = e / DS, d = e % DS;
                float v = 0.f;
                for (int q = 0; q < nw; q++) v += red[q * CT * DS + e];
                if (d < dn) st1(dx + (size_t)(ts + j) * H * D + d, v);
            }
        }
        // to the post side of the block before: the block's factors, then the gradient of its snapshot
        const bool take = live && R.dbuf != nullptr && (A.lim == nullptr || n <= A.lim[(size_t)lb * NB + jb]);
#pragma unroll
        for (int c = 0; c < DS; c += 4) {
            const float4 g = ld4(Gs + tid * SS + c);
            S[c] = take ? fmaf(ptot, S[c], g.x) : ptot * S[c];
            S[c + 1] = take ? fmaf(ptot, S[c + 1], g.y) : ptot * S[c + 1];
            S[c + 2] = take ? fmaf(ptot, S[c + 2], g.z) : ptot * S[c + 2];
            S[c + 3] = take ? fmaf(ptot, S[c + 3], g.w) : ptot * S[c + 3];
        }
    }
}

template <typename Tin>
static cudaError_t launch(const RowAdjArgs& A, cudaStream_t st) {
    const int nt = (A.N + 31) & ~31, ds = row_adjoint_ds(A.N);
    const int sl = row_adjoint_slices(A.N, A.t0.D) + (A.t1.D ? row_adjoint_slices(A.N, A.t1.D) : 0);
    auto go = [&](auto soft, auto hard, size_t sm) {
        auto kern = A.hard ? hard : soft;
        const cudaError_t e = opt_in_smem(kern, sm);
        if (e != cudaSuccess) return e;
        kern<<<dim3(sl, A.nbh), nt, sm, st>>>(A);
        return cudaGetLastError();
    };
    if (ds == 16) {
        if (A.G <= 4) return go(row_adjoint_kernel<Tin, 4, 16, false>, row_adjoint_kernel<Tin, 4, 16, true>, RowAdjShape<4, 16>::smem(nt));
        if (A.G <= 8) return go(row_adjoint_kernel<Tin, 8, 16, false>, row_adjoint_kernel<Tin, 8, 16, true>, RowAdjShape<8, 16>::smem(nt));
        return go(row_adjoint_kernel<Tin, 16, 16, false>, row_adjoint_kernel<Tin, 16, 16, true>, RowAdjShape<16, 16>::smem(nt));
    }
    if (A.G <= 4) return go(row_adjoint_kernel<Tin, 4, 32, false>, row_adjoint_kernel<Tin, 4, 32, true>, RowAdjShape<4, 32>::smem(nt));
    if (A.G <= 8) return go(row_adjoint_kernel<Tin, 8, 32, false>, row_adjoint_kernel<Tin, 8, 32, true>, RowAdjShape<8, 32>::smem(nt));
    return go(row_adjoint_kernel<Tin, 16, 32, false>, row_adjoint_kernel<Tin, 16, 32, true>, RowAdjShape<16, 32>::smem(nt));
}

// table[0] += table[1] + ... + table[slices - 1], element by element, in this order
__global__ void __launch_bounds__(256) row_dsum_kernel(float* __restrict__ dp, size_t n, int slices) {
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        float v = dp[i];
        for (int s = 1; s < slices; s++) v += dp[(size_t)s * n + i];
        dp[i] = v;
    }
}

cudaError_t run_row_adjoint(const RowAdjArgs& A, int in_dtype, cudaStream_t st) {
    return in_dtype == SLOTSCAN_F32 ? launch<float>(A, st) : launch<__nv_bfloat16>(A, st);
}

cudaError_t run_row_dsum(float* dp, size_t n, int slices, cudaStream_t st) {
    if (slices < 2) return cudaSuccess;
    row_dsum_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, st>>>(dp, n, slices);
    return cudaGetLastError();
}

}  // namespace slotscan
