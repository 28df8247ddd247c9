// Address backward for sequences that use MORE than 32 rows: token-parallel like the gather kernel, the two contractions
// as register-tiled products.
//
// A work item is 32 tokens of one sequence.  Every row version its tokens can see is in memory (slotscan_addr_gather.cuh):
// slot i < 32 is the undo row of token t0 + i, slot 32 + n row n as it is after the chunk.  All of them come into shared
// memory once, then
//   1. St[slot][j] = <row, q_j> for every slot and token (a thread holds NS rows x 4 tokens),
//   2. softmax adjoint, a warp per 4 tokens and 8 lanes per token; C[slot][j] = dz temp / |K_n| of the version token j
//      sees replaces St, 0 elsewhere,
//   3. dqn_j = sum over the slots C[slot][j] row (a thread holds 8 tokens x 4 columns, the slots in two halves), and
//      dq_j = (dqn_j - qn_j <qn_j, dqn_j>) / |q_j|.
// [reference addr_bwd, slotkern_cuda.py:264-443]
// Bound: 2 x (32 + rows) x DK multiply-adds per token on the CUDA cores (float32: the tensor cores' bf16 or tf32 operands
// would lose bits); the chunked resident-state kernel (slotscan_addr_bwd.cuh) walks 8-token chunks of a sequence one after
// another with five barriers each.  B = 32, T = 1024, H = 6, 192 rows x 128 all in use, bf16: 2.07 ms chunked, 1.33 ms here
// (1.44 with scalar multiply-adds);
// B = 4, T = 1000, H = 12, ~60 rows x 64, float32 (48 sequences, so that the chunked kernel had 48 CTAs): 1.29 -> 0.27 ms.
// Where all of many sequences use 33 to 96 rows and fill the chunked kernel's rounds of two to an SM, that one is ahead: T = 256,
// 60 rows x 128, chunked / tiles us: 148 sequences 229 / 196, 240: 264 / 309, 300: 456 / 391, 444: 509 / 551, 800: 759 / 976.
// Persistent: the CTAs share the items of the sequences that need this kernel, which they find from the forward's tfirst
// table (a launch whose sequences all use few rows returns after that look).
#pragma once
#include "slotscan_addr_gather.cuh"

namespace slotscan {

constexpr int TL_THREADS = 256;
constexpr int TL_WIN = 8192;                  // sequences looked over at a time (bitmap and its prefix sums)

template <int DK>
struct TilesLayout {
    static constexpr int RS = DK + 4;         // row stride (floats): 16-byte rows, conflict-free
    __host__ __device__ static int groups(int N) { return 1 + (N + 31) / 32; }
    static size_t smem(int N) {
        const size_t slots = 32 * (size_t)groups(N);
        return 4 * (slots * RS + 32 * RS + slots * 32 + 2 * slots + 4 * 32 + 32 + (size_t)((N + 3) & ~3)) + 32 * (size_t)((N + 3) & ~3) +
               4 * (TL_WIN / 32 * 2 + 8) + 16;
    }
};

// vend[bh][c][n]: first token >= (c + 1) * 32 that writes row n, or -1; only sequences that used more than GATHER_ROWS rows
static __global__ void __launch_bounds__(192) next_write_all_kernel(const slotscan_params p, const int* __restrict__ am,
                                                                    const int* __restrict__ tfirst, int* __restrict__ vend) {
    const int N = p.N, T = p.T, H = p.H, n = threadIdx.x;
    const int bh = blockIdx.x, b = bh / H, h = bh % H;
    if (gather_sequence(tfirst + (size_t)bh * N, N, T)) return;
    const int nc = (T + GC - 1) / GC;
    __shared__ int s_first[2][192];
    int ver = -1;
    s_first[0][n] = BIGI;
    s_first[1][n] = BIGI;
    int a_next = (n < GC && (nc - 1) * GC + n < T) ? am[((size_t)b * T + (nc - 1) * GC + n) * H + h] : -1;
    __syncthreads();
    for (int c = nc - 1; c >= 0; c--) {
        int* f = s_first[c & 1];
        if (n < N) vend[((size_t)bh * nc + c) * N + n] = ver;
        const int a = a_next;
        if (n < GC && c > 0) a_next = am[((size_t)b * T + (c - 1) * GC + n) * H + h];
        if (a >= 0 && a < N) atomicMin(&f[a], n);
        __syncthreads();
        if (f[n] != BIGI) ver = c * GC + f[n];
        f[n] = BIGI;                                         // this slot is written again two chunks on, after a barrier
    }
}

// step 1 for NS groups of 32 slots: thread = rows rg + 32 i, tokens tq + 8 k
template <int DK, int NS>
__device__ __forceinline__ void tiles_scores(const float* rows, const float* sq, float* St) {
    constexpr int RS = TilesLayout<DK>::RS;
    const int lane = threadIdx.x & 31, rg = (threadIdx.x >> 5) * 4 + (lane >> 3), tq = lane & 7;
    float tot[NS][4];
#pragma unroll
    for (int i = 0; i < NS; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) tot[i][k] = 0.f;
    // a quarter of the columns at a time: four short chains instead of one of DK, whose rounding showed in the gradients
#pragma unroll 1
    for (int d0 = 0; d0 < DK; d0 += DK / 4) {
        f32x2 acc[NS][4];                                    // even and odd columns
#pragma unroll
        for (int i = 0; i < NS; i++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[i][k] = 0ull;
#pragma unroll 2
        for (int d = d0; d < d0 + DK / 4; d += 4) {
            f32x4 q[4];
#pragma unroll
            for (int k = 0; k < 4; k++) q[k] = ld4x2(sq + (tq + 8 * k) * RS + d);
#pragma unroll
            for (int i = 0; i < NS; i++) {
                const f32x4 r = ld4x2(rows + (rg + 32 * i) * RS + d);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    acc[i][k] = fma2(r.a, q[k].a, acc[i][k]);
                    acc[i][k] = fma2(r.b, q[k].b, acc[i][k]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NS; i++)
#pragma unroll
            for (int k = 0; k < 4; k++) { const float2 v = unpack2(acc[i][k]); tot[i][k] += v.x + v.y; }
    }
#pragma unroll
    for (int i = 0; i < NS; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int s = rg + 32 * i, j = tq + 8 * k;
            St[s * 32 + ((((j >> 2) ^ (s & 7)) << 2) | (j & 3))] = tot[i][k];
        }
}
// place of (slot, token) in St / C: quads of tokens swapped around by slot, so that 8 neighbouring slots of one token (step
// 2) and 4 neighbouring tokens of one slot (step 3, one 16-byte load) both miss each other's banks
__device__ __forceinline__ int tiles_at(int s, int j) { return s * 32 + ((((j >> 2) ^ (s & 7)) << 2) | (j & 3)); }

template <int DK, typename Tin>
__global__ void __launch_bounds__(TL_THREADS) addr_bwd_tiles_kernel(
    const slotscan_params p, const Tin* __restrict__ q, const float* __restrict__ gate, const float* __restrict__ fr,
    const float* __restrict__ temp_p, const int* __restrict__ am, const float* __restrict__ kold,
    const float* __restrict__ oold, const float* __restrict__ kiold, const float* __restrict__ kfin,
    const float* __restrict__ ofin, const int* __restrict__ tfirst, const int* __restrict__ vend,
    const float* __restrict__ Din, Tin* __restrict__ dq, float* __restrict__ dg, float* __restrict__ dfr,
    float* __restrict__ part, const int part_stride) {
    constexpr int RS = TilesLayout<DK>::RS, CQ = DK / 4, SUB = 32 / CQ;    // column quads, slots side by side in a warp
    extern __shared__ __align__(128) unsigned char tl_sm[];
    const int N = p.N, T = p.T, H = p.H, BH = p.B * H, nc = (T + GC - 1) / GC;
    const int slots = 32 * TilesLayout<DK>::groups(N), NP = (N + 3) & ~3;
    float* rows = reinterpret_cast<float*>(tl_sm);           // [slots][RS]
    float* sq = rows + slots * RS;                           // [32][RS] queries
    float* St = sq + 32 * RS;                                // [slots][32]
    float* s_ki = St + slots * 32;                           // [slots] 1 / |row|
    float* s_oc = s_ki + slots;                              // [slots] occupancy
    float* s_g = s_oc + slots;                               // [32] gate, fr, 1 / |q|
    float* s_fr = s_g + 32;
    float* s_qi = s_fr + 32;
    int* s_am = reinterpret_cast<int*>(s_qi + 32);           // [32]
    float* s_red = reinterpret_cast<float*>(s_am + 32);      // [2][8] partial sums, [16] flags
    int* s_bad = reinterpret_cast<int*>(s_red + 16);         // a row version that is not finite
    unsigned* s_map = reinterpret_cast<unsigned*>(s_red + 32);               // [TL_WIN / 32] sequences of the window
    int* s_pre = reinterpret_cast<int*>(s_map + TL_WIN / 32);                // [TL_WIN / 32 + 1] its prefix sums
    int* s_tf = s_pre + TL_WIN / 32 + 8;                     // [NP] first token at which row n is a candidate
    unsigned char* s_slot = reinterpret_cast<unsigned char*>(s_tf + NP);     // [32][NP] slot of row n as token j sees it
    __shared__ __align__(8) uint64_t s_bar;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float temp = temp_p[0], eps = p.eps;
    if (tid == 0) { mbar_init(&s_bar, 1); mbar_fence_init(); }
    unsigned phase = 0;
    for (int w0 = 0; w0 < BH; w0 += TL_WIN) {
        const int wn = min(TL_WIN, BH - w0), nwords = (wn + 31) / 32;
        __syncthreads();
        for (int i = tid; i < nwords * 32; i += TL_THREADS) {            // warp-uniform trip count: 256 divides by 32
            const bool mine = i < wn && !gather_sequence(tfirst + (size_t)(w0 + i) * N, N, T);
            const unsigned m = __ballot_sync(FULL, mine);
            if (lane == 0) s_map[i >> 5] = m;
        }
        __syncthreads();
        if (warp == 0) {                                                 // prefix sums of the words' counts
            int run = 0;
            for (int i = 0; i < nwords; i += 32) {
                int v = i + lane < nwords ? __popc(s_map[i + lane]) : 0;
                int x = v;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) { const int y = __shfl_up_sync(FULL, x, off); if (lane >= off) x += y; }
                if (i + lane < nwords) s_pre[i + lane] = run + x - v;
                run += __shfl_sync(FULL, x, 31);
            }
            if (lane == 0) s_pre[nwords] = run;
        }
        __syncthreads();
        const long long items = (long long)s_pre[nwords] * nc;
        for (long long it = blockIdx.x; it < items; it += gridDim.x) {
            const int rank = (int)(it / nc), c = (int)(it % nc);
            int lo = 0, hi = nwords - 1;                                 // last word with prefix <= rank
            while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (s_pre[mid] <= rank) lo = mid; else hi = mid - 1; }
            const int bh = w0 + lo * 32 + (int)__fns(s_map[lo], 0, rank - s_pre[lo] + 1), b = bh / H, h = bh % H;
            const int t0 = c * GC, tc = min(GC, T - t0);
            const int* tf = tfirst + (size_t)bh * N;
            // candidate rows 0 .. lim at the chunk's last token (rows become candidates in index order)
            int lim;
            {
                int l = 0, r = N - 1;
                while (l < r) { const int mid = (l + r + 1) >> 1; if (tf[mid] < t0 + tc) l = mid; else r = mid - 1; }
                lim = l;
            }
            const int NS = 1 + lim / 32 + 1;                             // groups of 32 slots in use
            // ---- staging: warp 0..7 each take every eighth slot ----
            const size_t ix0 = ((size_t)b * T + t0) * H + h;             // token t0 + j: + j * H
            if (tid == 0) {
                *s_bad = 0;
                mbar_arrive_expect_tx(&s_bar, (unsigned)(tc + lim + 1) * (unsigned)(DK * 4));
            }
            if (tid < 32) {
                const bool in = tid < tc;
                const size_t ix = ix0 + (size_t)tid * H;
                s_am[tid] = in ? am[ix] : -1;
                s_g[tid] = in ? gate_eff(gate[ix], p.hard_gate) : 0.f;
                s_fr[tid] = in ? (p.fr_per_token ? fr[ix] : fr[0]) : 0.f;
            }
            for (int s = warp + 8 * lane; s < NS * 32; s += 256) {       // a slot per lane
                float* dst = rows + s * RS;
                if (s < 32 ? s < tc : s - 32 <= lim) {
                    const float* src;
                    if (s < 32) {
                        const size_t ix = ix0 + (size_t)s * H;
                        src = kold + ix * DK;
                        s_ki[s] = kiold[ix];
                        s_oc[s] = oold[ix];
                    } else {
                        const int n = s - 32, ve = vend[((size_t)bh * nc + c) * N + n];
                        const size_t vix = ((size_t)b * T + ve) * H + h;
                        src = ve < 0 ? kfin + ((size_t)bh * N + n) * DK : kold + vix * DK;
                        s_ki[s] = ve < 0 ? -1.f : kiold[vix];            // -1: from the row once it is here
                        s_oc[s] = ve < 0 ? ofin[(size_t)bh * N + n] : oold[vix];
                    }
                    bulk_g2s(dst, src, DK * 4, &s_bar);
                } else {                                                 // no version: weight 0 below, so it must be a number
                    s_ki[s] = 0.f;
                    s_oc[s] = 0.f;
                    for (int d = 0; d < DK; d += 4) st4(dst + d, make_float4(0.f, 0.f, 0.f, 0.f));
                }
            }
            for (int n = tid; n <= lim; n += TL_THREADS) s_tf[n] = tf[n];
            for (int i = tid; i < 32 * CQ; i += TL_THREADS) {
                const int j = i / CQ, d = (i % CQ) * 4;
                st4(sq + j * RS + d, j < tc ? ld4(q + (ix0 + (size_t)j * H) * DK + d) : make_float4(0.f, 0.f, 0.f, 0.f));
            }
            __syncthreads();
            for (int n = tid; n <= lim; n += TL_THREADS) {               // the version of row n that token j sees
                int s = 32 + n;
                for (int j = 31; j >= 0; j--) {
                    if (s_am[j] == n) s = j;
                    s_slot[j * NP + n] = (unsigned char)s;
                }
            }
            const bool landed = mbar_wait_bounded(&s_bar, phase);
            phase ^= 1u;
            if (!__syncthreads_and(landed ? 1 : 0)) {
                if (tid == 0) atomicExch(&g_gather_status, 1);
                return;
            }
            {   // 1 / |row| of rows that are final rows, 1 / |q|: 8 lanes per row
                const int r8 = tid >> 3, l8 = tid & 7;
                for (int s = r8; s < NS * 32 + 32; s += TL_THREADS / 8) {            // uniform within a warp's groups of 8
                    const bool isq = s >= NS * 32;
                    const bool need = isq || (s >= 32 && s - 32 <= lim && s_ki[s] == -1.f);
                    const float* row = isq ? sq + (s - NS * 32) * RS : rows + s * RS;
                    float a = 0.f;
                    if (need) {
#pragma unroll
                        for (int f = 0; f < DK / 32; f++) { const float4 v = ld4(row + (l8 + 8 * f) * 4); a += dot4(v, v); }
                    }
                    a += __shfl_xor_sync(FULL, a, 1); a += __shfl_xor_sync(FULL, a, 2); a += __shfl_xor_sync(FULL, a, 4);
                    __syncwarp();
                    if (l8 == 0) {
                        if (isq) s_qi[s - NS * 32] = fminf(rsqrtf(a), 1e6f);
                        else {
                            if (need) s_ki[s] = fminf(rsqrtf(a), 1e6f);
                            const float ki = s_ki[s];                    // of a NaN row: NaN, of an infinite one: 0
                            if ((s < 32 ? s < tc : s - 32 <= lim) && !(ki > 0.f)) *s_bad = 1;
                        }
                    }
                }
            }
            // ---- 1. scores ----
            switch (NS) {
                case 2: tiles_scores<DK, 2>(rows, sq, St); break;
                case 3: tiles_scores<DK, 3>(rows, sq, St); break;
                case 4: tiles_scores<DK, 4>(rows, sq, St); break;
                case 5: tiles_scores<DK, 5>(rows, sq, St); break;
                case 6: tiles_scores<DK, 6>(rows, sq, St); break;
                default: tiles_scores<DK, 7>(rows, sq, St); break;
            }
            __syncthreads();
            // ---- 2. softmax adjoint: warp w = tokens 4 w .. 4 w + 3, lane = token (low 2 bits) x row of 8 ----
            {
                const int j = warp * 4 + (lane & 3), r8 = lane >> 2;
                const bool tok = j < tc;
                const int t = t0 + min(j, tc - 1);
                int limj = 0;                                            // last candidate row of the token
                for (int r = lim; limj < r;) { const int mid = (limj + r + 1) >> 1; if (s_tf[mid] <= t) limj = mid; else r = mid - 1; }
                if (!tok) limj = -1;
                const size_t ix = ix0 + (size_t)min(j, tc - 1) * H;
                const size_t di = ((size_t)bh * T + t) * N, dv = (size_t)BH * T * N;
                const float g = s_g[j], frv = s_fr[j], tqi = temp * s_qi[j];
                constexpr int NR = 24;                                   // rows of a lane: r8 + 8 i
                float dwv[NR], zv[NR];
                int ei = BIGI;
                unsigned okm = 0u;                                       // rows of this lane that are occupied candidates
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int n = r8 + 8 * i;
                    dwv[i] = zv[i] = 0.f;
                    if (8 * i <= lim && n <= limj) { dwv[i] = Din[di + n]; zv[i] = Din[dv + di + n]; }   // loads only: all in flight
                }
#pragma unroll
                for (int i = 0; i < NR; i++) dwv[i] += zv[i];            // key part + value part
                float zmax = -INFINITY, smax = -INFINITY;
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int n = r8 + 8 * i;
                    zv[i] = -INFINITY;
                    if (8 * i <= lim && n <= limj) {
                        const int s = s_slot[j * NP + n];
                        const float oc = s_oc[s];
                        const bool occ = oc >= eps;
                        const float sc = tqi * (s_ki[s] * St[tiles_at(s, j)]);
                        zv[i] = sc - (occ ? frv : 0.f);
                        smax = fmaxf(smax, sc);
                        if (occ) { okm |= 1u << i; zmax = fmaxf(zmax, zv[i]); }
                        else if (oc < eps && n < ei) ei = n;
                    }
                }
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) ei = min(ei, __shfl_xor_sync(FULL, ei, off));     // lowest free row
#pragma unroll
                for (int i = 0; i < NR; i++)
                    if (r8 + 8 * i == ei) { okm |= 1u << i; zmax = fmaxf(zmax, zv[i]); }
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) {
                    zmax = fmaxf(zmax, __shfl_xor_sync(FULL, zmax, off));
                    smax = fmaxf(smax, __shfl_xor_sync(FULL, smax, off));
                }
                float se = 0.f, sd = 0.f;
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    if (8 * i <= lim) {
                        zv[i] = (okm >> i) & 1u ? __expf(zv[i] - zmax) : 0.f;
                        se += zv[i];
                        sd += zv[i] * dwv[i];
                    }
                }
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) {
                    se += __shfl_xor_sync(FULL, se, off);
                    sd += __shfl_xor_sync(FULL, sd, off);
                }
                const float inv = 1.f / se, sa = g * sd * inv;
                float f1 = 0.f, f2 = 0.f;
                const int a = s_am[j];
                // the token's column: first its scores, then the weights of the versions it sees; only these lanes touch it
                float cv[NR];
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int n = r8 + 8 * i;
                    cv[i] = 0.f;
                    if (8 * i <= lim && n <= limj) {
                        const int s = s_slot[j * NP + n];
                        const float dz = (okm >> i) & 1u ? (zv[i] * inv) * (g * dwv[i] - sa) : 0.f;
                        const float ki = s_ki[s];
                        // (the dz of a token add up to zero: against the largest score instead of zero the products cancel less)
                        f2 += (okm >> i) & 1u ? dz * (tqi * (ki * St[tiles_at(s, j)]) - smax) : 0.f;
                        if (s_oc[s] >= eps) f1 -= dz;
                        cv[i] = dz * temp * ki;
                        if (n == a) dg[ix] = dwv[i];
                    }
                }
                __syncwarp();
                for (int s = r8; s < NS * 32; s += 8) St[tiles_at(s, j)] = 0.f;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int n = r8 + 8 * i;
                    if (8 * i <= lim && n <= limj) St[tiles_at(s_slot[j * NP + n], j)] = cv[i];
                }
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) {
                    f1 += __shfl_xor_sync(FULL, f1, off);
                    f2 += __shfl_xor_sync(FULL, f2, off);
                }
                if (r8 == 0 && tok && p.fr_per_token) dfr[ix] = f1;
                f1 = tok ? f1 : 0.f;
                f2 = tok ? f2 / temp : 0.f;
                f1 += __shfl_xor_sync(FULL, f1, 1); f1 += __shfl_xor_sync(FULL, f1, 2);
                f2 += __shfl_xor_sync(FULL, f2, 1); f2 += __shfl_xor_sync(FULL, f2, 2);
                if (lane == 0) { s_red[warp] = f2; s_red[8 + warp] = p.fr_per_token ? 0.f : f1; }
            }
            __syncthreads();
            // ---- 3. query gradient: warp = 8 tokens x one half of the slots, lane = 4 columns (x SUB slots) ----
            {
                const int tg = (warp & 3) * 8, half = warp >> 2, cq = lane % CQ, sub = lane / CQ;
                const int sh = NS * 16, s_lo = half * sh + sub, s_hi = half * sh + sh;
                f32x2 tot[8][2];
#pragma unroll
                for (int j = 0; j < 8; j++) tot[j][0] = tot[j][1] = 0ull;
                const bool bad = *s_bad != 0;
#pragma unroll 1
                for (int sb = s_lo; sb < s_hi; sb += 16) {               // 16 slots at a time: short chains
                    f32x2 part2[8][2];
#pragma unroll
                    for (int j = 0; j < 8; j++) part2[j][0] = part2[j][1] = 0ull;
#pragma unroll 2
                    for (int s = sb; s < sb + 16; s += SUB) {            // half * sh is a multiple of 16
                        const f32x4 r = ld4x2(rows + s * RS + cq * 4);
                        const float4 c0 = ld4(St + tiles_at(s, tg)), c1 = ld4(St + tiles_at(s, tg + 4));
                        const float cv[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            if (bad && cv[j] == 0.f) continue;           // a version a token does not see stays out of its sum
                            const f32x2 c2 = pack2(cv[j], cv[j]);
                            part2[j][0] = fma2(c2, r.a, part2[j][0]);
                            part2[j][1] = fma2(c2, r.b, part2[j][1]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 8; j++) { tot[j][0] = add2(tot[j][0], part2[j][0]); tot[j][1] = add2(tot[j][1], part2[j][1]); }
                }
                float acc[8][4];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float2 lo = unpack2(tot[j][0]), hi = unpack2(tot[j][1]);
                    acc[j][0] = lo.x; acc[j][1] = lo.y; acc[j][2] = hi.x; acc[j][3] = hi.y;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
#pragma unroll
                        for (int off = 16; off >= CQ; off >>= 1) acc[j][k] += __shfl_xor_sync(FULL, acc[j][k], off);
                    }
                }
                __syncthreads();                                         // rows are free: the halves meet there
                if (half == 1 && sub == 0) {
#pragma unroll
                    for (int j = 0; j < 8; j++) st4(rows + (tg + j) * RS + cq * 4, make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]));
                }
                __syncthreads();
                if (half == 0) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int jt = tg + j;
                        const float4 o = ld4(rows + jt * RS + cq * 4), qv = ld4(sq + jt * RS + cq * 4);
                        const float qi = s_qi[jt];
                        const float4 x = make_float4(acc[j][0] + o.x, acc[j][1] + o.y, acc[j][2] + o.z, acc[j][3] + o.w);
                        const float4 qn = make_float4(qv.x * qi, qv.y * qi, qv.z * qi, qv.w * qi);
                        float pr = dot4(x, qn);
#pragma unroll
                        for (int off = CQ / 2; off > 0; off >>= 1) pr += __shfl_xor_sync(FULL, pr, off);
                        if (jt < tc && sub == 0) {
                            float4 out;                                  // qi = 1e6: |q| under its clamp, no projection
                            if (qi >= 1e6f) out = make_float4(qi * x.x, qi * x.y, qi * x.z, qi * x.w);
                            else out = make_float4(qi * (x.x - qn.x * pr), qi * (x.y - qn.y * pr), qi * (x.z - qn.z * pr), qi * (x.w - qn.w * pr));
                            st4(dq + (ix0 + (size_t)jt * H) * DK + cq * 4, out);
                        }
                    }
                }
            }
            if (tid == 0) {
                float a = 0.f, d = 0.f;
                for (int w = 0; w < 8; w++) { a += s_red[w]; d += s_red[8 + w]; }
                part[(size_t)bh * part_stride + c] = a;                              // dtemp partial
                part[((size_t)BH + bh) * part_stride + c] = d;                       // scalar dfr partial
            }
            // before the copies of the next item write over what generic stores filled here
            fence_proxy_async_smem();
            __syncthreads();
        }
    }
}

}  // namespace slotscan
