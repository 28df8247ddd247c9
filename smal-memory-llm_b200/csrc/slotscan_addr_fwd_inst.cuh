// Instantiation body of the forward address scan for one input dtype: included by slotscan_addr_fwd_{f32,bf16}.cu
// with SLOTSCAN_TIN and SLOTSCAN_SUFFIX defined.
#include <stdint.h>
#include <stdio.h>

#include "slotscan_addr_fwd.cuh"
#include "slotscan_addr_narrow.cuh"
#include "slotscan_addr_wide.cuh"
#include "slotscan_launch.h"

namespace slotscan {

#define SS_CAT_(a, b) a##b
#define SS_CAT(a, b) SS_CAT_(a, b)
typedef SLOTSCAN_TIN Tin;

template <int DK, int RPL>
static cudaError_t launch_one(const slotscan_params& p, const void* q, const void* k, const float* gate, const float* fr,
                              const float* temp, const slotscan_log& L, const AddrFwdState& S0, int ncap, int second, float* hand,
                              cudaStream_t st) {
    const size_t sm = sizeof(float) * (size_t)addr_fwd_layout(ncap, DK, RPL, (int)sizeof(Tin)).total;
    cudaError_t e = cudaSuccess;
#define AF_LAUNCH(OCCB_, CARRY_)                                                                                          \
    {                                                                                                                     \
        auto kern = addr_fwd_direct_kernel<DK, RPL, OCCB_, CARRY_, Tin>;                                                  \
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return e;                                                         \
        kern<<<p.B * p.H, AF_THREADS, sm, st>>>(p, (const Tin*)q, (const Tin*)k, gate, fr, temp, L.addr, L.oold, L.kiold, \
                                                L.ofin, L.tfirst, S0.K0, S0.o0, S0.nsq0, S0.nsqfin, ncap, second, hand);  \
    }
    const bool carry = S0.K0 != nullptr;
    if (p.occ_bin) { if (carry) AF_LAUNCH(true, true) else AF_LAUNCH(true, false) }
    else { if (carry) AF_LAUNCH(false, true) else AF_LAUNCH(false, false) }
#undef AF_LAUNCH
    return cudaGetLastError();
}

template <int DK, int RPL>
static cudaError_t launch_wide(const slotscan_params& p, const void* q, const void* k, const float* gate, const float* fr,
                               const float* temp, const slotscan_log& L, const AddrFwdState& S0, const float* hand, cudaStream_t st) {
    const size_t sm = sizeof(float) * (size_t)addr_wide_layout(RPL, DK).total;
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return e;
        kern<<<p.B * p.H, aw_threads(RPL), sm, st>>>(p, (const Tin*)q, (const Tin*)k, gate, fr, temp, L.addr, L.oold, L.kiold, L.ofin,
                                                     L.tfirst, S0.K0, S0.o0, S0.nsq0, S0.nsqfin, hand);
        return cudaGetLastError();
    };
    const bool carry = S0.K0 != nullptr;
    if (p.occ_bin) return carry ? go(addr_fwd_wide_kernel<DK, RPL, true, true, Tin>) : go(addr_fwd_wide_kernel<DK, RPL, true, false, Tin>);
    return carry ? go(addr_fwd_wide_kernel<DK, RPL, false, true, Tin>) : go(addr_fwd_wide_kernel<DK, RPL, false, false, Tin>);
}
// Which kernel takes the last pass.  The wide one fills an SM, so where more sequences may come than there are SMs and two or more
// CTAs of the direct one fit beside each other, the direct one needs fewer rounds (each kernel starting at token 0: 192 sequences,
// T = 256, all of 96 rows x 128 in use, 312 us against 396 wide, 296 sequences 429 against 517, rows of 64 (T = 512) 536 against 825).
// With at most a sequence per SM the wide one is ahead at every length, the direct kernel of 64 rows left out as well (us, narrow to
// wide / direct of 64 rows and wide / direct of 64 rows and of all; 192 rows x 128): 24 sequences x 96 tokens, all rows in use 70 / 79 /
// 84, x 128 93 / 105 / 113; 144 x 160, clustered, 125 / 141 / 147; x 64: 144 x 160 95 / 119 / 121.  Past 128 rows, where it has six
// resolver warps to wait for, more sequences than SMs take it from 192 tokens on (a sequence passes row 64 after 64 tokens at the
// earliest).  With a state carried in that has more rows in use every row is scanned from the first token on: the wide one takes a short
// call of however many sequences (8 tokens, 444 sequences, 96 rows x 128: 63 us against 77 direct; 192 rows x 64: 66 against 86; 192
// sequences, 96 rows x 64: 34 against 32), while in a long one the rounds count again (256 tokens, 296 sequences, 96 rows x 128: 362
// against 306).
template <int DK>
static bool wide_second_pass(const slotscan_params& p, bool carry) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t direct = sizeof(float) * (size_t)addr_fwd_layout(p.N, DK, 6, (int)sizeof(Tin)).total + 1024;
    if ((long long)p.B * p.H <= sms) return true;
    if (2 * direct <= 228 * 1024 && (!carry || p.T >= 192)) return false;
    return p.N <= 128 || carry || p.T >= 192;
}
template <int DK, int CTAS>
static cudaError_t launch_narrow(const slotscan_params& p, const void* q, const void* k, const float* gate, const float* fr,
                                 const float* temp, const slotscan_log& L, const AddrFwdState& S0, float* hand, cudaStream_t st) {
    const size_t sm = sizeof(float) * (size_t)addr_narrow_layout(DK).total;
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        if ((e = opt_in_smem(kern, sm)) != cudaSuccess) return e;
        kern<<<p.B * p.H, AN_THREADS, sm, st>>>(p, (const Tin*)q, (const Tin*)k, gate, fr, temp, L.addr, L.oold, L.kiold, L.ofin,
                                                L.tfirst, S0.K0, S0.o0, S0.nsq0, S0.nsqfin, hand);
        return cudaGetLastError();
    };
    const bool carry = S0.K0 != nullptr;
    if (p.occ_bin) return carry ? go(addr_fwd_narrow_kernel<DK, CTAS, true, true, Tin>) : go(addr_fwd_narrow_kernel<DK, CTAS, true, false, Tin>);
    return carry ? go(addr_fwd_narrow_kernel<DK, CTAS, false, true, Tin>) : go(addr_fwd_narrow_kernel<DK, CTAS, false, false, Tin>);
}
// The passes: keys 64 or 128 wide start with the narrow kernel (32 rows), the others with the direct one.  The direct one with 64
// rows, three CTAs to an SM, goes on with what the narrow one left, and the full-size one with the rest (slotscan_addr_fwd.cuh:
// AfResume).  With at most a sequence per SM the wide kernel follows the narrow one at once: the
// direct one between them costs a launch that does nothing where no sequence needs it (12 sequences x 256 tokens, 9 rows x 128: 71 us
// against 76; 48 x 1024, 11 rows: 255 against 259), and the wide one is as fast from row 32 on or nearly (us, narrow to wide / with the
// direct one between / direct to wide, no narrow one): 148 x 1024, 42 rows x 128 of 192: 820 / 745 / 626; of 96: 625 / 745 / 627;
// 148 x 1024, 39 rows x 64: 559 / 609 / 513; 148 x 1024, 32 rows x 128: 607 / 584 / 571; 24 x 512, all of 192 rows x 128: 401 / - / 449.
// Sequences that end between 32 and 64 rows are where a chain of passes is behind: each pass waits for the last sequence of the one
// before.  Up to 32 rows it is ahead by nearly half: 24 x 1024, 22 rows x 128: 305 against 535 without the narrow kernel.
// The exception, more than two sequences per SM from the empty memory: the zero-fill of the snapshots runs beside the scan (rows past
// the first replay tile), and the replay behind the scan contends with it for the memory.  Where the fill (4.66 MB per us beside a scan)
// outlasts the direct kernel (0.74 us per token and round of three CTAs to an SM) by a fifth, a faster scan only brings that on
// earlier.  Narrow first / direct first, us, forward and then forward and backward, few rows in use, fill over scan in front:
//   0.98  300 x 1024, 192 rows x 128, bf16      898 / 995     1732 / 1823     0.98  300 x 512, float32, stride 16   520 / 597    1000 / 1077
//   1.14  384 x 512, 96 x 128, float32          657 / 680     1250 / 1275     1.14  384 x 1024, 192 x 64, float32  1000 / 1051   1969 / 2077
//   1.25  384 x 1024, 192 x 128, bf16          1133 / 1112    2076 / 2055     1.96  300 x 512, 192 x 128, float32   865 / 845    1389 / 1381
// Short calls are ahead with it past the line too (1.25, 384 x 128: 214 / 233, 430 / 434); sequences that take a new row every second
// token are behind on both sides of it (0.98, 300 x 512: 1679 / 1626, 3832 / 3802).
static bool behind_the_fill(const slotscan_params& p, int sms) {
    const double snaps = (double)p.B * p.H * ((p.T + p.G - 1) / p.G), esz = p.snap_dtype == SLOTSCAN_F32 ? 4.0 : 2.0;
    const double cols = (double)(p.N - replay_tile_rows(p.DK)) * p.DK + (double)(p.N - replay_tile_rows(p.DV)) * p.DV;
    const long long rounds = ((long long)p.B * p.H + 3 * sms - 1) / (3 * sms);
    return snaps * cols * esz / 4.66e6 > 1.2 * 0.74 * (double)p.T * (double)rounds;
}
// Where a pass leaves key rows for the next one: the final rows' place, which the replay writes later.  NULL, so that the next pass
// starts again, where the caller gave no room for the norms or where it carries the state in place.
static float* hand_over_rows(const slotscan_params& p, const slotscan_log& L, const AddrFwdState& S0) {
    const size_t rows = (size_t)p.B * p.H * p.N;
    auto apart = [](const void* a, const void* b, size_t bytes) {
        const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
        return a == nullptr || x + bytes <= y || y + bytes <= x;
    };
    const bool ok = S0.nsqfin != nullptr && apart(S0.K0, L.kfin, rows * p.DK * sizeof(float)) && apart(S0.o0, L.ofin, rows * sizeof(float)) &&
                    apart(S0.nsq0, S0.nsqfin, rows * sizeof(double));
    return ok ? L.kfin : nullptr;
}
template <int DK>
static cudaError_t launch_dk(const slotscan_params& p, const void* q, const void* k, const float* gate, const float* fr,
                             const float* temp, const slotscan_log& L, const AddrFwdState& S0, cudaStream_t st) {
    cudaError_t e;
    float* hand = hand_over_rows(p, L, S0);
    if constexpr (DK >= 64) {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const long long BH = (long long)p.B * p.H;
        int second = 0;                                   // this pass takes the sequences that the one before it marked
        if (BH <= 2 * sms || S0.K0 != nullptr || p.N <= AF_NCAP1 || !behind_the_fill(p, sms)) {
            if (BH <= 2 * sms) e = launch_narrow<DK, 2>(p, q, k, gate, fr, temp, L, S0, hand, st);
            else e = launch_narrow<DK, 3>(p, q, k, gate, fr, temp, L, S0, hand, st);
            if (e != cudaSuccess || p.N <= AN_ROWS) return e;
            second = 1;
        }
        const bool wide = p.N > AF_NCAP1 && wide_second_pass<DK>(p, S0.K0 != nullptr);
        if (!wide || BH > sms) {
            e = launch_one<DK, 2>(p, q, k, gate, fr, temp, L, S0, p.N <= AF_NCAP1 ? p.N : AF_NCAP1, second, hand, st);
            if (e != cudaSuccess || p.N <= AF_NCAP1) return e;
        }
        if (wide) {
            if (p.N <= 128) return launch_wide<DK, 4>(p, q, k, gate, fr, temp, L, S0, hand, st);
            return launch_wide<DK, 6>(p, q, k, gate, fr, temp, L, S0, hand, st);
        }
    } else {
        e = launch_one<DK, 2>(p, q, k, gate, fr, temp, L, S0, p.N <= AF_NCAP1 ? p.N : AF_NCAP1, 0, hand, st);
        if (e != cudaSuccess || p.N <= AF_NCAP1) return e;
    }
    return launch_one<DK, 6>(p, q, k, gate, fr, temp, L, S0, p.N, 1, hand, st);         // N <= 192
}

cudaError_t SS_CAT(run_addr_fwd_, SLOTSCAN_SUFFIX)(const slotscan_params& p, const void* q, const void* k, const float* gate,
                                                  const float* fr, const float* temp, const slotscan_log& L,
                                                  const AddrFwdState& S0, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    SLOTSCAN_DISPATCH_D(p.DK, e = (launch_dk<DD>(p, q, k, gate, fr, temp, L, S0, st)));
    return e;
}

void SS_CAT(attrs_addr_fwd_, SLOTSCAN_SUFFIX)(slotscan_kernel_attr* out, int cap, int& n) {
    fill_attr(out, cap, n, "addr_fwd_narrow<128,rows<=32,2 CTAs>", addr_fwd_narrow_kernel<128, 2, true, false, Tin>);
    fill_attr(out, cap, n, "addr_fwd_narrow<128,rows<=32,3 CTAs>", addr_fwd_narrow_kernel<128, 3, true, false, Tin>);
    fill_attr(out, cap, n, "addr_fwd<128,rows<=64>", addr_fwd_direct_kernel<128, 2, true, false, Tin>);
    fill_attr(out, cap, n, "addr_fwd_wide<128,rows<=192>", addr_fwd_wide_kernel<128, 6, true, false, Tin>);
}

}  // namespace slotscan

