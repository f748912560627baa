// xengine.cu -- plain FP32 X-engine and the row scaling kernel.
//
// Replaces corr_kernel (corr-cuda/src/kernels.cu:194-265): for every baseline
// b = (j,k), j <= k, and channel c,
//     acc[b][c] += sum_f Y_j[f][c] * conj(Y_k[f][c])
// with the reference's complex multiply-accumulate convention
//     re += xr*yr + xi*yi,  im += xi*yr - xr*yi          (kernels.cu:243-245)
// in FP32. Even and odd frames (and, for small problems, up to eight runs of them)
// are summed apart, so a sum takes two fused multiply-adds per component and frame
// and still rounds less than one long sum with a rounding per frame: relative RMS
// against float64 at 24 inputs, n_freq 16384, 1024 frames 2.2e-7 (4.9e-7 with one
// sum per visibility and the product pair rounded first).
//
// Shape: a warp owns a 6 x 6 tile of the station matrix for 16 channels, one per
// lane of each half warp; the half warps take even and odd frames. 72 sums and 24
// operands per thread fit 128 registers, and a frame's 12 shared-memory loads feed
// 144 multiply-adds: 24 bank cycles against 36 FP32 cycles, where a 4 x 4 tile's 8
// loads per 64 take as long as its arithmetic. An 8 x 8 tile reads less still but
// needs 168 registers (12 warps) and spilled around its loop; f32x2 instructions
// want their operands broadcast and negated in pairs, one move per multiply-add.
// Diagonal tiles leave out k < j, tiles of the last column the stations past the
// end. Up to 15 such warps (every tile of a channel tile, then parts of the frames,
// then channel tiles) and one that loads share a CTA; CTAs are persistent, and the
// TMA ring runs on through their tiles, so that the end of one (two shuffles per
// value, then reductions at L2) overlaps the loads of the next.
//
// Bound by issue: at 24 inputs (10 tiles on 4 schedulers) and 256 frames a launch, ncu has
// 66 % of the issue slots and 52 % of the FP32 pipe busy and DRAM at 43 %; the rest goes
// to scheduler imbalance, waits for stages and the ends of tiles. Measured on one GB300,
// complex64 rows, before (4 x 4 tiles, 32 channels, cp.async, a CTA barrier per 2 to 12
// frames) -> now:
//   24 inputs, n_freq 16384, 1024 frames  1.88 -> 0.95 ms
//   40 inputs, n_freq  4096,  300 frames  0.392 -> 0.286 ms
//   15 inputs, n_freq 12288,  301 frames  0.228 -> 0.121 ms
//    4 inputs, n_freq 32768,   64 frames  25.4 -> 24.3 us
//    4 inputs, n_freq  2048,  300 frames  89.6 -> 8.1 us

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "ptx.cuh"
#include "tensor_map.h"

namespace corrgb {
namespace {

constexpr int kXch = 16;      // channels of a warp's tile, one per lane of each half warp
constexpr int kTile = 6;      // stations on each side of a warp's tile of the matrix
constexpr int kSub = 3;       // stations on each side of a tile's four sub-blocks
constexpr int kMaxWarps = 15; // summing warps per CTA; one more loads
constexpr int kMaxSlots = 8;  // TMA ring depth, at most
constexpr int kMaxParts = 8;  // runs of frames summed apart, at most
constexpr int kSumElems = kTile * kSub * 32;   // float2 of a tile's sum
constexpr int kMaxTiles = 253;   // 22 x 23 / 2 tiles of 128 stations

// Which tiles a launch has: whole ones only; whole ones and, in the last column,
// ones of at most kSub stations (n_station % kTile = 1 .. 3); any (some baselines
// only). A kernel for each keeps its code, and so its instruction fetches, short.
enum : int { kWhole = 0, kEdge = 1, kAny = 2 };

struct PlainParams {
    int n_station;
    int n_freq;
    int frames;
    int ytile;
    int seg;              // frames per part (contiguous runs of the launch's frames, even)
    int n_parts;
    int tiles;            // CTA shape: tiles x part slots x channel tiles, a warp each
    int slots_p;
    int slots_c;
    int fs;               // frames of each (channel tile, part) per ring slot, even
    int slot_shift;       // ring slots: 1 << slot_shift
    int n_tiles;          // tiles computed
    int tile_groups;      // ceil(n_tiles / tiles)
    int units;            // channel-tile groups x tile_groups
    int sums_at;          // float2 before the tiles' sums in shared memory
    int group_sums;       // sums kept of a (channel tile, tile): see the launch
    void *acc;
    int *err;
    // J | K << 5 | sub-block mask << 10, groups of `tiles` one after the other (bit
    // 2a + b of the mask: blocks of kSub stations 2J + a, 2K + b); mask 0: no tile
    uint16_t tile[kMaxTiles + kMaxWarps];
};

// row[at] += v, at L2; complex128 rows (ACC64): the FP32 sum added in double
template <bool ACC64>
__device__ __forceinline__ void add_to_row(void *row, size_t at, float2 v) {
    if constexpr (ACC64) {
        double *dst = static_cast<double *>(row) + 2 * at;
        red_add_f64(dst, widen(v.x));
        red_add_f64(dst + 1, widen(v.y));
    } else {
        red_add_f32x2(static_cast<float2 *>(row) + at, v);
    }
}

// ROW: a run of frames in the ring holds [frame][station][16 channels] (ytile >= 16);
// otherwise [spectra tile][frame][station][ytile], as the TMA box brings narrower tiles.
// KIND: which tiles a launch has (kWhole, kEdge, kAny below). ACC64: complex128 rows.
// A launch of few frames is bound by its instruction fetches, and both kinds of rows in
// one kernel made the epilogue half as long again: 20 stations, n_freq 14336, 1 frame
// 23.4 -> 17.2 us, 64 frames 95.7 -> 85.4 us.
template <bool ROW, int KIND, bool ACC64, bool SIDE>
__global__ void __launch_bounds__((kMaxWarps + 1) * 32, 1)
    xengine_plain_kernel(const __grid_constant__ CUtensorMap ymap,
                         const __grid_constant__ PlainParams p) {
    extern __shared__ __align__(128) float2 xs[];   // TMA ring, then the tiles' sums so far
    __shared__ uint64_t full[kMaxSlots], empty[kMaxSlots];
    __shared__ int s_abort;
    __shared__ float2 zeros[kTile * kXch];   // a frame of one tile's stations that is not there
    __shared__ int s_turn[kMaxWarps];   // per (channel tile, tile): parts summed
    // SIDE, per (channel tile, tile): the parts' sums are in shared memory, and have been
    // added up; and the rounds of them each warp has seen
    __shared__ uint64_t laid_down[kMaxWarps / 4], summed_up[kMaxWarps / 4];
    __shared__ volatile int s_rounds[kMaxWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_warps = (blockDim.x >> 5) - 1;
    const int N = p.n_station;
    const volatile int *abort_flag = &s_abort;
    const int slot_mask = (1 << p.slot_shift) - 1;

    if (tid == 0) {
        for (int s = 0; s <= slot_mask; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], n_warps);
        }
        if (SIDE)
            for (int s = 0; s < p.tiles * p.slots_c; ++s) {
                mbar_init(&laid_down[s], p.slots_p);
                mbar_init(&summed_up[s], p.slots_p);
            }
        s_abort = 0;
        fence_mbar_init();
    }
    if (tid < kMaxWarps) s_turn[tid] = s_rounds[tid] = 0;
    for (int i = tid; i < kTile * kXch; i += blockDim.x) zeros[i] = make_float2(0.f, 0.f);
    __syncthreads();

    // The CTA walks units (a tile group of a group of channel tiles), each in
    // n_parts / slots_p rounds, each round in stages of fs frames per part; the
    // ring of stages runs on through all of them.
    const int rounds = p.n_parts / p.slots_p;
    auto part_frames = [&](int t) { return max(0, min(p.seg, p.frames - t * p.seg)); };
    auto round_stages = [&](int r) {   // by its first, longest part
        return (part_frames(r * p.slots_p) + p.fs - 1) / p.fs;
    };
    const int run_elems = p.fs * N * kXch;
    const int slot_elems = p.slots_c * p.slots_p * run_elems;

    if (warp == n_warps) {
        // ------------------------------ loader ------------------------------
        if (lane == 0) {
            int n = 0;   // stages issued
            bool ok = true;
            for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const int ct0 = u / p.tile_groups * p.slots_c;
                const int n_ct = min(p.slots_c, p.n_freq / kXch - ct0);
                for (int r = 0; r < rounds && ok; ++r) {
                    const int stages = round_stages(r);
                    for (int s = 0; s < stages; ++s, ++n) {
                        const int slot = n & slot_mask;
                        if (n > slot_mask &&
                            !mbar_wait_bounded(&empty[slot],
                                               static_cast<uint32_t>((n >> p.slot_shift) - 1) & 1u,
                                               p.err, kErrXengineMmaTimeout, abort_flag)) {
                            s_abort = 1;
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(
                            &full[slot],
                            static_cast<uint32_t>(n_ct * p.slots_p * run_elems * sizeof(float2)));
                        // frames past the launch's arrive as zeros, those past their
                        // part are not used
                        float2 *dst = xs + slot * slot_elems;
                        for (int c = 0; c < n_ct; ++c) {
                            const int ch = (ct0 + c) * kXch;
                            for (int i = 0; i < p.slots_p; ++i, dst += run_elems)
                                tma_load_4d(dst, &ymap, ch % p.ytile, 0,
                                            (r * p.slots_p + i) * p.seg + s * p.fs, ch / p.ytile,
                                            &full[slot]);
                        }
                    }
                }
            }
            // Every load lands before this thread leaves, and with it the CTA's shared
            // memory, also where the summing warps have given up on the last ones.
            for (int s = 0; s <= slot_mask; ++s) {
                const uint32_t n_s = static_cast<uint32_t>(n + slot_mask - s) >> p.slot_shift;
                if (n_s > 0) mbar_wait_bounded(&full[s], (n_s - 1) & 1u, nullptr, 0);
            }
        }
        return;
    }

    // ------------------------------- sums -------------------------------
    // this warp's place in the CTA: tile, part slot, channel tile
    const int wt = warp % p.tiles, wp = (warp / p.tiles) % p.slots_p;
    const int wc = warp / (p.tiles * p.slots_p);
    volatile int *turn = &s_turn[wc * p.tiles + wt];   // the part to come
    float2 *const so_far = xs + p.sums_at + (wc * p.tiles + wt) * p.group_sums * kSumElems + lane;
    const int rs = ROW ? kXch : p.ytile;   // float2 between stations of a run
    const int half = lane >> 4, ch = lane & 15;   // half warp: even or odd frames of the part
    const int lane_off = ROW ? ch : (ch / rs) * (p.fs * N * rs) + ch % rs;
    int used = 0;   // stages of the ring read

    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
        const int ct = u / p.tile_groups * p.slots_c + wc;
        const int entry = ct < p.n_freq / kXch ? p.tile[u % p.tile_groups * p.tiles + wt] : 0;
        const int J = entry & 31, K = (entry >> 5) & 31, sub = entry >> 10;
        for (int r = 0; r < rounds; ++r) {
            const int t = r * p.slots_p + wp;
            const int n_mine = part_frames(t);
            // visibilities of stations j = 6J + i and k = 6K + l
            float re[kTile][kTile], im[kTile][kTile];
#pragma unroll
            for (int i = 0; i < kTile; ++i)
#pragma unroll
                for (int l = 0; l < kTile; ++l) re[i][l] = im[i][l] = 0.f;

            // The round's frames, two a step, one per half warp: the sub-blocks of
            // `mask`; on a tile of the diagonal (DIAG) the pairs k < j are left out. False,
            // to the whole warp, once a wait has run out: its lanes leave together, as the
            // shuffles and votes below take all of them.
            auto sum_frames = [&](auto mask_tag, auto diag_tag, int mask_arg) {
                constexpr int MASK = decltype(mask_tag)::value;
                constexpr bool DIAG = decltype(diag_tag)::value;
                const int mask = MASK != 0 ? MASK : mask_arg;
                const float2 *const run = xs + (wc * p.slots_p + wp) * run_elems + lane_off +
                                          (half * N + J * kTile) * rs;
                const int to_k = (K - J) * kTile * rs;
                const int step = 2 * N * rs;
                int n_left = n_mine;
                for (int s = round_stages(r); s > 0; --s, n_left -= p.fs, ++used) {
                    const int slot = used & slot_mask;
                    const bool landed = mbar_wait_bounded(
                        &full[slot], static_cast<uint32_t>(used >> p.slot_shift) & 1u, p.err,
                        kErrXengineMmaTimeout, abort_flag);
                    if (!__all_sync(0xffffffffu, landed)) {
                        s_abort = 1;
                        return false;
                    }
                    const float2 *xj = run + slot * slot_elems;
                    const int nf = MASK == 0 && KIND != kAny ? 0 : min(p.fs, n_left);
#pragma unroll 1
                    for (int f = 0; f < nf; f += 2, xj += step) {
                        // the odd frame of a last pair, which is not there, counts as
                        // zeros; zeros has one station after the other, whatever the
                        // layout of the ring (ch + (kTile - 1) * rs stays inside it)
                        const float2 *yk = f + half < nf ? xj + to_k : zeros + ch;
                        constexpr int NY = MASK == 0x5 || MASK == 0x1 ? kSub : kTile;
                        constexpr int NX = MASK == 0x1 ? kSub : kTile;
                        float2 x[kTile], y[kTile];
#pragma unroll
                        for (int l = 0; l < NY; ++l) y[l] = yk[l * rs];
#pragma unroll
                        for (int i = 0; i < NX; ++i) x[i] = DIAG ? y[i] : xj[i * rs];
                        // j = 6J + i against k = 6K + l, l0 <= l < l1
                        auto mac = [&](int i, int l0, int l1) {
#pragma unroll
                            for (int l = l0; l < l1; ++l) {
                                re[i][l] = fmaf(x[i].x, y[l].x, re[i][l]);
                                im[i][l] = fmaf(x[i].y, y[l].x, im[i][l]);
                            }
#pragma unroll
                            for (int l = l0; l < l1; ++l) {
                                re[i][l] = fmaf(x[i].y, y[l].y, re[i][l]);
                                im[i][l] = fmaf(-x[i].x, y[l].y, im[i][l]);
                            }
                        };
                        if constexpr (MASK != 0) {
#pragma unroll
                            for (int i = 0; i < NX; ++i) mac(i, DIAG ? i : 0, NY);
                        } else {
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if ((mask >> q) & 1) {
#pragma unroll
                                    for (int i = 0; i < kSub; ++i)
                                        mac(q / 2 * kSub + i, q % 2 * kSub, q % 2 * kSub + kSub);
                                }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[slot]);
                }
                return true;
            };
            using std::integral_constant;
            bool summed;
            if (sub == 0xf) {
                summed = sum_frames(integral_constant<int, 0xf>{}, std::false_type{}, 0);
            } else if (sub == 0xb && J == K) {   // a whole tile of the diagonal
                summed = sum_frames(integral_constant<int, 0xb>{}, std::true_type{}, 0);
            } else if (KIND == kAny) {
                summed = sum_frames(integral_constant<int, 0>{}, std::false_type{}, sub);
            } else if (KIND == kEdge && sub == 0x5) {   // the last column, of 1 to 3 stations
                summed = sum_frames(integral_constant<int, 0x5>{}, std::false_type{}, 0);
            } else if (KIND == kEdge && sub == 0x1) {   // and its diagonal tile
                summed = sum_frames(integral_constant<int, 0x1>{}, std::true_type{}, 0);
            } else {   // no tile: the slots only pass
                summed = sum_frames(integral_constant<int, 0>{}, std::false_type{}, 0);
            }
            if (!summed) return;
            if (sub == 0) continue;

            // The half warps' sums together (even + odd frames), each half warp
            // keeping three of the six rows. Then part after part (turn): each adds
            // to the sum so far of its tile, in shared memory, and the last one adds
            // the total to the row, as reductions at L2 (the launch's only ones to
            // those values), so that the result does not depend on the warps' timing.
            if (!SIDE && p.n_parts > 1) {   // part 0: until the tile before is through
                const long long t0 = clock64();
                bool mine = true;
                while (*turn != t) {
                    if (*abort_flag != 0 || clock64() - t0 > kWaitBudgetCycles) {
                        mine = false;
                        break;
                    }
                }
                if (!__all_sync(0xffffffffu, mine)) {
                    if (p.err != nullptr && *abort_flag == 0) atomicExch(p.err, kErrXengineMmaTimeout);
                    s_abort = 1;
                    return;
                }
                __threadfence_block();
            }
            const size_t c = static_cast<size_t>(ct) * kXch + ch;
#pragma unroll
            for (int i3 = 0; i3 < kSub; ++i3) {
                const int j = J * kTile + kSub * half + i3;
                // where baseline (j, 0) of a full square would be
                const size_t row = static_cast<size_t>(j * N - j * (j + 1) / 2) * p.n_freq + c;
#pragma unroll
                for (int l = 0; l < kTile; ++l) {
                    const float gr = half ? re[i3][l] : re[kSub + i3][l];   // the other's
                    const float gi = half ? im[i3][l] : im[kSub + i3][l];
                    const float ar = __shfl_xor_sync(0xffffffffu, gr, 16);
                    const float ai = __shfl_xor_sync(0xffffffffu, gi, 16);
                    const float mr = half ? re[kSub + i3][l] : re[i3][l];
                    const float mi = half ? im[kSub + i3][l] : im[i3][l];
                    float2 v = make_float2(mr + ar, mi + ai);
                    const int e = (i3 * kTile + l) * 32;
                    if constexpr (SIDE) {
                        so_far[wp * kSumElems + e] = v;
                        continue;
                    }
                    if (t > 0) v = cadd(so_far[e], v);
                    if (t < p.n_parts - 1) {
                        so_far[e] = v;
                        continue;
                    }
                    const int k = K * kTile + l;
                    if (j <= k && k < N && ((sub >> (2 * half + l / kSub)) & 1))
                        add_to_row<ACC64>(p.acc, row + static_cast<size_t>(k) * p.n_freq, v);
                }
            }
            if constexpr (!SIDE) {
                if (p.n_parts > 1) {
                    __threadfence_block();
                    __syncwarp();
                    if (lane == 0) *turn = (t + 1) % p.n_parts;
                }
                continue;
            }
            // Four or eight parts side by side (SIDE): each part's warp has laid its sums
            // down, and when all have, each adds up every slots_p-th of them. One warp
            // after the other took as long as the frames themselves: 4 stations, n_freq
            // 2048, 300 frames 14.6 -> 8.3 us; 7 stations, 14336, 64 frames 34 -> 26 us. Two are
            // faster in turn (15 stations, n_freq 14336, 100 frames 61 us, 74 side by side).
            const int group = wc * p.tiles + wt;
            const uint32_t sum_rounds = s_rounds[warp];
            __syncwarp();
            if (lane == 0) mbar_arrive(&laid_down[group]);
            const bool all_there = mbar_wait_bounded(&laid_down[group], sum_rounds & 1u, p.err,
                                                     kErrXengineMmaTimeout, abort_flag);
            if (!__all_sync(0xffffffffu, all_there)) {
                s_abort = 1;
                return;
            }
            float2 *const carried = so_far + p.slots_p * kSumElems;   // the rounds before
#pragma unroll 1
            for (int e = wp; e < kSub * kTile; e += p.slots_p) {
                float2 v = so_far[e * 32];
                if (r > 0) v = cadd(carried[e * 32], v);
                for (int q = 1; q < p.slots_p; ++q) v = cadd(v, so_far[q * kSumElems + e * 32]);
                if (r < rounds - 1) {
                    carried[e * 32] = v;
                    continue;
                }
                const int j = J * kTile + kSub * half + e / kTile, l = e % kTile;
                const int k = K * kTile + l;
                if (j <= k && k < N && ((sub >> (2 * half + l / kSub)) & 1))
                    add_to_row<ACC64>(
                        p.acc,
                        static_cast<size_t>(j * N - j * (j + 1) / 2 + k) * p.n_freq + c, v);
            }
            // all read before the next round's are laid down
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&summed_up[group]);
                s_rounds[warp] = sum_rounds + 1;
            }
            __syncwarp();
            const bool all_read = mbar_wait_bounded(&summed_up[group], sum_rounds & 1u, p.err,
                                                    kErrXengineMmaTimeout, abort_flag);
            if (!__all_sync(0xffffffffu, all_read)) {
                s_abort = 1;
                return;
            }
        }
    }
}

__global__ void scale_kernel(float2 *__restrict__ acc, size_t n, float s) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += stride) {
        float2 v = acc[i];
        v.x *= s;
        v.y *= s;
        acc[i] = v;
    }
}

__global__ void scale64_kernel(double2 *__restrict__ acc, size_t n, double s) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += stride) {
        double2 v = acc[i];
        v.x *= s;
        v.y *= s;
        acc[i] = v;
    }
}

__global__ void add64_kernel(double2 *__restrict__ dst, const double2 *__restrict__ src,
                             size_t n) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += stride) {
        double2 v = dst[i];
        const double2 w = src[i];
        v.x += w.x;
        v.y += w.y;
        dst[i] = v;
    }
}

// (float)(v * s), s = s_hi + s_lo; exact: s is a power of two. This GPU multiplies and
// converts doubles at 2 lanes per SM and cycle, so v is cut, in integer arithmetic, into
// its leading 24 bits and the next 23 (and whether any bit follows) and multiplied in
// FP32: hi * s_hi + tail, to 2^-44 of it, rounded once by the last FMA, as the double
// product is rounded (exactly, if s is a power of two). Where 2^-43 more or less would
// round another way, the double product decides. That happens once in 2^19 values; rows
// that hold little else than ties (v a few bits longer than a float and s a power of two)
// are the exact case. Zeros, numbers near or past FP32's range, infinities and NaN go the
// long way too.
__device__ __forceinline__ float scaled_to_float(double v, float s_hi, float s_lo, double s,
                                                 bool exact) {
    const uint32_t top = static_cast<uint32_t>(__double2hiint(v));
    const uint32_t low = static_cast<uint32_t>(__double2loint(v));
    const uint32_t e = (top >> 20) & 0x7ffu;   // 1023 + exponent
    if (e - 960u > 127u) return static_cast<float>(v * s);   // |v| outside [2^-63, 2^65)
    const uint32_t sign = top & 0x80000000u;
    const uint32_t f_exp = (e - 896u) << 23;
    const float hi = __uint_as_float(sign | f_exp | ((top & 0xfffffu) << 3) | (low >> 29));
    // the low 29 bits' first 23, in units of hi's last place (the last one also set
    // if any after it is, so that it decides which way a product rounds)
    const float frac =
        __uint_as_float(0x3f800000u | ((low >> 6) & 0x7fffffu) | ((low & 0x3fu) != 0u)) - 1.0f;
    const float lo = frac * __uint_as_float(sign | (f_exp - (23u << 23)));
    const float tail = fmaf(hi, s_lo, lo * s_hi);
    const float r = fmaf(hi, s_hi, tail), d = fabsf(r) * 0x1p-43f;
    const bool sure = exact || fmaf(hi, s_hi, tail + d) == fmaf(hi, s_hi, tail - d);
    if (!sure || fabsf(r) < 0x1p-60f) return static_cast<float>(v * s);
    return r;
}

// Two channels per thread and step: 32 bytes of complex128 in, 16 bytes of complex64
// out. Bound by those bytes since the arithmetic left the FP64 pipe: 24 inputs, n_freq
// 16384 48 -> 33 us with its launch, 40 inputs 108 -> 63 us. blockIdx.x = row * n_map + baseline, blockIdx.y strides over its channels.
__global__ void __launch_bounds__(256)
    dump64_kernel(float2 *__restrict__ out, size_t out_row, const double2 *__restrict__ src,
                  size_t src_row, const int32_t *__restrict__ gmap,
                  const int32_t *__restrict__ lmap, int n_map, int half_freq, float s_hi,
                  float s_lo, double s, bool exact) {
    const int r = blockIdx.x / n_map, m = blockIdx.x - r * n_map;
    const int gb = gmap ? gmap[m] : m;
    const int lb = lmap ? lmap[m] : m;
    const double2 *a = src + r * src_row + static_cast<size_t>(lb) * half_freq * 2;
    float4 *o = reinterpret_cast<float4 *>(out + r * out_row +
                                           static_cast<size_t>(gb) * half_freq * 2);
#pragma unroll 2
    for (int c = blockIdx.y * 256 + threadIdx.x; c < half_freq; c += gridDim.y * 256) {
        const double2 a0 = a[2 * c], a1 = a[2 * c + 1];
        o[c] = make_float4(scaled_to_float(a0.x, s_hi, s_lo, s, exact),
                           scaled_to_float(a0.y, s_hi, s_lo, s, exact),
                           scaled_to_float(a1.x, s_hi, s_lo, s, exact),
                           scaled_to_float(a1.y, s_hi, s_lo, s, exact));
    }
}

// One thread records the GPU's global nanosecond timer: the latency marks of a
// captured batch (a kernel node keeps its place in the graph's order, where an
// event recorded during capture would only express a dependency).
__global__ void stamp_kernel(unsigned long long *slot) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *slot = t;
}

// One thread waits on an mbarrier whose phase never completes (nothing arrives
// on it), with a caller-chosen budget; the bounded wait gives up and records
// kErrSelftestTimeout. The barrier is then retired by arriving on it so the CTA
// exits with nothing pending.
__global__ void watchdog_selftest_kernel(int *err, long long budget) {
    __shared__ uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    fence_mbar_init();
    const long long t0 = clock64();
    bool done = false;
    while (!(done = mbar_try_wait(&bar, 0u))) {
        if (clock64() - t0 > budget) break;
    }
    if (!done) atomicExch(err, kErrSelftestTimeout);
    mbar_arrive(&bar);
}

} // namespace

corr_status watchdog_selftest_launch(int *err, long long budget_cycles, cudaStream_t stream) {
    watchdog_selftest_kernel<<<1, 32, 0, stream>>>(err, budget_cycles);
    return cuda_check(cudaGetLastError(), "watchdog_selftest_kernel launch");
}

// Parts of a launch: its frames in contiguous runs, summed apart and then added up
// in order. One, or more where the channels alone leave warps idle and a part
// keeps 16 frames. A function of n_freq and frames alone, never of the station
// count or of the baselines computed: devices that hold different stations of one
// run sum the same sets of frames and agree to the bit. (Even and odd frames are
// summed apart too, so that no sum runs over more than half of the frames: its
// two roundings per frame then leave less error than one rounding per frame of a
// sum over all of them.)
static int plain_parts(int n_freq, int frames) {
    int h = 1;
    while (h < kMaxParts && n_freq / kXch * h < 152 * 12 && frames / (2 * h) >= 16) h *= 2;
    return h;
}

void xengine_plain_tiles(int n_station, const std::vector<int32_t> &baselines,
                         std::vector<uint16_t> *out) {
    const int nb = (n_station + kTile - 1) / kTile;
    std::vector<int> mask(static_cast<size_t>(nb) * nb, 0);
    auto mark = [&](int j, int k) {
        mask[static_cast<size_t>(j / kTile) * nb + k / kTile] |=
            1 << (2 * (j / kSub % 2) + k / kSub % 2);
    };
    int b = 0;
    size_t next = 0;   // into the (ascending) baselines
    for (int j = 0; j < n_station; ++j)
        for (int k = j; k < n_station; ++k, ++b) {
            if (next < baselines.size() && baselines[next] == b) {
                mark(j, k);
                ++next;
            }
        }
    out->clear();
    for (int J = 0; J < nb; ++J)
        for (int K = J; K < nb; ++K)
            if (const int m = mask[static_cast<size_t>(J) * nb + K])
                out->push_back(static_cast<uint16_t>(J | (K << 5) | (m << 10)));
}

// All of them, in the same order; out has room for kMaxTiles.
static int whole_matrix_tiles(int n_station, uint16_t *out) {
    const int nb = (n_station + kTile - 1) / kTile;
    // the last row and column of tiles may have stations in their first half only
    auto half_only = [&](int J) { return J * kTile + kSub >= n_station; };
    int n = 0;
    for (int J = 0; J < nb; ++J)
        for (int K = J; K < nb; ++K) {
            const int b = half_only(K) ? 0x5 : 0xf;             // sub-blocks with stations k
            const int a = half_only(J) ? 0x3 : 0xf;             // ... and j
            const int m = a & b & (J == K ? 0xb : 0xf);         // 0x4 lies below the diagonal
            out[n++] = static_cast<uint16_t>(J | (K << 5) | (m << 10));
        }
    return n;
}

// Multiply-accumulates per pair of frames of a tile entry, about.
static int tile_weight(uint16_t e) {
    const bool diag = (e & 31) == ((e >> 5) & 31);
    const int m = e >> 10;
    const int n = (m & 1) + (m >> 1 & 1) + (m >> 2 & 1) + (m >> 3);
    return (diag ? 6 * n + 3 * (m >> 1 & 1) : 9 * n) + 3;   // and the loads
}

// Deal the tiles to the groups, and inside a group to the warps, so that the SM's
// four schedulers (warp % 4) get shares as equal as may be: heaviest first, each
// to the group, then to the place, where the most loaded scheduler has least. Runs
// for every launch, so without allocations and over the four schedulers' next free
// places alone: a launch's host time at 24 / 64 / 128 stations (253 tiles)
// 4.1 / 9.6 / 35.9 -> 3.3 / 4.2 / 8.1 us.
static void place_tiles(const uint16_t *tiles, PlainParams *p) {
    constexpr int kHeaviest = 4 * 9 + 3, kMaxGroups = (kMaxTiles + kMaxWarps - 1) / kMaxWarps;
    int at[kHeaviest + 2] = {};   // counting sort, heaviest first
    uint16_t order[kMaxTiles];
    for (int i = 0; i < p->n_tiles; ++i) ++at[kHeaviest + 1 - tile_weight(tiles[i])];
    for (int w = 0; w < kHeaviest; ++w) at[w + 1] += at[w];
    for (int i = 0; i < p->n_tiles; ++i) order[at[kHeaviest - tile_weight(tiles[i])]++] = tiles[i];
    int size[kMaxGroups] = {}, load[kMaxGroups] = {};
    for (int i = 0; i < p->n_tiles; ++i) {
        int g = 0;   // a full group's load is out of reach
        for (int j = 1; j < p->tile_groups; ++j)
            if (load[j] < load[g]) g = j;
        p->tile[g * p->tiles + size[g]++] = order[i];
        load[g] += size[g] < p->tiles ? tile_weight(order[i]) : 1 << 20;
    }
    // copies of a place r on scheduler s
    int on[4][4] = {};
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < p->slots_p * p->slots_c; ++c) ++on[r][(r + c * p->tiles) % 4];
    for (int g = 0; g < p->tile_groups; ++g) {
        uint16_t *slot = p->tile + g * p->tiles;
        uint16_t mine[kMaxWarps];
        std::copy(slot, slot + size[g], mine);
        std::fill(slot, slot + p->tiles, uint16_t(0));
        int busy[4] = {0, 0, 0, 0};
        int next[4] = {0, 1, 2, 3};   // the first free place of each scheduler
        for (int i = 0; i < size[g]; ++i) {
            const int w = tile_weight(mine[i]);
            int best = -1, best_sq = 0;
            for (int r = 0; r < 4; ++r) {
                if (next[r] >= p->tiles) continue;
                int sq = 0;
                for (int s = 0; s < 4; ++s) {
                    const int v = busy[s] + w * on[r][s];
                    sq += v * v;
                }
                if (best < 0 || sq < best_sq || (sq == best_sq && next[r] < next[best])) {
                    best = r;
                    best_sq = sq;
                }
            }
            slot[next[best]] = mine[i];
            next[best] += 4;
            for (int s = 0; s < 4; ++s) busy[s] += w * on[best][s];
        }
    }
}

corr_status xengine_plain_launch(const XengineArgs &a, int num_sms, cudaStream_t stream) {
    if (a.frames <= 0) return CORR_OK;
    const int N = a.n_station;
    PlainParams p{};
    uint16_t whole[kMaxTiles];
    const uint16_t *tiles = whole;
    if (a.tiles != nullptr) {
        tiles = a.tiles->data();
        p.n_tiles = static_cast<int>(a.tiles->size());
    } else {
        p.n_tiles = whole_matrix_tiles(N, whole);
    }
    if (p.n_tiles == 0) return CORR_OK;
    const int n_ct = a.n_freq / kXch;
    p.n_parts = plain_parts(a.n_freq, a.frames);
    p.seg = ((a.frames + p.n_parts - 1) / p.n_parts + 1) / 2 * 2;
    // Ring: four slots (eight if they are small), each as long as fits; rows past
    // the last station are read (and dropped) by the last tile, hence the pad.
    const size_t pad = static_cast<size_t>(kTile) * kXch * sizeof(float2);
    const size_t run_pair = static_cast<size_t>(2) * N * kXch * sizeof(float2);
    // Sums of a (channel tile, tile) in shared memory: one that the parts' warps add to in
    // turn; four or eight side by side have one each, and one that the rounds carry on.
    auto group_sums = [&](int slots_p) {
        if (slots_p < 4) return p.n_parts > 1 ? 1 : 0;
        return slots_p + (slots_p < p.n_parts ? 1 : 0);
    };
    auto sums_of = [&](int slots_p, int slots_c) {
        return static_cast<size_t>(p.tiles) * slots_c * group_sums(slots_p) * kSumElems *
               sizeof(float2);
    };
    auto budget_of = [&](int slots_p, int slots_c, int ctas) -> size_t {
        const size_t sums = sums_of(slots_p, slots_c);
        const size_t sm = static_cast<size_t>(224 * 1024) / ctas, fixed = 2048 + pad + sums;
        return sm > fixed && (run_pair * slots_p * slots_c << 2) <= sm - fixed ? sm - fixed : 0;
    };
    // CTA shape: every tile of a channel tile if they fit, in tile groups (that
    // read the same spectra) otherwise; then parts side by side; then channel
    // tiles. Not wider than the ring has room for (a few baselines of many
    // stations: few tiles, long runs).
    p.tile_groups = (p.n_tiles + kMaxWarps - 1) / kMaxWarps;
    p.tiles = (p.n_tiles + p.tile_groups - 1) / p.tile_groups;
    p.slots_p = 1;
    while (p.slots_p < p.n_parts && p.tiles * p.slots_p * 2 <= kMaxWarps &&
           budget_of(p.slots_p * 2, 1, 1) > 0)
        p.slots_p *= 2;
    // Channel tiles side by side: as many as cost least. The busiest SM's tiles take
    // about their frames and 10 more for each part; every round of a CTA's units takes
    // another 100, since its first loads and its last sums have nothing beside them.
    // (100 and 10 come within 1.5 % of the best width over 550 launches: 1 to 40
    // stations, n_freq 1024 to 32768, 1 to 512 frames.) As wide as leaves each SM a
    // CTA, which was the rule, left a second round nearly empty: n_freq 32768, 4 stations
    // 64 frames 54 -> 25 us, 1 station 4 frames 10.2 -> 6.0.
    const int sms = std::max(1, num_sms);
    int per_sm = 1;
    int64_t least = -1;
    for (int c = 1; p.tiles * p.slots_p * c <= kMaxWarps; ++c) {
        int ctas = (kMaxWarps + 1) / (p.tiles * p.slots_p * c + 1);
        while (ctas > 1 && budget_of(p.slots_p, c, ctas) == 0) --ctas;
        if (budget_of(p.slots_p, c, ctas) == 0) break;
        const int units = (n_ct + c - 1) / c * p.tile_groups;
        const int rounds = (units + sms * ctas - 1) / (sms * ctas) * (p.n_parts / p.slots_p);
        const int64_t busiest = static_cast<int64_t>((units + sms - 1) / sms) * c * p.tiles;
        const int64_t cost = 100 * rounds + busiest * (10 * p.n_parts + a.frames);
        // as dear, the narrower; but the wider with six tiles or more, whose warps CTA by
        // CTA do not divide by the four schedulers (13 stations, n_freq 32768, 128 frames
        // 1.15 times as long)
        if (least >= 0 && (cost > least || (cost == least && p.tiles < 6))) continue;
        least = cost;
        per_sm = ctas;
        p.slots_c = c;
    }
    if (least < 0)
        return failf(CORR_ERR_ARG, "plain X-engine: %d stations do not fit in shared memory", N);
    p.units = (n_ct + p.slots_c - 1) / p.slots_c * p.tile_groups;
    place_tiles(tiles, &p);
    const size_t per_pair = run_pair * p.slots_p * p.slots_c;
    const int warps = p.tiles * p.slots_p * p.slots_c + 1;
    const size_t budget = budget_of(p.slots_p, p.slots_c, per_sm);
    const size_t sums = sums_of(p.slots_p, p.slots_c);
    p.group_sums = group_sums(p.slots_p);
    p.slot_shift = 8 * 16 * per_pair <= budget ? 3 : 2;
    p.fs = 2 * static_cast<int>(std::min<size_t>(16, (budget >> p.slot_shift) / per_pair));
    p.fs = std::min(p.fs, p.seg);   // no stages longer than a part: their rest would be zeros
    const size_t ring = ((per_pair * (p.fs / 2)) << p.slot_shift) + pad;
    p.sums_at = static_cast<int>(ring / sizeof(float2));
    const size_t smem = ring + sums;
    p.n_station = N;
    p.n_freq = a.n_freq;
    p.frames = a.frames;
    p.ytile = a.ytile;
    p.acc = a.acc;
    p.err = a.err;

    EncodeTiledFn enc = encode_tiled();
    if (enc == nullptr)
        return fail(CORR_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    // Spectra as (channel within its tile, station, frame, tile), 8 bytes a bin.
    const cuuint32_t box_c = static_cast<cuuint32_t>(std::min(a.ytile, kXch));
    const cuuint64_t row = static_cast<cuuint64_t>(a.ytile) * sizeof(float2);
    CUtensorMap map;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(a.ytile), static_cast<cuuint64_t>(N),
                                static_cast<cuuint64_t>(a.frames),
                                static_cast<cuuint64_t>(a.n_freq / a.ytile)};
    const cuuint64_t strides[3] = {row, row * N, row * N * a.y_frames};
    const cuuint32_t box[4] = {box_c, static_cast<cuuint32_t>(N), static_cast<cuuint32_t>(p.fs),
                               kXch / box_c};
    const CUresult cr =
        enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, const_cast<float2 *>(a.y), dims, strides,
            box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS)
        return failf(CORR_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(cr));

    using Kernel = void (*)(CUtensorMap, PlainParams);
    // [complex128 rows][parts' sums side by side][narrow spectra tiles][kind]
#define CORRGB_PLAIN_KINDS(ROW, ACC64, SIDE)                                                  \
    {xengine_plain_kernel<ROW, kWhole, ACC64, SIDE>, xengine_plain_kernel<ROW, kEdge, ACC64, SIDE>, \
     xengine_plain_kernel<ROW, kAny, ACC64, SIDE>}
    static constexpr Kernel kernels[2][2][2][3] = {
        {{CORRGB_PLAIN_KINDS(true, false, false), CORRGB_PLAIN_KINDS(false, false, false)},
         {CORRGB_PLAIN_KINDS(true, false, true), CORRGB_PLAIN_KINDS(false, false, true)}},
        {{CORRGB_PLAIN_KINDS(true, true, false), CORRGB_PLAIN_KINDS(false, true, false)},
         {CORRGB_PLAIN_KINDS(true, true, true), CORRGB_PLAIN_KINDS(false, true, true)}}};
#undef CORRGB_PLAIN_KINDS
    static PerDevice setup;   // the shared-memory limit is a per-device setting
    corr_status st = setup.run([](int) {
        for (int k = 0; k < 24; ++k) {
            corr_status s2 =
                cuda_check(cudaFuncSetAttribute(kernels[k / 12][k / 6 % 2][k / 3 % 2][k % 3], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                224 * 1024),
                           "cudaFuncSetAttribute(xengine_plain)");
            if (s2 != CORR_OK) return s2;
        }
        return CORR_OK;
    });
    if (st != CORR_OK) return st;
    const int grid = std::min(p.units, sms * per_sm);
    const int kind = a.tiles != nullptr ? kAny : (N - 1) % kTile < kSub ? kEdge : kWhole;
    const Kernel kernel = kernels[a.acc64 ? 1 : 0][p.slots_p >= 4][a.ytile < kXch][kind];
    kernel<<<grid, warps * 32, smem, stream>>>(map, p);
    return cuda_check(cudaGetLastError(), "xengine_plain_kernel launch");
}

corr_status scale_launch(float2 *acc, size_t n, float s, cudaStream_t stream) {
    if (n == 0) return CORR_OK;
    size_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    scale_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(acc, n, s);
    return cuda_check(cudaGetLastError(), "scale_kernel launch");
}

namespace {
unsigned grid_for(size_t n, unsigned cap) {
    size_t blocks = (n + 255) / 256;
    if (blocks > cap) blocks = cap;
    return static_cast<unsigned>(blocks < 1 ? 1 : blocks);
}
} // namespace

corr_status scale64_launch(double2 *acc, size_t n, double s, cudaStream_t stream) {
    if (n == 0) return CORR_OK;
    scale64_kernel<<<grid_for(n, 4096), 256, 0, stream>>>(acc, n, s);
    return cuda_check(cudaGetLastError(), "scale64_kernel launch");
}

corr_status add64_launch(double2 *dst, const double2 *src, size_t n, cudaStream_t stream) {
    if (n == 0) return CORR_OK;
    add64_kernel<<<grid_for(n, 4096), 256, 0, stream>>>(dst, src, n);
    return cuda_check(cudaGetLastError(), "add64_kernel launch");
}

corr_status dump64_launch(float2 *out, size_t out_row, const double2 *src, size_t src_row,
                          const int32_t *gmap, const int32_t *lmap, int n_map, int n_freq,
                          int rows, double s, cudaStream_t stream) {
    if (n_freq % 2 != 0) return fail(CORR_ERR_INTERNAL, "dump64: n_freq must be even");
    const int64_t lines = static_cast<int64_t>(n_map) * rows;
    if (lines <= 0) return CORR_OK;
    if (lines > 0x7fffffff) return fail(CORR_ERR_INTERNAL, "dump64: too many rows");
    // four steps a thread where there are lines enough to fill the GPU
    const int half = n_freq / 2;
    const int steps = lines * half >= (1 << 19) ? 4 : 1;
    const dim3 grid(static_cast<unsigned>(lines),
                    static_cast<unsigned>((half + 256 * steps - 1) / (256 * steps)));
    const float s_hi = static_cast<float>(s), s_lo = static_cast<float>(s - s_hi);
    int e;
    const bool exact = std::frexp(s, &e) == 0.5;
    dump64_kernel<<<grid, 256, 0, stream>>>(out, out_row, src, src_row, gmap, lmap, n_map, half,
                                            s_hi, s_lo, s, exact);
    return cuda_check(cudaGetLastError(), "dump64_kernel launch");
}

// MurmurHash3's 32-bit finaliser (a published integer mixing function).
__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

// Sum of four uniform bytes, centred and scaled: close to N(0, 24^2), in int8.
__global__ void synth_fill_kernel(int8_t *x, size_t n, uint32_t seed) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += stride) {
        const uint32_t h = mix32(static_cast<uint32_t>(i) ^ mix32(static_cast<uint32_t>(i >> 32) + seed));
        const int sum = static_cast<int>((h & 0xff) + ((h >> 8) & 0xff) + ((h >> 16) & 0xff) +
                                         (h >> 24)) - 510;
        const int v = __float2int_rn(static_cast<float>(sum) * 0.1624f);
        x[i] = static_cast<int8_t>(max(-127, min(127, v)));
    }
}

corr_status synth_fill_launch(int8_t *x, size_t n, uint32_t seed, cudaStream_t stream) {
    if (n == 0) return CORR_OK;
    size_t blocks = (n + 255) / 256;
    if (blocks > 16384) blocks = 16384;
    synth_fill_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(x, n, seed);
    return cuda_check(cudaGetLastError(), "synth_fill_kernel launch");
}

corr_status stamp_launch(unsigned long long *slot, cudaStream_t stream) {
    stamp_kernel<<<1, 1, 0, stream>>>(slot);
    return cuda_check(cudaGetLastError(), "stamp_kernel launch");
}

} // namespace corrgb
