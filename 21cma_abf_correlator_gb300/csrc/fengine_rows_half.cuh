// fengine_rows_half.cuh -- the F-engine kernel of n_freq 18432 .. 32768: the transform
// of fengine_rows.cuh twice per frame.
//
// n_freq = 2 M complex points do not fit in shared memory, so a radix-2 step of
// decimation in frequency splits the frame z into a[e] = z[e] + z[e + M], whose
// transform is the even bins, and b[e] = (z[e] - z[e + M]) exp(-pi i e / M), the odd
// ones, transformed one after the other. b's factor costs no pass of its own: with
// e = 16 a + b, a = 32 a1 + a0, it is half a bin more in the exponents of the three
// passes: exp(-pi i a1 / R0) on the samples, w_2L^(a0 (2 k1 + 1)) as second-pass
// twiddles (a table of their own in tensor memory) and w_2M^(b (2 j + 1)) in the last
// pass (a's table times w_2M^b; butterfly J-1-t's are conjugates of butterfly t's but
// for W_16^b, which only moves the DFT's outputs by one place).
//
// The data take 16 rows x 33 R0 points, the frame's regrouped samples (both halves of
// it) another 64 KB at M = 16384, so no landing buffer for a copy is left. The next
// frame is prefetched into L2 and regrouped straight from global memory in b's second
// pass: a lane loads four points of its row of 16, and stmatrix.trans turns 8 x 8
// blocks. Sample row 8 sel + c holds b = 4 (c / 2) + 2 sel + c % 2, as the loads bring
// them, so that its eight rows lie in different banks.
//
// Measured on one GB300, 24 stations, 512 frames, FP16 / hi-lo / FP32 output, the
// Stockham form (a landing buffer, a CTA barrier on each side of a pass) -> this one:
//   18432 1003 / 1214 / 1206 -> 898 / 1061 / 1052 us
//   20480 1121 / 1333 / 1319 -> 886 / 1117 / 1106 us
//   22528 1137 / 1374 / 1357 -> 971 / 1259 / 1234 us
//   24576 1250 / 1587 / 1487 -> 970 / 1313 / 1296 us
//   26624 1515 / 1937 / 1868 -> 1145 / 1463 / 1443 us
//   28672 1525 / 2057 / 2031 -> 1132 / 1563 / 1553 us
//   30720 2303 / 2642 / 2608 -> 1279 / 1617 / 1663 us
//   32768 1308 / 1666 / 1675 -> 1055 / 1596 / 1570 us
// (four frames of 18432: 16.5 -> 18.1 us.) Even and odd bins share 32-byte sectors and are
// written a transform apart, which costs DRAM 1.37 times the reads (FP16 output; ncu, 256
// frames of 32768) and the 8-byte formats most.
// Keeping the even ones in L2 until then took 32768 hi-lo from 1712 to 1565-1596 us;
// letting the odd ones go first 1642, and either for FP16 up to 9 % slower.

#ifndef CORR_GB300_FENGINE_ROWS_HALF_CUH
#define CORR_GB300_FENGINE_ROWS_HALF_CUH

#include "fengine_rows.cuh"

namespace corrgb {
namespace {

__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t *r) {
    asm volatile(
        "stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
        : "memory");
}

// A row's first pass: 18 .. 30 = 2 R2 (R2 odd), 4 R2 or 8 x 3, prime-factor form; 32.
template <int R>
__device__ __forceinline__ void dft_row(float2 *v) {
    if constexpr (R == 32)
        Dft<32>::run(v);
    else if constexpr (R == 24)
        DftPfa<8, 3>::run<false>(v);
    else if constexpr (R % 4 == 0)
        DftPfa<4, R / 4>::template run<false>(v);
    else
        DftPfa<2, R / 2>::template run<false>(v);
}

template <int MM>
struct FhCfg {
    using C = FrCfg<MM>;
    static_assert(C::RPW == 1 && C::G == 1 && C::CHAIN == 4, "a warp per row, a frame per CTA");
    static constexpr int T_HALF = C::ROWS * C::TROW;   // regrouped samples of half a frame
    static constexpr int OFF_D = 2 * T_HALF;
    static constexpr int OFF_HS = OFF_D + C::ROWS * C::DROW * 8;   // exp(-pi i r / R0)
    static constexpr int OFF_OM = OFF_HS + 32 * 8;                 // w_2M^r
    static constexpr int OFF_BAR = OFF_OM + 16 * 8;
    static constexpr int SMEM = OFF_BAR + 2 * 8 + 8;
    static_assert(SMEM <= 227 * 1024 && OFF_D % 16 == 0, "shared memory");
    static_assert((128 + 2 * (MM / 64)) * 8 <= C::ROWS * C::DROW * 8, "tables fit in the data");
    static constexpr int TM_ODD = C::TM_USED;          // b's second-pass twiddles
    static constexpr int TM_COLS = TM_ODD + 64 <= 256 ? 256 : 512;
    static_assert(TM_ODD + 64 <= 512, "tensor memory");
};

template <int MM, int FMT, bool CONTIG>
__global__ void __launch_bounds__(512, 1) fengine_rows_half_kernel(FengineArgs a, TwPtrs tw) {
    using C = FrCfg<MM>;
    using H2 = FhCfg<MM>;
    constexpr int M = C::M, R0 = C::R0, J = C::J, R = 16, H = R / 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float2 *const sd = reinterpret_cast<float2 *>(smem + H2::OFF_D);
    float2 *const hs = reinterpret_cast<float2 *>(smem + H2::OFF_HS);
    float2 *const om = reinterpret_cast<float2 *>(smem + H2::OFF_OM);
    uint64_t *const data_read = reinterpret_cast<uint64_t *>(smem + H2::OFF_BAR);
    uint64_t *const samples_read = data_read + 1;
    // as in fengine_rows_kernel: set before the threads meet, looked at after
    volatile int *const abort_flag = reinterpret_cast<volatile int *>(smem + H2::OFF_BAR + 16);
    __shared__ uint32_t s_tmem;
    const float out_scale = (FMT == kSpectraF32) ? 1.0f : a.y_scale;   // FP32 bins unscaled

    float2 *const plo = sd, *const phi = plo + 64;
    float2 *const qlo = phi + M / 64, *const qhi = qlo + 64;
    for (int i = t; i < 64; i += C::T) {
        plo[i] = tw.pass_lo[i];
        qlo[i] = tw.post_lo[i];
    }
    for (int i = t; i < M / 64; i += C::T) {
        phi[i] = tw.pass_hi[i];
        qhi[i] = tw.post_hi[i];
    }
    if (t < R0) hs[t] = tw.post_hi[8 * t];   // M / R0 = 512 = 8 x 64
    if (t < R) om[t] = tw.post_lo[t];
    const float2 odd_shift = *tw.odd_shift;
    if (t == 0) {
        mbar_init(data_read, C::WPF);
        mbar_init(samples_read, C::WPF);
        abort_flag[0] = abort_flag[1] = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, H2::TM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm_lane = s_tmem + (static_cast<uint32_t>(warp & 3) << 21);   // lane 32*(warp%4)
    const uint32_t tm_warp = tm_lane + 64 + C::TM_WARP * (warp >> 2);
    const bool last_active = t < J / 2;   // whole warps
    fill_twiddles<MM>(tm_lane, tm_warp, plo, phi, qlo, qhi, 0.5f * out_scale, lane, warp, t,
                      last_active);
    {
        const int c = warp >> 2, k1 = lane % R0;
        float2 w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            // w_2L^(a0 (2 k1 + 1)) = exp(-pi i u / M)
            int u = (8 * c + q) * (2 * k1 + 1) * C::ROWS;
            const bool neg = u >= M;
            u -= neg ? M : 0;
            const float2 x = cmul(qlo[u & 63], qhi[u >> 6]);
            w[q] = neg ? make_float2(-x.x, -x.y) : x;
        }
        tmem_store8(tm_lane + H2::TM_ODD + 16 * c, w);
        tmem_store_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // Even bins fill half of each sector: they wait in L2 for the odd ones. Samples are
    // read once.
    uint64_t keep, normal, once;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    const int n_items = a.frames * a.n_station, stride = gridDim.x;
    const int ytile_shift = __ffs(a.ytile) - 1;
    using Row = YRow<FMT, CONTIG, 2>;
    auto row_of = [&](int item, int odd) {
        return Row{reinterpret_cast<typename Row::T *>(a.y) + static_cast<size_t>(item) * a.ytile,
                   static_cast<uint32_t>(a.y_frames) * a.n_station * a.ytile, ytile_shift,
                   out_scale, 0.5f * out_scale, odd, odd ? normal : keep};
    };
    auto src_of = [&](int item) {
        const int f = item / a.n_station, s = item - f * a.n_station;
        return a.samples + static_cast<size_t>(s) * a.station_stride +
               static_cast<size_t>(f) * a.frame_stride;
    };
    // The first item from `item` on whose frame is there; the spectra of the
    // missing ones before it are zeros.
    auto next_present = [&](int item) {
        for (; item < n_items; item += stride) {
            const int f = item / a.n_station;
            if (frame_present<M>(a, f, item - f * a.n_station)) break;
            const Row even = row_of(item, 0), odd = row_of(item, 1);
            for (int k = t; k < M; k += C::T) {
                even.put(k, make_float2(0.f, 0.f));
                odd.put(k, make_float2(0.f, 0.f));
            }
        }
        return item;
    };
    const uint32_t t_at = smem_addr(smem);
    // A frame to rows, 16 a's (512 bytes) a step.
    constexpr int kPairs = 2 * C::L / 16, kSteps = (kPairs + C::WPF - 1) / C::WPF;
    auto regroup = [&](int item) {
        const int8_t *src = src_of(item) + lane * 8;
        uint2 x[kSteps][2];
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
            const int p = i * C::WPF + warp;
            if (kPairs % C::WPF != 0 && p >= kPairs) break;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.b32 {%0, %1}, [%2], %3;"
                             : "=r"(x[i][h].x), "=r"(x[i][h].y)
                             : "l"(src + p * 512 + h * 256), "l"(once));
        }
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
            const int p = i * C::WPF + warp;
            if (kPairs % C::WPF != 0 && p >= kPairs) break;
            const bool second = p >= kPairs / 2;
            const int a0 = (p - (second ? kPairs / 2 : 0)) * 16 + (lane >> 4) * 8;
            const uint32_t r[4] = {x[i][0].x, x[i][0].y, x[i][1].x, x[i][1].y};
            stmatrix_x4_trans(t_at + (second ? H2::T_HALF : 0) + (lane & 15) * C::TROW + a0 * 2, r);
        }
    };
    const int chain = warp >> 2;   // step of four warps into the last pass

    int cur = next_present(blockIdx.x);
    int nxt = n_items;
    if (cur < n_items) {
        regroup(cur);
        nxt = next_present(cur + stride);
        __syncthreads();
    }
    // this warp's row of points: sample row `warp`, data row b
    float2 *const drow = sd + (4 * ((warp & 7) >> 1) + 2 * (warp >> 3) + (warp & 1)) * C::DROW;
    const bool lane_used = lane < R0;
    const int k1 = lane_used ? lane : 0;

    // n counts half frames: even ones a, odd ones b
    for (uint32_t n = 0; cur < n_items; ++n) {
        const bool odd = n & 1;
        {
            float2 v[R0];
            const uint32_t at =
                t_at + warp * C::TROW +
                ((2 * (lane >> 3) + (lane & 1)) * 32 + ((lane >> 1) & 3) * 8) * 2;
            // a: (x + B) + ((y + B) - 2B), b: (x + B) - (y + B), exactly
            const float sgn = odd ? -1.0f : 1.0f, off = odd ? 0.0f : -2.0f * kInt8Bias;
#pragma unroll
            for (int q = 0; q < (R0 + 7) / 8; ++q) {
                // eight a1 a load; past the last one the first is read again
                uint32_t x[4], y[4];
                const bool over = R0 % 8 != 0 && 8 * q + 2 * (lane >> 3) >= R0;
                ldmatrix_x4_trans(at + (over ? 0 : q * 8 * 64), x);
                ldmatrix_x4_trans(at + H2::T_HALF + (over ? 0 : q * 8 * 64), y);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int r = 8 * q + 2 * m;
                    if (r >= R0) break;
                    const uint32_t ux = x[m] ^ 0x80808080u, uy = y[m] ^ 0x80808080u;
                    auto biased = [](uint32_t u, uint32_t sel) {
                        return __uint_as_float(__byte_perm(u, 0x4B000000u, sel));
                    };
                    v[r] = cadd(make_float2(biased(ux, 0x7440), biased(ux, 0x7441)),
                                fma2(make_float2(sgn, sgn),
                                     make_float2(biased(uy, 0x7440), biased(uy, 0x7441)),
                                     make_float2(off, off)));
                    v[r + 1] = cadd(make_float2(biased(ux, 0x7442), biased(ux, 0x7443)),
                                    fma2(make_float2(sgn, sgn),
                                         make_float2(biased(uy, 0x7442), biased(uy, 0x7443)),
                                         make_float2(off, off)));
                }
            }
            if (odd) {
                __syncwarp();
                if (lane == 0) mbar_arrive(samples_read);
#pragma unroll
                for (int r = 1; r < R0; ++r) v[r] = cmul(v[r], hs[r]);
            }
            dft_row<R0>(v);
            // the data of the half before must be read
            if (n > 0 && !mbar_wait_bounded(data_read, (n - 1) & 1, a.err, kErrFengineCopyTimeout))
                abort_flag[n & 1] = 1;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R0; ++r) drow[r * 33 + lane] = v[r];
        }
        __syncwarp();
        {
            float2 v[32];
#pragma unroll
            for (int r = 0; r < 32; ++r) v[r] = drow[k1 * 33 + 4 * (r & 7) + (r >> 3)];   // a0 = r
            if (odd) {   // row 0's twiddle is 1 in either table
                tmem_twiddles<32>(v, tm_lane + H2::TM_ODD);
            } else {
                tmem_twiddles<32>(v, tm_lane);
            }
            Dft<32>::run(v);
            __syncwarp();
            if (lane_used) {
#pragma unroll
                for (int r = 0; r < 32; ++r) drow[k1 + R0 * r] = v[r];
            }
        }
        if (nxt < n_items) {
            if (odd) {   // the samples have been read twice
                if (!mbar_wait_bounded(samples_read, (n >> 1) & 1, a.err, kErrFengineCopyTimeout))
                    abort_flag[n & 1] = 1;
                __syncwarp();
                regroup(nxt);
            } else if (t * 128 < 4 * M) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(src_of(nxt) + t * 128));
            }
        }
        __syncthreads();
        if (abort_flag[n & 1]) break;

        // Last pass and real-FFT split, as last_pass_store and last_pass_store_odd.
        if (chain > 0) named_wait(8 + chain - 1, 256);
        if (!last_active) {
            if (chain < C::CHAIN - 1) named_pass(8 + chain, 256);
            if (lane == 0) mbar_arrive(data_read);
        } else {
            const bool t0 = t == 0;
            const int j1 = t, j2 = odd ? J - 1 - t : t0 ? J / 2 : J - t;
            float2 x[R], y[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                x[r] = sd[r * C::DROW + j1];
                y[r] = sd[r * C::DROW + j2];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(data_read);
            if (odd) {
                __syncwarp();   // the loads take the whole warp
#pragma unroll
                for (int c = 0; c < R / 8; ++c) {
                    float2 w[8];
                    tmem_load8(tm_warp + 16 * c, w);
                    tmem_wait8(w);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int r = 8 * c + q;
                        if (r == 0) continue;
                        const float2 wb = cmul(w[q], om[r]);   // w_2M^(r (2 j1 + 1))
                        x[r] = cmul(x[r], wb);
                        y[r] = cmul(y[r], make_float2(wb.x, -wb.y));
                    }
                }
            } else {
                tmem_twiddles<R>(x, tm_warp);
            }
            Dft<R>::run(x);   // Z[j1 + r*J]
            if (chain < C::CHAIN - 1) named_pass(8 + chain, 256);
            if (!odd) tmem_twiddles<R>(y, tm_warp + 2 * R);
            Dft<R>::run(y);   // Z[j2 + r*J]; b: y[(r + 1) % R]
            const Row yrow = row_of(cur, odd);
            float2 w[2][8];
            __syncwarp();
            tmem_load8(tm_warp + 4 * R, w[0]);
            tmem_wait8(w[0]);
            tmem_load8(tm_warp + 4 * R + 16, w[1]);
            if (odd) {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    split_store(x[q], y[(R - q) % R], cmul(w[0][q], odd_shift), j1 + q * J, M - 1,
                                true, yrow);
                __syncwarp();
                tmem_wait8(w[1]);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    // thread 0's second half in the table is a's; b's is -i times the first
                    const float2 wq = t0 ? make_float2(w[0][q].y, -w[0][q].x) : w[1][q];
                    split_store(x[H + q], y[H - q], cmul(wq, odd_shift), j1 + (H + q) * J, M - 1,
                                true, yrow);
                }
            } else {
                // thread 0's butterflies 0 and J/2 pair with themselves
                const int kB = t0 ? J / 2 : j1 + H * J;
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    const float2 zmk = t0 ? x[(R - i) % R] : y[R - 1 - i];
                    split_store(x[i], zmk, w[0][i], j1 + i * J, M, !(t0 && i == 0), yrow);
                }
                __syncwarp();
                tmem_wait8(w[1]);
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    const float2 zk = t0 ? y[i] : x[H + i];
                    const float2 zmk = t0 ? y[R - 1 - i] : y[H - 1 - i];
                    split_store(zk, zmk, w[1][i], kB + i * J, M, true, yrow);
                }
                if (t0) yrow.put(M / 2, make_float2(x[H].x * yrow.scale, -x[H].y * yrow.scale));
            }
        }
        if (odd) {
            cur = nxt;
            nxt = next_present(nxt + stride);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(s_tmem, H2::TM_COLS);
}

template <int MM, int FMT, bool CONTIG>
corr_status launch_rows_half_one(const FengineArgs &a, const TwiddleTables &tw, int num_sms,
                                 cudaStream_t stream) {
    using H2 = FhCfg<MM>;
    static PerDevice setup;   // the shared-memory limit is a per-device setting
    corr_status st = setup.run([](int) {
        return cuda_check(cudaFuncSetAttribute(fengine_rows_half_kernel<MM, FMT, CONTIG>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               H2::SMEM),
                          "cudaFuncSetAttribute(fengine_rows_half)");
    });
    if (st != CORR_OK) return st;
    const int items = a.frames * a.n_station;
    if (items <= 0) return CORR_OK;
    TwPtrs p{tw.pass_lo, tw.pass_hi, tw.post_lo, tw.post_hi, tw.odd_shift};
    const int grid = std::min(items, num_sms);
    fengine_rows_half_kernel<MM, FMT, CONTIG><<<grid, 512, H2::SMEM, stream>>>(a, p);
    return cuda_check(cudaGetLastError(), "fengine_rows_half_kernel launch");
}

// n_freq = 2*MH above 16384: two MH-point transforms per frame.
template <int MH>
corr_status launch_rows_half(const FengineArgs &a, const TwiddleTables &tw, int num_sms,
                             cudaStream_t stream) {
    if (a.fplan != 0)
        return failf(CORR_ERR_ARG, "FFT plan %d is not available at n_freq=%d", a.fplan, 2 * MH);
    if (a.pmask != nullptr)
        return failf(CORR_ERR_ARG,
                     "n_freq=%d: packet masks cover frames of at most 32 packets (n_freq <= 16384)",
                     2 * MH);
    if (tw.odd_shift == nullptr)
        return failf(CORR_ERR_INTERNAL, "n_freq=%d: twiddle tables lack the odd-bin shift", 2 * MH);
    const bool contig = a.ytile == 2 * MH;
    if (a.y_fmt == kSpectraF16)
        return contig ? launch_rows_half_one<MH, kSpectraF16, true>(a, tw, num_sms, stream)
                      : launch_rows_half_one<MH, kSpectraF16, false>(a, tw, num_sms, stream);
    if (a.y_fmt == kSpectraF16Split)
        return contig ? launch_rows_half_one<MH, kSpectraF16Split, true>(a, tw, num_sms, stream)
                      : launch_rows_half_one<MH, kSpectraF16Split, false>(a, tw, num_sms, stream);
    return contig ? launch_rows_half_one<MH, kSpectraF32, true>(a, tw, num_sms, stream)
                  : launch_rows_half_one<MH, kSpectraF32, false>(a, tw, num_sms, stream);
}

} // namespace
} // namespace corrgb

#endif // CORR_GB300_FENGINE_ROWS_HALF_CUH
