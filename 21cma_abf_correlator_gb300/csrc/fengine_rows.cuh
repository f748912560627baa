// fengine_rows.cuh -- the F-engine kernel of n_freq 4096 .. 16384: the transform of
// fengine_impl.cuh decimated so that the first of its two exchanges stays inside a
// warp, with the twiddles in tensor memory.
//
// A frame is M complex points z[n], n = 16 a + b. Row b (16 of them) is the L = M/16
// points z[16 a + b]; a warp owns RPW whole rows:
//   first pass   radix R0 = L/32 over a1, a = 32 a1 + a0 (lane = a0), straight from
//                the int8 samples; exchange within the warp's rows;
//   second pass  radix 32 over a0 (lane = row and k1), twiddles w_L^(a0 k1);
//                -> Y_b[k1 + R0 k2] to shared memory; exchange between all warps;
//   last pass    radix 16 over b fused with the real-FFT split and the store, as
//                last_pass_store does: thread t owns k' = t and J - t (J = L).
// Only the second exchange needs the frame's warps to meet. The other waits are
// "the frame before has been read" (data and samples), on mbarriers that the
// readers arrive on as soon as their loads are done, half a frame early.
//
// What bounded the plain Stockham form: a pass between two CTA barriers is either
// shared-memory traffic (47 % of the time) or FP32 work (52 %), all warps in step,
// so the two added up. Here the last pass is entered by four warps after another
// (one per scheduler: `chain`), which keeps the warps a quarter pass apart for the
// whole frame; frames of 4096 or 8192 points go four or two to a CTA, each in its
// own group of warps. The twiddles (62 + 92 words a thread, constant over frames)
// come from tensor memory, off the shared-memory path, where a table read or a
// product per twiddle was.
//
// The int8 samples: the landed frame is regrouped into rows by ldmatrix.trans /
// stmatrix (8 x 8 blocks of sample pairs, 16 bits each) and read by ldmatrix.trans,
// which hands a thread the points a1, a1 + 1 of its a0 = 8 (lane % 4) + lane / 4.
//
// Measured on one GB300, 24 stations, 1024 frames, FP16 / hi-lo / FP32 output, the
// Stockham form -> this one: n_freq 16384 1051 / 1245 / 1150 -> 866 / 957 / 905 us,
// 8192 484 / 564 / 536 -> 433 / 527 / 490 us, 6144 480 / - / 498 -> 443 / - / 461 us,
// 4096 223 / 254 / - -> 211 / 243 / - us; 15 stations, n_freq 12288, 301 frames, FP32
// 232 -> 185 us. At 16384 the decimation alone gave nothing (1063 us), with the chained
// entry 1039, with the tables in tensor memory instead 1060, with both 923, with the
// read barriers and the regrouping moved into the second pass 867. Per SM and cycle
// now: issue 66 %, FP32 pipe about 55 %, shared-memory wavefronts 48 %; what is left
// is arithmetic with too few warps (4 per scheduler, 128 registers) to fill every gap.

#ifndef CORR_GB300_FENGINE_ROWS_CUH
#define CORR_GB300_FENGINE_ROWS_CUH

#include <algorithm>

#include "fengine_impl.cuh"

namespace corrgb {
namespace {

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t *r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, const uint32_t *r) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}

// Named barriers: `threads` of them meet (wait), or some only report (pass).
__device__ __forceinline__ void named_wait(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_pass(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <int MM>
struct FrCfg {
    static constexpr int M = MM, T = 512, ROWS = 16;
    static constexpr int L = M / ROWS;             // points of a row
    static constexpr int R0 = L / 32;              // radix of the first pass
    static_assert(L == 32 * R0 && R0 >= 8 && R0 <= 32, "row length");
    static constexpr int RPW = 32 / R0;            // rows per warp
    static constexpr int WPF = ROWS / RPW;         // warps per frame
    static constexpr int G = T / 32 / WPF;         // frames in flight, a group of warps each
    static_assert(WPF * RPW == ROWS && WPF * G * 32 == T && WPF % 4 == 0, "warp layout");
    static constexpr int FT = WPF * 32;            // threads per frame
    static constexpr int J = L;                    // butterflies of the last pass
    static constexpr int CHAIN = WPF / 4;          // steps of four warps into the last pass
    static constexpr int DROW = 33 * R0;           // float2 of a data row
    static constexpr int TROW = 2 * L + 16;        // bytes of a row of sample pairs
    // shared memory (bytes): per group the landed frame, the regrouped samples, the data
    static constexpr int OFF_T = 2 * M;
    static constexpr int OFF_D = OFF_T + ROWS * TROW;
    static constexpr int GROUP = OFF_D + ROWS * DROW * 8;
    static constexpr int OFF_BAR = G * GROUP;      // three mbarriers per group
    static constexpr int OFF_FLAG = OFF_BAR + 3 * 8 * G;   // two words per group
    static constexpr int SMEM = OFF_FLAG + 8 * G;
    static_assert(SMEM <= 227 * 1024 && GROUP % 16 == 0, "shared memory");
    // the twiddle tables the tensor-memory ones are made from, before the first frame
    static_assert((128 + 2 * (M / 64)) * 8 <= GROUP, "tables fit in a group's memory");
    // tensor-memory columns: the second pass's twiddles (per lane), then per warp of
    // a lane quarter the last pass's 2 x 16 and the split's 16
    static constexpr int TM_WARP = 96;
    static constexpr int TM_USED = 64 + TM_WARP * ((J / 2 + 127) / 128);
    static constexpr int TM_COLS = TM_USED <= 256 ? 256 : 512;
    static_assert(TM_USED <= 512, "tensor memory");
};

constexpr int inverse_mod(int a, int m) {
    int x = 1;
    while (a * x % m != 1) ++x;
    return x;
}

// Radix 2, 4 or 8 x R2 with an odd R2, prime-factor form (no twiddles): input n =
// (R2 n1 + R1 n2) mod R, output k = (R2 (R2^-1 mod R1) k1 + R1 (R1^-1 mod R2) k2) mod
// R. BIASED inputs carry the int8 unpacking's offset (Dft<4>::run_biased).
template <int R1, int R2>
struct DftPfa {
    static constexpr int R = R1 * R2;
    static constexpr int U1 = R2 * inverse_mod(R2, R1), U2 = R1 * inverse_mod(R1, R2);
    template <bool BIASED>
    static __device__ __forceinline__ void run(float2 *v, float2 two_b = float2{}) {
        static_assert(R1 > 2 || !BIASED, "radix 2 takes plain inputs");
        float2 y[R2][R1];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) y[n2][n1] = v[(R2 * n1 + R1 * n2) % R];
            if constexpr (R1 == 2) {
                const float2 s = cadd(y[n2][0], y[n2][1]);
                y[n2][1] = csub(y[n2][0], y[n2][1]);
                y[n2][0] = s;
            } else if constexpr (R1 == 4 && BIASED) {
                Dft<4>::run_biased(y[n2], two_b);
            } else if constexpr (R1 == 4) {
                Dft<4>::run(y[n2]);
            } else {
                Dft<R1>::template run<BIASED>(y[n2], two_b);
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            float2 t[R2];
#pragma unroll
            for (int n2 = 0; n2 < R2; ++n2) t[n2] = y[n2][k1];
            Dft<R2>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) v[(U1 * k1 + U2 * k2) % R] = t[k2];
        }
    }
};

template <int R>
__device__ __forceinline__ void dft_from_int8(float2 *v) {
    const float2 two_b = make_float2(2.0f * kInt8Bias, 2.0f * kInt8Bias);
    if constexpr (R == 12 || R == 20 || R == 28)
        DftPfa<4, R / 4>::template run<true>(v, two_b);
    else if constexpr (R == 24)
        DftPfa<8, 3>::run<true>(v, two_b);
    else
        Dft<R>::template run<true>(v, two_b);
}

// v[r] *= w[r], r = 1 .. R-1, w this thread's R twiddles in tensor memory at `tm`
// (w[0] unused). Chunks of eight, the next one loaded while one is multiplied.
template <int R>
__device__ __forceinline__ void tmem_twiddles(float2 *v, uint32_t tm) {
    static_assert(R % 8 == 0, "chunks of eight");
    float2 w[2][8];
    __syncwarp();
    tmem_load8(tm, w[0]);
#pragma unroll
    for (int c = 0; c < R / 8; ++c) {
        tmem_wait8(w[c & 1]);
        if (c + 1 < R / 8) tmem_load8(tm + 16 * (c + 1), w[(c + 1) & 1]);
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (c + r > 0) v[8 * c + r] = cmul(v[8 * c + r], w[c & 1][r]);
    }
}

// The second pass's twiddles of this lane (tm_lane) and, for the threads t < J/2 of
// the last pass, theirs: w_M^(r j1), w_M^(r j2) and the split's h w_2M^k in
// last_pass_store's order (tm_warp). Each is one product of two entries of the tables
// in shared memory. The warps that share a table write different parts of it.
template <int MM>
__device__ __forceinline__ void fill_twiddles(uint32_t tm_lane, uint32_t tm_warp,
                                              const float2 *plo, const float2 *phi,
                                              const float2 *qlo, const float2 *qhi, float half,
                                              int lane, int warp, int t, bool last) {
    using C = FrCfg<MM>;
    constexpr int R = 16, H = R / 2, J = C::J;
    {
        const int c = warp >> 2;   // four chunks, four warps of each lane quarter
        float2 w[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
            w[r] = tw_pass(plo, phi, (8 * c + r) * (lane % C::R0) * C::ROWS);
        tmem_store8(tm_lane + 16 * c, w);
    }
    if (last) {   // a whole warp or none (J/2 is a multiple of 32)
        const int part = warp / C::WPF;   // group
        // w^(r j2) = W_16^r conj(w^(r j1)) for j2 = J - j1; thread 0's j2 is J/2
        for (int c = part; c < R / 8; c += C::G) {
            float2 w[8], w2[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int r = 8 * c + q;
                w[q] = tw_pass(plo, phi, r * t);
                const float cr = c == 0 ? cos32(2 * q) : cos32(2 * q + 16);
                const float sr = c == 0 ? sin32(2 * q) : sin32(2 * q + 16);
                const float ch = c == 0 ? cos32(q) : cos32(q + 8);
                const float sh = c == 0 ? sin32(q) : sin32(q + 8);
                w2[q] = t == 0 ? make_float2(ch, -sh)
                               : cmul(make_float2(cr, -sr), make_float2(w[q].x, -w[q].y));
            }
            tmem_store8(tm_warp + 16 * c, w);
            tmem_store8(tm_warp + 2 * R + 16 * c, w2);
        }
        // the split's: k = j1 + i J, a 32nd root of unity apart (thread 0, second
        // half: k = J/2 + (i - H) J)
        for (int c = part; c < R / 8; c += C::G) {
            const int k = c == 0 ? t : t == 0 ? J / 2 : t + H * J;
            const float2 w0 = scale_tw(cmul(qlo[k & 63], qhi[k >> 6]), half);
            float2 w[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) w[q] = mul_w32(w0, q);
            tmem_store8(tm_warp + 4 * R + 16 * c, w);
        }
    }
    tmem_store_wait();
}

template <int MM, int FMT, bool CONTIG>
__global__ void __launch_bounds__(512, 1) fengine_rows_kernel(FengineArgs a, TwPtrs tw) {
    using C = FrCfg<MM>;
    constexpr int M = C::M, R0 = C::R0, RPW = C::RPW, FT = C::FT, J = C::J;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = warp / C::WPF;                   // group: a frame of its own
    const int t = threadIdx.x - g * FT;            // thread and warp within the group
    const int wf = warp - g * C::WPF;
    unsigned char *const raw = smem + g * C::GROUP;
    float2 *const sd = reinterpret_cast<float2 *>(raw + C::OFF_D);
    uint64_t *const bar = reinterpret_cast<uint64_t *>(smem + C::OFF_BAR) + 3 * g;
    uint64_t *const data_read = bar + 1, *const samples_read = bar + 2;
    // A wait of frame n that ran out sets word n & 1 of its group before the threads
    // meet, and all of them look at it after: they leave together, none at a barrier.
    volatile int *const abort_flag = reinterpret_cast<volatile int *>(smem + C::OFF_FLAG) + 2 * g;
    __shared__ uint32_t s_tmem;
    __shared__ volatile uint32_t entered[4];   // frames each group has taken into the last pass
    const float out_scale = (FMT == kSpectraF32) ? 1.0f : a.y_scale;   // FP32 bins unscaled

    float2 *const plo = reinterpret_cast<float2 *>(smem), *const phi = plo + 64;
    float2 *const qlo = phi + M / 64, *const qhi = qlo + 64;
    for (int i = threadIdx.x; i < 64; i += C::T) {
        plo[i] = tw.pass_lo[i];
        qlo[i] = tw.post_lo[i];
    }
    for (int i = threadIdx.x; i < M / 64; i += C::T) {
        phi[i] = tw.pass_hi[i];
        qhi[i] = tw.post_hi[i];
    }
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init(data_read, C::WPF);
        mbar_init(samples_read, C::WPF);
        abort_flag[0] = abort_flag[1] = 0;
        entered[g] = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, C::TM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm_lane = s_tmem + (static_cast<uint32_t>(warp & 3) << 21);   // lane 32*(warp%4)
    const uint32_t tm_warp = tm_lane + 64 + C::TM_WARP * (wf >> 2);
    const bool last_active = t < J / 2;   // whole warps
    fill_twiddles<MM>(tm_lane, tm_warp, plo, phi, qlo, qhi, 0.5f * out_scale, lane, warp, t,
                      last_active);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const int n_items = a.frames * a.n_station, stride = gridDim.x * C::G;
    const int ytile_shift = __ffs(a.ytile) - 1;
    using Row = YRow<FMT, CONTIG>;
    auto row_of = [&](int item) {
        return Row{reinterpret_cast<typename Row::T *>(a.y) + static_cast<size_t>(item) * a.ytile,
                   static_cast<uint32_t>(a.y_frames) * a.n_station * a.ytile, ytile_shift,
                   out_scale, 0.5f * out_scale};
    };
    // The first item from `item` on whose frame is there; the spectra of the
    // missing ones before it are zeros.
    auto next_present = [&](int item) {
        for (; item < n_items; item += stride) {
            const int f = item / a.n_station;
            if (frame_present<M>(a, f, item - f * a.n_station)) break;
            const Row yrow = row_of(item);
            for (int k = t; k < M; k += FT) yrow.put(k, make_float2(0.f, 0.f));
        }
        return item;
    };
    auto issue = [&](int item) {
        if (t == 0 && item < n_items) {
            const int f = item / a.n_station, s = item - f * a.n_station;
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(bar, 2 * M);
            bulk_copy_g2s(raw, a.samples + static_cast<size_t>(s) * a.station_stride +
                                   static_cast<size_t>(f) * a.frame_stride,
                          2 * M, bar);
        }
    };
    uint32_t parity = 0;
    const uint32_t raw_at = smem_addr(raw), t_at = raw_at + C::OFF_T;
    // The landed frame to rows. Points of lost packets (512 points, 32 a) become zeros.
    auto deinterleave = [&](int item, uint32_t n) {
        if (!mbar_wait_bounded(bar, parity, a.err, kErrFengineCopyTimeout)) abort_flag[n & 1] = 1;
        parity ^= 1u;
        const int f = item / a.n_station;
        const uint32_t kept = packets_kept<M>(a, f, item - f * a.n_station);
        const int bh = (lane >> 3) & 1, row = lane & 7;
        __syncwarp();
#pragma unroll
        for (int q0 = 0; q0 < C::L / 16; q0 += C::WPF) {   // 16 a each
            const int q = q0 + wf;
            if ((C::L / 16) % C::WPF != 0 && q >= C::L / 16) break;
            const int a0 = q * 16 + (lane >> 4) * 8;
            uint32_t r[4];
            ldmatrix_x4_trans(raw_at + (a0 + row) * 32 + bh * 16, r);
            if (!((kept >> (q / 2)) & 1u)) r[0] = r[1] = r[2] = r[3] = 0u;
            stmatrix_x4(t_at + (bh * 8 + row) * C::TROW + a0 * 2, r);
        }
    };
    auto meet = [&] {   // the frame's threads
        if constexpr (C::G == 1)
            __syncthreads();
        else
            named_wait(1 + g, FT);
    };
    const int chain = wf >> 2;                        // step of four warps
    const int chain_id = 8 + g * (C::CHAIN - 1);      // its named barriers (G*(CHAIN-1) of them)

    int cur = next_present(blockIdx.x + g * gridDim.x);   // few items: one per SM
    issue(cur);
    int nxt = n_items;
    if (cur < n_items) {
        deinterleave(cur, 0);
        nxt = next_present(cur + stride);
        meet();
        // no second copy on a barrier whose first has not landed: leave at frame 0's meeting
        if (abort_flag[0]) nxt = n_items;
        issue(nxt);
    }
    float2 *const drow = sd + wf * RPW * C::DROW;     // this warp's rows
    // second pass: lane = row and k1 (the lanes past RPW*R0 repeat lane 0's work)
    const bool lane_used = lane < RPW * R0;
    const int k1 = lane_used ? lane % R0 : 0;
    float2 *const lrow = drow + (lane_used ? lane / R0 : 0) * C::DROW;

    for (uint32_t n = 0; cur < n_items; ++n) {
        {
            float2 v[RPW][R0];
            const uint32_t at =
                t_at + wf * RPW * C::TROW +
                ((2 * (lane >> 3) + (lane & 1)) * 32 + ((lane >> 1) & 3) * 8) * 2;
#pragma unroll
            for (int w = 0; w < RPW; ++w) {
#pragma unroll
                for (int q = 0; q < (R0 + 7) / 8; ++q) {
                    // eight a1 a load; past the last one the first is read again
                    uint32_t x[4];
                    const bool over = R0 % 8 != 0 && 8 * q + 2 * (lane >> 3) >= R0;
                    ldmatrix_x4_trans(at + w * C::TROW + (over ? 0 : q * 8 * 64), x);
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const int r = 8 * q + 2 * m;
                        if (r >= R0) break;
                        const uint32_t u = x[m] ^ 0x80808080u;   // int8_pair_to_biased
                        v[w][r] = make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440)),
                                              __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7441)));
                        v[w][r + 1] =
                            make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7442)),
                                        __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7443)));
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(samples_read);
#pragma unroll
            for (int w = 0; w < RPW; ++w) dft_from_int8<R0>(v[w]);
            // the data of the frame before must be read
            if (n > 0 && !mbar_wait_bounded(data_read, (n - 1) & 1, a.err, kErrFengineCopyTimeout))
                abort_flag[n & 1] = 1;
            __syncwarp();
            // k1-major, lane (not a0) fastest: both sides free of bank conflicts
#pragma unroll
            for (int w = 0; w < RPW; ++w)
#pragma unroll
                for (int r = 0; r < R0; ++r) drow[w * C::DROW + r * 33 + lane] = v[w][r];
        }
        __syncwarp();
        {
            float2 v[32];
#pragma unroll
            for (int r = 0; r < 32; ++r) v[r] = lrow[k1 * 33 + 4 * (r & 7) + (r >> 3)];   // a0 = r
            if (nxt < n_items) {
                if (!mbar_wait_bounded(samples_read, n & 1, a.err, kErrFengineCopyTimeout))
                    abort_flag[n & 1] = 1;
                deinterleave(nxt, n);
            }
            tmem_twiddles<32>(v, tm_lane);
            Dft<32>::run(v);
            __syncwarp();
            if (lane_used) {
#pragma unroll
                for (int r = 0; r < 32; ++r) lrow[k1 + R0 * r] = v[r];
            }
        }
        meet();
        if (abort_flag[n & 1]) {   // let the copy last waited for land
            if (t == 0) mbar_wait_bounded(bar, parity ^ 1u, nullptr, 0);
            break;
        }
        const int after = next_present(nxt + stride);
        issue(after);

        // Last pass and real-FFT split, as last_pass_store.
        if (C::CHAIN > 1 && chain > 0) named_wait(chain_id + chain - 1, 256);
        if (C::G > 1 && chain == 0 && g > 0) {
            // behind the group before, if it is about as far (only for speed: a group
            // that is not is not waited for long)
            const long long since = clock64();
            while (static_cast<int>(entered[g - 1] - (n + 1)) < 0 && clock64() - since < 6000) {
            }
            __syncwarp();
        }
        if (!last_active) {
            if (C::CHAIN > 1 && chain < C::CHAIN - 1) named_pass(chain_id + chain, 256);
            if (lane == 0) mbar_arrive(data_read);
        } else {
            constexpr int R = 16, H = R / 2;
            const Row yrow = row_of(cur);
            const int j1 = t, j2 = t == 0 ? J / 2 : J - t;
            float2 x[R], y[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                x[r] = sd[r * C::DROW + j1];
                y[r] = sd[r * C::DROW + j2];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(data_read);
            tmem_twiddles<R>(x, tm_warp);
            Dft<R>::run(x);   // x[r] = Z[j1 + r*J]
            if (C::CHAIN > 1 && chain < C::CHAIN - 1) named_pass(chain_id + chain, 256);
            if (C::G > 1 && t == FT - 128) entered[g] = n + 1;
            tmem_twiddles<R>(y, tm_warp + 2 * R);
            Dft<R>::run(y);   // y[r] = Z[j2 + r*J]
            // thread 0's butterflies 0 and J/2 pair with themselves
            const bool t0 = t == 0;
            const int kB = t0 ? J / 2 : j1 + H * J;
            float2 w[2][8];
            __syncwarp();
            tmem_load8(tm_warp + 4 * R, w[0]);
#pragma unroll
            for (int c = 0; c < R / 8; ++c) {
                __syncwarp();
                tmem_wait8(w[c & 1]);
                if (c + 1 < R / 8) tmem_load8(tm_warp + 4 * R + 16 * (c + 1), w[(c + 1) & 1]);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int i = 8 * c + q;
                    if (i < H) {
                        const float2 zmk = t0 ? x[(R - i) % R] : y[R - 1 - i];
                        split_store(x[i], zmk, w[c & 1][q], j1 + i * J, M, !(t0 && i == 0), yrow);
                    } else {
                        const float2 zk = t0 ? y[i - H] : x[i];
                        const float2 zmk = t0 ? y[R - 1 - (i - H)] : y[R - 1 - i];
                        split_store(zk, zmk, w[c & 1][q], kB + (i - H) * J, M, true, yrow);
                    }
                }
            }
            if (t0) yrow.put(M / 2, make_float2(x[H].x * yrow.scale, -x[H].y * yrow.scale));
        }
        cur = nxt;
        nxt = after;
    }
    if (C::G > 1 && t == 0) entered[g] = 0x7fffffffu;   // no one waits for it any more
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(s_tmem, C::TM_COLS);
}

template <int MM, int FMT, bool CONTIG>
corr_status launch_rows_one(const FengineArgs &a, const TwiddleTables &tw, int num_sms,
                            cudaStream_t stream) {
    using C = FrCfg<MM>;
    static PerDevice setup;   // the shared-memory limit is a per-device setting
    corr_status st = setup.run([](int) {
        return cuda_check(cudaFuncSetAttribute(fengine_rows_kernel<MM, FMT, CONTIG>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               C::SMEM),
                          "cudaFuncSetAttribute(fengine_rows)");
    });
    if (st != CORR_OK) return st;
    const int items = a.frames * a.n_station;
    if (items <= 0) return CORR_OK;
    TwPtrs p{tw.pass_lo, tw.pass_hi, tw.post_lo, tw.post_hi, tw.odd_shift};
    const int grid = std::min(items, num_sms);
    fengine_rows_kernel<MM, FMT, CONTIG><<<grid, C::T, C::SMEM, stream>>>(a, p);
    return cuda_check(cudaGetLastError(), "fengine_rows_kernel launch");
}

template <int MM>
corr_status launch_rows(const FengineArgs &a, const TwiddleTables &tw, int num_sms,
                        cudaStream_t stream) {
    if (a.fplan != 0)
        return failf(CORR_ERR_ARG, "FFT plan %d is not available at n_freq=%d", a.fplan, MM);
    const bool contig = a.ytile == MM;
    if (a.y_fmt == kSpectraF16)
        return contig ? launch_rows_one<MM, kSpectraF16, true>(a, tw, num_sms, stream)
                      : launch_rows_one<MM, kSpectraF16, false>(a, tw, num_sms, stream);
    if (a.y_fmt == kSpectraF16Split)
        return contig ? launch_rows_one<MM, kSpectraF16Split, true>(a, tw, num_sms, stream)
                      : launch_rows_one<MM, kSpectraF16Split, false>(a, tw, num_sms, stream);
    return contig ? launch_rows_one<MM, kSpectraF32, true>(a, tw, num_sms, stream)
                  : launch_rows_one<MM, kSpectraF32, false>(a, tw, num_sms, stream);
}

} // namespace
} // namespace corrgb

#endif // CORR_GB300_FENGINE_ROWS_CUH
