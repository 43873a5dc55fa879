// Frame-group gather kernel for complex ensembles: LF = 2, 4, 8 or 16 neighbouring lanes own one voxel,
// eight frames each, and share the arithmetic of its delays.
//
// A warp-wide 256-bit load of the voxel-per-lane kernel touched as many 128-byte lines as its 32
// voxels had sample rows (about 16), and used 32 bytes of each: the L1 tag stage, not its data path,
// bounded the kernel (200-frame complex64 Doppler: data pipe 72 %, time unchanged with twice the
// loads in flight).  Here the lanes of a voxel read adjacent 32-byte pieces of one row, so a
// load touches fewer lines, and whole ones.  The delay arithmetic is not repeated by the
// lanes of a voxel: each takes one of LF consecutive elements, forms the receive path and then, per
// transmit, the tap row and weights of its own element; the LF points are then summed one after
// the other by all of the voxel's lanes, their four parameters broadcast by warp shuffles.
//
// Measured on B200, 8-frame chunks of the voxel-per-lane kernel -> 4 lanes per voxel, 192 frames x 5
// transmits on 256 x 256: complex64 3.80 -> 2.80 ms (nearest 2.87 -> 1.54, quadratic 5.70 -> 3.80),
// FP16 pairs 3.08 -> 2.07 ms, int16 pairs 3.39 -> 2.74 ms; 8 lanes 2.56 ms (complex64) and 1.96 ms
// (FP16 pairs); 128 frames with 4 / 8 / 16 lanes 1.84 / 1.70 / 1.57 ms and 1.39 / 1.31 / 1.26 ms; 16 frames
// x 3 with 2 lanes: complex64 223 -> 193 us, FP16 pairs 208 -> 174 us.  What is left is load latency
// (complex64 with 4 lanes: issue 0.46 per cycle) and issue (FP16 pairs: 0.73); rows that are no
// multiple of 128 bytes (200 frames) make a voxel's piece straddle one line more.
#pragma once

#include "das_lane_voxel.cuh"

namespace mach_b200 {

constexpr int kGroupLaneFrames = 8;  // frames per lane: 64 bytes of complex64, 32 of 4-byte pairs

template <int S, int INTERP, int LF, bool SPLIT>
__device__ __forceinline__ void frame_group_tile(const DasArgs& a, int64_t tile, float* smem_words, int chunk) {
    using T = typename Storage<S>::T;
    static_assert(Storage<S>::kComplex, "complex storage");
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kVoxels = kLaneVoxelThreads / LF;
    constexpr int kPiece = 32 / static_cast<int>(sizeof(T));  // frames of one 256-bit load
    constexpr int kPieces = kGroupLaneFrames / kPiece;
    constexpr int kTaps = INTERP == kNearest ? 1 : (INTERP == kLinear ? 2 : 3);
    // [tx_chunk][kVoxels] arrivals; split mode: sample base, fraction, phase cycles
    float* const s_arrival = smem_words;
    int* const s_base = reinterpret_cast<int*>(s_arrival + a.tx_chunk * kVoxels);
    float* const s_cyc = s_arrival + 2 * a.tx_chunk * kVoxels;

    const int lane = threadIdx.x & 31;
    const int sub = lane & (LF - 1);
    const int lv = threadIdx.x / LF;  // voxel of the tile
    const int64_t v = lane_voxel_index<kVoxels>(a, tile, lv);
    const bool vox_ok = v < a.n_vox;
    if (a.probed_fast != nullptr && !__syncthreads_or(vox_ok)) return;

    float vx = 0.f, vy = 0.f, vz = 0.f;
    if (vox_ok) {
        vx = __ldg(a.scan + 3 * v + 0);
        vy = __ldg(a.scan + 3 * v + 1);
        vz = __ldg(a.scan + 3 * v + 2);
    }
    const float radius = __fdiv_rn(vz, a.two_f_number);  // kernel.cu:583
    const float radius_sq = __fmul_rn(radius, radius);
    float bx0 = vox_ok ? vx : INFINITY, bx1 = vox_ok ? vx : -INFINITY;
    float by0 = vox_ok ? vy : INFINITY, by1 = vox_ok ? vy : -INFINITY;
    float rmax = vox_ok ? fabsf(radius) : 0.f;
#pragma unroll
    for (int off = 16; off >= LF; off >>= 1) {
        bx0 = fminf(bx0, __shfl_xor_sync(kFull, bx0, off));
        bx1 = fmaxf(bx1, __shfl_xor_sync(kFull, bx1, off));
        by0 = fminf(by0, __shfl_xor_sync(kFull, by0, off));
        by1 = fmaxf(by1, __shfl_xor_sync(kFull, by1, off));
        rmax = fmaxf(rmax, __shfl_xor_sync(kFull, rmax, off));
    }
    const float cand_r2 = rmax * rmax * 1.00001f + 1e-30f;

    // Piece i of this lane: frames first[i] .. first[i] + kPiece - 1 of the row.  Pieces past the
    // row's end read its first frames instead and are not written.
    const int f0 = a.frame_first + chunk * (LF * kGroupLaneFrames);
    const unsigned row_bytes = static_cast<unsigned>(a.row_frames) * static_cast<unsigned>(sizeof(T));
    int first[kPieces];
    const char* base[kPieces];
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
        first[i] = f0 + (i * LF + sub) * kPiece;
        base[i] = static_cast<const char*>(a.channel) + (first[i] < a.row_frames ? first[i] * static_cast<int>(sizeof(T)) : 0);
    }
    float2 acc[kPieces][kPiece];
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
#pragma unroll
        for (int q = 0; q < kPiece; ++q) acc[i][q] = make_float2(0.f, 0.f);
    }

    // Add one point: first tap row (quadratic: centre row), interpolation parameter, phasor.
    auto add_point = [&](int row, float w, float cw, float sw) {
        unsigned d[kPieces][kTaps][8];
        const int rows[3] = {INTERP == kQuadratic ? row - 1 : row,
                             INTERP == kQuadratic ? row : row + (w > 0.0f ? 1 : 0), row + 1};
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
#pragma unroll
            for (int k = 0; k < kTaps; ++k) {
                unsigned* r = d[i][k];
                asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                    : "l"(base[i] + static_cast<uint64_t>(static_cast<unsigned>(rows[k])) * row_bytes));
            }
        }
        float w0 = w, w1 = 0.f, w2 = 0.f;
        if constexpr (INTERP == kQuadratic) {
            const float hx = __fmul_rn(0.5f, w);
            const float q = __fmul_rn(hx, w);
            w0 = __fsub_rn(q, hx);             // x (x - 1) / 2
            w1 = __fmaf_rn(-2.0f, q, 1.0f);    // (1 - x)(1 + x)
            w2 = __fadd_rn(q, hx);             // x (x + 1) / 2
        }
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            float2 x[kPiece];
            if constexpr (INTERP == kLinear && (S == kCF16 || S == kCBF16)) {
#pragma unroll
                for (int q = 0; q < kPiece; ++q) x[q] = lerp_half_word<S>(d[i][0][q], d[i][1][q], w0);
            } else {
                float2 t[kTaps][kPiece];
#pragma unroll
                for (int k = 0; k < kTaps; ++k) {
#pragma unroll
                    for (int h = 0; h < 4; ++h) widen8<S>(make_uint2(d[i][k][2 * h], d[i][k][2 * h + 1]), t[k] + h * (kPiece / 4));
                }
#pragma unroll
                for (int q = 0; q < kPiece; ++q) {
                    if constexpr (INTERP == kNearest) {
                        x[q] = t[0][q];
                    } else if constexpr (INTERP == kLinear) {
                        x[q].x = __fmaf_rn(w0, __fsub_rn(t[1][q].x, t[0][q].x), t[0][q].x);
                        x[q].y = __fmaf_rn(w0, __fsub_rn(t[1][q].y, t[0][q].y), t[0][q].y);
                    } else {
                        x[q].x = __fmaf_rn(w2, t[kTaps - 1][q].x, __fmaf_rn(w0, t[0][q].x, __fmul_rn(w1, t[1][q].x)));
                        x[q].y = __fmaf_rn(w2, t[kTaps - 1][q].y, __fmaf_rn(w0, t[0][q].y, __fmul_rn(w1, t[1][q].y)));
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < kPiece; ++q) {
                acc[i][q].x = __fmaf_rn(x[q].x, cw, __fmaf_rn(-x[q].y, sw, acc[i][q].x));
                acc[i][q].y = __fmaf_rn(x[q].y, cw, __fmaf_rn(x[q].x, sw, acc[i][q].y));
            }
        }
    };

    const int tx_chunk = a.tx_chunk;
    for (int t0 = 0; t0 < a.n_tx; t0 += tx_chunk) {
        const int nt = min(tx_chunk, a.n_tx - t0);
        __syncthreads();
        for (int t = sub; t < nt; t += LF) {
            const int i = t * kVoxels + lv;
            const float txa = vox_ok ? __ldg(a.arrivals + static_cast<int64_t>(t0 + t) * a.n_vox + v) : 0.f;
            if constexpr (SPLIT) {
                const SplitPos sp = split_position((static_cast<double>(txa) - a.t0_d) * a.fs_d);
                s_base[i] = sp.base;
                s_arrival[i] = sp.frac;
                s_cyc[i] = reduced_cycles(static_cast<double>(txa) * a.fmod_d);
            } else {
                s_arrival[i] = txa;
            }
        }
        __syncthreads();

        for (int eb = a.e_begin; eb < a.e_end; eb += 32) {
            bool cand = false;
            if (eb + lane < a.e_end) {
                const float ex = __ldg(a.rx + 3 * (eb + lane) + 0);
                const float ey = __ldg(a.rx + 3 * (eb + lane) + 1);
                const float ddx = fmaxf(fmaxf(bx0 - ex, ex - bx1), 0.f);
                const float ddy = fmaxf(fmaxf(by0 - ey, ey - by1), 0.f);
                cand = ddx * ddx + ddy * ddy <= cand_r2;
            }
            const unsigned cmask = __ballot_sync(kFull, cand);
            // LF consecutive elements at a time, one per lane of a voxel, whatever the candidates are: the
            // order of a voxel's sum does not depend on which warp (tile) it is in.
            for (int eg = 0; eg < 32; eg += LF) {
                if (((cmask >> eg) & ((1u << LF) - 1u)) == 0u) continue;
                const bool e_ok = ((cmask >> (eg + sub)) & 1u) != 0u;
                const int e = e_ok ? eb + eg + sub : eb;
                PairRx rx{};
                const bool pair_ok = pair_receive<SPLIT ? 1 : 0>(a, __ldg(a.rx + 3 * e + 0), __ldg(a.rx + 3 * e + 1),
                                                                __ldg(a.rx + 3 * e + 2), vx, vy, vz, radius, radius_sq, rx) &&
                                     vox_ok && e_ok;
                if (!__any_sync(kFull, pair_ok)) continue;
                int row_e = (t0 * a.n_rx + e) * a.n_samples;
                const int row_step = a.n_rx * a.n_samples;
#pragma unroll 1
                for (int t = 0; t < nt; ++t, row_e += row_step) {
                    const int si = t * kVoxels + lv;
                    TapPosition tp{};
                    float w = 0.f, cw = rx.w, sw = 0.f;
                    bool ok;
                    if constexpr (SPLIT) {
                        int b = s_base[si] + rx.pos.base;
                        float frac = __fadd_rn(s_arrival[si], rx.pos.frac);
                        if (frac >= 1.0f) {
                            frac = __fsub_rn(frac, 1.0f);
                            b += 1;
                        }
                        ok = pair_ok && !(b < a.start_base || (b == a.start_base && frac < a.start_frac));
                        const bool inside = split_tap_position<INTERP>(b, frac, a.n_samples, tp);
                        ok = ok && inside;
                        w = INTERP == kQuadratic ? __fsub_rn(frac, static_cast<float>(tp.idx - b)) : tp.w0;
                        if (a.rotate) {
                            float sn, cs;
                            split_phasor(__fadd_rn(s_cyc[si], rx.cyc), sn, cs);
                            cw = __fmul_rn(cs, rx.w);
                            sw = __fmul_rn(sn, rx.w);
                        }
                    } else {
                        const float tau = __fmaf_rn(rx.dist, a.inv_c, s_arrival[si]);
                        const float s = __fmul_rn(__fsub_rn(tau, a.t0), a.fs);
                        ok = pair_ok && !(tau < 0.0f);
                        if constexpr (INTERP == kNearest) {
                            ok = ok && (s >= -0.5f) && (s <= a.hi_nearest);
                        } else if constexpr (INTERP == kLinear) {
                            ok = ok && (s >= 0.0f) && (s <= a.hi_linear);
                        } else {
                            ok = ok && (s >= 1.0f) && (s <= a.hi_quadratic);
                        }
                        tp = tap_position<INTERP>(s);
                        if constexpr (INTERP == kNearest) ok = ok && tp.idx < a.n_samples;
                        w = INTERP == kQuadratic ? __fsub_rn(s, static_cast<float>(tp.idx)) : tp.w0;
                        if (a.rotate) {
                            float sn, cs;
                            __sincosf(__fmul_rn(a.mod_rad, tau), &sn, &cs);  // kernel.cu:656-658
                            cw = __fmul_rn(cs, rx.w);
                            sw = __fmul_rn(sn, rx.w);
                        }
                    }
                    const int row = ok ? row_e + tp.idx : -1;
#pragma unroll
                    for (int k = 0; k < LF; ++k) {  // the point of lane k's element
                        const int rk = __shfl_sync(kFull, row, k, LF);
                        const float wk = __shfl_sync(kFull, w, k, LF);
                        const float ck = __shfl_sync(kFull, cw, k, LF), sk = __shfl_sync(kFull, sw, k, LF);
                        if (rk >= 0) add_point(rk, wk, ck, sk);
                    }
                }
            }
        }
    }

    if (!vox_ok) return;
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
#pragma unroll
        for (int q = 0; q < kPiece; ++q) {
            const int f = first[i] + q;
            if (f >= a.n_frames) continue;
            float2* out = static_cast<float2*>(a.out) + v * a.n_frames + f;
            float2 r = acc[i][q];
            if (a.accumulate) {
                const float2 prev = *out;
                r.x = __fadd_rn(prev.x, r.x);
                r.y = __fadd_rn(prev.y, r.y);
            }
            *out = r;
        }
    }
}

// CTAs per SM that the register budget is cut for: the kernel waits for its row loads, so it gains from
// every warp that fits (LF = 4, 192 frames on B200: complex64 6 / 7 / 8 CTAs 2.93 / 2.89 / 2.80 ms, FP16
// pairs 8 / 9 / 10 CTAs 2.14 / 2.12 / 2.07 ms; loading a point ahead in 128 registers was slower, 3.03
// and 2.35 ms), until the spills of the shorter loop of LF = 2 cost more (16 frames, 6 / 7 CTAs
// 193 / 233 us).
template <int S, int INTERP, int LF>
constexpr int frame_group_ctas() {
    if (INTERP == kQuadratic) return S == kC64 ? 5 : 8;
    if (LF >= 4) return S == kC64 ? 8 : 10;
    return S == kC64 ? 6 : 8;
}

template <int S, int INTERP, int LF, bool SPLIT>
__global__ void __launch_bounds__(kLaneVoxelThreads, frame_group_ctas<S, INTERP, LF>())
    das_frame_group_kernel(const __grid_constant__ DasArgs a) {
    extern __shared__ float smem_words[];
    const int64_t tile = blockIdx.x / a.frame_chunks;  // consecutive CTAs: the chunks of one tile, which share rows
    frame_group_tile<S, INTERP, LF, SPLIT>(a, tile, smem_words, static_cast<int>(blockIdx.x - tile * a.frame_chunks));
}

}  // namespace mach_b200
