// Analytic signal of contiguous columns (one frame per sample): the transform of das_hilbert.cu with
// its spectrum kept in digit order, for lengths that are products of small radices.
//
// n = R1 R2 .. Rm.  The forward transform is decimation in frequency, in place (Cooley and Tukey
// 1965; Gentleman and Sande 1966): stage j takes the DFTs of length R_j over digit j of the index
// and multiplies by the twiddles of the digits below; its output digit k_j stays where digit j was.
// After stage m, position (k1, .., km) holds bin k1 + R1 (k2 + R2 (k3 + ..)).  The inverse transform
// is the mirror image, stages m .. 1, and ends in time order.  So
//   * stage 1 reads its samples from global memory into registers, stage m of both directions and
//     the multiplier -i sgn(k) / n between them run on the same registers, and the last inverse stage
//     writes z = x + i y straight to global memory: 2 (m - 1) round trips through shared memory
//     instead of the 2 m + 2 of the out-of-place form, and no reordering;
//   * a thread's last stage covers the samples that its first stage read, so x waits in registers
//     (KEEP: every thread has at most one item of stage 1), and the next group's first stage may
//     start without a barrier;
//   * a column pair needs one buffer, not two.
// Two real columns are packed as x1 + i x2 as in das_hilbert.cu.  A CTA takes P pairs, P n about 4096,
// so that a stage has about one butterfly of 16 points per thread.  Buffer strides are padded so
// that the lanes of a half warp hit different banks.  Twiddles are FP64-rounded tables, computed
// once per CTA.
//
// Bound: the 12 bytes per sample of HBM traffic are 59 us for the compounding acquisition
// (32 M samples of 3328 = 16 16 13); instruction issue and the shared-memory round trips follow.
// Measured on B200 for that job: 0.52 ms out of place -> 0.22 ms in place (staging the next group with
// cp.async: 0.24 ms; three CTAs per SM without x in registers: 0.28 ms).  Out of place / in place for 16 M
// samples of other lengths, float32, acquisition order: 64 samples a column 542 / 183 us, 256 234 / 130 us,
// 2048 255 / 126 us, 5120 426 / 292 us (one CTA per SM, samples read twice), 8192 553 / 258 us; 1 M samples:
// 64 72 / 40 us, 2048 49 / 41 us, 8192 93 / 68 us.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

#include "das_device.cuh"
#include "das_launch.cuh"

namespace mach_b200 {
namespace {

constexpr int kThreads = 256;

// cos and sin of 2 pi m / R at compile time (Taylor series of the argument reduced to [-pi, pi]).
constexpr double kTwoPi = 6.283185307179586476925286766559;
__host__ __device__ constexpr double series(double x, double term, int k) {
    double sum = term;
    for (int i = 0; i < 20; ++i) {
        term *= -x * x / ((k + 1) * (k + 2));
        k += 2;
        sum += term;
    }
    return sum;
}
template <int R>
struct Roots {
    float c[R], s[R];
    __host__ __device__ constexpr Roots() : c(), s() {
        for (int m = 0; m < R; ++m) {
            const double x = kTwoPi * (2 * m > R ? m - R : m) / R;
            c[m] = static_cast<float>(series(x, 1.0, 0));
            s[m] = static_cast<float>(series(x, x, 1));
        }
    }
};

// Packed FP32x2, one instruction each (the difference as a + (-1) b, exact before its one rounding).
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
template <bool CONJ>
__device__ __forceinline__ float2 mul(float2 a, float2 w) {  // a w, or a conj(w)
    if (CONJ) return make_float2(fmaf(a.x, w.x, a.y * w.y), fmaf(a.y, w.x, -(a.x * w.y)));
    return make_float2(fmaf(a.x, w.x, -(a.y * w.y)), fmaf(a.x, w.y, a.y * w.x));
}
// a times W_R^m = exp(-2 pi i m / R) (forward) or its conjugate
template <int R, bool INV>
__device__ __forceinline__ float2 turn(float2 a, int m) {
    constexpr Roots<R> w{};
    m %= R;
    if (m == 0) return a;
    if (4 * m == R) return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
    if (2 * m == R) return make_float2(-a.x, -a.y);
    if (4 * m == 3 * R) return INV ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
    return mul<false>(a, make_float2(w.c[m], INV ? w.s[m] : -w.s[m]));
}

// First factor of a radix: 4, else 2, else an odd prime.
__host__ __device__ constexpr int first_factor(int r) {
    if (r % 4 == 0) return 4;
    for (int p = 2; p * p <= r; ++p)
        if (r % p == 0) return p;
    return r;
}

// DFT of R points in registers, natural order in and out.
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    constexpr int A = first_factor(R);
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const float2 a = v[0];
        v[0] = add(a, v[1]);
        v[1] = sub(a, v[1]);
    } else if constexpr (R == 4) {
        const float2 t0 = add(v[0], v[2]), t1 = sub(v[0], v[2]), t2 = add(v[1], v[3]);
        const float2 d = sub(v[1], v[3]);
        const float2 t3 = INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
        v[0] = add(t0, t2);
        v[2] = sub(t0, t2);
        v[1] = add(t1, t3);
        v[3] = sub(t1, t3);
    } else if constexpr (A < R) {  // R = A B: DFT_B over v[a + A b], twiddle W_R^(a c), DFT_A over a
        constexpr int B = R / A;
        float2 o[R];
        float2 t[A][B];
#pragma unroll
        for (int a = 0; a < A; ++a) {
            float2 u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) u[b] = v[a + A * b];
            dft<B, INV>(u);
#pragma unroll
            for (int c = 0; c < B; ++c) t[a][c] = turn<R, INV>(u[c], a * c);
        }
#pragma unroll
        for (int c = 0; c < B; ++c) {
            float2 u[A];
#pragma unroll
            for (int a = 0; a < A; ++a) u[a] = t[a][c];
            dft<A, INV>(u);
#pragma unroll
            for (int d = 0; d < A; ++d) o[c + B * d] = u[d];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = o[k];
    } else {  // odd prime, by the conjugate symmetry of the roots
        constexpr int H = (R - 1) / 2;
        constexpr Roots<R> w{};
        float2 x0 = v[0];
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            const float2 a = add(v[r], v[R - r]), b = sub(v[r], v[R - r]);
            v[r] = a;
            v[R - r] = b;
            x0 = add(x0, a);
        }
        float2 o[R];
        o[0] = x0;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            float2 p = v[0], s = make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 1; r <= H; ++r) {
                const int m = (r * q) % R;
                p.x = fmaf(v[r].x, w.c[m], p.x);
                p.y = fmaf(v[r].y, w.c[m], p.y);
                s.x = fmaf(v[R - r].x, w.s[m], s.x);
                s.y = fmaf(v[R - r].y, w.s[m], s.y);
            }
            const float2 is = make_float2(-s.y, s.x);
            o[q] = INV ? add(p, is) : sub(p, is);
            o[R - q] = INV ? sub(p, is) : add(p, is);
        }
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = o[k];
    }
}

// x / d and x % d for 0 <= x < 2^24: a float estimate off by at most one, then a correction.
__device__ __forceinline__ int div_mod(int x, int d, float rd, int& rem) {
    int q = __float2int_rz(__int2float_rn(x) * rd);
    rem = x - q * d;
    if (rem < 0) {
        --q;
        rem += d;
    } else if (rem >= d) {
        ++q;
        rem -= d;
    }
    return q;
}

// Buffer offset of index b < L[j] below digit j (digits j + 1 .. m - 1, counted from 0).
__device__ __forceinline__ int low_offset(const HilbertColsArgs& g, int j, int b) {
    int off = 0;
    for (int q = g.m - 1; q > j + 1; --q) {
        int d;
        b = div_mod(b, g.radix[q], g.r_radix[q], d);
        off += d * g.stride[q];
    }
    return j + 1 < g.m ? off + b * g.stride[j + 1] : 0;
}
// Buffer offset of digits 0 .. j - 1 of u (mixed radix, digit j - 1 fastest), and the frequency that
// they stand for.
__device__ __forceinline__ int high_offset(const HilbertColsArgs& g, int j, int u, int& freq) {
    int off = 0;
    freq = 0;
    for (int q = j - 1; q > 0; --q) {
        int d;
        u = div_mod(u, g.radix[q], g.r_radix[q], d);
        off += d * g.stride[q];
        freq += d * g.weight[q];
    }
    if (j > 0) {
        off += u * g.stride[0];
        freq += u;
    }
    return off;
}

// A middle stage: digit j of every pair's buffer.
template <int R, bool INV>
__device__ __forceinline__ void middle_stage(const HilbertColsArgs& g, int j, const float2* tw, float2* buf) {
    const int L = g.low[j], S = g.stride[j], items = g.items[j];
    for (int i = threadIdx.x; i < items << g.pairs_log2; i += kThreads) {
        int item = i, p = 0;
        if (g.pairs_log2) p = div_mod(i, items, g.r_items[j], item);
        int b, freq;
        const int u = div_mod(item, L, g.r_low[j], b);
        float2* at = buf + p * g.pair_size + high_offset(g, j, u, freq) + low_offset(g, j, b);
        const float2* w = tw + b;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            v[r] = at[r * S];
            if (INV && r > 0) v[r] = mul<true>(v[r], w[(r - 1) * L]);
        }
        dft<R, INV>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) at[r * S] = !INV && r > 0 ? mul<false>(v[r], w[(r - 1) * L]) : v[r];
    }
}

// Stage m of both directions with the multiplier -i sgn(k) / n between them.
template <int R>
__device__ __forceinline__ void turn_stage(const HilbertColsArgs& g, float2* buf) {
    const int j = g.m - 1, items = g.items[j], top = g.n / R;
    for (int i = threadIdx.x; i < items << g.pairs_log2; i += kThreads) {
        int item = i, p = 0;
        if (g.pairs_log2) p = div_mod(i, items, g.r_items[j], item);
        int freq;
        float2* at = buf + p * g.pair_size + high_offset(g, j, item, freq);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = at[r];
        dft<R, false>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int twice = 2 * (freq + r * top);
            const float f = twice == 0 || twice == g.n ? 0.f : (twice < g.n ? g.inv_n : -g.inv_n);
            v[r] = make_float2(v[r].y * f, -v[r].x * f);
        }
        dft<R, true>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) at[r] = v[r];
    }
}

template <typename T>
__device__ __forceinline__ float widen(T x) {
    return static_cast<float>(x);
}
template <>
__device__ __forceinline__ float widen(__half x) {
    return __half2float(x);
}
template <>
__device__ __forceinline__ float widen(__nv_bfloat16 x) {
    return __bfloat162float(x);
}

// R samples of a column pair, `step` samples apart (a column past the last one reads as 0).
template <typename In, int R>
__device__ __forceinline__ void load_pair(const HilbertColsArgs& g, int64_t off0, int64_t off1, int64_t step,
                                          float2 (&v)[R]) {
    const In* src = static_cast<const In*>(g.src);
    if (sizeof(In) == 4 && g.pair_vec) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = __ldg(reinterpret_cast<const float2*>(src + off0 + r * step));
        return;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        v[r].x = widen(__ldg(src + off0 + r * step));
        v[r].y = off1 >= 0 ? widen(__ldg(src + off1 + r * step)) : 0.f;
    }
}
template <int R>
__device__ __forceinline__ void load_any(const HilbertColsArgs& g, int64_t off0, int64_t off1, int64_t step,
                                         float2 (&v)[R]) {
    switch (g.src_code) {
        case kF32: load_pair<float>(g, off0, off1, step, v); break;
        case kF16: load_pair<__half>(g, off0, off1, step, v); break;
        case kBF16: load_pair<__nv_bfloat16>(g, off0, off1, step, v); break;
        default: load_pair<short>(g, off0, off1, step, v); break;
    }
}

__device__ __forceinline__ short saturate(float v) {
    return static_cast<short>(rintf(fminf(fmaxf(v, -32768.0f), 32767.0f)));
}
// One column's z = x + i y at R samples, `step` samples apart from sample `at`.
template <int R, bool SECOND>
__device__ __forceinline__ void store_column(const HilbertColsArgs& g, int64_t at, int step, const float2 (&x)[R],
                                             const float2 (&y)[R]) {
#define MACH_B200_PART(v) ((SECOND ? (v).y : (v).x) * g.scale)
    if (g.dst_code == kC64) {
        float2* d = static_cast<float2*>(g.dst) + at;
#pragma unroll
        for (int r = 0; r < R; ++r) d[r * step] = make_float2(MACH_B200_PART(x[r]), MACH_B200_PART(y[r]));
    } else if (g.dst_code == kCF16) {
        __half2* d = static_cast<__half2*>(g.dst) + at;
#pragma unroll
        for (int r = 0; r < R; ++r) d[r * step] = __floats2half2_rn(MACH_B200_PART(x[r]), MACH_B200_PART(y[r]));
    } else if (g.dst_code == kCBF16) {
        __nv_bfloat162* d = static_cast<__nv_bfloat162*>(g.dst) + at;
#pragma unroll
        for (int r = 0; r < R; ++r) d[r * step] = __floats2bfloat162_rn(MACH_B200_PART(x[r]), MACH_B200_PART(y[r]));
    } else {
        short2* d = static_cast<short2*>(g.dst) + at;
#pragma unroll
        for (int r = 0; r < R; ++r) d[r * step] = make_short2(saturate(MACH_B200_PART(x[r])), saturate(MACH_B200_PART(y[r])));
    }
#undef MACH_B200_PART
}

// Stage 1: samples from global memory, kept in x when KEEP; pairs fastest, so that neighbouring
// lanes read neighbouring columns of a sample.
template <int R, bool KEEP>
__device__ __forceinline__ void first_stage(const HilbertColsArgs& g, const float2* tw, float2* buf,
                                            const int64_t* off, float2 (&x)[16]) {
    const int L = g.low[0], S = g.stride[0];
    for (int i = threadIdx.x; i < L << g.pairs_log2; i += kThreads) {
        const int p = i & ((1 << g.pairs_log2) - 1), b = i >> g.pairs_log2;
        const int64_t off0 = off[2 * p], off1 = off[2 * p + 1];
        float2 v[R];
        if (off0 >= 0) {
            load_any<R>(g, off0 + b * g.src_sample, off1 >= 0 ? off1 + b * g.src_sample : -1, L * g.src_sample, v);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = make_float2(0.f, 0.f);
        }
        if (KEEP) {
#pragma unroll
            for (int r = 0; r < R; ++r) x[r] = v[r];
        }
        dft<R, false>(v);
        float2* at = buf + p * g.pair_size + low_offset(g, 0, b);
#pragma unroll
        for (int r = 0; r < R; ++r) at[r * S] = r > 0 ? mul<false>(v[r], tw[(r - 1) * L + b]) : v[r];
    }
}

template <int R, bool KEEP>
__device__ __forceinline__ void last_stage(const HilbertColsArgs& g, const float2* tw, const float2* buf,
                                           const int64_t* off, const int64_t* dst_off, const float2 (&x)[16]) {
    const int L = g.low[0], S = g.stride[0];
    for (int i = threadIdx.x; i < L << g.pairs_log2; i += kThreads) {
        const int p = i & ((1 << g.pairs_log2) - 1), b = i >> g.pairs_log2;
        const int64_t off0 = off[2 * p], off1 = off[2 * p + 1];
        if (off0 < 0) continue;
        const float2* at = buf + p * g.pair_size + low_offset(g, 0, b);
        float2 v[R], z[R];
        if (KEEP) {
#pragma unroll
            for (int r = 0; r < R; ++r) z[r] = x[r];
        } else {
            load_any<R>(g, off0 + b * g.src_sample, off1 >= 0 ? off1 + b * g.src_sample : -1, L * g.src_sample, z);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = r > 0 ? mul<true>(at[r * S], tw[(r - 1) * L + b]) : at[0];
        dft<R, true>(v);
        store_column<R, false>(g, dst_off[2 * p] + b, L, z, v);
        if (off1 >= 0) store_column<R, true>(g, dst_off[2 * p + 1] + b, L, z, v);
    }
}

#define MACH_B200_RADICES(X) X(16) X(13) X(12) X(11) X(10) X(8) X(7) X(6) X(5) X(4) X(3) X(2)
#define MACH_B200_FIRST_RADICES(X) X(16) X(12) X(10) X(8)

template <bool KEEP>
__global__ void __launch_bounds__(kThreads, 2) hilbert_cols_kernel(const __grid_constant__ HilbertColsArgs g) {
    extern __shared__ float2 smem[];
    constexpr int kMaxCols = 2 << kHilColsMaxPairsLog2;
    __shared__ int64_t s_src[2][kMaxCols], s_dst[2][kMaxCols];
    float2* const buf = smem + g.twiddles;
    // twiddles of stage j: W_(R_j L_j)^(k b) at [(k - 1) L_j + b]
    for (int j = 0, at = 0; j + 1 < g.m; ++j) {
        const int L = g.low[j], count = (g.radix[j] - 1) * L;
        for (int i = threadIdx.x; i < count; i += kThreads) {
            int b;
            const int k = div_mod(i, L, g.r_low[j], b) + 1;
            double sn, cs;
            sincospi(-2.0 * (static_cast<double>(k) * b) / (static_cast<double>(g.radix[j]) * L), &sn, &cs);
            smem[at + i] = make_float2(static_cast<float>(cs), static_cast<float>(sn));
        }
        at += count;
    }
    const int cols = 2 << g.pairs_log2;
    const int64_t n_groups = (g.n_cols + cols - 1) / cols;
    auto set_offsets = [&](int64_t grp, int slot) {
        if (static_cast<int>(threadIdx.x) < cols) {
            const int64_t c = grp * cols + threadIdx.x;
            int64_t so = -1, d = 0;
            if (c < g.n_cols) {
                const int64_t c1 = c % g.n1, c2 = c / g.n1;
                so = c1 * g.src_stride[0] + c2 * g.src_stride[1];
                d = c1 * g.dst_stride[0] + c2 * g.dst_stride[1];
            }
            s_src[slot][threadIdx.x] = so;
            s_dst[slot][threadIdx.x] = d;
        }
    };
    int64_t grp = blockIdx.x;
    if (grp < n_groups) set_offsets(grp, 0);
    __syncthreads();
    float2 x[16];
    for (int slot = 0; grp < n_groups; grp += gridDim.x, slot ^= 1) {
        const float2* tw = smem;
        switch (g.radix[0]) {
#define X(R) \
    case R: first_stage<R, KEEP>(g, tw, buf, s_src[slot], x); break;
            MACH_B200_FIRST_RADICES(X)
#undef X
        }
        __syncthreads();
        // (after the barrier: a slower warp's last stage of the group before may have read this slot)
        if (grp + gridDim.x < n_groups) set_offsets(grp + gridDim.x, slot ^ 1);
        for (int j = 1; j + 1 < g.m; ++j) {
            tw += (g.radix[j - 1] - 1) * g.low[j - 1];
            switch (g.radix[j]) {
#define X(R) \
    case R: middle_stage<R, false>(g, j, tw, buf); break;
                MACH_B200_RADICES(X)
#undef X
            }
            __syncthreads();
        }
        switch (g.radix[g.m - 1]) {
#define X(R) \
    case R: turn_stage<R>(g, buf); break;
            MACH_B200_RADICES(X)
#undef X
        }
        __syncthreads();
        for (int j = g.m - 2; j > 0; --j) {
            switch (g.radix[j]) {
#define X(R) \
    case R: middle_stage<R, true>(g, j, tw, buf); break;
                MACH_B200_RADICES(X)
#undef X
            }
            tw -= (g.radix[j - 1] - 1) * g.low[j - 1];
            __syncthreads();
        }
        // This stage reads what the same thread's next first stage overwrites: no barrier between.
        switch (g.radix[0]) {
#define X(R) \
    case R: last_stage<R, KEEP>(g, tw, buf, s_src[slot], s_dst[slot], x); break;
            MACH_B200_FIRST_RADICES(X)
#undef X
        }
    }
}

// Fewest stages of the kernel's radices, the largest first (stage 1 must be 16, 12, 10 or 8; the last
// stage, which holds both directions, is the smallest).
bool split_radices(int n, int max_r, int left, int* out, int count, int& best, int* best_out) {
    static const int kRadices[] = {16, 13, 12, 11, 10, 8, 7, 6, 5, 4, 3, 2};
    if (n == 1) {
        if (count < best) {
            best = count;
            std::copy(out, out + count, best_out);
        }
        return true;
    }
    if (left == 0 || count + 1 >= best) return false;
    bool any = false;
    for (int r : kRadices) {
        if (r > max_r || n % r != 0) continue;
        out[count] = r;
        any |= split_radices(n / r, r, left - 1, out, count + 1, best, best_out);
    }
    return any;
}

}  // namespace

bool hilbert_cols_plan(int n, HilbertColsArgs& g) {
    int out[kHilColsMaxStages], best_out[kHilColsMaxStages], best = kHilColsMaxStages + 1;
    if (n < 64 || n > (1 << 16)) return false;
    split_radices(n, 16, kHilColsMaxStages, out, 0, best, best_out);
    if (best > kHilColsMaxStages || best < 2) return false;
    // stage 1 from {16, 12, 10, 8}: the first of them in the list moves to the front
    int first = -1;
    for (int j = 0; j < best && first < 0; ++j) {
        const int r = best_out[j];
        if (r == 16 || r == 12 || r == 10 || r == 8) first = j;
    }
    if (first < 0) return false;
    std::rotate(best_out, best_out + first, best_out + first + 1);
    g.n = n;
    g.m = best;
    int low = n, weight = 1;
    for (int j = 0; j < g.m; ++j) {
        g.radix[j] = best_out[j];
        g.r_radix[j] = 1.0f / g.radix[j];
        g.weight[j] = weight;
        weight *= g.radix[j];
        low /= g.radix[j];
        g.low[j] = low;
        g.r_low[j] = 1.0f / low;
        g.items[j] = n / g.radix[j];
        g.r_items[j] = 1.0f / g.items[j];
    }
    g.twiddles = 0;
    for (int j = 0; j + 1 < g.m; ++j) g.twiddles += (g.radix[j] - 1) * g.low[j];
    // Strides: 1 for the last digit, an odd stride above it (stage m: lanes along digit m - 1), and
    // above that the stride that continues the run of the digits below (mod the 16 float2 of a bank row).
    g.stride[g.m - 1] = 1;
    for (int j = g.m - 2; j >= 0; --j) {
        int s = g.radix[j + 1] * g.stride[j + 1];
        if (j == g.m - 2) {
            s |= 1;
        } else {
            while (s % 16 != g.low[j + 1] % 16) ++s;
        }
        g.stride[j] = s;
    }
    g.pairs_log2 = 0;
    while (g.pairs_log2 < kHilColsMaxPairsLog2 && (n << (g.pairs_log2 + 1)) <= 4096) ++g.pairs_log2;
    g.pair_size = g.radix[0] * g.stride[0];
    while (g.pairs_log2 && g.pair_size % 16 != 16 >> g.pairs_log2) ++g.pair_size;
    return true;
}

size_t hilbert_cols_smem(const HilbertColsArgs& g) {
    return sizeof(float2) * (static_cast<size_t>(g.twiddles) + (static_cast<size_t>(g.pair_size) << g.pairs_log2));
}

cudaError_t launch_hilbert_cols(const HilbertColsArgs& g, cudaStream_t st) {
    const size_t smem = hilbert_cols_smem(g);
    const bool keep = (g.low[0] << g.pairs_log2) <= kThreads;
    auto k = keep ? hilbert_cols_kernel<true> : hilbert_cols_kernel<false>;
    cudaError_t e = allow_smem(k, smem);
    if (e != cudaSuccess) return e;
    int device = 0, sms = 0, per_sm = 0;
    if ((e = cudaGetDevice(&device)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem)) != cudaSuccess) return e;
    const int64_t cols = int64_t{2} << g.pairs_log2, groups = (g.n_cols + cols - 1) / cols;
    const int64_t resident = static_cast<int64_t>(std::max(1, per_sm)) * sms;
    k<<<static_cast<unsigned>(std::min(groups, resident)), kThreads, smem, st>>>(g);
    return cudaGetLastError();
}

}  // namespace mach_b200
