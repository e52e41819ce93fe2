// FFT path in one block per pair: transform of the right matrix, product with the left spectrum, inverse
// transform and the result's layout without leaving shared memory.
//
// For sizes whose half spectrum fits one SM's shared memory.  The transform size is free (any P x Q of at
// least 2H-1 x 2W-1 gives the same linear correlation), so P and Q are products of a power of two and at most one
// 3 and one 5, of few passes: no slow prime lengths.  Every pass is in place -- decimation in frequency
// forwards, the same network backwards -- so spectra stay in the passes' digit-reversed order, in which the
// product does not care, and nothing is ever reordered.  Real rows are transformed two at a time as real and
// imaginary part; the two half spectra are separated (and joined again on the way back) inside the storage of
// the row pair.
//
// Storage: P rows of K = Q/2 + 1 complex numbers, a row pair every 2K + 1: neighbouring lanes take neighbouring
// columns in the column passes and neighbouring row pairs in the row passes, free of bank conflicts in both.
// Twiddles come from tables computed once per block (sincospif).
// Bound by shared-memory traffic, 16 bytes a point and pass, and the latency of a pass between two barriers; the
// result is written once, the inputs read once.  Measured on B200 against pad, cuFFT, product, cuFFT, unpack (us):
// 64 x 64 1 x 512 106 -> 60, 90 x 75 4 x 48 55 -> 35, 60 x 60 1 x 1500 285 -> 141, one 60 x 60 pair 33 -> 26.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "xcorr_launch.h"
#include "xcorr_smem.h"

namespace xcorr {

namespace {

struct Dim { int n, passes, radix[4]; };

struct FftBlockArgs {
    const float* right;            // matrices (the forward kernel's inputs)
    const float2* left_spectra;    // pair kernel
    const float2* right_spectra;   // pair kernel: spectra made before, or nullptr: transform `right`
    float2* spectra;               // forward kernel
    float* out;
    int H, W, K;
    Dim rows, cols;                // lengths Q (along a row) and P (along a column)
    unsigned m, right_stride;      // pair = l * m + j: right matrix l * right_stride + j
    float scale;
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template<bool INV> __device__ __forceinline__ float2 rot(float2 a) {      // times -i (forwards) or i
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template<bool INV> __device__ __forceinline__ float2 twisted(float2 a, float c, float s) {   // times c - i s, or c + i s
    return INV ? make_float2(a.x * c - a.y * s, a.y * c + a.x * s) : make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
}

// Discrete transforms of R points in natural order.
template<int R, bool INV> struct Dft;
template<bool INV> struct Dft<2, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[2]) { const float2 a = v[0]; v[0] = cadd(a, v[1]); v[1] = csub(a, v[1]); }
};
template<bool INV> struct Dft<3, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[3]) {
        const float2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        const float2 m = make_float2(v[0].x - 0.5f * s.x, v[0].y - 0.5f * s.y);
        const float2 e = rot<INV>(make_float2(d.x * 0.86602540378443865f, d.y * 0.86602540378443865f));
        v[0] = cadd(v[0], s); v[1] = cadd(m, e); v[2] = csub(m, e);
    }
};
template<bool INV> struct Dft<4, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[4]) {
        const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = rot<INV>(csub(v[1], v[3]));
        v[0] = cadd(a, c); v[1] = cadd(b, d); v[2] = csub(a, c); v[3] = csub(b, d);
    }
};
template<bool INV> struct Dft<5, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[5]) {
        constexpr float r = 0.55901699437494742f, s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;   // sqrt(5) / 4, sines
        const float2 a = cadd(v[1], v[4]), b = csub(v[1], v[4]), c = cadd(v[2], v[3]), d = csub(v[2], v[3]), z = v[0];
        const float2 t = cadd(a, c), m = make_float2(z.x - 0.25f * t.x, z.y - 0.25f * t.y);
        const float2 p = make_float2(m.x + r * (a.x - c.x), m.y + r * (a.y - c.y));
        const float2 q = make_float2(m.x - r * (a.x - c.x), m.y - r * (a.y - c.y));
        const float2 e = rot<INV>(make_float2(s1 * b.x + s2 * d.x, s1 * b.y + s2 * d.y));
        const float2 f = rot<INV>(make_float2(s2 * b.x - s1 * d.x, s2 * b.y - s1 * d.y));
        v[0] = cadd(z, t); v[1] = cadd(p, e); v[4] = csub(p, e); v[2] = cadd(q, f); v[3] = csub(q, f);
    }
};
template<bool INV> struct Dft<8, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[8]) {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4, INV>::run(e);
        Dft<4, INV>::run(o);
        constexpr float h = 0.70710678118654752f;
        o[1] = twisted<INV>(o[1], h, h);
        o[2] = rot<INV>(o[2]);
        o[3] = twisted<INV>(o[3], -h, h);
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[i] = cadd(e[i], o[i]); v[i + 4] = csub(e[i], o[i]); }
    }
};
template<bool INV> struct Dft<16, INV> {
    static __device__ __forceinline__ void run(float2 (&v)[16]) {
        float2 e[8], o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) { e[i] = v[2 * i]; o[i] = v[2 * i + 1]; }
        Dft<8, INV>::run(e);
        Dft<8, INV>::run(o);
        constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
        o[1] = twisted<INV>(o[1], c1, s1); o[2] = twisted<INV>(o[2], h, h); o[3] = twisted<INV>(o[3], s1, c1);
        o[4] = rot<INV>(o[4]);
        o[5] = twisted<INV>(o[5], -s1, c1); o[6] = twisted<INV>(o[6], -h, h); o[7] = twisted<INV>(o[7], -c1, s1);
#pragma unroll
        for (int i = 0; i < 8; ++i) { v[i] = cadd(e[i], o[i]); v[i + 8] = csub(e[i], o[i]); }
    }
};

// Lengths of two coprime factors without twiddles (Good and Thomas): element (n1, n2) stands at N2 n1 + N1 n2,
// frequency (k1, k2) at the residue that is k1 mod N1 and k2 mod N2.
template<int N1, int N2, bool INV> struct DftPair {
    static __device__ __forceinline__ void run(float2 (&v)[N1 * N2]) {
        constexpr int N = N1 * N2;
        float2 u[N1][N2];
#pragma unroll
        for (int a = 0; a < N1; ++a) {
#pragma unroll
            for (int b = 0; b < N2; ++b) u[a][b] = v[(N2 * a + N1 * b) % N];
            Dft<N2, INV>::run(u[a]);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (k >= N2) continue;
            float2 c[N1];
#pragma unroll
            for (int a = 0; a < N1; ++a) c[a] = u[a][k];
            Dft<N1, INV>::run(c);
#pragma unroll
            for (int a = 0; a < N1; ++a) u[a][k] = c[a];
        }
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = u[k % N1][k % N2];
    }
};
template<bool INV> struct Dft<6, INV> : DftPair<2, 3, INV> {};
template<bool INV> struct Dft<10, INV> : DftPair<2, 5, INV> {};
template<bool INV> struct Dft<12, INV> : DftPair<3, 4, INV> {};

// quotient of small non-negative integers by a number of at most 512
__device__ __forceinline__ int quotient(int a, float inv) { return (int)(((float)a + 0.5f) * inv); }

// One pass of radix R over `count` transforms of length n in place.  Lanes run over the transforms.
// COLS: transform = column, element = row; else transform = row pair, element = position in the pair's storage.
// LAST: the network's last pass forwards, its first backwards (neighbouring elements, no twiddles).
// live: elements from there on are zeros that need not be read (forwards, the first pass).
// MUL (backwards, the first pass): what is loaded is the product of the spectra: left * conj(right), the
// right one from global memory or from where it stands.
template<int R, bool INV, bool COLS, bool LAST, bool MUL>
__device__ __forceinline__ void fft_pass(float2* s, const float2* __restrict__ tw, int n, int len, int live, int count, int K,
                                         const float2* left, const float2* right) {
    const int sub = LAST ? 1 : len / R, total = n / R * count, step = n / len;
    const float inv_count = 1.0f / (float)count, inv_sub = 1.0f / (float)sub;
    // distance of a butterfly's elements in storage: odd factors come first, so `sub` is even but in the last pass,
    // where an even radix takes whole row pairs
    const int stride = COLS ? (LAST ? 2 * K + 1 : (sub >> 1) * (2 * K + 1)) : sub;
    for (int item = threadIdx.x; item < total; item += blockDim.x) {
        const int b = quotient(item, inv_count), i = item - b * count;
        const int blk = LAST ? b : quotient(b, inv_sub), j = LAST ? 0 : b - blk * sub, first = blk * len + j;
        float2* base = s + (COLS ? (first >> 1) * (2 * K + 1) + (first & 1) * K + i : i * (2 * K + 1) + first);
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int at = COLS && LAST ? (q >> 1) * stride + (q & 1) * K : q * stride;
            if (MUL) {
                // (not through the read-only path: the launch before this one wrote the spectra)
                const int g = (first + q) * K + i;
                const float2 l = __ldcg(left + g), r = right ? __ldcg(right + g) : base[at];
                v[q] = make_float2(l.x * r.x + l.y * r.y, l.y * r.x - l.x * r.y);
            } else {
                v[q] = INV || first + q * sub < live ? base[at] : make_float2(0.f, 0.f);
            }
        }
        if (INV && !LAST) {
#pragma unroll
            for (int q = 1; q < R; ++q) { const float2 w = tw[j * q * step]; v[q] = cmul(v[q], make_float2(w.x, -w.y)); }
        }
        Dft<R, INV>::run(v);
        if (!INV && !LAST) {
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[j * q * step]);
        }
#pragma unroll
        for (int q = 0; q < R; ++q) base[COLS && LAST ? (q >> 1) * stride + (q & 1) * K : q * stride] = v[q];
    }
}

template<bool INV, bool COLS>
__device__ __forceinline__ void fft_inner(int radix, float2* s, const float2* tw, int n, int len, int live, int count, int K) {
    switch (radix) {
    case 2: fft_pass<2, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 3: fft_pass<3, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 4: fft_pass<4, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 5: fft_pass<5, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 6: fft_pass<6, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 10: fft_pass<10, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 12: fft_pass<12, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    case 8: fft_pass<8, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    default: fft_pass<16, INV, COLS, false, false>(s, tw, n, len, live, count, K, nullptr, nullptr); break;
    }
    __syncthreads();
}
template<bool INV, bool COLS, bool MUL>
__device__ __forceinline__ void fft_last(int radix, float2* s, const float2* tw, int n, int live, int count, int K,
                                         const float2* left, const float2* right) {
    switch (radix) {
    case 2: fft_pass<2, INV, COLS, true, MUL>(s, tw, n, 2, live, count, K, left, right); break;
    case 4: fft_pass<4, INV, COLS, true, MUL>(s, tw, n, 4, live, count, K, left, right); break;
    case 8: fft_pass<8, INV, COLS, true, MUL>(s, tw, n, 8, live, count, K, left, right); break;
    default: fft_pass<16, INV, COLS, true, MUL>(s, tw, n, 16, live, count, K, left, right); break;
    }
    __syncthreads();
}

// Forwards, `live` elements of a transform not being zero; backwards, MUL as above.
template<bool COLS>
__device__ __forceinline__ void fft_forward(const Dim& d, float2* s, const float2* tw, int live, int count, int K) {
    int len = d.n;
    for (int p = 0; p < d.passes - 1; ++p) {
        fft_inner<false, COLS>(d.radix[p], s, tw, d.n, len, p == 0 ? live : d.n, count, K);
        len /= d.radix[p];
    }
    fft_last<false, COLS, false>(len, s, tw, d.n, d.passes == 1 ? live : d.n, count, K, nullptr, nullptr);
}
template<bool COLS, bool MUL>
__device__ __forceinline__ void fft_backward(const Dim& d, float2* s, const float2* tw, int count, int K, const float2* left, const float2* right) {
    int len = d.radix[d.passes - 1];
    fft_last<true, COLS, MUL>(len, s, tw, d.n, d.n, count, K, left, right);
    for (int p = d.passes - 2; p >= 0; --p) { len *= d.radix[p]; fft_inner<true, COLS>(d.radix[p], s, tw, d.n, len, d.n, count, K); }
}

// Separate the half spectra of the two rows of `pairs` row pairs (JOIN: the way back).  Everything of a batch of
// pairs is read before anything of it is written.
template<bool JOIN>
__device__ __forceinline__ void row_pairs(float2* s, const unsigned short* __restrict__ place, int pairs, int Q, int K) {
    constexpr int kItems = 8;
    const int batch = max(1, kItems * (int)blockDim.x / K);
    for (int t0 = 0; t0 < pairs; t0 += batch) {
        const int n = min(batch, pairs - t0), total = n * K;
        const float inv_n = 1.0f / (float)n;
        float2 a[kItems], b[kItems];
#pragma unroll
        for (int z = 0; z < kItems; ++z) {
            const int item = threadIdx.x + z * blockDim.x;
            if (item >= total) continue;
            const int k = quotient(item, inv_n), t = t0 + item - k * n;
            const float2* base = s + t * (2 * K + 1);
            if (JOIN) {
                a[z] = base[k]; b[z] = base[K + k];
            } else {
                a[z] = base[place[k]]; b[z] = base[place[k == 0 ? 0 : Q - k]];
            }
        }
        __syncthreads();
#pragma unroll
        for (int z = 0; z < kItems; ++z) {
            const int item = threadIdx.x + z * blockDim.x;
            if (item >= total) continue;
            const int k = quotient(item, inv_n), t = t0 + item - k * n;
            float2* base = s + t * (2 * K + 1);
            const float2 u = a[z], v = b[z];
            if (JOIN) {
                // X_a + i X_b, and at Q - k conj X_a + i conj X_b; both are real at 0 and Q / 2
                const bool real = k == 0 || 2 * k == Q;
                base[place[k]] = real ? make_float2(u.x, v.x) : make_float2(u.x - v.y, u.y + v.x);
                if (!real) base[place[Q - k]] = make_float2(u.x + v.y, v.x - u.y);
            } else {
                base[k] = make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
                base[K + k] = make_float2(0.5f * (u.y + v.y), 0.5f * (v.x - u.x));
            }
        }
        __syncthreads();
    }
}

// PAIR = false: the spectrum of matrix blockIdx.x.  PAIR = true: result blockIdx.x.
template<int THREADS, int BLOCKS, bool PAIR>
__global__ void __launch_bounds__(THREADS, BLOCKS) fft_block_kernel(const __grid_constant__ FftBlockArgs a) {
    extern __shared__ __align__(16) float2 fft_smem[];
    const int Q = a.rows.n, P = a.cols.n, K = a.K, H = a.H, W = a.W;
    float2* s = fft_smem;
    float2* tw_rows = s + (P / 2) * (2 * K + 1);
    float2* tw_cols = tw_rows + Q;
    unsigned short* place = reinterpret_cast<unsigned short*>(tw_cols + P);
    for (int i = threadIdx.x; i < Q; i += THREADS) {
        float sn, cs;
        sincospif(-2.0f * (float)i / (float)Q, &sn, &cs);
        tw_rows[i] = make_float2(cs, sn);
        // where the passes leave frequency i
        int k = i, at = 0, span = Q;
        for (int p = 0; p < a.rows.passes; ++p) { const int r = a.rows.radix[p]; span /= r; at += (k % r) * span; k /= r; }
        place[i] = (unsigned short)at;
    }
    for (int i = threadIdx.x; i < P; i += THREADS) {
        float sn, cs;
        sincospif(-2.0f * (float)i / (float)P, &sn, &cs);
        tw_cols[i] = make_float2(cs, sn);
    }
    if (!PAIR) asm volatile("griddepcontrol.launch_dependents;");
    const unsigned pair = blockIdx.x, l = PAIR ? pair / a.m : 0u;
    const size_t mat = PAIR ? (size_t)l * a.right_stride + (pair - l * a.m) : pair;
    const size_t spectrum = (size_t)P * K;
    const float2* right_spectrum = PAIR && a.right_spectra ? a.right_spectra + mat * spectrum : nullptr;
    if (!right_spectrum) {
        const float* src = a.right + mat * H * W;
        const int full = (H + 1) / 2;
        const float inv_w = 1.0f / (float)W;
        for (int i = threadIdx.x; i < full * W; i += THREADS) {
            const int t = quotient(i, inv_w), x = i - t * W;
            s[t * (2 * K + 1) + x] = make_float2(__ldg(src + (2 * t) * W + x), 2 * t + 1 < H ? __ldg(src + (2 * t + 1) * W + x) : 0.f);
        }
        __syncthreads();
        fft_forward<false>(a.rows, s, tw_rows, W, full, K);
        row_pairs<false>(s, place, full, Q, K);
        fft_forward<true>(a.cols, s, tw_cols, 2 * full, K, K);
    } else {
        __syncthreads();
    }
    if (!PAIR) {
        float2* to = a.spectra + pair * spectrum;
        const float inv_k = 1.0f / (float)K;
        for (int i = threadIdx.x; i < P * K; i += THREADS) {
            const int r = quotient(i, inv_k), k = i - r * K;
            to[i] = s[(r >> 1) * (2 * K + 1) + (r & 1) * K + k];
        }
        return;
    }
    // the spectra of the launch before this one (a block may start while that is still running)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    fft_backward<true, true>(a.cols, s, tw_cols, K, K, a.left_spectra + l * spectrum, right_spectrum);
    row_pairs<true>(s, place, P / 2, Q, K);
    fft_backward<false, false>(a.rows, s, tw_rows, P / 2, K, nullptr, nullptr);
    // shift (sy, sx) stands in row sy mod P, column sx mod Q
    const int OW = 2 * W - 1, OH = 2 * H - 1;
    float* out = a.out + (size_t)pair * OH * OW;
    const float inv_ow = 1.0f / (float)OW;
    for (int i = threadIdx.x; i < (P / 2) * OW; i += THREADS) {
        const int t = quotient(i, inv_ow), ox = i - t * OW, sx = ox - (W - 1);
        const float2 v = s[t * (2 * K + 1) + (sx < 0 ? sx + Q : sx)];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const int r = 2 * t + z, sy = r < H ? r : r - P;
            if (sy > -H) out[(sy + H - 1) * OW + ox] = (z ? v.y : v.x) * a.scale;
        }
    }
}

// Passes of a length 2^a, 3 * 2^a, 5 * 2^a or 15 * 2^a (a >= 1): as few as there can be, odd factors first (an
// even radix of a power of two last).
Dim passes_of(int n, int odd) {
    Dim d{};
    d.n = n;
    int twos = n / odd;
    const auto take = [&](int r) { d.radix[d.passes++] = r; };
    const auto passes = [](int t) { return t <= 16 ? 1 : t <= 256 ? 2 : 3; };
    if (odd == 15) { take(5); odd = 3; }
    if (odd == 3 || odd == 5) {
        // 12, 10 or 6 where the rest then needs one pass less
        int with = 1;
        if (twos >= 4 && passes(twos / 2) < passes(twos)) with = 2;
        else if (odd == 3 && twos >= 8 && passes(twos / 4) < passes(twos)) with = 4;
        take(odd * with);
        twos /= with;
    }
    while (twos > 1) {
        const int r = twos <= 16 ? twos : twos == 32 || twos == 64 ? 8 : 16;
        take(r);
        twos /= r;
    }
    return d;
}

// The length of at least `need` with the fewest points times passes, or (small) the smallest.
bool pick_dim(int need, bool small, Dim* d) {
    int best = 1 << 30;
    for (int odd : {1, 3, 5, 15})
        for (int v = 2 * odd; v <= 512; v *= 2) {
            if (v < need) continue;
            const Dim c = passes_of(v, odd);
            const int cost = small ? v : v * (c.passes + 1);
            if (cost < best) { best = cost; *d = c; }
        }
    return best < 1 << 30;
}

size_t smem_bytes(const Dim& rows, const Dim& cols) {
    const size_t K = rows.n / 2 + 1;
    return (cols.n / 2 * (2 * K + 1) + rows.n + cols.n) * sizeof(float2) + rows.n * sizeof(unsigned short);
}

template<int THREADS, int BLOCKS, bool PAIR>
cudaError_t launch(const FftBlockArgs& a, unsigned grid, size_t bytes, int device, cudaStream_t stream) {
    static SmemLimit limit;
    const cudaError_t e = limit.allow(device, bytes, [](size_t size) {
        return cudaFuncSetAttribute(fft_block_kernel<THREADS, BLOCKS, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)size);
    });
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = bytes;
    config.stream = stream;
    // the pair kernel transforms its right matrix while the left spectra are still being made
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &early;
    config.numAttrs = PAIR ? 1 : 0;
    return cudaLaunchKernelEx(&config, fft_block_kernel<THREADS, BLOCKS, PAIR>, a);
}

}  // namespace

bool fft_block_run(const float* left, const float* right, float* out, int H, int W, const PairMap& pm, unsigned n_right,
                   void* workspace, size_t workspace_bytes, int device, int sm_count, cudaStream_t stream, cudaError_t* err, FftRoute* route) {
    FftBlockArgs a{};
    size_t bytes = 0;
    for (int small = 0; small < 2; ++small) {
        if (!pick_dim(2 * W - 1, small, &a.rows) || !pick_dim(2 * H - 1, small, &a.cols)) return false;
        bytes = smem_bytes(a.rows, a.cols);
        if (bytes <= (size_t)kSmemLimit) break;
    }
    if (bytes > (size_t)kSmemLimit) return false;
    a.H = H; a.W = W; a.K = a.rows.n / 2 + 1;
    a.m = pm.m;
    a.right_stride = pm.right_stride;
    a.scale = 1.0f / ((float)a.rows.n * (float)a.cols.n);
    const size_t spectrum = (size_t)a.cols.n * a.K, pairs = (size_t)pm.n_left * pm.m;
    // One block takes 17 us and 1.2 us per thousand points (256 x 81 points: 41 us), whatever else runs; cuFFT
    // spreads a few large transforms over the GPU (one 200 x 40 pair: 37 us against 43).
    if (spectrum > 14000 && pairs < 24) return false;
    // A right matrix that meets several lefts is transformed once, in a launch of its own, where there is more than
    // a wave of pairs; below that every pair transforms it again beside the others (64 x 64 9 x 14: one launch less).
    const size_t wave = (size_t)sm_count * (bytes <= 75 * 1024 ? 3 : bytes <= 113 * 1024 ? 2 : 1);
    const bool shared_rights = pm.n_left > 1 && pm.right_stride == 0 && pairs > wave;
    const size_t spectra = pm.n_left + (shared_rights ? (size_t)n_right : 0);
    if (spectra * spectrum * sizeof(float2) > workspace_bytes || pairs > 0x7fffffffull || n_right > 0x7fffffffu) return false;
    *route = FftRoute{1, a.cols.n, a.rows.n, shared_rights ? 1 : 0, 0};
    float2* store = static_cast<float2*>(workspace);
    const auto run = [&](bool pair, unsigned grid) -> cudaError_t {
        ++route->launches;
        // three blocks of 256 threads per SM where they fit, two of 384, else one of 512; no more blocks than SMs:
        // 512 threads, the time is one block's (one 60 x 60 pair 29 -> 26 us, 64 x 64 9 x 14 43 -> 27 us with the
        // launch saved below; the left spectra of 64 x 64 1 x 512, one block before all others, 62 -> 60 us)
        if (grid <= (unsigned)sm_count && bytes > 12 * 1024)
            return pair ? launch<512, 1, true>(a, grid, bytes, device, stream) : launch<512, 1, false>(a, grid, bytes, device, stream);
        if (bytes <= 75 * 1024)
            return pair ? launch<256, 3, true>(a, grid, bytes, device, stream) : launch<256, 3, false>(a, grid, bytes, device, stream);
        if (bytes <= 113 * 1024)
            return pair ? launch<384, 2, true>(a, grid, bytes, device, stream) : launch<384, 2, false>(a, grid, bytes, device, stream);
        return pair ? launch<512, 1, true>(a, grid, bytes, device, stream) : launch<512, 1, false>(a, grid, bytes, device, stream);
    };
    a.right = left;
    a.spectra = store;
    *err = run(false, pm.n_left);
    if (*err == cudaSuccess && shared_rights) {
        a.right = right;
        a.spectra = store + (size_t)pm.n_left * spectrum;
        *err = run(false, n_right);
        a.right_spectra = a.spectra;
    }
    if (*err != cudaSuccess) return true;
    a.right = right;
    a.left_spectra = store;
    a.out = out;
    *err = run(true, (unsigned)pairs);
    return true;
}

}  // namespace xcorr
