// Long-range PM force: CIC deposit, 3D real FFT with the Green's function,
// FD4 gradient and CIC interpolation, all on the device.
//
// Reference: pmforce_periodic (pm_periodic.c:67-314), which deposits and
// interpolates on the host and round-trips the grid through cuFFT.  Here:
//   k_deposit      CIC mass assignment (pm_periodic.c:97-132): each weight as
//                  the integer w * 2^32, added with 64-bit integer atomics into
//                  an M^3 grid, so the grid is the same whatever order the
//                  particles land in (float atomics are not associative).  A
//                  box deposits in original particle order (beside the sort)
//                  or, where that is scattered, in cell order.
//   k_fft_z_r2c    real->complex along z; its load converts the integer sums to
//                  mass (one rounding) and writes zero back, so the grid is
//                  clean for the next deposit.  Two real rows are packed as the
//                  real and imaginary parts of one complex row, transformed
//                  together and separated (X1 = (Z + conj Z_-k)/2,
//                  X2 = (Z - conj Z_-k)/2i).
//   k_fft_axis     complex transforms along y, and along x fused with the
//                  Green's-function multiply and the inverse x transform: the
//                  x pass is the last forward and the first inverse pass, so the
//                  spectrum is multiplied in shared memory and never stored.
//   k_fft_z_c2r    the inverse of k_fft_z_r2c (Hermitian extension of each row,
//                  imaginary parts of the self-conjugate points dropped).
//   k_interp       the FD4 gradient of the potential (pm_periodic.c:205-270) at
//                  the 8 CIC corners of each particle and the CIC interpolation
//                  (pm_periodic.c:272-309), fused: the three force grids the
//                  reference builds are never materialised.
// All transforms are unnormalised with cuFFT's sign conventions.  Power-of-two
// meshes up to 1024 use a two-level transform with the points in registers
// (RegFFT; the one-box axis passes with their column batch fixed at compile
// time, fft_axis_reg_fixed); other meshes M = 2^a 3^b 5^c use a shared-memory
// Stockham FFT over a batch of columns with stages of radix 3 to 24.  Twiddles
// come from an FP64-built table.
// The Green's function factorises: smth(k) = -g(kx) g(ky) g(kz) / k^2 with
// g(k) = exp(-k^2 (2 pi asmth / L)^2) / sinc(pi k / M)^4, built in FP64.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace cuco {

namespace {

constexpr int kFFTThreads = 256;
constexpr size_t kMaxSmem = 227 * 1024;  // shared memory a CTA can have
constexpr int kLoadBatch = 8;  // global loads issued per thread before use

// complex a + b, a - b: one packed instruction each (every element rounded as
// the scalar operation rounds it)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(make_float2(-1.f, -1.f), b, a); }

// Points from one (x, y) row of the half spectrum to the next.  (Rounded up to
// whole 32-byte sectors the axis passes gained 3 % at M = 512 and the inverse
// z pass lost a quarter.)
__host__ __device__ constexpr int spec_stride(int M) { return M / 2 + 1; }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// The stages of a mesh's Stockham transform, five bits each (0 ends): the
// fewest stages, of those the ones with the most factors of two in a single
// radix, which goes first, of those the smallest radix sum.  Every stage is one
// round trip through shared memory and one CTA barrier, which is what these
// passes spend their time on: M = 200 takes 3 (8 5 5) instead of the 4 of
// radices to 5, most meshes to 240 take 2.  Radices 18 and 24 make it 2 for 384
// (16 24) and a few others, where 16 and less need 3: the five passes at 384
// 1.08 -> 0.97 ms.  Their kernels hold 80 registers a thread instead of 64, so
// only such meshes run them (0.4 % slower at 200 with them compiled in; 200 as
// 20 10 was 2 % slower than 8 5 5).
//
// The factors of two go first for the rounding: the mesh of a hardly displaced
// lattice is large harmonics of the lattice that cancel, and radices 4 and 2
// take their sums before any twiddle.  Against 64 bits, over 20 such states of
// 18^3 on 36^3, the largest error relative to that of 4 3 3 (and the mean):
// 6 6 1.42 (1.03), 9 4 1.36 (1.05), 4 9 1.03 (0.99).
constexpr int kRadices[] = {24, 18, 16, 15, 12, 10, 9, 8, 6, 5, 4, 3};  // (no even mesh to 1024 wants a 2)
// Whether a plan has a radix above 16.
__host__ __device__ __forceinline__ bool wide_plan(uint32_t plan) {
    for (; plan; plan >>= 5)
        if ((plan & 31) > 16) return true;
    return false;
}
uint32_t stage_plan(int M) {
    constexpr int kMaxStages = 6;
    struct Plan {
        int stages = 0, twos = 0, sum = 0, radix[kMaxStages] = {};
    } best, cur;
    best.stages = kMaxStages + 1;
    auto search = [&](auto &&self, int rem, int from) -> void {
        if (rem == 1) {
            if (cur.stages != best.stages ? cur.stages < best.stages
                                          : (cur.twos != best.twos ? cur.twos > best.twos : cur.sum < best.sum))
                best = cur;
            return;
        }
        if (cur.stages == kMaxStages) return;
        for (int i = from; i < (int)(sizeof kRadices / sizeof kRadices[0]); ++i) {
            const int R = kRadices[i];
            if (rem % R) continue;
            const Plan before = cur;
            cur.radix[cur.stages++] = R;
            cur.sum += R;
            cur.twos = std::max(cur.twos, R & -R);
            self(self, rem / R, i);
            cur = before;
        }
    };
    search(search, M, 0);
    // the radix with the most factors of two first, the others largest first
    int first = 0;
    while (first < best.stages && (best.radix[first] & -best.radix[first]) != best.twos) ++first;
    uint32_t plan = first < best.stages ? (uint32_t)best.radix[first] : 0u;
    for (int k = 0, at = 5; k < best.stages; ++k)
        if (k != first) plan |= (uint32_t)best.radix[k] << at, at += 5;
    return plan;
}

// Division by a runtime d without a divide instruction: j / d is
// umulhi(j, ceil(2^32 / d)), exact for j, d < 2^16 (checked exhaustively for
// d <= 2048; every index here is below 2^16).
struct FastDiv {
    uint32_t d, inv;
    __device__ __forceinline__ explicit FastDiv(uint32_t d_) : d(d_), inv(d_ > 1 ? (uint32_t)((0x100000000ull + d_ - 1) / d_) : 0u) {}
    __device__ __forceinline__ uint32_t div(uint32_t j) const { return d > 1 ? __umulhi(j, inv) : j; }
};

template <int R>
__device__ __forceinline__ void dft_small(float2 (&v)[R], int sign) {
    if (R == 4) {
        const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]), a2 = cadd(v[1], v[3]), d = csub(v[1], v[3]);
        // (v1 - v3) * (sign * i)
        const float2 a3 = sign < 0 ? make_float2(d.y, -d.x) : make_float2(-d.y, d.x);
        v[0] = cadd(a0, a2);
        v[1] = make_float2(a1.x + a3.x, a1.y + a3.y);
        v[2] = csub(a0, a2);
        v[3] = make_float2(a1.x - a3.x, a1.y - a3.y);
    } else if (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if (R == 3) {
        // y1,2 = v0 - (v1+v2)/2 +- i s (v1-v2), s = sign sqrt(3)/2
        const float s3 = sign * 0.866025403784438647f;
        const float2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        const float2 m = __ffma2_rn(make_float2(-0.5f, -0.5f), t, v[0]);
        v[0] = cadd(v[0], t);
        v[1] = make_float2(m.x - s3 * d.y, m.y + s3 * d.x);
        v[2] = make_float2(m.x + s3 * d.y, m.y - s3 * d.x);
    } else {
        // five-point DFT by the conjugate pairs (1,4), (2,3)
        const float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f;
        const float s1 = sign * 0.951056516295153572f, s2 = sign * 0.587785252292473129f;
        const float2 a1 = cadd(v[1], v[R - 1]), b1 = csub(v[1], v[R - 1]);
        const float2 a2 = cadd(v[2], v[R - 2]), b2 = csub(v[2], v[R - 2]);
        auto dup = [](float c) { return make_float2(c, c); };
        const float2 t1 = __ffma2_rn(dup(c2), a2, __ffma2_rn(dup(c1), a1, v[0]));
        const float2 t2 = __ffma2_rn(dup(c1), a2, __ffma2_rn(dup(c2), a1, v[0]));
        const float2 u1 = __ffma2_rn(dup(s2), b2, __fmul2_rn(dup(s1), b1));
        const float2 u2 = __ffma2_rn(dup(-s1), b2, __fmul2_rn(dup(s2), b1));
        v[0] = cadd(cadd(v[0], a1), a2);
        v[1] = make_float2(t1.x - u1.y, t1.y + u1.x);      // t1 + i u1
        v[2] = make_float2(t2.x - u2.y, t2.y + u2.x);      // t2 + i u2
        v[R - 2] = make_float2(t2.x + u2.y, t2.y - u2.x);  // t2 - i u2
        v[R - 1] = make_float2(t1.x + u1.y, t1.y - u1.x);  // t1 - i u1
    }
}

// sin(2 pi j / n) in double at compile time (Taylor, the angle reduced to
// [-pi/4, pi/4] and an octant)
constexpr double kTau = 6.283185307179586476925286766559;
constexpr double taylor(double x, bool cosine) {
    double term = cosine ? 1.0 : x, sum = term;
    for (int k = cosine ? 1 : 2; k < 24; k += 2) {
        term *= -x * x / (k * (k + 1));
        sum += term;
    }
    return sum;
}
constexpr double sin_turns(int j, int n) {
    j = ((j % n) + n) % n;
    // octant q of 8 j / n, rounded; the rest of the angle
    const int q = (16 * j + n) / (2 * n);
    const double x = kTau * ((double)j / n - q / 8.0);
    const double c = taylor(x, true), s = taylor(x, false), h = 0.70710678118654752440084436210485;
    switch (q & 7) {
        case 0: return s;
        case 1: return h * (c + s);
        case 2: return c;
        case 3: return h * (c - s);
        case 4: return -s;
        case 5: return -h * (c + s);
        case 6: return -c;
        default: return h * (s - c);
    }
}
template <int N>
struct Roots {
    float c[N], s[N];
    constexpr Roots() : c(), s() {
        for (int j = 0; j < N; ++j) c[j] = (float)sin_turns(4 * j + N, 4 * N), s[j] = (float)sin_turns(j, N);
    }
};

// In-register DFT of N points (5-smooth), X[k] = sum_n v[n] exp(S 2 pi i n k / N):
// N = A Q by Cooley-Tukey with A in {4, 3, 2, 5}; the roots are constants.
template <int N, int S>
__device__ __forceinline__ void dft_any(float2 (&v)[N]) {
    if constexpr (N <= 5) {
        dft_small<N>(v, S);
    } else {
        constexpr int A = N % 4 == 0 ? 4 : N % 3 == 0 ? 3 : N % 2 == 0 ? 2 : 5, Q = N / A;
        constexpr Roots<N> root;
        float2 w[N];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) {
            float2 t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) t[n1] = v[Q * n1 + n2];
            dft_small<A>(t, S);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1)
                w[Q * k1 + n2] = n2 * k1 ? cmul(t[k1], make_float2(root.c[n2 * k1 % N], S * root.s[n2 * k1 % N])) : t[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            float2 u[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) u[n2] = w[Q * k1 + n2];
            dft_any<Q, S>(u);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) v[k1 + A * k2] = u[k2];
        }
    }
}

// One Stockham stage of radix R over Ns already-combined points, for B = 2^bs
// columns: reads x[j + p M/R] (p < R), twiddles it by w^{p k M/(Ns R)} (k = j
// mod Ns), and writes the R-point DFT to y[(j/Ns) Ns R + k + q Ns].
template <int R, int S>
__device__ __forceinline__ void stockham_stage(const float2 *in, float2 *out, const float2 *tw, int M, int Ns,
                                               int bs, int pitch) {
    const int nb = M / R, step = M / (Ns * R);
    const FastDiv dns((uint32_t)Ns);
    const int total = nb << bs, bmask = (1 << bs) - 1;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int b = e & bmask, j = e >> bs;
        const int g = (int)dns.div((uint32_t)j), k = j - g * Ns;
        const int dst = g * Ns * R + k;
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = in[(j + q * nb) * pitch + b];
        if (k) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                float2 w = tw[q * k * step];
                if (S > 0) w.y = -w.y;
                v[q] = cmul(v[q], w);
            }
        }
        dft_any<R, S>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) out[(dst + q * Ns) * pitch + b] = v[q];
    }
}

// Transform B = 2^bs columns of length M held in x[m*pitch + b] by the stages
// of `plan`; returns the buffer holding the result.  S = -1: forward (e^{-i}),
// +1: inverse.
template <int S, bool WIDE>
__device__ float2 *fft_columns(float2 *x, float2 *y, const float2 *tw, int M, uint32_t plan, int bs, int pitch) {
    int Ns = 1;
    float2 *in = x, *out = y;
    for (; plan; plan >>= 5) {
        const int r = plan & 31;
        switch (r) {
#define CUCO_STAGE(R) \
    case R: stockham_stage<R, S>(in, out, tw, M, Ns, bs, pitch); break
            CUCO_STAGE(3);
            CUCO_STAGE(4);
            CUCO_STAGE(5);
            CUCO_STAGE(6);
            CUCO_STAGE(8);
            CUCO_STAGE(9);
            CUCO_STAGE(10);
            CUCO_STAGE(12);
            CUCO_STAGE(15);
            case 18:
                if (WIDE) stockham_stage<18, S>(in, out, tw, M, Ns, bs, pitch);
                break;
            case 24:
                if (WIDE) stockham_stage<24, S>(in, out, tw, M, Ns, bs, pitch);
                break;
            default: stockham_stage<16, S>(in, out, tw, M, Ns, bs, pitch); break;
#undef CUCO_STAGE
        }
        __syncthreads();
        float2 *t = in;
        in = out;
        out = t;
        Ns *= r;
    }
    return in;
}

__host__ __device__ constexpr int ilog2(int v) {
    int l = 0;
    while ((1 << (l + 1)) <= v) ++l;
    return l;
}

__device__ __forceinline__ void load_twiddles(float2 *tw_s, const float2 *tw, int M) {
    for (int i = threadIdx.x; i < M; i += blockDim.x) tw_s[i] = tw[i];
}

// ------------------------------------------------ register transforms
// Power-of-two meshes M = M1 * M2 (M1, M2 <= 32) take a two-level
// Cooley-Tukey transform with the points in registers: one DFT over M1
// points strided by M2, a twiddle, one shared-memory exchange, one DFT over
// M2 contiguous points.  Each column is handled by max(M1, M2) threads and
// visits shared memory twice instead of once per radix-4 stage.  The
// forward transform leaves X[k] in slot M2 (k mod M1) + k / M1; the inverse
// starts from that layout and ends in natural order, so a forward pass, a
// multiply and an inverse pass (the x pass with the Green's function) need
// no reordering in between.

// cos and sin of 2 pi j / 32, j < 32
__host__ __device__ constexpr float cos32(int j) {
    constexpr float c[32] = {1.0f, 9.807852804e-01f, 9.238795325e-01f, 8.314696123e-01f, 7.071067812e-01f,
                             5.555702330e-01f, 3.826834324e-01f, 1.950903220e-01f, 0.0f, -1.950903220e-01f,
                             -3.826834324e-01f, -5.555702330e-01f, -7.071067812e-01f, -8.314696123e-01f,
                             -9.238795325e-01f, -9.807852804e-01f, -1.0f, -9.807852804e-01f, -9.238795325e-01f,
                             -8.314696123e-01f, -7.071067812e-01f, -5.555702330e-01f, -3.826834324e-01f,
                             -1.950903220e-01f, 0.0f, 1.950903220e-01f, 3.826834324e-01f, 5.555702330e-01f,
                             7.071067812e-01f, 8.314696123e-01f, 9.238795325e-01f, 9.807852804e-01f};
    return c[j & 31];
}
__host__ __device__ constexpr float sin32(int j) { return cos32(j - 8); }

// exp(S 2 pi i m / N) for N dividing 32
template <int N, int S>
__device__ __forceinline__ float2 wconst(int m) {
    const int j = (m * (32 / N)) & 31;
    return make_float2(cos32(j), S * sin32(j));
}

// In-register DFT of N = 2^a <= 32 points, X[k] = sum_n v[n] exp(S 2 pi i n k / N),
// as radix-4 Cooley-Tukey (N = 4 Q: DFTs over n1 of v[Q n1 + n2], twiddle,
// DFTs over n2; X[k1 + 4 k2]).  All indices are compile-time constants.
template <int N, int S>
__device__ __forceinline__ void dft_reg(float2 (&v)[N]) {
    if constexpr (N == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (N == 4) {
        dft_small<4>(v, S);
    } else {
        constexpr int Q = N / 4;
        float2 w[N];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) {
            float2 t[4] = {v[n2], v[n2 + Q], v[n2 + 2 * Q], v[n2 + 3 * Q]};
            dft_small<4>(t, S);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) w[Q * k1 + n2] = (n2 * k1) ? cmul(t[k1], wconst<N, S>(n2 * k1)) : t[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            float2 u[Q];
#pragma unroll
            for (int j = 0; j < Q; ++j) u[j] = w[Q * k1 + j];
            dft_reg<Q, S>(u);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) v[k1 + 4 * k2] = u[k2];
        }
    }
}

// Shared memory: point `row` of column b is at (row + row / M2) * pitch + b, one
// spare row after every M2.  The second level's threads read rows M2 apart;
// without the spare row those are a multiple of 16 float2 apart and all fall
// on one bank.
template <int M1, int M2>
struct RegFFT {
    static constexpr int M = M1 * M2, N1 = M1, N2 = M2, T = M1 > M2 ? M1 : M2;
    static constexpr int ROWS = M + M1;  // a column's rows with the spare ones
    // a column takes T threads
    __device__ static int slot(int k) { return M2 * (k & (M1 - 1)) + k / M1; }
    __device__ static int at(int row, int pitch) { return (row + row / M2) * pitch; }
    // twiddle exp(S 2 pi i j / M) from the table of exp(-2 pi i j / M)
    template <int S>
    __device__ static float2 tw(const float2 *tw_s, int j) {
        float2 w = tw_s[j];
        if (S > 0) w.y = -w.y;
        return w;
    }
    // first level: the M1-point transforms over points M2 apart, twiddled
    template <int S>
    __device__ static void forward_first(float2 *x, const float2 *tw_s, int pitch, int b, int n2) {
        float2 v[M1];
#pragma unroll
        for (int n1 = 0; n1 < M1; ++n1) v[n1] = x[at(M2 * n1 + n2, pitch) + b];
        dft_reg<M1, S>(v);
#pragma unroll
        for (int k1 = 0; k1 < M1; ++k1) x[at(M2 * k1 + n2, pitch) + b] = k1 ? cmul(v[k1], tw<S>(tw_s, n2 * k1)) : v[k1];
    }
    // second level: u[k2] = X[k1 + M1 k2]
    template <int S>
    __device__ static void forward_second(const float2 *x, int pitch, int b, int k1, float2 (&u)[M2]) {
#pragma unroll
        for (int n2 = 0; n2 < M2; ++n2) u[n2] = x[at(M2 * k1 + n2, pitch) + b];
        dft_reg<M2, S>(u);
    }
    // the inverse's first level, from u[k2] = X[k1 + M1 k2]
    template <int S>
    __device__ static void inverse_first(float2 *x, const float2 *tw_s, int pitch, int b, int k1, float2 (&u)[M2]) {
        dft_reg<M2, S>(u);
#pragma unroll
        for (int n2 = 0; n2 < M2; ++n2) x[at(M2 * k1 + n2, pitch) + b] = k1 ? cmul(u[n2], tw<S>(tw_s, n2 * k1)) : u[n2];
    }
    template <int S>
    __device__ static void inverse_second(float2 *x, int pitch, int b, int n2) {
        float2 v[M1];
#pragma unroll
        for (int k1 = 0; k1 < M1; ++k1) v[k1] = x[at(M2 * k1 + n2, pitch) + b];
        dft_reg<M1, S>(v);
#pragma unroll
        for (int n1 = 0; n1 < M1; ++n1) x[at(M2 * n1 + n2, pitch) + b] = v[n1];
    }
    // the 2^lb columns of x: natural order in, slot order out
    template <int S>
    __device__ static void forward(float2 *x, const float2 *tw_s, int pitch, int lb) {
        const int b = threadIdx.x & ((1 << lb) - 1), r = threadIdx.x >> lb;
        if (r < M2) forward_first<S>(x, tw_s, pitch, b, r);
        __syncthreads();
        if (r < M1) {
            float2 u[M2];
            forward_second<S>(x, pitch, b, r, u);
#pragma unroll
            for (int k2 = 0; k2 < M2; ++k2) x[at(M2 * r + k2, pitch) + b] = u[k2];
        }
        __syncthreads();
    }
    // slot order in, natural order out
    template <int S>
    __device__ static void inverse(float2 *x, const float2 *tw_s, int pitch, int lb) {
        const int b = threadIdx.x & ((1 << lb) - 1), r = threadIdx.x >> lb;
        if (r < M1) {
            float2 u[M2];
#pragma unroll
            for (int k2 = 0; k2 < M2; ++k2) u[k2] = x[at(M2 * r + k2, pitch) + b];
            inverse_first<S>(x, tw_s, pitch, b, r, u);
        }
        __syncthreads();
        if (r < M2) inverse_second<S>(x, pitch, b, r);
        __syncthreads();
    }
    // natural order in and out: forward transform, each X[m] times mul(m),
    // inverse transform; the spectrum stays in the second level's registers
    template <typename Mul>
    __device__ static void filter(float2 *x, const float2 *tw_s, int pitch, int lb, Mul mul) {
        const int b = threadIdx.x & ((1 << lb) - 1), r = threadIdx.x >> lb;
        if (r < M2) forward_first<-1>(x, tw_s, pitch, b, r);
        __syncthreads();
        if (r < M1) {
            float2 u[M2];
            forward_second<-1>(x, pitch, b, r, u);
#pragma unroll
            for (int k2 = 0; k2 < M2; ++k2) {
                const float g = mul(r + M1 * k2);
                u[k2] = make_float2(u[k2].x * g, u[k2].y * g);
            }
            inverse_first<+1>(x, tw_s, pitch, b, r, u);
        }
        __syncthreads();
        if (r < M2) inverse_second<+1>(x, pitch, b, r);
        __syncthreads();
    }
};

// Whether M takes the register transforms with `cols` columns per CTA (the
// one-box and many-box passes decide alike, so a box's transform is the same
// in both).  512 and 1024 use 32-point register DFTs, which need twice the
// registers: the many-box passes run those boxes in kernels of their own.
__host__ __device__ inline bool reg_fft_ok(int M, int cols) {
    int T;
    switch (M) {
        case 16: T = 4; break;
        case 32: T = 8; break;
        case 64: T = 8; break;
        case 128: T = 16; break;
        case 256: T = 16; break;
        case 512: T = 32; break;
        case 1024: T = 32; break;
        default: return false;
    }
    return T * cols <= kFFTThreads;
}

// The passes below with the register transforms (M = FT::M; one buffer of
// FT::ROWS * pitch points, the twiddle table after it).
//
// z passes: the pitch P + 1 keeps a row's consecutive points on different
// banks where global rows are read or written along m or k, and (M2 + 1)
// (P + 1), odd, does so for the slot order: the two rows' spectra are taken
// straight from the transform's slots, and the inverse's slots filled
// straight from the rows, with no staging block.
template <typename FT>
__device__ __forceinline__ void fft_z_r2c_reg(unsigned long long *__restrict__ rho64, float mscale,
                                              float2 *__restrict__ spec, const float2 *tw, int P, int blk) {
    constexpr int M = FT::M, stride = spec_stride(M), kBatch = 4;
    extern __shared__ float2 sm[];
    const int pitch = P + 1;
    float2 *x = sm, *tw_s = sm + FT::ROWS * pitch;
    const size_t r0 = (size_t)blk * 2 * P;
    load_twiddles(tw_s, tw, M);
    chain_wait();
    // rows 2pr and 2pr+1 packed as one complex column, two points a thread
    // and load; every sum read is cleared for the next deposit
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
    for (int e0 = threadIdx.x; e0 < P * (M / 2); e0 += kBatch * blockDim.x) {
        ulonglong2 a[kBatch], c[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * (M / 2)) {
                const int pr = e / (M / 2), m = 2 * (e & (M / 2 - 1));
                const ulonglong2 *g = reinterpret_cast<const ulonglong2 *>(rho64 + (r0 + 2 * pr) * M + m);
                a[u] = g[0];
                c[u] = g[M / 2];
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * (M / 2)) {
                const int pr = e / (M / 2), m = 2 * (e & (M / 2 - 1));
                ulonglong2 *g = reinterpret_cast<ulonglong2 *>(rho64 + (r0 + 2 * pr) * M + m);
                g[0] = zero;
                g[M / 2] = zero;
                x[FT::at(m, pitch) + pr] = make_float2(__fmul_rn(__ull2float_rn(a[u].x), mscale),
                                                       __fmul_rn(__ull2float_rn(c[u].x), mscale));
                x[FT::at(m + 1, pitch) + pr] = make_float2(__fmul_rn(__ull2float_rn(a[u].y), mscale),
                                                           __fmul_rn(__ull2float_rn(c[u].y), mscale));
            }
        }
    }
    __syncthreads();
    FT::template forward<-1>(x, tw_s, pitch, ilog2(P));
    chain_next();
    // both rows of a pair from the same two transform values, consecutive k
    for (int e = threadIdx.x; e < P * (M / 2); e += blockDim.x) {
        const int pr = e / (M / 2), k = e & (M / 2 - 1);
        auto put = [&](int k) {
            const float2 z = x[FT::at(FT::slot(k), pitch) + pr];
            float2 zc = x[FT::at(FT::slot((M - k) & (M - 1)), pitch) + pr];
            zc.y = -zc.y;
            float2 *row = spec + (r0 + 2 * pr) * stride + k;
            row[0] = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y + zc.y));
            // (z - zc) / (2i)
            row[stride] = make_float2(0.5f * (z.y - zc.y), -0.5f * (z.x - zc.x));
        };
        put(k);
        if (k == 0) put(M / 2);
    }
}

template <typename FT>
__device__ __forceinline__ void fft_z_c2r_reg(const float2 *__restrict__ spec, float *__restrict__ out,
                                              const float2 *tw, int P, int blk) {
    constexpr int M = FT::M, stride = spec_stride(M);
    extern __shared__ float2 sm[];
    const int pitch = P + 1;
    float2 *x = sm, *tw_s = sm + FT::ROWS * pitch;
    const size_t r0 = (size_t)blk * 2 * P;
    load_twiddles(tw_s, tw, M);
    chain_wait();
    // row pair pr packed as one complex column a + i b (a, b the Hermitian
    // rows 2pr and 2pr+1, imaginary parts at k = 0 and M/2 dropped), placed
    // in the slot order the inverse transform starts from: a pair's values at
    // k give the column's at k and M - k
    for (int e0 = threadIdx.x; e0 < P * (M / 2); e0 += kLoadBatch * blockDim.x) {
        float2 a[kLoadBatch], b[kLoadBatch];
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * (M / 2)) {
                const float2 *row = spec + (r0 + 2 * (e / (M / 2))) * stride + (e & (M / 2 - 1));
                a[u] = row[0];
                b[u] = row[stride];
            }
        }
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * (M / 2)) {
                const int pr = e / (M / 2), k = e & (M / 2 - 1);
                if (k) {
                    x[FT::at(FT::slot(k), pitch) + pr] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);      // a + i b
                    x[FT::at(FT::slot(M - k), pitch) + pr] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);  // conj a + i conj b
                } else {
                    const float2 *row = spec + (r0 + 2 * pr) * stride + M / 2;
                    x[FT::at(FT::slot(0), pitch) + pr] = make_float2(a[u].x, b[u].x);
                    x[FT::at(FT::slot(M / 2), pitch) + pr] = make_float2(row[0].x, row[stride].x);
                }
            }
        }
    }
    __syncthreads();
    FT::template inverse<+1>(x, tw_s, pitch, ilog2(P));
    chain_next();
    // the pair's two real rows from one transform value
    for (int e = threadIdx.x; e < P * M; e += blockDim.x) {
        const int pr = e / M, m = e & (M - 1);
        const float2 z = x[FT::at(m, pitch) + pr];
        out[(r0 + 2 * pr) * M + m] = z.x;
        out[(r0 + 2 * pr + 1) * M + m] = z.y;
    }
}

// The Green's factor of the transform index m along x for one (ky, kz):
// -g(kx) g(ky) g(kz) / k^2, 0 at k = 0.
struct GreenColumn {
    const float *green1d;
    float gy, gz;
    int c, M;
    __device__ __forceinline__ GreenColumn(const float *g1, int M_, int o, int kz, bool valid) : green1d(g1), M(M_) {
        const int ky = o <= M / 2 ? o : M - o;
        gy = g1[ky];
        gz = valid ? g1[kz] : 0.f;
        c = ky * ky + kz * kz;
    }
    __device__ __forceinline__ float operator()(int m) const {
        const int kx = m <= M / 2 ? m : M - m;
        const int k2 = kx * kx + c;
        return k2 > 0 ? -green1d[kx] * gy * gz * __frcp_rn((float)k2) : 0.f;
    }
};

template <typename FT>
__device__ __forceinline__ void fft_axis_reg(float2 *__restrict__ spec, const float2 *tw,
                                             const float *__restrict__ green1d, int B, int axis, int sign,
                                             int green, int bx, int by) {
    constexpr int M = FT::M, Mh = M / 2 + 1;
    extern __shared__ float2 sm[];
    const int pitch = B;
    float2 *x = sm, *tw_s = sm + FT::ROWS * pitch;
    const int o = by, kz0 = bx * B, bsh = ilog2(B), nb = min(B, Mh - kz0);
    const size_t sm_stride = axis == 1 ? (size_t)spec_stride(M) : (size_t)M * spec_stride(M);
    const size_t base = (size_t)o * (axis == 1 ? M : 1) * spec_stride(M);
    // an inverse-only pass starts from the slot order
    const bool to_slots = sign > 0;
    load_twiddles(tw_s, tw, M);
    chain_wait();
    for (int e0 = threadIdx.x; e0 < M * B; e0 += kLoadBatch * blockDim.x) {
        float2 v[kLoadBatch];
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            const int m = e >> bsh, b = e & (B - 1);
            v[u] = (e < M * B && b < nb) ? spec[base + m * sm_stride + kz0 + b] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < M * B) {
                const int m = e >> bsh, b = e & (B - 1);
                x[FT::at(to_slots ? FT::slot(m) : m, pitch) + b] = v[u];
            }
        }
    }
    __syncthreads();
    bool natural = true;
    if (sign < 0 && green) {
        const int b = threadIdx.x & (B - 1);
        FT::filter(x, tw_s, pitch, bsh, GreenColumn(green1d, M, o, kz0 + b, b < nb));
    } else if (sign < 0) {
        FT::template forward<-1>(x, tw_s, pitch, bsh);
        natural = false;
    } else {
        FT::template inverse<+1>(x, tw_s, pitch, bsh);
    }
    for (int e = threadIdx.x; e < M * B; e += blockDim.x) {
        const int m = e >> bsh, b = e & (B - 1);
        if (b < nb) spec[base + m * sm_stride + kz0 + b] = x[FT::at(natural ? m : FT::slot(m), pitch) + b];
    }
}

// rows r0 .. r0+2P-1 of the M^3 real grid (row = x*M + y) -> spectrum rows,
// as fft_z_r2c_reg
template <bool WIDE>
__device__ __forceinline__ void fft_z_r2c(unsigned long long *__restrict__ rho64, float mscale,
                                          float2 *__restrict__ spec, const float2 *tw, int M, uint32_t plan, int P,
                                          int blk) {
    constexpr int kBatch = 4;
    extern __shared__ float2 sm[];
    const int pitch = P + 1, half = M / 2, stride = spec_stride(M);
    float2 *x = sm, *y = sm + M * pitch, *tw_s = sm + 2 * M * pitch;
    const size_t r0 = (size_t)blk * 2 * P;
    const FastDiv dH((uint32_t)half);
    load_twiddles(tw_s, tw, M);
    chain_wait();
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
    for (int e0 = threadIdx.x; e0 < P * half; e0 += kBatch * blockDim.x) {
        ulonglong2 a[kBatch], c[kBatch];
        ulonglong2 *g[kBatch];
        int at[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * half) {
                const int pr = (int)dH.div((uint32_t)e), m = 2 * (e - pr * half);
                g[u] = reinterpret_cast<ulonglong2 *>(rho64 + (r0 + 2 * pr) * M + m);
                at[u] = m * pitch + pr;
                a[u] = g[u][0];
                c[u] = g[u][half];
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (e0 + u * blockDim.x < P * half) {
                g[u][0] = zero;  // cleared for the next deposit
                g[u][half] = zero;
                // the deposit's exact integer sums, rounded once to float
                x[at[u]] = make_float2(__fmul_rn(__ull2float_rn(a[u].x), mscale),
                                       __fmul_rn(__ull2float_rn(c[u].x), mscale));
                x[at[u] + pitch] = make_float2(__fmul_rn(__ull2float_rn(a[u].y), mscale),
                                               __fmul_rn(__ull2float_rn(c[u].y), mscale));
            }
        }
    }
    __syncthreads();
    float2 *res = fft_columns<-1, WIDE>(x, y, tw_s, M, plan, ilog2(P), pitch);
    chain_next();
    for (int e = threadIdx.x; e < P * half; e += blockDim.x) {
        const int pr = (int)dH.div((uint32_t)e), k = e - pr * half;
        auto put = [&](int k) {
            const float2 z = res[k * pitch + pr];
            float2 zc = res[(k ? M - k : 0) * pitch + pr];
            zc.y = -zc.y;
            float2 *row = spec + (r0 + 2 * pr) * stride + k;
            row[0] = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y + zc.y));
            // (z - zc) / (2i)
            row[stride] = make_float2(0.5f * (z.y - zc.y), -0.5f * (z.x - zc.x));
        };
        put(k);
        if (k == 0) put(half);
    }
}

template <bool WIDE>
__device__ __forceinline__ void fft_z_c2r(const float2 *__restrict__ spec, float *__restrict__ out,
                                          const float2 *tw, int M, uint32_t plan, int P, int blk) {
    extern __shared__ float2 sm[];
    const int pitch = P + 1, half = M / 2, stride = spec_stride(M);
    float2 *x = sm, *y = sm + M * pitch, *tw_s = sm + 2 * M * pitch;
    const size_t r0 = (size_t)blk * 2 * P;
    const FastDiv dH((uint32_t)half), dM((uint32_t)M);
    load_twiddles(tw_s, tw, M);
    chain_wait();
    for (int e0 = threadIdx.x; e0 < P * half; e0 += kLoadBatch * blockDim.x) {
        float2 a[kLoadBatch], b[kLoadBatch];
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * half) {
                const int pr = (int)dH.div((uint32_t)e);
                const float2 *row = spec + (r0 + 2 * pr) * stride + (e - pr * half);
                a[u] = row[0];
                b[u] = row[stride];
            }
        }
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < P * half) {
                const int pr = (int)dH.div((uint32_t)e), k = e - pr * half;
                if (k) {
                    x[k * pitch + pr] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);        // a + i b
                    x[(M - k) * pitch + pr] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);  // conj a + i conj b
                } else {
                    const float2 *row = spec + (r0 + 2 * pr) * stride + half;
                    x[pr] = make_float2(a[u].x, b[u].x);
                    x[half * pitch + pr] = make_float2(row[0].x, row[stride].x);
                }
            }
        }
    }
    __syncthreads();
    float2 *res = fft_columns<+1, WIDE>(x, y, tw_s, M, plan, ilog2(P), pitch);
    chain_next();
    for (int e = threadIdx.x; e < P * M; e += blockDim.x) {
        const int pr = (int)dM.div((uint32_t)e), m = e - pr * M;
        const float2 z = res[m * pitch + pr];
        out[(r0 + 2 * pr) * M + m] = z.x;
        out[(r0 + 2 * pr + 1) * M + m] = z.y;
    }
}

// axis 1: y transform for fixed x = by; axis 0: x transform for fixed y = by,
// with the Green's multiply and inverse transform when green != 0; columns
// kz0 = bx * B ...
template <bool WIDE>
__device__ __forceinline__ void fft_axis(float2 *__restrict__ spec, const float2 *tw,
                                         const float *__restrict__ green1d, int M, uint32_t plan, int B, int axis,
                                         int sign, int green, int bx, int by) {
    extern __shared__ float2 sm[];
    const int pitch = B;
    float2 *x = sm, *y = sm + M * pitch, *tw_s = sm + 2 * M * pitch;
    const int Mh = M / 2 + 1;
    const int o = by;
    const int kz0 = bx * B;
    const int bsh = ilog2(B);  // B is a power of two
    const int nb = min(B, Mh - kz0);
    const size_t sm_stride = axis == 1 ? (size_t)spec_stride(M) : (size_t)M * spec_stride(M);
    const size_t base = (size_t)o * (axis == 1 ? M : 1) * spec_stride(M);
    load_twiddles(tw_s, tw, M);
    chain_wait();
    for (int e0 = threadIdx.x; e0 < M * B; e0 += kLoadBatch * blockDim.x) {
        float2 v[kLoadBatch];
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            int e = e0 + u * blockDim.x;
            const int m = e >> bsh, b = e & (B - 1);
            v[u] = (e < M * B && b < nb) ? spec[base + m * sm_stride + kz0 + b] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u) {
            int e = e0 + u * blockDim.x;
            if (e < M * B) x[e] = v[u];  // pitch == B
        }
    }
    __syncthreads();
    float2 *res = sign < 0 ? fft_columns<-1, WIDE>(x, y, tw_s, M, plan, bsh, pitch)
                           : fft_columns<+1, WIDE>(x, y, tw_s, M, plan, bsh, pitch);
    if (green) {
        // res holds the full forward transform: k index m along x, y index o, kz0+b
        const int ky = o <= M / 2 ? o : M - o;
        const float gy = green1d[ky];
        for (int e = threadIdx.x; e < M * B; e += blockDim.x) {
            const int m = e >> bsh, b = e & (B - 1);
            int kx = m <= M / 2 ? m : M - m;
            int kz = kz0 + b;
            float2 v = res[m * pitch + b];
            float g = 0.f;
            if (b < nb) {
                int k2 = kx * kx + ky * ky + kz * kz;
                if (k2 > 0) g = -green1d[kx] * gy * green1d[kz] * __frcp_rn((float)k2);
            }
            res[m * pitch + b] = make_float2(v.x * g, v.y * g);
        }
        __syncthreads();
        float2 *other = res == x ? y : x;
        res = fft_columns<+1, WIDE>(res, other, tw_s, M, plan, bsh, pitch);
    }
    chain_next();
    for (int e = threadIdx.x; e < M * B; e += blockDim.x) {
        const int m = e >> bsh, b = e & (B - 1);
        if (b < nb) spec[base + m * sm_stride + kz0 + b] = res[m * pitch + b];
    }
}

template <bool WIDE>
__global__ void __launch_bounds__(kFFTThreads)
    k_fft_z_r2c(unsigned long long *__restrict__ rho64, float mscale, float2 *__restrict__ spec,
                const float2 *tw, int M, uint32_t plan, int P) {
    fft_z_r2c<WIDE>(rho64, mscale, spec, tw, M, plan, P, blockIdx.x);
}

template <bool WIDE>
__global__ void __launch_bounds__(kFFTThreads)
    k_fft_z_c2r(const float2 *__restrict__ spec, float *__restrict__ out, const float2 *tw, int M, uint32_t plan, int P) {
    fft_z_c2r<WIDE>(spec, out, tw, M, plan, P, blockIdx.x);
}

template <bool WIDE>
__global__ void __launch_bounds__(kFFTThreads)
    k_fft_axis(float2 *__restrict__ spec, const float2 *tw, const float *__restrict__ green1d, int M,
               uint32_t plan, int B, int axis, int sign, int green) {
    fft_axis<WIDE>(spec, tw, green1d, M, plan, B, axis, sign, green, blockIdx.x, blockIdx.y);
}

// fft_axis_reg for one box, with the batch B a compile-time constant
// (B divides the block and M * B is a multiple of it): each thread keeps one
// column b and visits the points m = r0 + j * (threads / B), so the index
// arithmetic of the loads, stores and transforms folds to constants and the
// Green's factor's column terms are computed once.  Same transforms and the
// same operations per point as fft_axis_reg.
template <typename FT, int B>
__device__ __forceinline__ void fft_axis_reg_fixed(float2 *__restrict__ spec, const float2 *tw,
                                                   const float *__restrict__ green1d, int axis, int sign,
                                                   int green, int bx, int by) {
    constexpr int M = FT::M, Mh = M / 2 + 1;
    constexpr int bsh = ilog2(B), rs = kFFTThreads / B, per = M * B / kFFTThreads;
    static_assert(kFFTThreads % B == 0 && (M * B) % kFFTThreads == 0, "batch layout");
    extern __shared__ float2 sm[];
    float2 *x = sm, *tw_s = sm + FT::ROWS * B;
    const int o = by, kz0 = bx * B, nb = min(B, Mh - kz0);
    const int b = threadIdx.x & (B - 1), r0 = threadIdx.x >> bsh;
    const bool valid = b < nb;
    const size_t sm_stride = axis == 1 ? (size_t)spec_stride(M) : (size_t)M * spec_stride(M);
    float2 *col = spec + (size_t)o * (axis == 1 ? M : 1) * spec_stride(M) + kz0 + b;
    // an inverse-only pass starts from the slot order
    const bool to_slots = sign > 0;
    load_twiddles(tw_s, tw, M);
    chain_wait();
#pragma unroll
    for (int j0 = 0; j0 < per; j0 += kLoadBatch) {
        float2 v[kLoadBatch];
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u)
            if (j0 + u < per) v[u] = valid ? col[(size_t)(r0 + (j0 + u) * rs) * sm_stride] : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kLoadBatch; ++u)
            if (j0 + u < per) {
                const int m = r0 + (j0 + u) * rs;
                x[FT::at(to_slots ? FT::slot(m) : m, B) + b] = v[u];
            }
    }
    __syncthreads();
    bool natural = true;
    if (sign < 0 && green) {
        FT::filter(x, tw_s, B, bsh, GreenColumn(green1d, M, o, kz0 + b, valid));
    } else if (sign < 0) {
        FT::template forward<-1>(x, tw_s, B, bsh);
        natural = false;
    } else {
        FT::template inverse<+1>(x, tw_s, B, bsh);
    }
    chain_next();
    if (valid) {
#pragma unroll 4
        for (int j = 0; j < per; ++j) {
            const int m = r0 + j * rs;
            col[(size_t)m * sm_stride] = x[FT::at(natural ? m : FT::slot(m), B) + b];
        }
    }
}

// One box, power-of-two mesh M = M1 * M2: the register transforms, one
// instantiation per split (its registers sized for its DFT lengths).
// The z passes' CTAs are as many threads as the batch's transforms take (P = 8
// pairs; 4 at M = 1024), which leaves none idle and more CTAs an SM.
constexpr int kMaxP = 8;
__host__ __device__ constexpr int z_threads(int M1, int M2) {
    const int T = M1 > M2 ? M1 : M2, P = M1 * M2 == 1024 ? 4 : kMaxP;
    return T * P < 128 ? 128 : T * P;
}

template <int M1, int M2>
__global__ void __launch_bounds__(z_threads(M1, M2), M1 * M2 == 1024 ? 4 : M1 * M2 == 512 ? 2 : 6)
    k_fft_z_r2c_r(unsigned long long *__restrict__ rho64, float mscale, float2 *__restrict__ spec,
                  const float2 *tw, int P) {
    fft_z_r2c_reg<RegFFT<M1, M2>>(rho64, mscale, spec, tw, P, blockIdx.x);
}

template <int M1, int M2>
__global__ void __launch_bounds__(z_threads(M1, M2), M1 * M2 == 1024 ? 4 : M1 * M2 == 512 ? 2 : 6)
    k_fft_z_c2r_r(const float2 *__restrict__ spec, float *__restrict__ out, const float2 *tw, int P) {
    fft_z_c2r_reg<RegFFT<M1, M2>>(spec, out, tw, P, blockIdx.x);
}

// the one-box batch of the axis passes, fft_batch_axis(M)
__host__ __device__ constexpr int axis_batch(int M) { return M == 1024 ? 8 : (4096 / M > 16 ? 16 : 4096 / M); }

template <int M1, int M2>
__global__ void __launch_bounds__(kFFTThreads, M1 * M2 >= 512 ? 2 : 4)
    k_fft_axis_r(float2 *__restrict__ spec, const float2 *tw, const float *__restrict__ green1d, int axis,
                 int sign, int green) {
    fft_axis_reg_fixed<RegFFT<M1, M2>, axis_batch(M1 * M2)>(spec, tw, green1d, axis, sign, green, blockIdx.x,
                                                            blockIdx.y);
}

// The five transform passes of one box with the register transforms.
template <int M1, int M2>
cuco_status_t fft_passes_reg(const PMPlan &plan, int P, bool chain, cudaStream_t stream) {
    constexpr int M = M1 * M2, Mh = M / 2 + 1, B = axis_batch(M);
    // the transform buffer and the twiddles
    constexpr int rows = RegFFT<M1, M2>::ROWS, zt = z_threads(M1, M2);
    const size_t smz = sizeof(float2) * ((size_t)rows * (P + 1) + M), sma = sizeof(float2) * ((size_t)rows * B + M);
    static OncePerDevice limit;
    CUCO_TRY_CUDA(limit.run([] {
        cudaError_t e = raise_smem_limit(k_fft_z_r2c_r<M1, M2>, kMaxSmem);
        if (e == cudaSuccess) e = raise_smem_limit(k_fft_z_c2r_r<M1, M2>, kMaxSmem);
        if (e == cudaSuccess) e = raise_smem_limit(k_fft_axis_r<M1, M2>, kMaxSmem);
        return e;
    }));
    const unsigned zblocks = (unsigned)((size_t)M * M / (2 * P));
    CUCO_TRY_CUDA(launch_chained(chain, k_fft_z_r2c_r<M1, M2>, zblocks, zt, smz, stream, plan.rho64,
                                 ldexpf(plan.mass, -32), plan.spec, plan.twiddle, P));
    dim3 ag((Mh + B - 1) / B, M);
    CUCO_TRY_CUDA(launch_chained(chain, k_fft_axis_r<M1, M2>, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                 plan.green1d, 1, -1, 0));
    CUCO_TRY_CUDA(launch_chained(chain, k_fft_axis_r<M1, M2>, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                 plan.green1d, 0, -1, 1));
    CUCO_TRY_CUDA(launch_chained(chain, k_fft_axis_r<M1, M2>, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                 plan.green1d, 1, +1, 0));
    CUCO_TRY_CUDA(launch_chained(chain, k_fft_z_c2r_r<M1, M2>, zblocks, zt, smz, stream, plan.spec, plan.rho,
                                 plan.twiddle, P));
    return CUCO_OK;
}

// Many boxes in one launch: map[blockIdx.x] = (box, the box's own block
// index).  BIG: only the boxes with 32-point register transforms (meshes 512
// and 1024), every other block returns; !BIG: every other box.
// What bounds them is latency: at four CTAs an SM (64 registers, a few spilled)
// instead of three (80) a step of 64 mixed boxes takes 6.15 instead of 6.31 ms,
// of 16 boxes of 16^3 to 64^3 1.31 instead of 1.33.
__device__ __forceinline__ bool big_box(const PMBoxDesc &d, int cols) {
    return d.M >= 512 && reg_fft_ok(d.M, cols);
}

template <bool BIG, bool WIDE>
__global__ void __launch_bounds__(kFFTThreads, BIG ? 2 : 4)
    k_fft_z_r2c_multi(const PMBoxDesc *__restrict__ boxes, const uint2 *__restrict__ map) {
    const uint2 m = map[blockIdx.x];
    const PMBoxDesc &d = boxes[m.x];
    if (big_box(d, d.P) != BIG) return;
    if (BIG) {
        if (d.M == 512)
            fft_z_r2c_reg<RegFFT<16, 32>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y);
        else
            fft_z_r2c_reg<RegFFT<32, 32>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y);
    } else if (reg_fft_ok(d.M, d.P)) {
        switch (d.M) {
            case 16: fft_z_r2c_reg<RegFFT<4, 4>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y); break;
            case 32: fft_z_r2c_reg<RegFFT<4, 8>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y); break;
            case 64: fft_z_r2c_reg<RegFFT<8, 8>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y); break;
            case 128: fft_z_r2c_reg<RegFFT<8, 16>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y); break;
            default: fft_z_r2c_reg<RegFFT<16, 16>>(d.rho64, d.mscale, d.spec, d.twiddle, d.P, m.y); break;
        }
    } else {
        fft_z_r2c<WIDE>(d.rho64, d.mscale, d.spec, d.twiddle, d.M, d.stages, d.P, m.y);
    }
}

template <bool BIG, bool WIDE>
__global__ void __launch_bounds__(kFFTThreads, BIG ? 2 : 4)
    k_fft_z_c2r_multi(const PMBoxDesc *__restrict__ boxes, const uint2 *__restrict__ map) {
    const uint2 m = map[blockIdx.x];
    const PMBoxDesc &d = boxes[m.x];
    if (big_box(d, d.P) != BIG) return;
    if (BIG) {
        if (d.M == 512)
            fft_z_c2r_reg<RegFFT<16, 32>>(d.spec, d.rho, d.twiddle, d.P, m.y);
        else
            fft_z_c2r_reg<RegFFT<32, 32>>(d.spec, d.rho, d.twiddle, d.P, m.y);
    } else if (reg_fft_ok(d.M, d.P)) {
        switch (d.M) {
            case 16: fft_z_c2r_reg<RegFFT<4, 4>>(d.spec, d.rho, d.twiddle, d.P, m.y); break;
            case 32: fft_z_c2r_reg<RegFFT<4, 8>>(d.spec, d.rho, d.twiddle, d.P, m.y); break;
            case 64: fft_z_c2r_reg<RegFFT<8, 8>>(d.spec, d.rho, d.twiddle, d.P, m.y); break;
            case 128: fft_z_c2r_reg<RegFFT<8, 16>>(d.spec, d.rho, d.twiddle, d.P, m.y); break;
            default: fft_z_c2r_reg<RegFFT<16, 16>>(d.spec, d.rho, d.twiddle, d.P, m.y); break;
        }
    } else {
        fft_z_c2r<WIDE>(d.spec, d.rho, d.twiddle, d.M, d.stages, d.P, m.y);
    }
}

template <bool BIG, bool WIDE>
__global__ void __launch_bounds__(kFFTThreads, BIG ? 2 : 4)
    k_fft_axis_multi(const PMBoxDesc *__restrict__ boxes, const uint2 *__restrict__ map, int axis, int sign,
                     int green) {
    const uint2 m = map[blockIdx.x];
    const PMBoxDesc &d = boxes[m.x];
    if (big_box(d, d.B) != BIG) return;
    const int nbx = (d.M / 2 + 1 + d.B - 1) / d.B;
    const int bx = m.y % nbx, by = m.y / nbx;
    if (BIG) {
        if (d.M == 512)
            fft_axis_reg<RegFFT<16, 32>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by);
        else
            fft_axis_reg<RegFFT<32, 32>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by);
    } else if (reg_fft_ok(d.M, d.B)) {
        switch (d.M) {
            case 16: fft_axis_reg<RegFFT<4, 4>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by); break;
            case 32: fft_axis_reg<RegFFT<4, 8>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by); break;
            case 64: fft_axis_reg<RegFFT<8, 8>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by); break;
            case 128: fft_axis_reg<RegFFT<8, 16>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by); break;
            default: fft_axis_reg<RegFFT<16, 16>>(d.spec, d.twiddle, d.green1d, d.B, axis, sign, green, bx, by); break;
        }
    } else {
        fft_axis<WIDE>(d.spec, d.twiddle, d.green1d, d.M, d.stages, d.B, axis, sign, green, bx, by);
    }
}

__device__ __forceinline__ void cic_axis(float to_slab_fac, float p, int M, int *s, int *ss,
                                         float *d) {
    float t = __fmul_rn(to_slab_fac, p);  // pm_periodic.c:99 in float
    int sl = (int)t;
    if (sl >= M) sl = M - 1;
    if (sl < 0) sl = 0;
    *d = __fsub_rn(t, (float)sl);
    *s = sl;
    *ss = sl + 1 >= M ? sl + 1 - M : sl + 1;
}

// The same for a 32-bit fixed-point coordinate x (units of L / 2^32): the
// mesh coordinate x * M / 2^32 is exact in 32.32 fixed point, so the cell and
// the fraction (rounded once, to float) need no float product.
__device__ __forceinline__ void cic_axis_fixed(uint32_t x, int M, int *s, int *ss, float *d) {
    const uint64_t t = (uint64_t)x * (uint32_t)M;
    const int sl = (int)(t >> 32);  // < M
    *d = (float)(uint32_t)t * 2.3283064365386963e-10f;  // 2^-32
    *s = sl;
    *ss = sl + 1 >= M ? sl + 1 - M : sl + 1;
}

template <bool FIXED>
__device__ __forceinline__ void cic_point(const float4 &p, float to_slab_fac, int M, int s[3][2], float d[3]) {
    if (FIXED) {
        cic_axis_fixed(__float_as_uint(p.x), M, &s[0][0], &s[0][1], &d[0]);
        cic_axis_fixed(__float_as_uint(p.y), M, &s[1][0], &s[1][1], &d[1]);
        cic_axis_fixed(__float_as_uint(p.z), M, &s[2][0], &s[2][1], &d[2]);
    } else {
        cic_axis(to_slab_fac, p.x, M, &s[0][0], &s[0][1], &d[0]);
        cic_axis(to_slab_fac, p.y, M, &s[1][0], &s[1][1], &d[1]);
        cic_axis(to_slab_fac, p.z, M, &s[2][0], &s[2][1], &d[2]);
    }
}

// CIC weights w in [0, 1] are added as the integers w * 2^32 (rounded once):
// integer atomics are associative, so the deposited grid does not depend on
// the order in which particles land, and it is the exact sum of the rounded
// weights.
constexpr unsigned kFullWarp = 0xffffffffu;
__device__ __forceinline__ unsigned long long weight_u64(float w) {
    return __float2ull_rn(__fmul_rn(w, 4294967296.0f));
}

// The eight CIC corners of a particle, warp-aggregated: particles of one warp
// in the same mesh cell share all eight corners, so one __match_any_sync on
// the cell finds them; each group adds its members' integer weights with
// shuffles into its lowest lane, which has the atomics issued.  When no two
// active lanes share a cell (lattice-ordered particles at high redshift) every
// lane keeps its own weights.  Integer sums are associative, so the grid is
// the same either way, bit for bit.  Called by every active lane of the warp
// together.
//
// What bounds it is the atomics in L2, which work on 32-byte sectors.  The two
// corners along z are neighbours there, so a full warp issues them from two
// lanes side by side, sixteen particles an instruction: neighbours in lattice
// or cell order then fill whole sectors (a lane issuing its eight corners
// touched each sector in two instructions).  Lanes of different boxes, and a
// partial warp, issue their own eight.  Measured as eight a lane / so:
// 512^3 lattice order on 1024^3 7.42 / 6.83 ms, 192^3 uniform in cell order on
// 384^3 0.271 / 0.224 ms, 100^3 clustered on 200^3 59 / 46 us.
template <bool FIXED, bool MANY>
__device__ __forceinline__ void deposit_one(float4 p, unsigned long long *__restrict__ rho64, int M,
                                            float to_slab_fac) {
    int s[3][2];
    float d[3];
    cic_point<FIXED>(p, to_slab_fac, M, s, d);
    const int sx = s[0][0], sxx = s[0][1], sy = s[1][0], syy = s[1][1], sz = s[2][0], szz = s[2][1];
    const float dx = d[0], dy = d[1], dz = d[2];
    const float m0 = 1.f - dx, m1 = dx;
    unsigned long long w[8] = {weight_u64(m0 * (1.f - dy) * (1.f - dz)), weight_u64(m0 * dy * (1.f - dz)),
                               weight_u64(m0 * (1.f - dy) * dz),        weight_u64(m0 * dy * dz),
                               weight_u64(m1 * (1.f - dy) * (1.f - dz)), weight_u64(m1 * dy * (1.f - dz)),
                               weight_u64(m1 * (1.f - dy) * dz),        weight_u64(m1 * dy * dz)};
    const unsigned active = __activemask(), lane = threadIdx.x & 31;
    const unsigned cell = ((unsigned)sx * (unsigned)M + (unsigned)sy) * (unsigned)M + (unsigned)sz;
    unsigned peers;
    bool mixed = false;  // a warp whose lanes hold particles of two boxes
    if (MANY) {
        int same;
        __match_all_sync(active, (unsigned long long)rho64, &same);
        mixed = !same;
    }
    if (mixed)
        peers = 1u << lane;  // (equal cells of different boxes are not the same cell)
    else
        peers = __match_any_sync(active, cell);
    bool lead = true;
    if (!__all_sync(active, peers == (1u << lane))) {
        // sum the group's weights into its lowest lane (every member runs the
        // same number of shuffles, named by the group's own mask)
        const unsigned first = (unsigned)__ffs(peers) - 1;
        lead = lane == first;
        unsigned long long sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (unsigned rest = peers; rest; rest &= rest - 1) {
            const int src = __ffs(rest) - 1;
#pragma unroll
            for (int c = 0; c < 8; ++c) sum[c] += __shfl_sync(peers, w[c], src);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] = sum[c];
    }
    [[maybe_unused]] const uint32_t M3 = (uint32_t)M * M * M;  // the bounds checks' grid size
    if (active == kFullWarp && !mixed) {
        // lane 2 j + h of an instruction: corner z + h of particle j
        const unsigned leads = __ballot_sync(kFullWarp, lead);
        const unsigned xs = (unsigned)sx | (unsigned)sxx << 16, ys = (unsigned)sy | (unsigned)syy << 16,
                       zs = (unsigned)sz | (unsigned)szz << 16;
        const bool hi = lane & 1;
#pragma unroll
        for (unsigned h = 0; h < 32; h += 16) {
            const unsigned src = h + (lane >> 1);
            const unsigned x = __shfl_sync(kFullWarp, xs, src), y = __shfl_sync(kFullWarp, ys, src),
                           zz = __shfl_sync(kFullWarp, zs, src), z = hi ? zz >> 16 : zz & 0xffffu;
            const bool on = leads >> src & 1u;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int lo = (c & 2) * 2 + (c & 1);
                const unsigned long long w0 = __shfl_sync(kFullWarp, w[lo], src), w1 = __shfl_sync(kFullWarp, w[lo + 2], src);
                const unsigned cx = c & 2 ? x >> 16 : x & 0xffffu, cy = c & 1 ? y >> 16 : y & 0xffffu;
                if (on) atomicAdd(&rho64[CUCO_IDX((cx * M + cy) * M + z, M3)], hi ? w1 : w0);
            }
        }
    } else if (lead) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const unsigned cx = c & 4 ? sxx : sx, cy = c & 1 ? syy : sy, cz = c & 2 ? szz : sz;
            atomicAdd(&rho64[CUCO_IDX((cx * M + cy) * M + cz, M3)], w[c]);
        }
    }
}

__device__ __forceinline__ int wrapi(int a, int M) { return a < 0 ? a + M : (a >= M ? a - M : a); }

template <bool FIXED>
__device__ __forceinline__ float4 interp_one(float4 p, const float *__restrict__ phi, int M, float to_slab_fac,
                                             float fac) {
    int s[3][2];
    float d[3];
    cic_point<FIXED>(p, to_slab_fac, M, s, d);
    float wx[2] = {1.f - d[0], d[0]}, wy[2] = {1.f - d[1], d[1]}, wz[2] = {1.f - d[2], d[2]};
    // Per dimension the six mesh planes s-2 .. s+3 (periodic), as offsets:
    // the two corners are planes 2 and 3, and along each dimension the two
    // corners' stencils (c-2, c-1, c+1, c+2) share one line of six points,
    // so every potential value loaded is one sum of three offsets.
    int off[3][6];
#pragma unroll
    for (int dim = 0; dim < 3; ++dim) {
        const int scale = dim == 0 ? M * M : (dim == 1 ? M : 1);
#pragma unroll
        for (int q = 0; q < 6; ++q) off[dim][q] = wrapi(s[dim][0] - 2 + q, M) * scale;
    }
    // What bounds it is L1: the loads a particle.  The eight corners are on a
    // line of every dimension and are loaded once, 56 loads instead of 72:
    // 192^3 uniform in cell order on 384^3 0.354 -> 0.325 ms, 128^3 clustered on
    // 256^3 0.123 -> 0.115, 100^3 clustered on 200^3 63 -> 57 us; lattice order
    // the same (512^3 on 1024^3 3.25 ms).
    float corner[2][2][2];
#pragma unroll
    for (int cx = 0; cx < 2; ++cx)
#pragma unroll
        for (int cy = 0; cy < 2; ++cy)
#pragma unroll
            for (int cz = 0; cz < 2; ++cz)
                corner[cx][cy][cz] =
                    __ldg(&phi[CUCO_IDX(off[0][2 + cx] + off[1][2 + cy] + off[2][2 + cz], (uint32_t)M * M * M)]);
    float out[3];
#pragma unroll
    for (int dim = 0; dim < 3; ++dim) {
        // 4 lines x 4 loads and 2 corners instead of 32 loads
        float F[2][2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                // the two other dimensions' corner planes
                const int d1 = (dim + 1) % 3, d2 = (dim + 2) % 3;
                const int base = off[d1][2 + u] + off[d2][2 + v];
                float f[6];
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    int at[3];
                    at[dim] = q - 2;
                    at[d1] = u;
                    at[d2] = v;
                    f[q] = q == 2 || q == 3 ? corner[at[0]][at[1]][at[2]]
                                            : __ldg(&phi[CUCO_IDX(base + off[dim][q], (uint32_t)M * M * M)]);
                }
                // corner at s0 (f[2]) and at s0 + 1 (f[3])
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float fm1 = f[1 + h], fp1 = f[3 + h], fm2 = f[h], fp2 = f[4 + h];
                    const float Fv = fac * ((4.0f / 3.0f) * (fm1 - fp1) - (1.0f / 6.0f) * (fm2 - fp2));
                    // F indexed by (cx, cy, cz)
                    int idx[3];
                    idx[dim] = h;
                    idx[d1] = u;
                    idx[d2] = v;
                    F[idx[0]][idx[1]][idx[2]] = Fv;
                }
            }
        float a = 0.f;
#pragma unroll
        for (int cx = 0; cx < 2; ++cx)
#pragma unroll
            for (int cy = 0; cy < 2; ++cy)
#pragma unroll
                for (int cz = 0; cz < 2; ++cz) a += F[cx][cy][cz] * wx[cx] * wy[cy] * wz[cz];
        out[dim] = a;
    }
    return make_float4(out[0], out[1], out[2], 0.f);
}

template <bool FIXED>
__global__ void k_deposit(const float4 *__restrict__ pos, uint32_t n, unsigned long long *__restrict__ rho64,
                          int M, float to_slab_fac) {
    chain_next();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) deposit_one<FIXED, false>(pos[i], rho64, M, to_slab_fac);
}

// perm (or null): where each result goes, for positions in cell order
template <bool FIXED>
__global__ void k_interp(const float4 *__restrict__ pos, const uint32_t *__restrict__ perm, uint32_t n,
                         const float *__restrict__ phi, int M, float to_slab_fac, float fac,
                         float4 *__restrict__ acc) {
    chain_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) acc[perm ? perm[i] : i] = interp_one<FIXED>(pos[i], phi, M, to_slab_fac, fac);
}

template <bool FIXED>
__global__ void k_deposit_multi(const float4 *__restrict__ pos, uint32_t n, const PMBoxDesc *__restrict__ boxes,
                                const uint32_t *__restrict__ pbeg, int nbox) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const PMBoxDesc &d = boxes[find_box(pbeg, nbox, i)];
    deposit_one<FIXED, true>(pos[i], d.rho64, d.M, d.to_slab_fac);
}

template <bool FIXED>
__global__ void k_interp_multi(const float4 *__restrict__ pos, uint32_t n, const PMBoxDesc *__restrict__ boxes,
                               const uint32_t *__restrict__ pbeg, int nbox, float4 *__restrict__ acc) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const PMBoxDesc &d = boxes[find_box(pbeg, nbox, i)];
    acc[i] = interp_one<FIXED>(pos[i], d.rho, d.M, d.to_slab_fac, d.fd_fac);
}

// Batch sizes are powers of two: the transforms split a flat index into
// (row, column) with a shift and a mask.
int fft_batch_z(int M) {
    int P = 4096 / M;
    if (P > 16) P = 16;
    if (P > M / 2) P = M / 2;
    if (P < 1) P = 1;
    P = 1 << ilog2(P);
    // P pairs per CTA must divide the M*M/2 row pairs
    while (P > 1 && ((M * M / 2) % P)) P >>= 1;
    return P;
}

int fft_batch_axis(int M) {
    // M = 1024: 8 columns, not 4096 / M = 4.  Its register transform gives a
    // column 32 threads, so 8 columns keep all 256 threads of a CTA busy, and
    // each row of the batch is 64 contiguous bytes (the five passes of one
    // force took 21.2 instead of 26.2 ms)
    if (M == 1024) return 8;
    int B = 4096 / M;
    if (B > 16) B = 16;
    if (B < 1) B = 1;
    return 1 << ilog2(B);
}

}  // namespace

bool pm_big_fft(int M, int P, int B) { return M >= 512 && reg_fft_ok(M, P) && reg_fft_ok(M, B); }

// A power-of-two mesh must take the register transforms in every pass (as one
// box does): its batches may not exceed what they hold.
bool pm_fft_batches_ok(int M, int P, int B) {
    const bool pow2 = M >= 16 && M <= 1024 && (M & (M - 1)) == 0;
    return !pow2 || (reg_fft_ok(M, P) && reg_fft_ok(M, B));
}

bool pm_wide_stages(uint32_t stages) { return wide_plan(stages); }
size_t pm_spec_points(int M) { return (size_t)M * M * spec_stride(M); }
uint32_t pm_stage_plan(int M) { return stage_plan(M); }
int pm_batch_z(int M) { return fft_batch_z(M); }
int pm_batch_axis(int M) { return fft_batch_axis(M); }

void pm_tables(int M, float boxsize, float asmth, float *green1d, float2 *twiddle) {
    const size_t Mh = M / 2 + 1;
    double asmth2 = (2 * M_PI) * (double)asmth / (double)boxsize;
    asmth2 *= asmth2;
    for (size_t k = 0; k < Mh; ++k) {
        double e = exp(-(double)(k * k) * asmth2);
        double f = 1.0;
        if (k) {
            f = (M_PI * (double)k) / M;
            f = sin(f) / f;
        }
        green1d[k] = (float)(e / (f * f * f * f));
    }
    for (int t = 0; t < M; ++t)
        twiddle[t] = make_float2((float)cos(2 * M_PI * t / M), (float)-sin(2 * M_PI * t / M));
}

float pm_fd_fac(int M, float boxsize, double G) {
    double fac = G / (M_PI * (double)boxsize);
    fac *= (double)(1.0f / (2.0f * boxsize / (float)M));
    return (float)fac;
}

size_t pm_smem_z(int M, int P) { return sizeof(float2) * (2 * (size_t)M * (P + 1) + M); }
size_t pm_smem_axis(int M, int B) { return sizeof(float2) * (2 * (size_t)M * B + M); }

cuco_status_t pm_forces_multi(const PMMulti &m, const float4 *pos, uint32_t n, float4 *acc,
                              cudaStream_t stream, int *launches) {
    static OncePerDevice limit;
    CUCO_TRY_CUDA(limit.run([] {
        cudaError_t e = cudaSuccess;
        auto set = [&](auto kernel) {
            if (e == cudaSuccess) e = raise_smem_limit(kernel, kMaxSmem);
        };
        set(k_fft_z_r2c_multi<true, false>), set(k_fft_z_c2r_multi<true, false>), set(k_fft_axis_multi<true, false>);
        set(k_fft_z_r2c_multi<false, false>), set(k_fft_z_c2r_multi<false, false>), set(k_fft_axis_multi<false, false>);
        set(k_fft_z_r2c_multi<false, true>), set(k_fft_z_c2r_multi<false, true>), set(k_fft_axis_multi<false, true>);
        return e;
    }));
    CUCO_TRY_CUDA(cudaMemsetAsync(m.rho64_all, 0, sizeof(unsigned long long) * m.rho_all_count, stream));
    if (n) {
        if (m.fixed)
            k_deposit_multi<true><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, m.boxes, m.pbeg, m.nbox);
        else
            k_deposit_multi<false><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, m.boxes, m.pbeg, m.nbox);
    }
    // each pass: the boxes of the common kernels, then (when the ensemble has
    // any) the boxes of the large register transforms
    const auto r2c = m.wide ? k_fft_z_r2c_multi<false, true> : k_fft_z_r2c_multi<false, false>;
    const auto c2r = m.wide ? k_fft_z_c2r_multi<false, true> : k_fft_z_c2r_multi<false, false>;
    const auto along = m.wide ? k_fft_axis_multi<false, true> : k_fft_axis_multi<false, false>;
    r2c<<<m.nz_blocks, kFFTThreads, m.smz, stream>>>(m.boxes, m.map_z);
    if (m.big) k_fft_z_r2c_multi<true, false><<<m.nz_blocks, kFFTThreads, m.smz, stream>>>(m.boxes, m.map_z);
    for (int pass = 0; pass < 3; ++pass) {
        const int axis = pass == 1 ? 0 : 1, sign = pass == 2 ? +1 : -1, green = pass == 1;
        along<<<m.naxis_blocks, kFFTThreads, m.sma, stream>>>(m.boxes, m.map_axis, axis, sign, green);
        if (m.big)
            k_fft_axis_multi<true, false><<<m.naxis_blocks, kFFTThreads, m.sma, stream>>>(m.boxes, m.map_axis, axis, sign,
                                                                                   green);
    }
    c2r<<<m.nz_blocks, kFFTThreads, m.smz, stream>>>(m.boxes, m.map_z);
    if (m.big) k_fft_z_c2r_multi<true, false><<<m.nz_blocks, kFFTThreads, m.smz, stream>>>(m.boxes, m.map_z);
    if (n) {
        if (m.fixed)
            k_interp_multi<true><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, m.boxes, m.pbeg, m.nbox, acc);
        else
            k_interp_multi<false><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, m.boxes, m.pbeg, m.nbox, acc);
    }
    CUCO_TRY_CUDA(cudaGetLastError());
    if (launches) *launches += m.big ? 12 : 7;
    return CUCO_OK;
}

bool pm_mesh_supported(int M) {
    if (M < 8 || M > 1024 || (M & 1)) return false;
    int r = M;
    for (int f : {2, 3, 5})
        while (r % f == 0) r /= f;
    return r == 1;
}

cuco_status_t pm_plan_create(PMPlan *plan, int M, float boxsize, float asmth, float mass,
                             double G, bool fixed) {
    if (!pm_mesh_supported(M)) {
        set_error("PM mesh size must be even, in [8, 1024], with no prime factor above 5");
        return CUCO_ERR_UNSUPPORTED;
    }
    plan->M = M;
    plan->stages = stage_plan(M);
    plan->fixed = fixed;
    plan->boxsize = boxsize;
    plan->to_slab_fac = (float)M / boxsize;
    plan->mass = mass;
    double fac = G / (M_PI * (double)boxsize);
    fac *= (double)(1.0f / (2.0f * boxsize / (float)M));
    plan->fd_fac = (float)fac;
    const size_t Mh = M / 2 + 1;
    CUCO_TRY_CUDA(cudaMalloc(&plan->rho, sizeof(float) * (size_t)M * M * M));
    CUCO_TRY_CUDA(cudaMalloc(&plan->rho64, sizeof(unsigned long long) * (size_t)M * M * M));
    plan->rho64_dirty = true;
    CUCO_TRY_CUDA(cudaMalloc(&plan->spec, sizeof(float2) * pm_spec_points(M)));
    CUCO_TRY_CUDA(cudaMalloc(&plan->green1d, sizeof(float) * Mh));
    CUCO_TRY_CUDA(cudaMalloc(&plan->twiddle, sizeof(float2) * M));
    std::vector<float> g(Mh);
    double asmth2 = (2 * M_PI) * (double)asmth / (double)boxsize;
    asmth2 *= asmth2;
    for (size_t k = 0; k < Mh; ++k) {
        double e = exp(-(double)(k * k) * asmth2);
        double f = 1.0;
        if (k) {
            f = (M_PI * (double)k) / M;
            f = sin(f) / f;
        }
        g[k] = (float)(e / (f * f * f * f));
    }
    std::vector<float2> tw(M);
    for (int t = 0; t < M; ++t) tw[t] = make_float2((float)cos(2 * M_PI * t / M), (float)-sin(2 * M_PI * t / M));
    CUCO_TRY_CUDA(cudaMemcpy(plan->green1d, g.data(), sizeof(float) * Mh, cudaMemcpyHostToDevice));
    CUCO_TRY_CUDA(cudaMemcpy(plan->twiddle, tw.data(), sizeof(float2) * M, cudaMemcpyHostToDevice));
    // The shared-memory limit is an attribute of the kernel, not of a launch:
    // it is set once to the most a CTA can have, so that boxes of different
    // meshes in one process (a serving loop's) never lower it under each
    // other's launches.
    const int P = fft_batch_z(M), B = fft_batch_axis(M);
    const size_t smz = sizeof(float2) * (2 * (size_t)M * (P + 1) + M);
    const size_t sma = sizeof(float2) * (2 * (size_t)M * B + M);
    if (smz > kMaxSmem || sma > kMaxSmem) {
        set_error("PM: the transform of this mesh needs more shared memory than a CTA has");
        return CUCO_ERR_UNSUPPORTED;
    }
    static OncePerDevice limit;
    CUCO_TRY_CUDA(limit.run([] {
        cudaError_t e = cudaSuccess;
        auto set = [&](auto kernel) {
            if (e == cudaSuccess) e = raise_smem_limit(kernel, kMaxSmem);
        };
        set(k_fft_z_r2c<false>), set(k_fft_z_c2r<false>), set(k_fft_axis<false>);
        set(k_fft_z_r2c<true>), set(k_fft_z_c2r<true>), set(k_fft_axis<true>);
        return e;
    }));
    return CUCO_OK;
}

void pm_plan_destroy(PMPlan *plan) {
    cudaFree(plan->rho);
    cudaFree(plan->rho64);
    plan->rho64 = nullptr;
    cudaFree(plan->spec);
    cudaFree(plan->green1d);
    cudaFree(plan->twiddle);
    plan->rho = nullptr;
    plan->spec = nullptr;
}

// Meshes below this launch the PM's kernels after the deposit chained
// (launch_chained): ten steps of 24^3 to 64^3 particles on twice the mesh take
// 745 -> 590, 745 -> 605, 1060 -> 900, 1300 -> 1185 and 1930 -> 1800 us, 80^3
// and 100^3 3655 -> 3455 and 6335 -> 6175; at 128^3 on 256^3 their launches
// are nothing beside the kernels, and the blocks that wait take places from
// the sort's (10.81 -> 10.83 ms).  A block lets the next kernel start when it
// begins its stores: as it ended its loads, 100^3 clustered lost 3 %.
constexpr int kChainMaxMesh = 256;

cuco_status_t pm_forces(PMPlan &plan, const float4 *pos, const uint32_t *perm, uint32_t n, float4 *acc,
                        cudaStream_t stream, cudaEvent_t *ev_deposit_done, cudaEvent_t *ev_fft_done,
                        int *launches) {
    const int M = plan.M, Mh = M / 2 + 1;
    // at most 8 row pairs per z-pass CTA: half the shared memory of 16, so
    // more CTAs fit beside the sort's (9 us faster per force at M = 256)
    const int P = std::min(fft_batch_z(M), kMaxP), B = fft_batch_axis(M);
    const size_t smz = sizeof(float2) * (2 * (size_t)M * (P + 1) + M);
    const size_t sma = sizeof(float2) * (2 * (size_t)M * B + M);
    // The z r2c pass clears the sums it reads, so the grid is zero again when
    // the previous call enqueued its passes; otherwise (first call, or a call
    // that stopped at an error) it is cleared here.
    const bool chain = M < kChainMaxMesh;
    if (plan.rho64_dirty)
        CUCO_TRY_CUDA(cudaMemsetAsync(plan.rho64, 0, sizeof(unsigned long long) * (size_t)M * M * M, stream));
    plan.rho64_dirty = true;
    if (n) {
        if (plan.fixed)
            k_deposit<true><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, plan.rho64, M, plan.to_slab_fac);
        else
            k_deposit<false><<<(n + 255) / 256, 256, 0, stream>>>(pos, n, plan.rho64, M, plan.to_slab_fac);
    }
    CUCO_TRY_CUDA(cudaGetLastError());
    if (ev_deposit_done) CUCO_TRY_CUDA(cudaEventRecord(*ev_deposit_done, stream));
    if (reg_fft_ok(M, P) && reg_fft_ok(M, B)) {
        cuco_status_t s;
        switch (M) {
            case 16: s = fft_passes_reg<4, 4>(plan, P, chain, stream); break;
            case 32: s = fft_passes_reg<4, 8>(plan, P, chain, stream); break;
            case 64: s = fft_passes_reg<8, 8>(plan, P, chain, stream); break;
            case 128: s = fft_passes_reg<8, 16>(plan, P, chain, stream); break;
            case 256: s = fft_passes_reg<16, 16>(plan, P, chain, stream); break;
            case 512: s = fft_passes_reg<16, 32>(plan, P, chain, stream); break;
            default: s = fft_passes_reg<32, 32>(plan, P, chain, stream); break;
        }
        CUCO_TRY(s);
    } else {
        const unsigned zblocks = (unsigned)((size_t)M * M / (2 * P));
        const bool wide = wide_plan(plan.stages);
        const auto r2c = wide ? k_fft_z_r2c<true> : k_fft_z_r2c<false>;
        const auto along = wide ? k_fft_axis<true> : k_fft_axis<false>;
        const auto c2r = wide ? k_fft_z_c2r<true> : k_fft_z_c2r<false>;
        CUCO_TRY_CUDA(launch_chained(chain, r2c, zblocks, kFFTThreads, smz, stream, plan.rho64, ldexpf(plan.mass,
                                     -32), plan.spec, plan.twiddle, M, plan.stages, P));
        dim3 ag((Mh + B - 1) / B, M);
        CUCO_TRY_CUDA(launch_chained(chain, along, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                     plan.green1d, M, plan.stages, B, 1, -1, 0));
        CUCO_TRY_CUDA(launch_chained(chain, along, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                     plan.green1d, M, plan.stages, B, 0, -1, 1));
        CUCO_TRY_CUDA(launch_chained(chain, along, ag, kFFTThreads, sma, stream, plan.spec, plan.twiddle,
                                     plan.green1d, M, plan.stages, B, 1, +1, 0));
        CUCO_TRY_CUDA(launch_chained(chain, c2r, zblocks, kFFTThreads, smz, stream, plan.spec, plan.rho,
                                     plan.twiddle, M, plan.stages, P));
        CUCO_TRY_CUDA(cudaGetLastError());
    }
    plan.rho64_dirty = false;
    if (ev_fft_done) CUCO_TRY_CUDA(cudaEventRecord(*ev_fft_done, stream));
    if (n) {
        if (plan.fixed)
            CUCO_TRY_CUDA(launch_chained(chain, k_interp<true>, (n + 255) / 256, 256, 0, stream, pos, perm, n,
                                         plan.rho, M, plan.to_slab_fac, plan.fd_fac, acc));
        else
            CUCO_TRY_CUDA(launch_chained(chain, k_interp<false>, (n + 255) / 256, 256, 0, stream, pos, perm, n,
                                         plan.rho, M, plan.to_slab_fac, plan.fd_fac, acc));
    }
    CUCO_TRY_CUDA(cudaGetLastError());
    if (launches) *launches += 5 + (n ? 2 : 0);  // five transform passes, deposit and interpolation
    return CUCO_OK;
}

uint32_t bounds_violations_pm() { return bounds_violations_take(); }

}  // namespace cuco
