// Kernel (b): a hand-written Stockham 3-D real FFT, the replacement of the
// FFTPACK5 halfcomplex transforms (PMP2mod_fft5.f90) used by POTENTfft5
// (PMP2main.f90:705-867) and POWERfft5 (PMP2mod_power.f90:209-463).
//
// The reference transforms FI with separable real halfcomplex FFTs and divides
// every coefficient by the eigenvalue of the 7-point Laplacian,
//   A1 = GREENf(i) + GREENf(j) + GREENf(k) - 6,  GREENf = 2 cos(2 pi m / N),
// keeping the DC coefficient (A1 := 1, PMP2main.f90:815).  Because the kernel
// depends only on |m| along each axis, the same operator is diagonal in the
// complex Fourier basis, so a real-to-complex 3-D transform with the same A1
// reproduces it up to rounding.  Pipeline (each pass one kernel, FP32 data
// between passes; the lines of a pass are computed in FP64 on the plain path,
// as FFTPACK5's real(kind=8), and in FP32 in the precision form, with twiddles
// tabulated in FP64):
//   x  : real rows -> half spectrum (N/2 complex FFT + split),      R2C
//   y  : complex lines along y,                                       forward
//   z  : forward along z, * trfi / A1 * 2 / N^3, inverse along z      (fused)
//   y  : inverse
//   x  : half spectrum -> real rows (merge + N/2 complex FFT),        C2R
// Lines live in registers: Stockham autosort stages of radix 4 to 32 on 4 to 32
// values per thread, straight from and to global memory, with one exchange through
// shared memory between two stages (one or two per line).
#include "mgg_internal.cuh"
#include "fft.cuh"
#include <map>
#include <mutex>
#include "reduce.cuh"

namespace mgg {

namespace {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by SIGN * i
template <int SIGN>
__device__ __forceinline__ float2 mul_si(float2 a) {
    return SIGN < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}
// the same in FP64 (the plain path's line arithmetic, as FFTPACK5's real(kind=8))
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
template <int SIGN>
__device__ __forceinline__ double2 mul_si(double2 a) {
    return SIGN < 0 ? make_double2(a.y, -a.x) : make_double2(-a.y, a.x);
}
// scalar type of a complex type; FP32 storage <-> the arithmetic type
template <class C> struct Scal;
template <> struct Scal<float2> { typedef float T; };
template <> struct Scal<double2> { typedef double T; };
template <class C> __device__ __forceinline__ C from_f2(float2 v);
template <> __device__ __forceinline__ float2 from_f2<float2>(float2 v) { return v; }
template <> __device__ __forceinline__ double2 from_f2<double2>(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ float2 to_f2(float2 v) { return v; }
__device__ __forceinline__ float2 to_f2(double2 v) { return make_float2((float)v.x, (float)v.y); }
template <class C> __device__ __forceinline__ C czero();
template <> __device__ __forceinline__ float2 czero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }

constexpr int ilog2c(int v) { return v <= 1 ? 0 : 1 + ilog2c(v >> 1); }

// W16^p = exp(-2 pi i p / 16) for p = 0..15, as (cos, sin) pairs
__device__ __forceinline__ float w16c(int p) {
    constexpr float c[16] = {1.0f, 0.92387953251f, 0.70710678119f, 0.38268343237f, 0.0f, -0.38268343237f,
                             -0.70710678119f, -0.92387953251f, -1.0f, -0.92387953251f, -0.70710678119f,
                             -0.38268343237f, 0.0f, 0.38268343237f, 0.70710678119f, 0.92387953251f};
    return c[p & 15];
}
__device__ __forceinline__ float w16s(int p) { return w16c(p + 12); }   // sin(2 pi p/16) = cos(2 pi (p-4)/16)
__device__ __forceinline__ double w16c_d(int p) {
    constexpr double c[16] = {1.0, 0.92387953251128674, 0.70710678118654752, 0.38268343236508977, 0.0,
                              -0.38268343236508977, -0.70710678118654752, -0.92387953251128674, -1.0,
                              -0.92387953251128674, -0.70710678118654752, -0.38268343236508977, 0.0,
                              0.38268343236508977, 0.70710678118654752, 0.92387953251128674};
    return c[p & 15];
}
// v * exp(SIGN 2 pi i p / 16), p a compile-time constant after unrolling
template <int SIGN>
__device__ __forceinline__ float2 rot16(float2 v, int p) {
    if ((p & 15) == 0) return v;
    if ((p & 15) == 4) return mul_si<SIGN>(v);
    if ((p & 15) == 8) return make_float2(-v.x, -v.y);
    if ((p & 15) == 12) return mul_si<-SIGN>(v);
    const float c = w16c(p), sn = (float)SIGN * w16s(p);
    return make_float2(v.x * c - v.y * sn, v.x * sn + v.y * c);
}
template <int SIGN>
__device__ __forceinline__ double2 rot16(double2 v, int p) {
    if ((p & 15) == 0) return v;
    if ((p & 15) == 4) return mul_si<SIGN>(v);
    if ((p & 15) == 8) return make_double2(-v.x, -v.y);
    if ((p & 15) == 12) return mul_si<-SIGN>(v);
    const double c = w16c_d(p), sn = (double)SIGN * w16c_d(p + 12);
    return make_double2(v.x * c - v.y * sn, v.x * sn + v.y * c);
}

// v * exp(SIGN 2 pi i p / 32), p in 0..15 a compile-time constant after unrolling
template <int SIGN, class C>
__device__ __forceinline__ C rot32(C v, int p) {
    if ((p & 1) == 0) return rot16<SIGN>(v, p >> 1);
    using T = typename Scal<C>::T;
    constexpr double c32[9] = {1.0, 0.98078528040323044, 0.0, 0.83146961230254524, 0.0,
                               0.55557023301960222, 0.0, 0.19509032201612827, 0.0};
    const T c = (T)(p <= 8 ? c32[p & 7] : -c32[16 - p]), sn = (T)(SIGN * (p <= 8 ? c32[8 - p] : c32[p - 8]));
    C r;
    r.x = v.x * c - v.y * sn;
    r.y = v.x * sn + v.y * c;
    return r;
}

// In-register DFTs of size R = 2, 4, 8, 16, 32, natural order in and out:
// X[m] = sum_r v[r] exp(SIGN 2 pi i r m / R)
template <int SIGN, class C>
__device__ __forceinline__ void dft4(C& v0, C& v1, C& v2, C& v3) {
    const C a = cadd(v0, v2), bb = csub(v0, v2), cc = cadd(v1, v3);
    const C d = mul_si<SIGN>(csub(v1, v3));
    v0 = cadd(a, cc);
    v2 = csub(a, cc);
    v1 = cadd(bb, d);
    v3 = csub(bb, d);
}
template <int SIGN, int R, class C>
__device__ __forceinline__ void dft(C* v) {
    if (R == 2) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if (R == 4) {
        dft4<SIGN>(v[0], v[1], v[2], v[3]);
    } else if (R == 8) {   // r = r1 + 2 r2, m = m1 + 4 m2
        C y[2][4];
#pragma unroll
        for (int r1 = 0; r1 < 2; ++r1) {
            y[r1][0] = v[r1]; y[r1][1] = v[r1 + 2]; y[r1][2] = v[r1 + 4]; y[r1][3] = v[r1 + 6];
            dft4<SIGN>(y[r1][0], y[r1][1], y[r1][2], y[r1][3]);
#pragma unroll
            for (int m1 = 0; m1 < 4; ++m1) y[r1][m1] = rot16<SIGN>(y[r1][m1], 2 * r1 * m1);
        }
#pragma unroll
        for (int m1 = 0; m1 < 4; ++m1) {
            v[m1] = cadd(y[0][m1], y[1][m1]);
            v[m1 + 4] = csub(y[0][m1], y[1][m1]);
        }
    } else if (R == 32) {  // r = r1 + 2 r2, m = m1 + 16 m2
        C y[2][16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            y[0][r] = v[(2 * r) & (R - 1)];
            y[1][r] = v[(2 * r + 1) & (R - 1)];
        }
        dft<SIGN, 16>(y[0]);
        dft<SIGN, 16>(y[1]);
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const C w = rot32<SIGN>(y[1][m], m);
            v[m & (R - 1)] = cadd(y[0][m], w);
            v[(m + 16) & (R - 1)] = csub(y[0][m], w);
        }
    } else if (R == 16) {  // r = r1 + 4 r2, m = m1 + 4 m2
        C y[4][4];
#pragma unroll
        for (int r1 = 0; r1 < 4; ++r1) {
            y[r1][0] = v[r1]; y[r1][1] = v[r1 + 4]; y[r1][2] = v[r1 + 8]; y[r1][3] = v[r1 + 12];
            dft4<SIGN>(y[r1][0], y[r1][1], y[r1][2], y[r1][3]);
#pragma unroll
            for (int m1 = 0; m1 < 4; ++m1) y[r1][m1] = rot16<SIGN>(y[r1][m1], r1 * m1);
        }
#pragma unroll
        for (int m1 = 0; m1 < 4; ++m1) {
            dft4<SIGN>(y[0][m1], y[1][m1], y[2][m1], y[3][m1]);
            v[m1] = y[0][m1]; v[m1 + 4] = y[1][m1]; v[m1 + 8] = y[2][m1]; v[m1 + 12] = y[3][m1];
        }
    }
}

// ------------------------------------------------ lines in registers ----
// A line of L elements is held by T = L / E threads, E elements each, and goes
// through two (three) radix-R Stockham stages in registers; between two stages
// it is exchanged once through shared memory.  Element e + r L/R of a line (r <
// R) belongs to thread e mod T before a radix-R stage and after the last one, so
// the first stage's elements come straight from global memory (or from the
// previous transform of the line) and the last stage's go straight back.
//
// What bounds a pass is memory traffic, then shared memory and barriers: stages
// that each read and wrote a shared-memory tile, between a load into it and a
// store from it, moved a line 7 to 13 times through shared memory (the x pass at
// 92 % of that pipe), this form 2 to 4 times.  Per launch, before -> after (of the
// measured copy bandwidth), plain path at 512^3: x 0.965 -> 0.311 ms (0.53) and
// 1.014 -> 0.299, y 0.799 -> 0.305 (0.54), z with the Green's multiply 1.391 ->
// 0.555 (0.30); precision form at 1024^3: x 3.76 -> 1.62 ms (0.81) and 4.01 ->
// 1.77, y 2.11 -> 1.90 (0.69), z 4.81 -> 3.50 (0.38; two transforms of a pencil at
// 16 warps per SM).  Staging the next pencil by tensor copies, as the y and z
// passes did, is worth less than the registers' shorter path.
//
// Rad: the radices; REV runs them in reverse order, so that a forward transform
// followed by a reversed inverse needs no exchange in between.
template <int L_, int E_, int R1, int R2, int R3 = 1>
struct Rad {
    static constexpr int L = L_, E = E_, T = L_ / E_, NST = R3 > 1 ? 3 : 2;
    static_assert(R1 * R2 * R3 == L_ && E_ >= R1 && E_ >= R2 && E_ >= R3, "radices of the line");
    static constexpr int at(int i) { return i == 0 ? R1 : (i == 1 ? R2 : R3); }
    template <bool REV>
    static constexpr int radix(int i) { return REV ? at(NST - 1 - i) : at(i); }
    static constexpr int FIRST = R1, LAST = NST == 3 ? R3 : R2;
};

// The element of a line that register i of thread t holds around a radix-R stage
template <class F, int R>
__device__ __forceinline__ int elem_of(int t, int i) { return t + (i / R) * F::T + (i & (R - 1)) * (F::L / R); }

// Stages I, I+1, ... of a line: s is the line's first word in shared memory,
// element e at s[(e + e / PADU) * ES] (PADU spreads the strided writes of a
// stage over the banks; 0: none).  BLOCK: the lines of a block are exchanged
// together (block barriers), else a line stays within a warp.  tw[k] = exp(-2 pi
// i k / (L TWM)).  BUSY: earlier reads of the exchange buffer may be under way.
template <int SIGN, class F, bool REV, int TWM, int ES, int PADU, bool BLOCK, bool BUSY, int I = 0, int LGNS = 0, class C>
__device__ __forceinline__ void fft_regs(C (&v)[F::E], C* s, int t, const C* __restrict__ tw) {
    constexpr int R = F::template radix<REV>(I), LGR = ilog2c(R), NS = 1 << LGNS, Q = F::E / R;
    constexpr int TSTEP = (F::L / (R * NS)) * TWM;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        if (LGNS > 0) {
            const int k = (t + q * F::T) & (NS - 1);
#pragma unroll
            for (int r = 1; r < R; ++r) {
                C w = __ldg(tw + r * k * TSTEP);
                if (SIGN > 0) w = cconj(w);
                v[q * R + r] = cmul(v[q * R + r], w);
            }
        }
        dft<SIGN, R>(v + q * R);
    }
    if constexpr (I + 1 < F::NST) {
        constexpr int RN = F::template radix<REV>(I + 1);
        auto word = [](int e) { return (PADU ? e + e / (PADU ? PADU : 1) : e) * ES; };
        if (BUSY || I > 0) { if (BLOCK) __syncthreads(); else __syncwarp(); }
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
            const int j = t + (i / R) * F::T;
            s[word(((j >> LGNS) << (LGNS + LGR)) + (j & (NS - 1)) + (i & (R - 1)) * NS)] = v[i];
        }
        if (BLOCK) __syncthreads(); else __syncwarp();
#pragma unroll
        for (int i = 0; i < F::E; ++i) v[i] = s[word(elem_of<F, RN>(t, i))];
        fft_regs<SIGN, F, REV, TWM, ES, PADU, BLOCK, BUSY, I + 1, LGNS + LGR>(v, s, t, tw);
    }
}

// Radices per line length, FP32 and FP64.  A line's values are what a thread has
// registers for, 64 words: 32 FP32 values (two stages, one exchange, up to 1024
// points), 16 FP64 values.  Measured against fewer values and a third stage: FP32
// 1024 points at 16 values y 2.21 against 1.89 ms, x 2.14 against 1.62; FP64 256
// points at 8 values y 0.046 against 0.035, 512 points at 8 values 0.313 against 0.304.
template <int L, bool F64> struct RadOf;
#define MGG_RAD(L, ...) template <> struct RadOf<L, false> { using F = Rad<L, __VA_ARGS__>; };
#define MGG_RAD64(L, ...) template <> struct RadOf<L, true> { using F = Rad<L, __VA_ARGS__>; };
MGG_RAD(8, 4, 4, 2) MGG_RAD(16, 4, 4, 4) MGG_RAD(32, 8, 8, 4) MGG_RAD(64, 8, 8, 8) MGG_RAD(128, 16, 16, 8)
MGG_RAD(256, 16, 16, 16)
MGG_RAD(512, 32, 32, 16) MGG_RAD(1024, 32, 32, 32)
MGG_RAD64(8, 4, 4, 2) MGG_RAD64(16, 4, 4, 4) MGG_RAD64(32, 8, 8, 4) MGG_RAD64(64, 8, 8, 8) MGG_RAD64(128, 16, 16, 8)
MGG_RAD64(256, 16, 16, 16) MGG_RAD64(512, 16, 16, 16, 2) MGG_RAD64(1024, 16, 16, 16, 4)
#undef MGG_RAD
#undef MGG_RAD64

// blocks per SM that the register budget of a line kernel is set for: E complex
// values, their butterflies and addresses.  One rule for every mode; it was set on the
// plain passes, which do not spill.  The z pass with the Green's multiply holds FP64
// factors beside its line and spills at some sizes (FP32 lines of 1024 and 256
// values 0.26 and 0.19 KB, FP64 ones of 256 and 64 0.14 and 0.06 KB, LM_DISP of 512
// and 1024 24 bytes), at 0.40 to 0.95 of the time of the shared-memory passes
// it replaced at every size; budgets per mode are not measured.
template <class F, class C>
constexpr int fft_min_blocks(int threads) {
    constexpr int words = F::E * (int)sizeof(C) / 4;                    // 32-bit registers of the line
    const int budget = words >= 64 ? 128 : (words >= 32 ? (threads >= 512 ? 64 : 72) : 48);
    const int b = 65536 / (budget * threads);
    return b < 1 ? 1 : (b > 16 ? 16 : b);
}

// --------------------------------------------------------------- x pass ----
// Rows of N reals = L = N/2 complex values; a row stays within a warp, so its
// exchanges need no block barrier.
template <int N, class C>
struct XShape {
    using F = typename RadOf<N / 2, sizeof(C) == 16>::F;
    static constexpr int NT = 128, RB = NT / F::T;              // rows per block
    static constexpr int PADU = F::FIRST, LS = F::L + F::L / PADU;   // padded row
    static constexpr size_t SMEM = (size_t)RB * LS * sizeof(C);
    static_assert(F::T <= 32, "a row stays within a warp");
};

template <int N, class C>
__global__ void __launch_bounds__(XShape<N, C>::NT, fft_min_blocks<typename XShape<N, C>::F, C>(XShape<N, C>::NT))
    k_fft_x_r2c(const float* __restrict__ in, float2* __restrict__ out, int nxp, const C* __restrict__ tw) {
    using X = XShape<N, C>;
    using F = typename X::F;
    using T = typename Scal<C>::T;
    constexpr int L = F::L;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int q = threadIdx.x / F::T, t = threadIdx.x & (F::T - 1);
    C* s = reinterpret_cast<C*>(sm_raw) + q * X::LS;
    const int row = blockIdx.x * X::RB + q;   // N^2 rows: a multiple of RB
    const float2* src = reinterpret_cast<const float2*>(in) + (int64_t)row * L;
    C v[F::E];
#pragma unroll
    for (int i = 0; i < F::E; ++i) v[i] = from_f2<C>(__ldg(src + elem_of<F, F::FIRST>(t, i)));
    fft_regs<-1, F, false, 2, 1, X::PADU, false, false>(v, s, t, tw);
    auto word = [](int e) { return e + e / X::PADU; };
    __syncwarp();
#pragma unroll
    for (int i = 0; i < F::E; ++i) s[word(elem_of<F, F::LAST>(t, i))] = v[i];
    __syncwarp();
    // split: X[k] = Fe + W^k Fo, X[L-k] = conj(Fe - W^k Fo) with Fe = (Z[k] + conj Z[L-k]) / 2,
    // Fo = -i (Z[k] - conj Z[L-k]) / 2
    float2* dst = out + (int64_t)row * nxp;
#pragma unroll
    for (int i = 0; i <= F::E / 2; ++i) {
        const int k = t + i * F::T;
        if (i == F::E / 2 && t != 0) break;   // k = L/2
        const C zk = s[word(k)], zc = cconj(s[word(k == 0 ? 0 : L - k)]);
        const C fe = cscale(cadd(zk, zc), (T)0.5);
        const C fo = cmul(__ldg(tw + k), mul_si<-1>(cscale(csub(zk, zc), (T)0.5)));
        dst[k] = to_f2(cadd(fe, fo));
        dst[L - k] = to_f2(cconj(csub(fe, fo)));
    }
}

// Half spectrum rows -> real rows.  Output = (N/2) * x (unnormalised inverse / 2).
template <int N, class C>
__global__ void __launch_bounds__(XShape<N, C>::NT, fft_min_blocks<typename XShape<N, C>::F, C>(XShape<N, C>::NT))
    k_fft_x_c2r(const float2* __restrict__ in, float* __restrict__ out, int nxp, const C* __restrict__ tw) {
    using X = XShape<N, C>;
    using F = typename X::F;
    using T = typename Scal<C>::T;
    constexpr int L = F::L;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int q = threadIdx.x / F::T, t = threadIdx.x & (F::T - 1);
    C* s = reinterpret_cast<C*>(sm_raw) + q * X::LS;
    const int row = blockIdx.x * X::RB + q;
    const float2* src = in + (int64_t)row * nxp;
    C v[F::E];
    // merge: Z[k] = Fe + i Fo, Fe = (X[k] + conj X[L-k]) / 2, Fo = (X[k] - conj X[L-k]) conj(W^k) / 2
#pragma unroll
    for (int i = 0; i < F::E; ++i) {
        const int k = elem_of<F, F::FIRST>(t, i);
        const C xk = from_f2<C>(__ldg(src + k)), xl = cconj(from_f2<C>(__ldg(src + (L - k))));
        const C fe = cscale(cadd(xk, xl), (T)0.5);
        const C fo = cscale(cmul(csub(xk, xl), cconj(__ldg(tw + k))), (T)0.5);
        v[i] = cadd(fe, mul_si<1>(fo));
    }
    fft_regs<1, F, false, 2, 1, X::PADU, false, false>(v, s, t, tw);
    float2* dst = reinterpret_cast<float2*>(out) + (int64_t)row * L;
#pragma unroll
    for (int i = 0; i < F::E; ++i) dst[elem_of<F, F::LAST>(t, i)] = to_f2(v[i]);
}

// ---------------------------------------------------------- y / z lines ----
// Tile: TX consecutive kx columns x N elements of one line set.
//   element (x, e) of tile o at buf[o*ostride + e*estride + x0 + x]
// C: the arithmetic type of the lines (float2, or double2 for the plain path's
// FP64 line arithmetic); the spectrum is stored as float2 either way.

// LM_POWER's fixed-point sums of a block, per pair of (linear, log) bin: a value of
// up to 2^61 is added as three 32-bit words (19, 19 and the remaining bits: a block
// has at most 8192 modes, so the lower words cannot overflow, and the upper word's
// sum is right modulo 2^26, all of it that the 64-bit sum keeps), each one
// shared-memory operation that nothing waits for.  The 64-bit adds it replaces are
// compare-and-swap loops, which had to be summed over a warp first, a handful of
// distinct bins one after the other: z pass of P(k) at 512^3 (plain path, a late
// snapshot) 2.70 -> 0.93 ms.
__device__ __forceinline__ void limb_add(uint32_t* h, int npair, int p, unsigned long long v) {
    atomicAdd(h + p, (uint32_t)v & 0x7ffffu);
    atomicAdd(h + npair + p, (uint32_t)(v >> 19) & 0x7ffffu);
    atomicAdd(h + 2 * npair + p, (uint32_t)(v >> 38));
}
__device__ __forceinline__ unsigned long long limb_sum(const uint32_t* h, int npair, int p) {
    return (unsigned long long)h[p] + ((unsigned long long)h[npair + p] << 19) + ((unsigned long long)h[2 * npair + p] << 38);
}

// entries of the bin table before its pairs (an even number, so that the pairs are aligned)
__host__ __device__ constexpr int bin_table_m2(int N) { return (3 * (N / 2) * (N / 2) + 2) / 2 * 2; }

template <int N, class C>
struct LShape {   // y / z lines: TX kx columns x N elements per block
    using F = typename RadOf<N, sizeof(C) == 16>::F;
    static constexpr int TX = 8, NT = TX * F::T;
    static constexpr int PADU = sizeof(C) == 8 ? F::FIRST : 0;   // 128-byte FP64 rows cover the banks without padding
    static constexpr size_t WORDS = (size_t)TX * (N + (PADU ? N / (PADU ? PADU : 1) : 0));
};

template <int MODE, int N, class C>
__global__ void __launch_bounds__(LShape<N, C>::NT, fft_min_blocks<typename LShape<N, C>::F, C>(LShape<N, C>::NT))
    k_fft_lines(float2* __restrict__ buf, int64_t estride, int64_t ostride, const C* __restrict__ tw, LineExtra ex) {
    using S = LShape<N, C>;
    using F = typename S::F;
    using T = typename Scal<C>::T;
    constexpr int TX = S::TX, NT = S::NT, nxh = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int x = threadIdx.x & (TX - 1), t = threadIdx.x / TX;
    C* s = reinterpret_cast<C*>(sm_raw) + x;
    const int x0 = blockIdx.x * TX, o = blockIdx.y, kx = x0 + x;
    const bool valid = kx < nxh;
    const float2* src = (MODE == LM_DISP ? ex.src : buf) + (int64_t)o * ostride + kx;
    C v[F::E];
    constexpr int RIN = MODE == LM_DISP ? F::LAST : F::FIRST;
#pragma unroll
    for (int i = 0; i < F::E; ++i)
        v[i] = valid ? from_f2<C>(__ldg(src + elem_of<F, RIN>(t, i) * estride)) : czero<C>();
    float2* dst = buf + (int64_t)o * ostride + kx;
    auto put = [&](int i, int e) { if (valid) dst[e * estride] = to_f2(v[i]); };
    if constexpr (MODE == LM_FWD || MODE == LM_INV) {
        fft_regs<MODE == LM_FWD ? -1 : 1, F, false, 1, TX, S::PADU, true, false>(v, s, t, tw);
#pragma unroll
        for (int i = 0; i < F::E; ++i) put(i, elem_of<F, F::LAST>(t, i));
    } else if constexpr (MODE == LM_DISP) {
        // spectrum -> displacement component: psi_c(k) = i k_c / k^2 * T(k) * delta(k)
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
            const int kz = elem_of<F, F::LAST>(t, i), ky = o;
            const int mx = kx, my = ky <= N / 2 ? ky : ky - N, mz = kz <= N / 2 ? kz : kz - N;
            const int m2 = mx * mx + my * my + mz * mz;
            T f = (T)0;
            if (m2 > 0 && valid) {
                int mc = ex.comp == 0 ? mx : (ex.comp == 1 ? my : mz);
                // Nyquist planes carry no odd (sine) part
                if ((ex.comp == 0 && kx == N / 2) || (ex.comp == 1 && ky == N / 2) || (ex.comp == 2 && kz == N / 2)) mc = 0;
                f = (T)(__ldg(ex.tk + m2) * (float)mc / (float)m2);
            }
            v[i] = mul_si<1>(cscale(v[i], f));
        }
        fft_regs<1, F, true, 1, TX, S::PADU, true, false>(v, s, t, tw);
#pragma unroll
        for (int i = 0; i < F::E; ++i) put(i, elem_of<F, F::FIRST>(t, i));
    } else if constexpr (MODE == LM_GREEN) {
        // axis == 2: o = ky, element = kz
        fft_regs<-1, F, false, 1, TX, S::PADU, true, false>(v, s, t, tw);
        const double go = (__ldg(ex.green + o) - 6.0) , gx = __ldg(ex.green + min(kx, N / 2));
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
            double A1 = (go + gx) + __ldg(ex.green + elem_of<F, F::LAST>(t, i));
            if (fabs(A1) < 1.0e-7) A1 = 1.0;
            v[i] = cscale(v[i], (T)(ex.green_scale * green_reciprocal(A1)));
        }
        fft_regs<1, F, true, 1, TX, S::PADU, true, true>(v, s, t, tw);
#pragma unroll
        for (int i = 0; i < F::E; ++i) put(i, elem_of<F, F::FIRST>(t, i));
    } else {   // LM_POWER
        // linear bins, log bins, quadrupole-weighted linear bins (two's-complement sums)
        static_assert(TX * N <= 8192, "limb_add");
        uint32_t* hl = reinterpret_cast<uint32_t*>(sm_raw + S::WORDS * sizeof(C));
        uint32_t* hq = hl + 3 * ex.npair;
        const int nh = (ex.quad ? 6 : 3) * ex.npair;
        for (int e = threadIdx.x; e < nh; e += NT) hl[e] = 0u;
        __syncthreads();
        fft_regs<-1, F, false, 1, TX, S::PADU, true, false>(v, s, t, tw);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < F::E; ++i) s[elem_of<F, F::LAST>(t, i) * TX] = v[i];   // read back by this thread only
        const int ky = o;
        const double w = ((kx == 0 || kx == N / 2) ? 1.0 : 2.0) * ex.amp_scale;   // amp_scale times a power of two
#pragma unroll 1
        for (int i = 0; i < F::E; ++i) {
            const int kz = elem_of<F, F::LAST>(t, i);
            const C f = s[kz * TX];
            const int my = ky <= N / 2 ? ky : N - ky, mz = kz <= N / 2 ? kz : N - kz;
            const int m2 = kx * kx + my * my + mz * mz;
            if (!valid || m2 == 0) continue;
            const int p = __ldg(ex.bins + m2);
            const double amp = ((double)f.x * f.x + (double)f.y * f.y) * w;
            const unsigned long long fx = __double2ull_rn(amp);
            if (fx == 0ull) continue;   // and so is its quadrupole, smaller by |P2| <= 1
            limb_add(hl, ex.npair, p, fx);
            if (ex.quad) {
                // P2(mu) about z in Real*4 as the reference (cosmu2 = MI/RK**2, P2 = 1.5 cosmu2 - 0.5,
                // PMP2mod_power.f90:386-388, its MI being the z index after its x<->z transposition)
                const float RK = sqrtf((float)m2);
                const float cosmu2 = __fdiv_rn((float)(mz * mz), __fmul_rn(RK, RK));
                const float p2 = __fsub_rn(__fmul_rn(1.5f, cosmu2), 0.5f);
                limb_add(hq, ex.npair, p, (unsigned long long)__double2ll_rn(amp * (double)p2));
            }
        }
        __syncthreads();
        const ushort2* pair = reinterpret_cast<const ushort2*>(ex.bins + bin_table_m2(N));
        for (int p = threadIdx.x; p < ex.npair; p += NT) {
            const unsigned long long a = limb_sum(hl, ex.npair, p);
            const ushort2 b = __ldg(pair + p);
            if (a) {
                atomicAdd(ex.hist + b.x, a);
                atomicAdd(ex.hist + (N + 1) + b.y, a);
            }
            if (ex.quad) {
                const unsigned long long q = limb_sum(hq, ex.npair, p);
                if (q) atomicAdd(ex.hist + 2 * (N + 1) + b.x, q);
            }
        }
    }
}

#define MGG_FFT_SIZES(F) F(16) F(32) F(64) F(128) F(256) F(512) F(1024)

template <int N, class C>
void set_attrs_n() {
    const int big = 200 * 1024;
    MGG_CUDA(cudaFuncSetAttribute(k_fft_x_r2c<N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    MGG_CUDA(cudaFuncSetAttribute(k_fft_x_c2r<N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    MGG_CUDA(cudaFuncSetAttribute(k_fft_lines<LM_FWD, N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    MGG_CUDA(cudaFuncSetAttribute(k_fft_lines<LM_INV, N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    MGG_CUDA(cudaFuncSetAttribute(k_fft_lines<LM_GREEN, N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    MGG_CUDA(cudaFuncSetAttribute(k_fft_lines<LM_POWER, N, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    if (sizeof(C) == 8)
        MGG_CUDA(cudaFuncSetAttribute(k_fft_lines<LM_DISP, N, float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
}

template <int N, class C>
void x_r2c_c(const FftPlan& p, const C* tw, const float* in, float2* out, cudaStream_t s) {
    using X = XShape<N, C>;
    k_fft_x_r2c<N, C><<<N * N / X::RB, X::NT, X::SMEM, s>>>(in, out, p.nxp, tw);
    MGG_CHECK_LAUNCH();
}

template <int N, class C>
void x_c2r_c(const FftPlan& p, const C* tw, const float2* in, float* out, cudaStream_t s) {
    using X = XShape<N, C>;
    k_fft_x_c2r<N, C><<<N * N / X::RB, X::NT, X::SMEM, s>>>(in, out, p.nxp, tw);
    MGG_CHECK_LAUNCH();
}

template <int N>
void x_r2c_n(const FftPlan& p, const float* in, float2* out, cudaStream_t s) {
    if (p.tw64) x_r2c_c<N>(p, p.tw64, in, out, s);
    else x_r2c_c<N>(p, p.tw, in, out, s);
}

template <int N>
void x_c2r_n(const FftPlan& p, const float2* in, float* out, cudaStream_t s) {
    if (p.tw64) x_c2r_c<N>(p, p.tw64, in, out, s);
    else x_c2r_c<N>(p, p.tw, in, out, s);
}

template <int N, class C>
void lines_c(const FftPlan& p, const C* tw, float2* buf, int axis, int mode, const LineExtra& ex, cudaStream_t s) {
    using S = LShape<N, C>;
    const dim3 grid(div_up(N / 2 + 1, S::TX), N);
    int64_t estride, ostride;
    if (axis == 1) { estride = p.nxp; ostride = (int64_t)N * p.nxp; }       // o = z
    else { estride = (int64_t)N * p.nxp; ostride = p.nxp; }                  // o = y
    size_t smem = S::WORDS * sizeof(C);
    switch (mode) {
    case LM_FWD: k_fft_lines<LM_FWD, N, C><<<grid, S::NT, smem, s>>>(buf, estride, ostride, tw, ex); break;
    case LM_INV: k_fft_lines<LM_INV, N, C><<<grid, S::NT, smem, s>>>(buf, estride, ostride, tw, ex); break;
    case LM_GREEN: k_fft_lines<LM_GREEN, N, C><<<grid, S::NT, smem, s>>>(buf, estride, ostride, tw, ex); break;
    case LM_POWER:
        smem += (ex.quad ? 6 : 3) * (size_t)ex.npair * sizeof(uint32_t);
        k_fft_lines<LM_POWER, N, C><<<grid, S::NT, smem, s>>>(buf, estride, ostride, tw, ex);
        break;
    case LM_DISP:
        if constexpr (sizeof(C) == 8) {
            k_fft_lines<LM_DISP, N, C><<<grid, S::NT, smem, s>>>(buf, estride, ostride, tw, ex);
            break;
        }
        throw Error{MGG_ERR_ARG, "fft_lines: no FP64 form of this mode"};
    default: throw Error{MGG_ERR_ARG, "fft_lines: bad mode"};
    }
    MGG_CHECK_LAUNCH();
}

template <int N>
void lines_n(const FftPlan& p, float2* buf, int axis, int mode, const LineExtra& ex, cudaStream_t s) {
    if (p.tw64) lines_c<N>(p, p.tw64, buf, axis, mode, ex, s);   // FP64 line arithmetic
    else lines_c<N>(p, p.tw, buf, axis, mode, ex, s);
}

}  // namespace

void fft_set_attributes() {
#define MGG_F(N) set_attrs_n<N, float2>(); set_attrs_n<N, double2>();
    MGG_FFT_SIZES(MGG_F)
#undef MGG_F
}

#define MGG_FFT_SWITCH(n, CALL)                                              \
    switch (n) {                                                             \
    case 16: CALL(16); break;                                                \
    case 32: CALL(32); break;                                                \
    case 64: CALL(64); break;                                                \
    case 128: CALL(128); break;                                              \
    case 256: CALL(256); break;                                              \
    case 512: CALL(512); break;                                              \
    case 1024: CALL(1024); break;                                            \
    default: throw Error{MGG_ERR_ARG, "fft: NGRID must be a power of two in [16, 1024]"}; \
    }

void fft_x_r2c(const FftPlan& p, const float* in, float2* out, cudaStream_t s) {
#define MGG_C(N) x_r2c_n<N>(p, in, out, s)
    MGG_FFT_SWITCH(p.n, MGG_C)
#undef MGG_C
}

void fft_x_c2r(const FftPlan& p, const float2* in, float* out, cudaStream_t s) {
#define MGG_C(N) x_c2r_n<N>(p, in, out, s)
    MGG_FFT_SWITCH(p.n, MGG_C)
#undef MGG_C
}

void fft_lines(const FftPlan& p, float2* buf, int axis, int mode, const LineExtra& ex, cudaStream_t s) {
#define MGG_C(N) lines_n<N>(p, buf, axis, mode, ex, s)
    MGG_FFT_SWITCH(p.n, MGG_C)
#undef MGG_C
}

// ------------------------------------------------------------- context ----
int fft_pitch(int N) { return ((N / 2 + 1) + 15) / 16 * 16; }

float2* make_twiddles(int N) {
    std::vector<float2> tw(N);
    for (int k = 0; k < N; ++k) {
        const double a = -2.0 * M_PI * (double)k / (double)N;
        tw[k] = make_float2((float)cos(a), (float)sin(a));
    }
    float2* d = nullptr;
    MGG_CUDA(cudaMalloc(&d, sizeof(float2) * N));
    MGG_CUDA(cudaMemcpy(d, tw.data(), sizeof(float2) * N, cudaMemcpyHostToDevice));
    return d;
}

double2* make_twiddles64(int N) {
    std::vector<double2> tw(N);
    for (int k = 0; k < N; ++k) {
        const double a = -2.0 * M_PI * (double)k / (double)N;
        tw[k] = make_double2(cos(a), sin(a));
    }
    double2* d = nullptr;
    MGG_CUDA(cudaMalloc(&d, sizeof(double2) * N));
    MGG_CUDA(cudaMemcpy(d, tw.data(), sizeof(double2) * N, cudaMemcpyHostToDevice));
    return d;
}

// Bins per integer |k|^2 with the reference's Real*4 arithmetic: linear
// MP = max(INT(RK + 0.5), 1), log MPlog = max(1, min(NPOWER, INT(Log10(RK)/dLog +
// 1000.) - 1000)) (PMP2mod_power.f90:396), and the distinct pairs of them (few, since
// both grow with |k|): pair index per |k|^2, then (linear, log) per pair.
struct BinTable {
    std::vector<uint16_t> table;
    int npair = 0;
    int lin(int m2) const { return table[m2bins + 2 * table[m2]]; }
    int log(int m2) const { return table[m2bins + 2 * table[m2] + 1]; }
    int m2bins = 0;
};
static BinTable bin_table(int N) {
    const int m2max = 3 * (N / 2) * (N / 2);
    BinTable b;
    b.m2bins = bin_table_m2(N);
    b.table.assign(b.m2bins, 0);
    std::vector<uint16_t> pairs;
    int last = -1;
    for (int m2 = 1; m2 <= m2max; ++m2) {
        const float RK = sqrtf((float)m2);
        int mp = (int)(RK + 0.5f);
        mp = mp < 1 ? 1 : mp;
        int ml = (int)(log10f(RK) / 0.02f + 1000.0f) - 1000;
        ml = ml < 1 ? 1 : (ml > N ? N : ml);
        if (ml > 255) ml = 255;
        if (last < 0 || pairs[2 * last] != mp || pairs[2 * last + 1] != ml) {
            pairs.push_back((uint16_t)mp);
            pairs.push_back((uint16_t)ml);
            ++last;
        }
        b.table[m2] = (uint16_t)last;
    }
    b.npair = last + 1;
    b.table.insert(b.table.end(), pairs.begin(), pairs.end());
    return b;
}

uint16_t* make_bins(int N) {
    const BinTable b = bin_table(N);
    uint16_t* d = nullptr;
    MGG_CUDA(cudaMalloc(&d, sizeof(uint16_t) * b.table.size()));
    MGG_CUDA(cudaMemcpy(d, b.table.data(), sizeof(uint16_t) * b.table.size(), cudaMemcpyHostToDevice));
    return d;
}

void fft_alloc(Ctx& c) {
    const int N = c.N;
    c.nxp = fft_pitch(N);
    MGG_CUDA(cudaMalloc(&c.cbuf, sizeof(float2) * (size_t)c.nxp * N * N));
    c.tw_n = make_twiddles(N);
    c.tw64_n = make_twiddles64(N);
    // GREENf of PMP2main.f90:736-742 mapped to the complex index k (m = min(k, N-k)),
    // with the reference's 2*pi constant P16 = 6.28318530718
    const double P16 = 6.28318530718;
    std::vector<double> g(N);
    for (int k = 0; k < N; ++k) {
        const int m = k <= N / 2 ? k : N - k;
        if (m == 0) g[k] = 2.0;
        else if (m == N / 2) g[k] = -2.0;
        else g[k] = 2.0 * cos(P16 * m / N);
    }
    MGG_CUDA(cudaMalloc(&c.green, sizeof(double) * N));
    MGG_CUDA(cudaMemcpy(c.green, g.data(), sizeof(double) * N, cudaMemcpyHostToDevice));
    c.pk_bins = make_bins(N);
    MGG_CUDA(cudaMalloc(&c.pk_hist, sizeof(unsigned long long) * 3 * (N + 1)));
    fft_set_attributes();
}

void poisson_solve(Ctx& c) {
    BucketScope bs(c, MGG_T_FORCE);
    const int N = c.N;
    FftPlan p;
    p.n = N;
    p.nxp = c.nxp;
    p.tw = c.tw_n;
    if (c.cfg.precision == MGG_PREC_PLAIN) p.tw64 = c.tw64_n;   // FP64 lines, as FFTPACK5
    const double cells = (double)c.ncell;
    const double cplx = 8.0 * (double)N * N * (N / 2 + 1);
    // trfi (PMP2main.f90:728-732), Real*4
    float trfi;
    if (c.cfg.omb < 0.005f) trfi = 1.5f * (c.cfg.om - c.cfg.omb) / c.aexpn;
    else trfi = 1.5f * c.cfg.om / c.aexpn;
    LineExtra ex;
    ex.green = c.green;
    ex.green_scale = (double)trfi * 2.0 / (cells);
    {
        ProfScope ps(c, K_FFT_X_R2C, 4.0 * cells + cplx);
        fft_x_r2c(p, c.fi, c.cbuf, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_Y, 2.0 * cplx);
        fft_lines(p, c.cbuf, 1, LM_FWD, ex, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_Z_GREEN, 2.0 * cplx);
        fft_lines(p, c.cbuf, 2, LM_GREEN, ex, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_Y, 2.0 * cplx);
        fft_lines(p, c.cbuf, 1, LM_INV, ex, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_X_C2R, 4.0 * cells + cplx);
        fft_x_c2r(p, c.cbuf, c.fi, c.stream);
    }
}

namespace {
__global__ void k_sumsq(const float* __restrict__ f, int64_t n, double* __restrict__ part) {
    double v = 0.0;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const double a = f[q];
        v += a * a;
    }
    v = block_sum_fixed(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}
}  // namespace

// Mode counts per integer |k|^2 over the full N^3 spectrum (each axis index
// m in [0, N/2] stands for 1 (m = 0, N/2) or 2 halfcomplex entries), the
// reference's iVolume/dk sums (PMP2mod_power.f90:406-409), computed once.
static void mode_counts(int N, std::vector<double>& cnt) {
    const int h = N / 2;
    const int m2max = 3 * h * h;
    cnt.assign(m2max + 1, 0.0);
    for (int a = 0; a <= h; ++a) {
        const double ca = (a == 0 || a == h) ? 1.0 : 2.0;
        for (int b = 0; b <= h; ++b) {
            const double cb = (b == 0 || b == h) ? 1.0 : 2.0;
            const int ab = a * a + b * b;
            for (int d = 0; d <= h; ++d) {
                const double cd = (d == 0 || d == h) ? 1.0 : 2.0;
                cnt[ab + d * d] += ca * cb * cd;
            }
        }
    }
}

namespace {
// Mode counts and sums of |k| per linear and log bin: they depend on the mesh size alone
// (powers of two up to 1024), so they are formed once per size and process (2 ms of
// host time at 512^3, as much as the transform, when every call did).
struct BinCounts {
    std::vector<double> iV, dk, iVl, dkl;
    int npair = 0;   // of the bin table
};
const BinCounts& bin_counts(int N) {
    static std::mutex mu;
    static std::map<int, BinCounts> all;
    std::lock_guard<std::mutex> lk(mu);
    BinCounts& b = all[N];
    if (!b.iV.empty()) return b;
    std::vector<double> cnt;
    mode_counts(N, cnt);
    const BinTable bt = bin_table(N);
    BinCounts r;
    r.npair = bt.npair;
    for (auto* v : {&r.iV, &r.dk, &r.iVl, &r.dkl}) v->assign(N + 1, 0.0);
    for (size_t m2 = 1; m2 < cnt.size(); ++m2) {
        if (cnt[m2] == 0.0) continue;
        const float RK = sqrtf((float)m2);
        const int MP = bt.lin((int)m2), ML = bt.log((int)m2);
        r.iV[MP] += cnt[m2];
        r.dk[MP] += cnt[m2] * (double)RK;
        r.iVl[ML] += cnt[m2];
        r.dkl[ML] += cnt[m2] * (double)RK;
    }
    return b = std::move(r);
}
}  // namespace

void power_bins(Ctx& c, const float* grid, int N, const float2* tw, const double2* tw64, const uint16_t* bins,
                bool quad, PkBins& out) {
    const double cells = (double)N * N * N;
    // Parseval bound for the fixed-point scale: sum_k |delta_k|^2 = sum delta^2 / N^3
    const int blocks = 148 * 8;
    ensure_partials(c, blocks);
    {
        ProfScope ps(c, K_GRID_OP, 4.0 * cells);
        k_sumsq<<<blocks, 256, 0, c.stream>>>(grid, (int64_t)cells, c.red_partial);
        MGG_CHECK_LAUNCH();
    }
    const double s2 = reduce_sum_blocks(c, blocks);
    const double total = s2 / cells;   // >= any bin sum (and any |quadrupole bin sum|)
    double scale = 1.0;
    if (total > 0.0) {
        int e;
        frexp(total, &e);                    // total < 2^e
        scale = ldexp(1.0, 61 - e);          // sums stay below 2^61
    }
    FftPlan p;
    p.n = N;
    p.nxp = fft_pitch(N);
    p.tw = tw;
    p.tw64 = tw64;
    LineExtra ex;
    const BinCounts& bc = bin_counts(N);   // exact, data independent
    ex.bins = bins;
    ex.npair = bc.npair;
    ex.hist = c.pk_hist;
    ex.amp_scale = scale / (cells * cells);
    ex.quad = quad ? 1 : 0;
    const int nh = 3 * (N + 1);
    MGG_CUDA(cudaMemsetAsync(c.pk_hist, 0, sizeof(unsigned long long) * nh, c.stream));
    const double cplx = 8.0 * (double)N * N * (N / 2 + 1);
    {
        ProfScope ps(c, K_FFT_X_R2C, 4.0 * cells + cplx);
        fft_x_r2c(p, grid, c.cbuf, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_Y, 2.0 * cplx);
        fft_lines(p, c.cbuf, 1, LM_FWD, ex, c.stream);
    }
    {
        ProfScope ps(c, K_FFT_Z_POWER, cplx);
        fft_lines(p, c.cbuf, 2, LM_POWER, ex, c.stream);
    }
    std::vector<unsigned long long> h(nh);
    MGG_CUDA(cudaMemcpyAsync(h.data(), c.pk_hist, sizeof(unsigned long long) * nh, cudaMemcpyDeviceToHost, c.stream));
    MGG_CUDA(cudaStreamSynchronize(c.stream));
    const std::vector<double>&iV = bc.iV, &dk = bc.dk, &iVl = bc.iVl, &dkl = bc.dkl;
    const float Pi = 3.141592653f;
    const float Scale = 2.0f * Pi / c.cfg.box;
    const float b3 = c.cfg.box * c.cfg.box * c.cfg.box;
    const double unfix = 1.0 / scale;
    const int nb = N / 2;
    for (auto* v : {&out.k, &out.n, &out.p, &out.kl, &out.nl, &out.pl, &out.q}) v->assign(nb + 1, 0.0);
    for (int I = 1; I <= nb; ++I) {
        if (iV[I] > 0) {
            out.k[I] = (float)(dk[I] / iV[I] * (double)Scale);
            out.n[I] = (float)iV[I];
            out.p[I] = (float)((double)b3 * ((double)h[I] * unfix) / iV[I]);
            // iPol = 1: DPOWER = 2.5 DPOWER ((2L+1)/2, PMP2mod_power.f90:420)
            if (quad) out.q[I] = (float)((double)b3 * (2.5 * ((double)(int64_t)h[2 * (N + 1) + I] * unfix)) / iV[I]);
        }
        if (iVl[I] > 0) {
            out.kl[I] = (float)(dkl[I] / iVl[I] * (double)Scale);
            out.nl[I] = (float)iVl[I];
            out.pl[I] = (float)((double)b3 * ((double)h[(N + 1) + I] * unfix) / iVl[I]);
        }
    }
}

void power_spectrum(Ctx& c, int nbins, double* k_out, double* n_out, double* p_out, double* kl_out,
                    double* nl_out, double* pl_out) {
    BucketScope bs(c, MGG_T_POWER);
    PkBins b;
    power_bins(c, c.fi, c.N, c.tw_n, c.cfg.precision == MGG_PREC_PLAIN ? c.tw64_n : nullptr, c.pk_bins, false, b);
    for (int I = 1; I <= nbins && I <= c.N / 2; ++I) {
        if (k_out) k_out[I - 1] = b.k[I];
        if (n_out) n_out[I - 1] = b.n[I];
        if (p_out) p_out[I - 1] = b.p[I];
        if (kl_out) kl_out[I - 1] = b.kl[I];
        if (nl_out) nl_out[I - 1] = b.nl[I];
        if (pl_out) pl_out[I - 1] = b.pl[I];
    }
}

}  // namespace mgg
