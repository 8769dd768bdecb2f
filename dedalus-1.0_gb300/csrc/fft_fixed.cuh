// FP64 pencil transforms on the integer pipes.
//
// GB300 issues 2 FP64 operations per clock and SM against 64 integer
// multiply-adds (32 x 32 + 64 bits) and 64 to 128 integer additions, and
// its FP64 <-> integer conversion instructions run at the FP64 rate too.  A
// transform is linear and its growth is known, so a pencil of doubles is
// transformed as block fixed point: one power-of-two scale per pencil, 64-bit
// integer values, FP64 bit patterns taken apart and put together with integer
// instructions.  Additions are exact; a twiddle product rounds once.
//
// Scale.  m = largest |re|, |im| of the pencil, read off the high words.  The
// first pass (radix R1) is bounded by R1 sqrt(2) m, and the scale is the
// power of two that puts this bound at 2^62.  Every later pass looks at the
// largest value that the pass before it wrote and divides (or multiplies) by
// the power of two that keeps its own bound at 2^62; the twiddle product's
// final shift does the division.  So the words stay filled whether the pencil
// is a few large modes or noise, the rounding errors of the earlier passes
// shrink with each division, and the result, rounded to FP64 once at the end,
// is closer to the exact transform than an FP64 FFT's.
//
// Conversions.  On the way in, real parts go through the conversion instruction
// (FP64 pipe) and imaginary parts are taken apart with integer instructions, so
// that both pipes work; on the way out everything is integer.
//
// Values below 2^-62 of the bound vanish, as they do in an FP64 sum with the
// larger ones.  A pencil whose largest value is outside 2^-895 .. 2^49, subnormal
// ones included, is scaled by 2^512 or 2^-975 on the way in and back on the way out.
// One that holds a NaN or an infinity gives NaN everywhere.
#pragma once
#include <type_traits>

#include "fft_engine.cuh"

namespace dd {

typedef long long fx;      // one fixed-point value

// --------------------------------------------------- scales
// 1 - largest |x| high word of a pencil (0 = zeros and subnormals) to its bound: every
// component is below 2^(e2 - 1022.5), a pair's modulus below 2^(e2 - 1022).
// rare: 0, or 1 (times 2^512 on the way in), 2 (times 2^-975), 3 (not finite).
struct FxScale {
    int e2, rare;
};

__host__ __device__ __forceinline__ FxScale fx_scale(unsigned m) {
    FxScale s;
    // exponent of sqrt(2) (m + 1): carries where the 20 mantissa bits exceed sqrt(2) - 1
    s.e2 = (int)((m + 614242u) >> 20);
    s.rare = 0;
    if (m >= 0x7ff00000u) { s.rare = 3; s.e2 = 1023; }
    else if (s.e2 < 128) { s.rare = 1; s.e2 = (s.e2 > 1 ? s.e2 : 1) + 512; }
    else if (s.e2 > 1072) { s.rare = 2; s.e2 -= 975; }
    return s;
}
__host__ __device__ __forceinline__ double fx_pre(int rare) {
    return rare == 1 ? 0x1p512 : rare == 2 ? 0x1p-975 : 1.0;
}
__device__ __forceinline__ double fx_post(int rare) {
    return rare == 1 ? 0x1p-512 : rare == 2 ? 0x1p975 : __longlong_as_double(0x7ff8000000000000ll);
}

// v[i] *= f behind a branch: FP64 instructions take 64 clocks of their pipe
// per warp even where a predicate turns them off, and a branch around each
// single one becomes such a predicate.  Zeros skip it: pencils of zeros are
// among the pre-scaled ones.
template <int N>
__device__ __forceinline__ void fx_scale_all(C<double>* v, double f) {
    unsigned nz = 0;
#pragma unroll
    for (int i = 0; i < N; i++)
        nz |= (unsigned)__double2hiint(v[i].x) | (unsigned)__double2loint(v[i].x) | (unsigned)__double2hiint(v[i].y) |
              (unsigned)__double2loint(v[i].y);
    if (nz == 0u) return;
#pragma unroll
    for (int i = 0; i < N; i++) { v[i].x *= f; v[i].y *= f; }
}

// --------------------------------------------------- conversions
__device__ __forceinline__ unsigned fx_absword(double x) { return (unsigned)__double2hiint(x) << 1; }
__device__ __forceinline__ unsigned fx_max(unsigned h, C<double> v) {   // words shifted left by one: no mask for the sign
    return max(h, max(fx_absword(v.x), fx_absword(v.y)));
}

// x times 2^(1085 - K), for |x| below that scale's 2^62 (K - the biased
// exponent of x is at least 2, and K <= 1085).  fx_in takes the bit pattern
// apart (truncating), fx_in64 adds to the exponent and converts (rounding).
__device__ __forceinline__ fx fx_in(double x, int K) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int k = min(K - (int)((hi << 1) >> 21), 63);
    const unsigned mh = (hi & 0xfffffu) | 0x100000u;
    const unsigned H = __funnelshift_l(lo, mh, 10), L = lo << 10;     // mantissa in bits 62 .. 10
    const unsigned rl = __funnelshift_rc(__funnelshift_rc(L, H, k), 0u, max(k - 32, 0));
    const unsigned rh = __funnelshift_rc(H, 0u, k);
    const fx v = (fx)(((unsigned long long)rh << 32) | rl);
    return (int)hi < 0 ? -v : v;
}
__device__ __forceinline__ fx fx_in64(double x, int K) {
    return __double2ll_rn(__hiloint2double(__double2hiint(x) + ((1085 - K) << 20), __double2loint(x)));
}
__device__ __forceinline__ C<fx> fx_in(C<double> v, int K) { return mk<fx>(fx_in64(v.x, K), fx_in(v.y, K)); }

// The double nearest to x 2^(eb - 1085): x in sign and magnitude, normalised,
// the exponent added to the high word (the leading one adds the last 1 of it).
// (The two FP64 additions that would join the words as mantissas of two doubles
// take longer than these instructions in the x pass and as long elsewhere.)
__device__ __forceinline__ double fx_out(fx x, int eb) {
    const int sgn = (int)(x >> 32);
    const unsigned long long a = (unsigned long long)(sgn < 0 ? -x : x);
    const unsigned hi = (unsigned)(a >> 32), lo = (unsigned)a;
    int n = __clz((int)hi);
    unsigned H = __funnelshift_lc(lo, hi, n), L = __funnelshift_lc(0u, lo, n);
    if (n == 32) {                             // below 2^32
        const int n2 = __clz((int)H);
        if (n2 == 32) return 0.0;
        H <<= n2;
        n += n2;
    }
    const unsigned long long r = (((unsigned long long)H << 32) | L) >> 11;
    const unsigned long long v = r + ((L >> 10) & 1u) + ((unsigned long long)(unsigned)((eb - n) << 20) << 32);
    return __hiloint2double((int)((unsigned)(v >> 32) | ((unsigned)sgn & 0x80000000u)), (int)(unsigned)v);
}
__device__ __forceinline__ C<double> fx_out(C<fx> v, int eb) { return mk<double>(fx_out(v.x, eb), fx_out(v.y, eb)); }

// --------------------------------------------------- products
__device__ __forceinline__ fx fx_mad(int a, int b, fx c) { return (fx)a * b + c; }

struct FxHL {
    int h, l;              // value = h 2^32 + l, both signed
};
__device__ __forceinline__ FxHL fx_split(fx a) {
    FxHL s;
    s.l = (int)a;
    s.h = (int)(a >> 32) + (int)((unsigned)s.l >> 31);
    return s;
}

__device__ __forceinline__ fx fx_shr(fx a, int n) {       // 0 <= n < 32
    const unsigned lo = (unsigned)a;
    const int hi = (int)(a >> 32);
    return (fx)(((unsigned long long)(unsigned)(hi >> n) << 32) | __funnelshift_r(lo, (unsigned)hi, n));
}
__device__ __forceinline__ fx fx_shl(fx a, int n) {       // 0 <= n < 32
    const unsigned lo = (unsigned)a, hi = (unsigned)(a >> 32);
    return (fx)(((unsigned long long)__funnelshift_l(lo, hi, n) << 32) | (lo << n));
}

// a (c + i s) / 2^(2 + n) for a twiddle c + i s = (w.x 2^32 + w.y + i (w.z 2^32 + w.w)) 2^-62
// (signed halves), half = 2^(31 + n): rounded to nearest up to the product of
// the low halves (below one unit before the division).  |a| < 2^62, n <= 1.
__device__ __forceinline__ C<fx> fx_twiddle(C<fx> a, int4 w, int n, fx half) {
    const FxHL x = fx_split(a.x), y = fx_split(a.y);
    fx re = fx_mad(x.h, w.y, half), im = fx_mad(x.h, w.w, half);
    re = fx_mad(x.l, w.x, re);
    im = fx_mad(x.l, w.z, im);
    re = fx_mad(y.h, -w.w, re);
    im = fx_mad(y.h, w.y, im);
    re = fx_mad(y.l, -w.z, re) >> 32;
    im = fx_mad(y.l, w.x, im) >> 32;
    re = fx_mad(x.h, w.x, re);
    im = fx_mad(x.h, w.z, im);
    re = fx_mad(y.h, -w.z, re);
    im = fx_mad(y.h, w.x, im);
    return mk<fx>(fx_shr(re, n), fx_shr(im, n));
}

// a times the constant (CH 2^32 + CL) 2^-63, rounded to nearest; |a| < 2^62.
__device__ __forceinline__ fx fx_mul63(fx a, int ch, int cl) {
    const FxHL x = fx_split(a);
    const fx t = fx_mad(x.l, ch, fx_mad(x.h, cl, 1ll << 30)) >> 31;
    return fx_mad(2 * x.h, ch, t);
}

// sqrt(1/2) and sqrt(3)/2 in units of 2^-63
#define DD_FX_R2H 1518500250
#define DD_FX_R2L (-51432894)
#define DD_FX_S3H 1859775393
#define DD_FX_S3L 1630710223

// a W_8^M (forward) or its conjugate (inverse), M = 1 or 3; |a| < 2^61.
template <int M, bool INV>
__device__ __forceinline__ C<fx> fx_rot8(C<fx> a) {
    static_assert(M == 1 || M == 3, "rotations of the radix-8 butterfly");
    if constexpr (M == 1) {                    // (1 -+ i) / sqrt 2
        const fx p = fx_mul63(a.x + a.y, DD_FX_R2H, DD_FX_R2L), d = fx_mul63(a.y - a.x, DD_FX_R2H, DD_FX_R2L);
        return INV ? mk<fx>(-d, p) : mk<fx>(p, d);
    } else {                                   // (-1 -+ i) / sqrt 2
        const fx p = fx_mul63(a.x + a.y, DD_FX_R2H, DD_FX_R2L), d = fx_mul63(a.y - a.x, DD_FX_R2H, DD_FX_R2L);
        return INV ? mk<fx>(-p, -d) : mk<fx>(d, -p);
    }
}

// --------------------------------------------------- in-register DFTs
template <int R, bool INV>
__device__ __forceinline__ void fx_dft(C<fx>* v) {
    if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        C<fx> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        C<fx> o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        dft4<INV>(e0, e1, e2, e3);
        dft4<INV>(o0, o1, o2, o3);
        o1 = fx_rot8<1, INV>(o1);
        o2 = mul_mi<INV>(o2);
        o3 = fx_rot8<3, INV>(o3);
        v[0] = e0 + o0; v[4] = e0 - o0;
        v[1] = e1 + o1; v[5] = e1 - o1;
        v[2] = e2 + o2; v[6] = e2 - o2;
        v[3] = e3 + o3; v[7] = e3 - o3;
    } else {
        static_assert(R == 3, "unsupported radix");
        const C<fx> t1 = v[1] + v[2], r = mul_mi<INV>(v[1] - v[2]);
        const C<fx> m1 = mk<fx>(v[0].x - ((t1.x + 1) >> 1), v[0].y - ((t1.y + 1) >> 1));
        const C<fx> m2 = mk<fx>(fx_mul63(r.x, DD_FX_S3H, DD_FX_S3L), fx_mul63(r.y, DD_FX_S3H, DD_FX_S3L));
        v[0] = v[0] + t1;
        v[1] = m1 + m2;
        v[2] = m1 - m2;
    }
}

// --------------------------------------------------- pencils
// Default schedules: P pencils of TPP threads, radices, and MB resident blocks
// per SM (__launch_bounds__).  Radix 8 and 4 passes of one butterfly per thread
// need 64 registers, so that 1024 threads fit an SM: at 256 points the y passes
// of a 256^3 step took 248 / 150 us (forward / inverse) against 281 / 178 us for
// two radix-16 passes (116 registers, 512 threads).  8-pencil tiles keep global
// accesses at 128 bytes; 4 pencils took 327 / 182 us.  Wider tiles are padded more
// where a row keeps few modes: with 8 pencils for 16 the y passes of 6 fields of
// 128^3 (43 modes) take 43.5 / 42.1 us against 46.2 / 45.1, with 8 for 32 those of
// 64^3 (22 modes) 8.6 / 8.5 us against 10.7 / 10.6, and with 16 for 64 those of 32^3
// (11 modes) 6.3 / 6.5 us against 8.4 / 8.5.  Forward schedules end
// with radix 8, whose outputs in the removed band are skipped, inverse ones begin
// with it.
template <int L> struct FxCfg;
template <> struct FxCfg<8>   { static constexpr int P = 64, TPP = 1,  MB = 8, R[3] = {8, 1, 1}, RF[3] = {8, 1, 1}; };
template <> struct FxCfg<16>  { static constexpr int P = 64, TPP = 4,  MB = 4, R[3] = {4, 4, 1}, RF[3] = {4, 4, 1}; };
template <> struct FxCfg<24>  { static constexpr int P = 64, TPP = 4,  MB = 4, R[3] = {8, 3, 1}, RF[3] = {8, 3, 1}; };
template <> struct FxCfg<32>  { static constexpr int P = 16, TPP = 4,  MB = 16, R[3] = {8, 4, 1}, RF[3] = {4, 8, 1}; };
template <> struct FxCfg<48>  { static constexpr int P = 16, TPP = 16, MB = 4, R[3] = {4, 4, 3}, RF[3] = {4, 4, 3}; };
template <> struct FxCfg<64>  { static constexpr int P = 8,  TPP = 8,  MB = 14, R[3] = {8, 8, 1}, RF[3] = {8, 8, 1}; };
template <> struct FxCfg<96>  { static constexpr int P = 16, TPP = 12, MB = 5, R[3] = {8, 4, 3}, RF[3] = {8, 4, 3}; };
template <> struct FxCfg<128> { static constexpr int P = 8,  TPP = 16, MB = 7, R[3] = {8, 4, 4}, RF[3] = {4, 4, 8}; };
template <> struct FxCfg<192> { static constexpr int P = 8,  TPP = 24, MB = 5, R[3] = {8, 8, 3}, RF[3] = {8, 8, 3}; };
template <> struct FxCfg<256> { static constexpr int P = 8,  TPP = 32, MB = 4, R[3] = {8, 8, 4}, RF[3] = {8, 4, 8}; };
template <> struct FxCfg<512> { static constexpr int P = 8,  TPP = 64, MB = 2, R[3] = {8, 8, 8}, RF[3] = {8, 8, 8}; };

template <int L, bool INV, int P = FxCfg<L>::P, class CC = FxCfg<L>>
using FxS = Sched<L, P, P * CC::TPP, INV ? CC::R[0] : CC::RF[0], INV ? CC::R[1] : CC::RF[1], INV ? CC::R[2] : CC::RF[2]>;

// Bits of growth of a pass: log2 R, and 2 for R = 3.
constexpr int fx_bits(int R) { return R == 8 ? 3 : 2; }

// Radix-R butterflies per thread of a pencil's TPP threads: j = jt + b TPP for
// those with fx_has.
template <class S, int R>
constexpr int fx_bpt() { return (S::L / R + S::TPP - 1) / S::TPP; }
template <class S, int R>
__device__ __forceinline__ bool fx_has(int b, int jt) {
    constexpr int NB = S::L / R;
    return NB % S::TPP == 0 || jt + b * S::TPP < NB;
}

// Tile offset of row base + r STEP for a compile-time r: off() is additive where
// STEP or (BASE8) base is a multiple of 8 rows, so that the constant part folds
// into the access.
template <class S, int STEP, bool BASE8 = false>
__device__ __forceinline__ int fx_row(int base, int r) {
    if constexpr (S::SKD == 0 || STEP % 8 == 0 || BASE8) return S::off(base) + S::off(r * STEP);
    else return S::off(base + r * STEP);
}

// K of fx_in for a pencil of bound e2 (packed: of sums of two such values).
template <class S>
__host__ __device__ constexpr int fx_kin(int e2, bool packed) {
    static_assert(S::R1 == 4 || S::R1 == 8, "first radix");
    return e2 + 1 + fx_bits(S::R1) + (packed ? 1 : 0);
}

// Scaling of a later pass of radix R from the largest high word h (or ~h) of
// its inputs: times 2^l (l >= 0) and 2^-(2 + n), net 2^-d, so that the bound
// R sqrt(2) (h + 1) 2^32 comes to at most 2^62.
struct FxStep {
    int l, n, d;
};
template <int R>
__device__ __forceinline__ FxStep fx_step(int h) {
    const unsigned m = (unsigned)h + 1u + (((unsigned)h + 1u) >> 1);
    const int d = min(32 - __clz((int)m) + fx_bits(R) - 30, fx_bits(R));
    FxStep s;
    s.l = max(2 - d, 0);
    s.n = max(d - 2, 0);
    s.d = d;
    return s;
}

// Shared words per pencil: the largest doubled high word of its input, and the
// largest high words after the first and the second pass.
constexpr int FX_WORDS = 3;

// Stage the twiddle table (cos, sin of 2 pi m / L as 2^-62 (h 2^32 + l) pairs)
// with the sign of one direction, and clear the n pencil maxima.
template <int L, bool INV>
__device__ __forceinline__ void fx_stage_twiddles(int4* s_tw, const int4* g_tw) {
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        int4 w = g_tw[i];
        if (!INV) { w.z = -w.z; w.w = -w.w; }
        s_tw[i] = w;
    }
}

// Where pencil_fx takes its input from and leaves its output.
enum FxIn { FX_IN_GLOBAL, FX_IN_TILE };                  // ld(e); the tile
enum FxOut { FX_OUT_GLOBAL, FX_OUT_TILE, FX_OUT_FIXED }; // st(e, value); the tile: doubles; the tile: fixed point

// Scaling, twiddles and DFTs of a later pass.
template <int R, int NS, int STEP, bool INV, int TPP, int BPT>
__device__ __forceinline__ void fx_twiddles(C<fx> (&v)[BPT][R], const int4* tw, int jt, FxStep st) {
    const fx half = (fx)(1ull << 31) << st.n;
#pragma unroll
    for (int b = 0; b < BPT; b++) {
        const int k = (jt + TPP * b) & (NS - 1);
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[b][r] = mk<fx>(fx_shl(v[b][r].x, st.l), fx_shl(v[b][r].y, st.l));
            if (r > 0) v[b][r] = fx_twiddle(v[b][r], tw[(r * k) * STEP], st.n, half);
            else v[b][r] = mk<fx>(fx_shr(v[b][r].x + (2 << st.n), st.n + 2), fx_shr(v[b][r].y + (2 << st.n), st.n + 2));
        }
        fx_dft<R, INV>(v[b]);
    }
}

// One later pass of radix R after NS: read, (barrier), scale, twiddle and DFT;
// the results stay in v.  Adds the net division to eb.
template <class S, int R, int NS, bool INV, bool SYNC>
__device__ __forceinline__ void fx_later_pass(C<fx> (&v)[fx_bpt<S, R>()][R], const C<fx>* tile, const int4* tw, int p,
                                              int jt, const int* hmax, int& eb) {
    constexpr int NB = S::L / R, BPT = fx_bpt<S, R>(), STEP = S::L / (NS * R);
#pragma unroll
    for (int b = 0; b < BPT; b++)
#pragma unroll
        for (int r = 0; r < R; r++)
            v[b][r] = fx_has<S, R>(b, jt) ? tile[fx_row<S, NB>(jt + S::TPP * b, r) + p] : mk<fx>(0, 0);
    const FxStep st = fx_step<R>(hmax[p]);
    if (SYNC) __syncthreads();
    eb += st.d;
    fx_twiddles<R, NS, STEP, INV, S::TPP, BPT>(v, tw, jt, st);
}

// Index of output r of butterfly j of a pass of radix R after NS.
template <int R, int NS>
__device__ __forceinline__ int fx_dest(int j) {
    const int k = j & (NS - 1);
    return (j - k) * R + k;
}

template <class S, int R, int NS>
__device__ __forceinline__ void fx_write(C<fx>* tile, const C<fx> (&v)[fx_bpt<S, R>()][R], int p, int jt, unsigned zout,
                                         int* hmax) {
    int hi = 0, lo = 0;
#pragma unroll
    for (int b = 0; b < fx_bpt<S, R>(); b++) {
        if (!fx_has<S, R>(b, jt)) continue;
        const int d = fx_dest<R, NS>(jt + S::TPP * b);
#pragma unroll
        for (int r = 0; r < R; r++)
            if (!((zout >> r) & 1u)) {
                tile[fx_row<S, NS, NS == 1 && R % 8 == 0>(d, r) + p] = v[b][r];
                const int x = (int)(v[b][r].x >> 32), y = (int)(v[b][r].y >> 32);
                hi = max(hi, max(x, y));
                lo = min(lo, min(x, y));
            }
    }
    if (hmax) atomicMax(hmax + p, max(hi, ~lo));
}

// The last pass's results: to st or the tile as doubles, or to the tile as they are.
template <class S, int R, int NS, FxOut OUT, unsigned ZOUT, class St>
__device__ __forceinline__ void fx_finish(C<double>* tile, const C<fx> (&v)[fx_bpt<S, R>()][R], int p, int jt,
                                          FxScale sc, int eb, St st) {
    if constexpr (OUT == FX_OUT_FIXED) {
        fx_write<S, R, NS>(reinterpret_cast<C<fx>*>(tile), v, p, jt, ZOUT, nullptr);
    } else {
        constexpr int BPT = fx_bpt<S, R>();
        C<double> o[BPT][R];
#pragma unroll
        for (int b = 0; b < BPT; b++)
#pragma unroll
            for (int r = 0; r < R; r++)
                o[b][r] = ((ZOUT >> r) & 1u) ? mk<double>(0., 0.) : fx_out(v[b][r], eb);
        if (sc.rare) fx_scale_all<BPT * R>(&o[0][0], fx_post(sc.rare));
#pragma unroll
        for (int b = 0; b < BPT; b++) {
            if (!fx_has<S, R>(b, jt)) continue;
            const int d = fx_dest<R, NS>(jt + S::TPP * b);
#pragma unroll
            for (int r = 0; r < R; r++) {
                if constexpr (OUT == FX_OUT_TILE) { if (!((ZOUT >> r) & 1u)) tile[fx_row<S, NS, NS == 1 && R % 8 == 0>(d, r) + p] = o[b][r]; }
                else st(d + r * NS, o[b][r]);
            }
        }
    }
}

// Transform S::P pencils (thread: pencil p, butterflies jt + b TPP).  smax:
// FX_WORDS arrays of P shared words, zero on entry (the first may hold a high word already).  The caller synchronises
// before, except that FX_IN_GLOBAL does so itself once its loads are issued
// (staged twiddles and cleared maxima become visible there); FX_OUT_TILE returns
// synchronised.  PRUNE as in pencil_fft_s: inputs of the removed band are taken
// as zero, outputs in it are not computed (st gets zeros).
template <class S, bool INV, bool PRUNE, FxIn IN, FxOut OUT, class Ld, class St>
__device__ __forceinline__ void pencil_fx(C<double>* tile, const int4* tw, unsigned* smax, Ld ld, St st) {
    constexpr int L = S::L, R1 = S::R1, NB1 = L / R1, BPT1 = fx_bpt<S, R1>();
    constexpr int NPASS = S::R3 > 1 ? 3 : S::R2 > 1 ? 2 : 1;
    constexpr int RL = NPASS == 3 ? S::R3 : S::R2;
    constexpr unsigned ZI = (PRUNE && INV && NPASS > 1) ? band_mask<L, R1>() : 0u;
    constexpr unsigned ZO = (PRUNE && !INV && NPASS > 1) ? band_mask<L, RL>() : 0u;
    const int p = threadIdx.x % S::P, jt = threadIdx.x / S::P;
    C<fx>* ft = reinterpret_cast<C<fx>*>(tile);
    C<fx> v[BPT1][R1];
    FxScale sc;
    {
        C<double> d[BPT1][R1];
#pragma unroll
        for (int b = 0; b < BPT1; b++)
#pragma unroll
            for (int r = 0; r < R1; r++) {
                if (((ZI >> r) & 1u) || !fx_has<S, R1>(b, jt)) d[b][r] = mk<double>(0., 0.);
                else if constexpr (IN == FX_IN_GLOBAL) d[b][r] = ld(jt + S::TPP * b + r * NB1);
                else d[b][r] = tile[fx_row<S, NB1>(jt + S::TPP * b, r) + p];
            }
        if (IN == FX_IN_GLOBAL) __syncthreads();
        unsigned h = 0;
#pragma unroll
        for (int b = 0; b < BPT1; b++)
#pragma unroll
            for (int r = 0; r < R1; r++)
                if (!((ZI >> r) & 1u)) h = fx_max(h, d[b][r]);
        atomicMax(smax + p, h);
        __syncthreads();
        sc = fx_scale(smax[p] >> 1);
        if (sc.rare) fx_scale_all<BPT1 * R1>(&d[0][0], fx_pre(sc.rare));
        const int K = fx_kin<S>(sc.e2, false);
#pragma unroll
        for (int b = 0; b < BPT1; b++)
#pragma unroll
            for (int r = 0; r < R1; r++) v[b][r] = ((ZI >> r) & 1u) ? mk<fx>(0, 0) : fx_in(d[b][r], K);
    }
#pragma unroll
    for (int b = 0; b < BPT1; b++) fx_dft<R1, INV>(v[b]);
    int eb = fx_kin<S>(sc.e2, false);
    int* hm = reinterpret_cast<int*>(smax + S::P);
    constexpr bool TO_TILE = OUT != FX_OUT_GLOBAL;
    if constexpr (NPASS == 1) {
        fx_finish<S, R1, 1, OUT, 0u>(tile, v, p, jt, sc, eb, st);
    } else {
        fx_write<S, R1, 1>(ft, v, p, jt, 0u, hm);
        __syncthreads();
        constexpr bool LAST2 = NPASS == 2;
        C<fx> v2[fx_bpt<S, S::R2>()][S::R2];
        fx_later_pass<S, S::R2, R1, INV, !LAST2 || TO_TILE>(v2, ft, tw, p, jt, hm, eb);
        if constexpr (LAST2) {
            fx_finish<S, S::R2, R1, OUT, ZO>(tile, v2, p, jt, sc, eb, st);
        } else {
            fx_write<S, S::R2, R1>(ft, v2, p, jt, 0u, hm + S::P);
            __syncthreads();
            C<fx> v3[fx_bpt<S, S::R3>()][S::R3];
            fx_later_pass<S, S::R3, R1 * S::R2, INV, TO_TILE>(v3, ft, tw, p, jt, hm + S::P, eb);
            fx_finish<S, S::R3, R1 * S::R2, OUT, ZO>(tile, v3, p, jt, sc, eb, st);
        }
    }
    if (TO_TILE) __syncthreads();
}

// --------------------------------------------------- rows: one thread group per pencil
// The x passes' pencils are contiguous in memory, so a pencil can belong to one
// group of TPP threads (a warp at 256 points, part of one or two warps elsewhere)
// that loads, packs, transforms and stores it with no block barrier: consecutive
// threads of a group take consecutive rows of the tile.  Tile rows have an odd
// stride and a skew of one entry every 8 rows, which keeps row sequences of step 1
// and 8 free of bank conflicts.  (With the pencils spread over all warps, as in
// the y and z passes, the 256-point hydro pass waited at 12 block barriers: 3.6 of
// 12.5 stalled warps per issue, 783 us per launch of a 256^3 step.)
template <int L> struct FxRowTPP { static constexpr int v = L == 192 ? 32 : L == 96 ? 16 : FxCfg<L>::TPP; };
template <int L, bool INV, int P, class CC = FxCfg<L>>
using FxR = Sched<L, P, P * FxRowTPP<L>::v, INV ? CC::R[0] : CC::RF[0], INV ? CC::R[1] : CC::RF[1],
                  INV ? CC::R[2] : CC::RF[2], (P | 1), 1>;

// Shared words of a block of P groups of two warps (three reductions).  Such groups
// synchronise on the named barriers 1 to 15, one each.
template <class S>
constexpr int fx_group_words() {
    static_assert(S::TPP <= 32 || S::P <= 15, "more groups of two warps than named barriers");
    return S::TPP > 32 ? 6 * S::P : 0;
}

template <int TPP>
__device__ __forceinline__ unsigned fx_group_mask() {
    if constexpr (TPP >= 32) return 0xffffffffu;
    else return ((1u << TPP) - 1u) << (threadIdx.x & 31 & ~(TPP - 1));
}

template <int TPP>
__device__ __forceinline__ void fx_group_sync(int g) {
    static_assert(TPP == 64 || (TPP <= 32 && 32 % TPP == 0), "groups of part of a warp or of two warps");
    if constexpr (TPP == 64) asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory");
    else __syncwarp(fx_group_mask<TPP>());
}

// Largest v of the group, for every thread of it; red: two shared words of this
// use alone (groups of two warps).
template <int TPP>
__device__ __forceinline__ unsigned fx_group_max(unsigned v, int g, unsigned* red) {
    if constexpr (TPP >= 32) {
        v = __reduce_max_sync(0xffffffffu, v);
    } else {
#pragma unroll
        for (int o = TPP / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(fx_group_mask<TPP>(), v, o));
    }
    if constexpr (TPP == 64) {
        if ((threadIdx.x & 31) == 0) red[(threadIdx.x >> 5) & 1] = v;
        fx_group_sync<64>(g);
        v = max(red[0], red[1]);
    }
    return v;
}

// Write the results of a pass and return the group's largest high word (or its
// complement); the group synchronises.
template <class S, int R, int NS>
__device__ __forceinline__ int fx_group_write(C<fx>* tile, const C<fx> (&v)[fx_bpt<S, R>()][R], int p, int jt, unsigned* red) {
    int hi = 0, lo = 0;
#pragma unroll
    for (int b = 0; b < fx_bpt<S, R>(); b++) {
        if (!fx_has<S, R>(b, jt)) continue;
        const int d = fx_dest<R, NS>(jt + S::TPP * b);
#pragma unroll
        for (int r = 0; r < R; r++) {
            tile[fx_row<S, NS, NS == 1 && R % 8 == 0>(d, r) + p] = v[b][r];
            const int x = (int)(v[b][r].x >> 32), y = (int)(v[b][r].y >> 32);
            hi = max(hi, max(x, y));
            lo = min(lo, min(x, y));
        }
    }
    const int h = (int)fx_group_max<S::TPP>((unsigned)max(hi, ~lo), p, red);
    fx_group_sync<S::TPP>(p);
    return h;
}

// Radix-R pass after NS of the group's pencil: read, synchronise, scale, twiddle, DFT.
template <class S, int R, int NS, bool INV>
__device__ __forceinline__ void fx_group_pass(C<fx> (&v)[fx_bpt<S, R>()][R], const C<fx>* tile, const int4* tw, int p, int jt,
                                              int hmax, int& eb) {
    constexpr int NB = S::L / R, BPT = fx_bpt<S, R>(), STEP = S::L / (NS * R);
#pragma unroll
    for (int b = 0; b < BPT; b++)
#pragma unroll
        for (int r = 0; r < R; r++)
            v[b][r] = fx_has<S, R>(b, jt) ? tile[fx_row<S, NB>(jt + S::TPP * b, r) + p] : mk<fx>(0, 0);
    const FxStep st = fx_step<R>(hmax);
    fx_group_sync<S::TPP>(p);
    eb += st.d;
    fx_twiddles<R, NS, STEP, INV, S::TPP, BPT>(v, tw, jt, st);
}

// The later passes of the group's pencil from the results v of the first one.
// FIXED: the tile ends up with the fixed-point transform, otherwise with doubles;
// outputs in the band of ZOUT are left out.  Synchronised on return.
template <class S, bool INV, bool FIXED, bool PRUNE>
__device__ __forceinline__ void fx_group_later(C<double>* tile, C<fx> (&v)[fx_bpt<S, S::R1>()][S::R1], const int4* tw, int p,
                                               int jt, FxScale sc, int& eb, unsigned* red) {
    constexpr int R1 = S::R1, NPASS = S::R3 > 1 ? 3 : S::R2 > 1 ? 2 : 1;
    constexpr int RL = NPASS == 3 ? S::R3 : S::R2;
    constexpr unsigned ZO = (PRUNE && !INV && NPASS > 1) ? band_mask<S::L, RL>() : 0u;
    constexpr FxOut OUT = FIXED ? FX_OUT_FIXED : FX_OUT_TILE;
    C<fx>* ft = reinterpret_cast<C<fx>*>(tile);
    const auto none = [](int, C<double>) {};
#pragma unroll
    for (int b = 0; b < fx_bpt<S, R1>(); b++) fx_dft<R1, INV>(v[b]);
    if constexpr (NPASS == 1) {
        fx_finish<S, R1, 1, OUT, 0u>(tile, v, p, jt, sc, eb, none);
    } else {
        int h = fx_group_write<S, R1, 1>(ft, v, p, jt, red + 2);
        C<fx> v2[fx_bpt<S, S::R2>()][S::R2];
        fx_group_pass<S, S::R2, R1, INV>(v2, ft, tw, p, jt, h, eb);
        if constexpr (NPASS == 2) {
            fx_finish<S, S::R2, R1, OUT, ZO>(tile, v2, p, jt, sc, eb, none);
        } else {
            h = fx_group_write<S, S::R2, R1>(ft, v2, p, jt, red + 4);
            C<fx> v3[fx_bpt<S, S::R3>()][S::R3];
            fx_group_pass<S, S::R3, R1 * S::R2, INV>(v3, ft, tw, p, jt, h, eb);
            fx_finish<S, S::R3, R1 * S::R2, OUT, ZO>(tile, v3, p, jt, sc, eb, none);
        }
    }
    fx_group_sync<S::TPP>(p);
}

// c2r: two half spectra A, B (kx < Kx) into the packed sequence Z = A + iB in
// fixed point (each mode is loaded and converted once for both of its places in
// Z), then the inverse transform, whose real and imaginary parts are the two rows
// (doubles in the tile).  get(k, A, B) loads; the imaginary parts at kx = 0 and
// kx = L/2 are dropped, as a c2r transform does.  kx = L/2 is kept by plans with
// Kx = L/2 + 1 only, which the 2/3 rule (PRUNE) never is.
template <class S, bool PRUNE, class Get>
__device__ __forceinline__ void fx_group_c2r(C<double>* tile, const int4* tw, int p, int jt, int Kx, unsigned* red, Get get) {
    constexpr int L = S::L, H = L / 2, TPP = S::TPP, NPT = (H + TPP - 1) / TPP, R1 = S::R1, NB1 = L / R1;
    constexpr unsigned ZI = (PRUNE && S::R2 > 1) ? band_mask<L, R1>() : 0u;
    C<fx>* ft = reinterpret_cast<C<fx>*>(tile);
    FxScale sc;
    {
        C<double> AB[NPT][2], last = mk<double>(0., 0.);   // last: real parts of both rows at kx = L/2
        unsigned h = 0;
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int k = jt + TPP * i;
            AB[i][0] = AB[i][1] = mk<double>(0., 0.);
            if (k < Kx) get(k, AB[i][0], AB[i][1]);
            if (k == 0) { AB[i][0].y = 0.; AB[i][1].y = 0.; }
        }
        if constexpr (!PRUNE) {
            if (Kx > H && jt == 0) {
                C<double> A = mk<double>(0., 0.), B = mk<double>(0., 0.);
                get(H, A, B);
                last = mk<double>(A.x, B.x);
                h = fx_max(h, last);
            }
        }
#pragma unroll
        for (int i = 0; i < NPT; i++) h = fx_max(fx_max(h, AB[i][0]), AB[i][1]);
        sc = fx_scale(fx_group_max<TPP>(h, p, red) >> 1);
        if (sc.rare) {
            fx_scale_all<2 * NPT>(&AB[0][0], fx_pre(sc.rare));
            if constexpr (!PRUNE) fx_scale_all<1>(&last, fx_pre(sc.rare));
        }
        const int K = fx_kin<S>(sc.e2, true);
        C<fx> lastf = mk<fx>(0, 0);
        if constexpr (!PRUNE) {
            if (Kx > H) lastf = fx_in(last, K);
        }
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int k = jt + TPP * i;
            if (H % TPP != 0 && k >= H) continue;
            const C<fx> a = fx_in(AB[i][0], K), b = fx_in(AB[i][1], K);
            ft[S::off(k) + p] = mk<fx>(a.x - b.y, a.y + b.x);
            ft[S::off(k == 0 ? H : L - k) + p] = k == 0 ? lastf : mk<fx>(a.x + b.y, b.x - a.y);
        }
    }
    fx_group_sync<TPP>(p);
    C<fx> v[fx_bpt<S, R1>()][R1];
#pragma unroll
    for (int b = 0; b < fx_bpt<S, R1>(); b++)
#pragma unroll
        for (int r = 0; r < R1; r++)
            v[b][r] = ((ZI >> r) & 1u) || !fx_has<S, R1>(b, jt) ? mk<fx>(0, 0) : ft[fx_row<S, NB1>(jt + TPP * b, r) + p];
    fx_group_sync<TPP>(p);
    int eb = fx_kin<S>(sc.e2, true);
    fx_group_later<S, true, false, PRUNE>(tile, v, tw, p, jt, sc, eb, red);
}

// r2c: the forward transform of the packed rows ld(e) (real and imaginary part),
// then their half spectra times 2^sexp smul: put0(k, value), put1(k, value) for
// kx < Kx.
template <class S, bool PRUNE, class Ld, class Put0, class Put1>
__device__ __forceinline__ void fx_group_r2c(C<double>* tile, const int4* tw, int p, int jt, int Kx, int sexp, double smul,
                                             unsigned* red, Ld ld, Put0 put0, Put1 put1) {
    constexpr int L = S::L, TPP = S::TPP, R1 = S::R1, NB1 = L / R1, BPT = fx_bpt<S, R1>();
    FxScale sc;
    C<fx> v[BPT][R1];
    {
        C<double> d[BPT][R1];
        unsigned h = 0;
#pragma unroll
        for (int b = 0; b < BPT; b++)
#pragma unroll
            for (int r = 0; r < R1; r++) d[b][r] = fx_has<S, R1>(b, jt) ? ld(jt + TPP * b + r * NB1) : mk<double>(0., 0.);
#pragma unroll
        for (int b = 0; b < BPT; b++)
#pragma unroll
            for (int r = 0; r < R1; r++) h = fx_max(h, d[b][r]);
        sc = fx_scale(fx_group_max<TPP>(h, p, red) >> 1);
        if (sc.rare) fx_scale_all<BPT * R1>(&d[0][0], fx_pre(sc.rare));
        const int K = fx_kin<S>(sc.e2, false);
#pragma unroll
        for (int b = 0; b < BPT; b++)
#pragma unroll
            for (int r = 0; r < R1; r++) v[b][r] = fx_in(d[b][r], K);
    }
    fx_group_sync<TPP>(p);                 // ld may read the tile
    int eb = fx_kin<S>(sc.e2, false);
    fx_group_later<S, false, true, PRUNE>(tile, v, tw, p, jt, sc, eb, red);
    const C<fx>* ft = reinterpret_cast<const C<fx>*>(tile);
    eb += sexp - 1;
    const bool plain = smul == 1.0 && !sc.rare;
    const double post = sc.rare ? fx_post(sc.rare) : 1.0;
    for (int k = jt; k < Kx; k += TPP) {
        const C<fx> z = ft[S::off(k) + p], w = ft[S::off(k == 0 ? 0 : L - k) + p];
        // A = (z + conj w) / 2, B = (z - conj w) / 2i
        C<double> o[2] = {fx_out(mk<fx>(z.x + w.x, z.y - w.y), eb), fx_out(mk<fx>(z.y + w.y, w.x - z.x), eb)};
        if (!plain) {
            fx_scale_all<2>(o, smul);
            fx_scale_all<2>(o, post);
        }
        put0(k, o[0]);
        put1(k, o[1]);
    }
}

// scale = 2^sexp smul with smul = 1 for a power of two and sexp = 0 otherwise.
inline void fx_split_scale(double scale, int& sexp, double& smul) {
    int e;
    const bool two = frexp(scale, &e) == 0.5;
    sexp = two ? e - 1 : 0;
    smul = two ? 1.0 : scale;
}

}  // namespace dd
