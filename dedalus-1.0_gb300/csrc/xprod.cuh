// Fused x-direction pass: NI half-spectrum fields -> c2r -> pointwise
// nonlinear products in shared memory -> r2c of NO fields, for Q rows per block.
//
// Real rows are paired into complex pencils in row-major (row, field) order:
// real row t = r*NI + f lives in pencil t/2, real part if t is even, imaginary
// part if odd.  The forward side pairs its outputs the same way with NO.  The
// inverse and forward transforms use their own schedules (SI, SF) so the
// pencil slots of the block can be filled on both sides.
//
// Op provides: static NI, NO; __device__ void operator()(const T* in, T* out,
// int run) on the NI grid values of one point, producing NO values.  Blocks
// are (row block, run): run b's fields start at win.p[f] + b * in_rs and
// wout.p[g] + b * out_rs (complex entries).
#pragma once
#include "launch_len.cuh"

namespace dd {

template <int L, int NI, int NO>
struct ProdCfg {
    using SI = DefSched<L>;
    using SF = DefSched<L>;
    static constexpr int q_of(int n) { return ((2 * SI::P) / n) & ~1; }
    static constexpr int Q = (q_of(NI) < q_of(NO) ? q_of(NI) : q_of(NO));
    static constexpr int NT = SI::NT;
};
// Hydro (6 -> 3) and MHD (12 -> 6): forward pencils are half the inverse
// ones, so SF doubles the threads per pencil and both sides are full.
template <> struct ProdCfg<64, 6, 3> {
    using SI = Sched<64, 24, 192, 8, 8, 1>;  using SF = Sched<64, 12, 192, 4, 4, 4>;
    static constexpr int Q = 8, NT = 192;
};
template <> struct ProdCfg<128, 6, 3> {
    using SI = Sched<128, 24, 192, 16, 8, 1>;  using SF = Sched<128, 12, 192, 8, 4, 4>;
    static constexpr int Q = 8, NT = 192;
};
template <> struct ProdCfg<256, 6, 3> {
    using SI = Sched<256, 12, 192, 16, 16, 1>;  using SF = Sched<256, 6, 192, 8, 8, 4>;
    static constexpr int Q = 4, NT = 192;
};
template <> struct ProdCfg<512, 6, 3> {
    using SI = Sched<512, 6, 192, 8, 8, 8>;  using SF = Sched<512, 3, 192, 8, 8, 8>;
    static constexpr int Q = 2, NT = 192;
};
// Hydro in divergence form (3 -> 5): the forward side has 5/3 of the inverse
// pencils; 4 rows per block fill 6 inverse pencils (32 threads each) and 10
// forward pencils (16 threads each).
template <> struct ProdCfg<256, 3, 5> {
    using SI = Sched<256, 6, 192, 8, 8, 4>;  using SF = Sched<256, 10, 160, 16, 16, 1>;
    static constexpr int Q = 4, NT = 192;
};
// 2D hydro (3 -> 2) on 64- and 128-point rows: 2 rows per block (3 inverse
// and 2 forward pencils of 16 threads), so that one 128^2 run has 64 blocks.
template <> struct ProdCfg<64, 3, 2> {
    using SI = Sched<64, 3, 48, 4, 4, 4>;  using SF = Sched<64, 2, 32, 4, 4, 4>;
    static constexpr int Q = 2, NT = 48;
};
template <> struct ProdCfg<128, 3, 2> {
    using SI = Sched<128, 3, 48, 8, 4, 4>;  using SF = Sched<128, 2, 32, 8, 4, 4>;
    static constexpr int Q = 2, NT = 48;
};
template <> struct ProdCfg<64, 12, 6> {
    using SI = Sched<64, 24, 192, 8, 8, 1>;  using SF = Sched<64, 12, 192, 4, 4, 4>;
    static constexpr int Q = 4, NT = 192;
};
template <> struct ProdCfg<128, 12, 6> {
    using SI = Sched<128, 24, 192, 16, 8, 1>;  using SF = Sched<128, 12, 192, 8, 4, 4>;
    static constexpr int Q = 4, NT = 192;
};
template <> struct ProdCfg<256, 12, 6> {
    using SI = Sched<256, 12, 192, 16, 16, 1>;  using SF = Sched<256, 6, 192, 8, 8, 4>;
    static constexpr int Q = 2, NT = 192;
};
template <> struct ProdCfg<512, 12, 6> {
    using SI = Sched<512, 12, 384, 8, 8, 8>;  using SF = Sched<512, 6, 384, 8, 8, 8>;
    static constexpr int Q = 2, NT = 384;
};

// The schedule a precision runs (ProdCfg unless specialised).  per_point:
// the tile fill, the product phase and the output unpacking are organised by
// grid point, with the pencils, rows and fields of a point in compile-time
// loops.  A thread fills and multiplies whole tile rows (complex entries, not
// their halves), and the field pointers are fixed per loop step instead of
// selected at run time.  Otherwise each thread takes one tile entry or one
// point of one row at a time.
template <typename T, int L, int NI, int NO>
struct ProdCfgT : ProdCfg<L, NI, NO> {
    static constexpr bool per_point = false;
    static constexpr int min_blocks = std::is_same<T, df64>::value ? 5 : 1;   // __launch_bounds__
};
// FP64 (fixed-point transforms, a thread group per pencil): exactly the pencils
// that the fields fill, the largest power of two of rows (2 to 16) whose pencils take
// at most 192 threads, and registers for 1024 threads per SM.  Small blocks keep
// fewer threads waiting at the block's barriers: on a 128^3 grid the MHD products (6
// fields in, 8 out) take 190 us at 2 rows (128 threads), 201 at 4 and 235 at 8, hydro's
// (3 and 5) 93 at 4 rows (160 threads), 99 at 6, 103 at 8 and 112 at 2; on 64^3 MHD
// 27.0 at 4, 31.1 at 6 and 29.1 at 8, hydro 16.8 at 8 and 18.8 at 12.  256 threads for
// the 2D products: alone they are 4% faster with 128, but an ensemble runs them
// beside those of other lengths, where its step takes 2941 us against 2885 (128
// uneven convection runs).
constexpr int prod_rows_fx(int threads_per_row, int most) {
    int q = 16;
    while (q > 2 && q * threads_per_row > most) q /= 2;
    return q;
}
template <int L, int NI, int NO>
struct ProdCfgT<double, L, NI, NO> {
    static constexpr int NM = NI > NO ? NI : NO;
    static constexpr int Q = prod_rows_fx(NM * FxRowTPP<L>::v / 2, NM <= 4 ? 256 : 192);
    using SI = FxR<L, true, NI * Q / 2>;
    using SF = FxR<L, false, NO * Q / 2>;
    static constexpr int NT = ((SI::NT > SF::NT ? SI::NT : SF::NT) + 31) / 32 * 32;
    static constexpr int min_blocks = NT > 512 ? 1 : 1024 / NT;
};
// 2D hydro on 64- and 128-point rows: 2 rows per block as for a single FP32 run
template <int L>
struct ProdCfg2Rows {
    static constexpr int Q = 2, NT = (3 * FxRowTPP<L>::v + 31) / 32 * 32, min_blocks = 1;
    using SI = FxR<L, true, 3>;
    using SF = FxR<L, false, 2>;
};
template <> struct ProdCfgT<double, 64, 3, 2> : ProdCfg2Rows<64> {};
template <> struct ProdCfgT<double, 128, 3, 2> : ProdCfg2Rows<128> {};
// FP32 hydro in divergence form on 256-point rows: 6 inverse and 10 forward
// pencils in tiles with unpadded rows and a skew every 8 rows (P / 2 entries),
// and the per-point product phase.  With the odd strides 7 and 11, 41% of the
// shared-memory wavefronts of a launch were bank conflicts (23.3 M of 57.2 M);
// a model of every access of the kernel puts this layout at 37% fewer
// wavefronts.  (Tiles 16 pencils wide, 9 inverse and 15 forward pencils per
// 6 rows, cut the conflicts to 4% but ran slower: their idle pencil slots cost
// more than the conflicts.)
template <>
struct ProdCfgT<float, 256, 3, 5> {
    using SI = Sched<256, 6, 192, 8, 8, 4, 6, 3>;
    using SF = Sched<256, 10, 160, 16, 16, 1, 10, 5>;
    static constexpr int Q = 4, NT = 192;
    static constexpr bool per_point = true;
    static constexpr int min_blocks = 6;   // 56 registers: 6 blocks per SM (72 and 4 blocks without the bound)
};

// FP32 MHD in divergence form (6 -> 8) on 256-point rows: the default 16-pencil
// tiles (12 inverse, 16 forward pencils for 4 rows), point-major phases.
template <>
struct ProdCfgT<float, 256, 6, 8> : ProdCfg<256, 6, 8> {
    static constexpr bool per_point = true;
    static constexpr int min_blocks = 4;   // 64 registers (90 unbounded: 2 blocks per SM, 565 vs 348 us)
};

// FP32 2D Boussinesq in divergence form (3 -> 4) on 256- and 512-point rows:
// the default tiles (16 pencils, 8 rows per block; 8 pencils, 4 rows),
// point-major phases.
template <>
struct ProdCfgT<float, 256, 3, 4> : ProdCfg<256, 3, 4> {
    static constexpr bool per_point = true;
    static constexpr int min_blocks = 4;   // 64 registers (72 unbounded, 3 blocks per SM)
};
template <>
struct ProdCfgT<float, 512, 3, 4> : ProdCfg<512, 3, 4> {
    static constexpr bool per_point = true;
    static constexpr int min_blocks = 1;
};

template <typename T, int L, int NI, int NO>
constexpr size_t prod_smem(size_t csize) {
    using CC = ProdCfgT<T, L, NI, NO>;
    const size_t a = (size_t)CC::SI::span, b = (size_t)CC::SF::span;
    return csize * ((a > b ? a : b) + L);
}

template <typename T, int L, class Op>
__global__ void __launch_bounds__(ProdCfgT<T, L, Op::NI, Op::NO>::NT, ProdCfgT<T, L, Op::NI, Op::NO>::min_blocks)
k_x_prod(int nrows, int Kx, CPtrs win, Ptrs wout, int64_t in_rs, int64_t out_rs,
         const typename TwVec<T>::type* gtw, T scale, const Op op) {
    using V = typename Vec2<T>::type;
    constexpr int NI = Op::NI, NO = Op::NO;
    static_assert(NI <= DD_MAXF && NO <= DD_MAXF, "too many fields for Ptrs");
    using CC = ProdCfgT<T, L, NI, NO>;
    using SI = typename CC::SI;
    using SF = typename CC::SF;
    extern __shared__ __align__(16) unsigned char dd_smem[];
    constexpr int NT = CC::NT, Q = CC::Q;
    static_assert(Q >= 2 && Q % 2 == 0, "need an even number of rows per block");
    static_assert((NI * Q + 1) / 2 <= SI::P && (NO * Q + 1) / 2 <= SF::P, "schedule too small for Q rows");
    static_assert(SI::NT == NT && SF::NT <= NT, "schedules must fit the block");
    C<T>* tile = reinterpret_cast<C<T>*>(dd_smem);
    constexpr size_t TA = (size_t)SI::span, TB = (size_t)SF::span;
    C<T>* tw = tile + (TA > TB ? TA : TB);
    load_twiddles<T, L>(tw, gtw);
    grid_wait();
    const int row0 = blockIdx.x * Q;
    const int nr = min(Q, nrows - row0);
    const int64_t ib = blockIdx.y * in_rs, ob = blockIdx.y * out_rs;  // run (batch) offsets
    constexpr int NPI = (NI * Q + 1) / 2;  // inverse pencils in use
    if constexpr (CC::per_point) {
        // tile row e = grid point e of the block's rows: all NPI pencils of a
        // row, the loads of a thread's rows in flight together
        constexpr int NE = (L + NT - 1) / NT;
        C<T> zv[NE][NPI];
#pragma unroll
        for (int i = 0; i < NE; i++) {
            const int e = threadIdx.x + i * NT;
#pragma unroll
            for (int pj = 0; pj < NPI; pj++) {
                const int ta = 2 * pj, tb = 2 * pj + 1;
                const int ra = ta / NI, fa = ta % NI, rb = tb / NI, fb = tb % NI;
                const bool va = ra < nr, vb = tb < NI * Q && rb < nr;
                C<T> z = zero<T>();
                if ((NE * NT == L || e < L) && (va || vb)) {
                    const V* pa = (const V*)win.p[fa] + ib + (int64_t)(row0 + ra) * Kx;
                    const V* pb = (const V*)win.p[tb < NI * Q ? fb : fa] + ib + (int64_t)(row0 + rb) * Kx;
                    z = pack_rows<T>(va ? pa : pb, vb ? pb : pa, e, L, Kx);
                    if (!va) z.x = T(0);
                    if (!vb) z.y = T(0);
                }
                zv[i][pj] = z;
            }
        }
#pragma unroll
        for (int i = 0; i < NE; i++) {
            const int e = threadIdx.x + i * NT;
            if (NE * NT == L || e < L) {
#pragma unroll
                for (int pj = 0; pj < NPI; pj++) tile[SI::off(e) + pj] = zv[i][pj];
#pragma unroll
                for (int pj = NPI; pj < SI::P; pj++) tile[SI::off(e) + pj] = zero<T>();
            }
        }
    } else {
        // the loads of a group of GX entries are in flight together (see load_tile)
        constexpr int NLD = L * SI::P, NPL = (NLD + NT - 1) / NT;
        constexpr int GX0 = (int)(128 / sizeof(C<T>)), GX = NPL < GX0 ? NPL : GX0;
#pragma unroll
        for (int i0 = 0; i0 < NPL; i0 += GX) {
            C<T> zv[GX];
#pragma unroll
            for (int i = 0; i < GX; i++) {
                const int idx = threadIdx.x + (i0 + i) * NT;
                const int e = idx % L, pj = idx / L;
                C<T> z = zero<T>();
                if (i0 + i < NPL && idx < NLD && pj < NPI) {
                    const int ta = 2 * pj, tb = 2 * pj + 1;
                    const int ra = ta / NI, fa = ta % NI, rb = tb / NI, fb = tb % NI;
                    const bool va = ra < nr, vb = tb < NI * Q && rb < nr;
                    if (va || vb) {
                        const V* pa = (const V*)pick_ptr<NI>(win.p, fa) + ib + (int64_t)(row0 + (va ? ra : rb)) * Kx;
                        const V* pb =
                            (const V*)pick_ptr<NI>(win.p, vb ? fb : fa) + ib + (int64_t)(row0 + (vb ? rb : ra)) * Kx;
                        z = pack_rows<T>(pa, pb, e, L, Kx);
                        if (!va) z.x = T(0);
                        if (!vb) z.y = T(0);
                    }
                }
                zv[i] = z;
            }
#pragma unroll
            for (int i = 0; i < GX; i++) {
                const int idx = threadIdx.x + (i0 + i) * NT;
                if (i0 + i < NPL && idx < NLD) tile[SI::off(idx % L) + idx / L] = zv[i];
            }
        }
    }
    __syncthreads();
    // kept kx <= Kx - 1: under the 2/3 rule the packed pencils are zero in the
    // removed band and the unpacking never reads it
    // (double-float has no pruned butterflies: one copy of its transform)
    const bool prune = IsLF<T>::value && Kx - 1 == kept23(L);
    if constexpr (IsLF<T>::value) {
        if (prune) pencil_fft_s<T, SI, true, true>(tile, tw);
        else pencil_fft_s<T, SI, true>(tile, tw);
    } else {
        pencil_fft_s<T, SI, true>(tile, tw);
    }
    if constexpr (CC::per_point) {
        // one grid point of all Q rows per thread: the NPI inverse pencils of a
        // row of the tile in, the NPF forward pencils out (the last one's
        // imaginary half zero when NO Q is odd)
        constexpr int NPP = (L + NT - 1) / NT, NPF = (NO * Q + 1) / 2;
        T outv[NPP][NO * Q];
#pragma unroll
        for (int i = 0; i < NPP; i++) {
            const int e = threadIdx.x + i * NT;
            if (e < L) {
                C<T> pin[NPI];
#pragma unroll
                for (int pj = 0; pj < NPI; pj++) pin[pj] = tile[SI::off(e) + pj];
#pragma unroll
                for (int r = 0; r < Q; r++) {
                    T in[NI];
#pragma unroll
                    for (int f = 0; f < NI; f++) {
                        const int t = r * NI + f;
                        in[f] = (t & 1) ? pin[t / 2].y : pin[t / 2].x;
                    }
                    op(in, &outv[i][r * NO], blockIdx.y);
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NPP; i++) {
            const int e = threadIdx.x + i * NT;
            if (e < L) {
#pragma unroll
                for (int pj = 0; pj < NPF; pj++)
                    tile[SF::off(e) + pj] = mk<T>(outv[i][2 * pj], 2 * pj + 1 < NO * Q ? outv[i][2 * pj + 1] : T(0));
            }
        }
    } else {
        constexpr int NPT = (L * Q + NT - 1) / NT;
        T outv[NPT][NO];
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int idx = threadIdx.x + i * NT;
            if (idx < L * Q) {
                const int e = idx % L, r = idx / L;
                T in[NI];
#pragma unroll
                for (int f = 0; f < NI; f++) {
                    const int t = r * NI + f;
                    const C<T> c = tile[SI::off(e) + t / 2];
                    in[f] = (t & 1) ? c.y : c.x;
                }
                op(in, outv[i], blockIdx.y);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int idx = threadIdx.x + i * NT;
            if (idx < L * Q) {
                const int e = idx % L, r = idx / L;
#pragma unroll
                for (int g = 0; g < NO; g++) {
                    const int t = r * NO + g;
                    if (t & 1) tile[SF::off(e) + t / 2].y = outv[i][g];
                    else tile[SF::off(e) + t / 2].x = outv[i][g];
                }
            }
        }
        if constexpr ((NO * Q) & 1) {  // the last pencil's imaginary half is unused
            for (int e = threadIdx.x; e < L; e += NT) tile[SF::off(e) + (NO * Q) / 2].y = T(0);
        }
    }
    __syncthreads();
    if constexpr (IsLF<T>::value) {
        if (prune) pencil_fft_s<T, SF, false, true>(tile, tw, threadIdx.x < SF::NT);
        else pencil_fft_s<T, SF, false>(tile, tw, threadIdx.x < SF::NT);
    } else {
        pencil_fft_s<T, SF, false>(tile, tw, threadIdx.x < SF::NT);
    }
    if constexpr (CC::per_point) {
        // two halves of the block take the rows r < Q/2 and r >= Q/2; within a
        // half consecutive threads take consecutive kx of one output row
        constexpr int KG = NT / 2;
        const int half = threadIdx.x / KG;
        for (int k = threadIdx.x % KG; k < Kx; k += KG) {
            const C<T>* zr = tile + SF::off(k);
            const C<T>* znr = tile + SF::off(k == 0 ? 0 : L - k);
#pragma unroll
            for (int r2 = 0; r2 < Q / 2; r2++) {
                const int r = half * (Q / 2) + r2;
                if (r >= nr) continue;
#pragma unroll
                for (int g = 0; g < NO; g++) {
                    const int t = r * NO + g;
                    C<T> A, B;
                    unpack_pair<T>(zr[t / 2], znr[t / 2], scale, A, B);
                    stc<T>((V*)wout.p[g] + ob + (int64_t)(row0 + r) * Kx + k, (t & 1) ? B : A);
                }
            }
        }
    } else {
        // field-major order: consecutive threads write the block's Q consecutive rows
        // of one output field, a contiguous range, so a 32-byte sector shared by two
        // rows (complex64 rows of an odd number of half-sectors) is written whole by
        // one warp instead of in two halves at different times
        for (int idx = threadIdx.x; idx < Kx * Q * NO; idx += NT) {
            const int k = idx % Kx, u = idx / Kx;
            const int g = u / Q, r = u % Q;
            if (r >= nr) continue;
            const int t = r * NO + g;              // its real row in the packed tile
            C<T> A, B;
            unpack_pair<T>(tile[SF::off(k) + t / 2], tile[SF::off(k == 0 ? 0 : L - k) + t / 2], scale, A, B);
            stc<T>((V*)pick_ptr<NO>(wout.p, g) + ob + (int64_t)(row0 + r) * Kx + k, (t & 1) ? B : A);
        }
    }
}

// The same pass for FP64 in fixed point (fft_fixed.cuh): a thread group loads,
// packs and transforms a pencil's two half spectra, the block forms the grid-point
// products in FP64, and the groups transform, unpack and store theirs.
template <int L, class Op>
constexpr int prod_words_fx() {
    using CC = ProdCfgT<double, L, Op::NI, Op::NO>;
    return fx_group_words<typename CC::SI>() + fx_group_words<typename CC::SF>();
}
template <int L, class Op>
constexpr size_t prod_smem_fx() {
    using CC = ProdCfgT<double, L, Op::NI, Op::NO>;
    const size_t a = (size_t)CC::SI::span, b = (size_t)CC::SF::span;
    return 16 * ((a > b ? a : b) + 2 * L) + sizeof(unsigned) * prod_words_fx<L, Op>();
}

template <int L, bool PRUNE, class Op>
__device__ __forceinline__ void x_prod_fx_body(int nrows, int Kx, const CPtrs& win, const Ptrs& wout, int64_t ib, int64_t ob,
                                               C<double>* tile, const int4* twi, const int4* twf, unsigned* words,
                                               int sexp, double smul, const Op& op) {
    constexpr int NI = Op::NI, NO = Op::NO;
    using CC = ProdCfgT<double, L, NI, NO>;
    using SI = typename CC::SI;
    using SF = typename CC::SF;
    constexpr int NT = CC::NT, Q = CC::Q, NPI = NI * Q / 2, NPF = NO * Q / 2, TPP = SI::TPP;
    const int row0 = blockIdx.x * Q;
    const int nr = min(Q, nrows - row0);
    const int p = threadIdx.x / TPP, jt = threadIdx.x % TPP;
    if (p < NPI) {
        const int ra = (2 * p) / NI, rb = (2 * p + 1) / NI;
        const double2* pa = (const double2*)pick_ptr<NI>(win.p, (2 * p) % NI) + ib + (int64_t)(row0 + ra) * Kx;
        const double2* pb = (const double2*)pick_ptr<NI>(win.p, (2 * p + 1) % NI) + ib + (int64_t)(row0 + rb) * Kx;
        fx_group_c2r<SI, PRUNE>(tile, twi, p, jt, Kx, words + 6 * p, [&](int k, C<double>& A, C<double>& B) {
            if (ra < nr) A = ldc<double>(pa + k);
            if (rb < nr) B = ldc<double>(pb + k);
        });
    }
    __syncthreads();
    constexpr int NPP = (L + NT - 1) / NT;
    if constexpr (NPP * NPF <= 12) {
        // a grid point of all rows per thread, whole tile entries in and out
        C<double> outv[NPP][NPF];
#pragma unroll
        for (int i = 0; i < NPP; i++) {
            const int e = threadIdx.x + i * NT;
            if (L % NT != 0 && e >= L) continue;
            double in[2 * NPI], out[2 * NPF];
#pragma unroll
            for (int pj = 0; pj < NPI; pj++) {
                const C<double> c = tile[SI::off(e) + pj];
                in[2 * pj] = c.x;
                in[2 * pj + 1] = c.y;
            }
#pragma unroll
            for (int r = 0; r < Q; r++) op(in + r * NI, out + r * NO, blockIdx.y);
#pragma unroll
            for (int pj = 0; pj < NPF; pj++) outv[i][pj] = mk<double>(out[2 * pj], out[2 * pj + 1]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NPP; i++) {
            const int e = threadIdx.x + i * NT;
            if (L % NT != 0 && e >= L) continue;
#pragma unroll
            for (int pj = 0; pj < NPF; pj++) tile[SF::off(e) + pj] = outv[i][pj];
        }
    } else {
        constexpr int NPT = (L * Q + NT - 1) / NT;
        double outv[NPT][NO];
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int idx = threadIdx.x + i * NT;
            if (idx < L * Q) {
                const int e = idx % L, r = idx / L;
                double in[NI];
#pragma unroll
                for (int f = 0; f < NI; f++) {
                    const int t = r * NI + f;
                    const double* c = &tile[SI::off(e) + t / 2].x;
                    in[f] = c[t & 1];
                }
                op(in, outv[i], blockIdx.y);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int idx = threadIdx.x + i * NT;
            if (idx < L * Q) {
                const int e = idx % L, r = idx / L;
#pragma unroll
                for (int g = 0; g < NO; g++) {
                    const int t = r * NO + g;
                    double* c = &tile[SF::off(e) + t / 2].x;
                    c[t & 1] = outv[i][g];
                }
            }
        }
    }
    __syncthreads();
    if (p < NPF) {
        const int ra = (2 * p) / NO, rb = (2 * p + 1) / NO;
        double2* pa = (double2*)pick_ptr<NO>(wout.p, (2 * p) % NO) + ob + (int64_t)(row0 + ra) * Kx;
        double2* pb = (double2*)pick_ptr<NO>(wout.p, (2 * p + 1) % NO) + ob + (int64_t)(row0 + rb) * Kx;
        fx_group_r2c<SF, PRUNE>(tile, twf, p, jt, Kx, sexp, smul, words + fx_group_words<SI>() + 6 * p,
                                [&](int e) { return tile[SF::off(e) + p]; },
                                [&](int k, C<double> c) { if (ra < nr) stc<double>(pa + k, c); },
                                [&](int k, C<double> c) { if (rb < nr) stc<double>(pb + k, c); });
    }
}

template <int L, class Op>
__global__ void __launch_bounds__(ProdCfgT<double, L, Op::NI, Op::NO>::NT, ProdCfgT<double, L, Op::NI, Op::NO>::min_blocks)
k_x_prod_fx(int nrows, int Kx, CPtrs win, Ptrs wout, int64_t in_rs, int64_t out_rs, const int4* gtw, int sexp, double smul,
            const Op op) {
    using CC = ProdCfgT<double, L, Op::NI, Op::NO>;
    extern __shared__ __align__(16) unsigned char dd_smem[];
    constexpr int Q = CC::Q, NT = CC::NT;
    static_assert(Q >= 2 && Q % 2 == 0, "need an even number of rows per block");
    static_assert(Op::NI * Q / 2 == CC::SI::P && Op::NO * Q / 2 == CC::SF::P, "a thread group per pencil");
    static_assert(CC::SI::NT <= NT && CC::SF::NT <= NT && CC::SI::TPP == CC::SF::TPP, "schedules must fit the block");
    C<double>* tile = reinterpret_cast<C<double>*>(dd_smem);
    constexpr size_t TA = (size_t)CC::SI::span, TB = (size_t)CC::SF::span;
    int4* twi = reinterpret_cast<int4*>(tile + (TA > TB ? TA : TB));
    int4* twf = twi + L;
    unsigned* words = reinterpret_cast<unsigned*>(twf + L);
    fx_stage_twiddles<L, true>(twi, gtw);
    fx_stage_twiddles<L, false>(twf, gtw);
    grid_wait();
    __syncthreads();
    const int64_t ib = blockIdx.y * in_rs, ob = blockIdx.y * out_rs;  // run (batch) offsets
    if (Kx - 1 == kept23(L)) x_prod_fx_body<L, true>(nrows, Kx, win, wout, ib, ob, tile, twi, twf, words, sexp, smul, op);
    else x_prod_fx_body<L, false>(nrows, Kx, win, wout, ib, ob, tile, twi, twf, words, sexp, smul, op);
}

template <typename T, int L, class Op>
int launch_x_prod(const char* name, int nrows, int Kx, const CPtrs& win, const Ptrs& wout, int nrun, int64_t in_rs,
                  int64_t out_rs, const typename TwVec<T>::type* tw, T scale, const Op& op, cudaStream_t st) {
    using CC = ProdCfgT<T, L, Op::NI, Op::NO>;
    if constexpr (std::is_same<T, double>::value) {
        constexpr size_t smem = prod_smem_fx<L, Op>();
        static std::atomic<unsigned long long> configured{0};
        DD_TRY(ensure_smem((const void*)k_x_prod_fx<L, Op>, smem, configured));
        static const std::string label = std::string(name) + "_" + std::to_string(L) + PrecName<T>::s;
        int sexp;
        double smul;
        fx_split_scale(scale, sexp, smul);
        DD_KT(label.c_str(), st,
              launch(k_x_prod_fx<L, Op>, dim3(cdiv(nrows, CC::Q), nrun), CC::NT, smem, st, nrows, Kx, win, wout, in_rs, out_rs, tw,
                                                                                       sexp, smul, op));
        DD_LAUNCH_CHECK();
        return DD_OK;
    } else {
    const size_t smem = prod_smem<T, L, Op::NI, Op::NO>(sizeof(C<T>));
    static std::atomic<unsigned long long> configured{0};
    DD_TRY(ensure_smem((const void*)k_x_prod<T, L, Op>, smem, configured));
    static const std::string label = std::string(name) + "_" + std::to_string(L) + PrecName<T>::s;
    DD_KT(label.c_str(), st,
          launch(k_x_prod<T, L, Op>, dim3(cdiv(nrows, CC::Q), nrun), CC::NT, smem, st, nrows, Kx, win, wout, in_rs, out_rs,
                                                                                  tw, scale, op));
    DD_LAUNCH_CHECK();
    return DD_OK;
    }
}

template <typename T, class Op>
int launch_x_prod_len(const char* name, int L, int nrows, int Kx, const CPtrs& win, const Ptrs& wout, int nrun,
                      int64_t in_rs, int64_t out_rs, const typename TwVec<T>::type* tw, T scale, const Op& op,
                      cudaStream_t st) {
    DD_CHECK_SUPPORTED(nrun >= 1 && nrun <= 65535, "run batch of %d not supported", nrun);
#define DD_XP(N) (launch_x_prod<T, N>(name, nrows, Kx, win, wout, nrun, in_rs, out_rs, tw, scale, op, st))
    switch (L) {
        DD_LEN_CASE(8, DD_XP(8))
        DD_LEN_CASE(16, DD_XP(16))
        DD_LEN_CASE(24, DD_XP(24))
        DD_LEN_CASE(48, DD_XP(48))
        DD_LEN_CASE(96, DD_XP(96))
        DD_LEN_CASE(192, DD_XP(192))
        DD_LEN_CASE(32, DD_XP(32))
        DD_LEN_CASE(64, DD_XP(64))
        DD_LEN_CASE(128, DD_XP(128))
        DD_LEN_CASE(256, DD_XP(256))
        DD_LEN_CASE(512, DD_XP(512))
        default: break;
    }
#undef DD_XP
    set_error("x length %d is not supported for %s%s", L, name, PrecName<T>::s);
    return DD_ERR_UNSUPPORTED;
}

}  // namespace dd
