// Transform passes: one kernel template moves a tile of pencils between
// global memory and shared memory around the pencil FFT engine.  The source
// and destination layouts (pruned/dealiased loads, compact intermediates,
// Hermitian packing of real rows, scaling) live in small "Op" structs whose
// load/store members are inlined into the kernel, so every pass is a single
// read and a single write of its data.
//
// Grid: x = (pencil tile) * nfield + field, y = slow index (up to 65535), z =
// slow index / 65535.  The field index varies fastest so that the blocks
// working on the same tile for different fields run together and re-reads of
// a shared input hit L2.
// LD_E / ST_E select whether consecutive threads walk elements (the pencil is
// contiguous in memory) or pencils (pencils are adjacent in memory), so global
// accesses stay coalesced.  Contiguous pencils are staged in the tile; adjacent
// ones go straight from global memory to the registers of the first butterflies
// and from those of the last ones back, so that the tile is written and read once
// per pass boundary only (FP32 at 256 points: y passes 97 -> 84 and 62 -> 50 us,
// z passes 68 -> 56 and 43 -> 34 us per launch of a 256^3 step, 3.5-3.9 -> 4.4-4.6
// TB/s).
#pragma once
#include <type_traits>
#include <utility>

#include "fft_fixed.cuh"
#include "geometry.cuh"

namespace dd {

// An Op whose pencils follow the 2/3 rule along the transform axis says so
// with kept() (its largest kept |mode index| there): an inverse Op's load then
// returns zero in the removed band and a forward Op's store never reads it,
// and the transform prunes that band when kept() == kept23(L).
template <class Op, class = void> struct HasKept : std::false_type {};
template <class Op>
struct HasKept<Op, std::void_t<decltype(std::declval<const Op&>().kept())>> : std::true_type {};

template <typename T, class S, bool INV, bool DIN, bool DOUT, class Op, class Ld, class St>
__device__ __forceinline__ void pass_fft(const Op& op, C<T>* tile, const C<T>* tw, Ld ld, St st) {
    if constexpr (HasKept<Op>::value && IsLF<T>::value) {   // one copy of the transform for double-float
        if (op.kept() == kept23(S::L)) { pencil_fft_io<T, S, INV, true, DIN, DOUT>(tile, tw, ld, st); return; }
    }
    pencil_fft_io<T, S, INV, false, DIN, DOUT>(tile, tw, ld, st);
}

// Global -> tile: the P contiguous pencils of L elements starting at pencil f0,
// pencils beyond npen zero.  Each thread loads its elements in groups of G into
// registers before storing any of the group to shared memory, so a group's
// global loads are in flight together (element-by-element load / store keeps
// one load in flight per thread: the shared stores may not move above the
// loads of generic pointers).
template <typename T, int L, int P, int PS, int NT, class Op>
__device__ __forceinline__ void load_tile(const Op& op, C<T>* tile, int fld, int s, int f0, int npen) {
    constexpr int N = L * P;
    constexpr int NPT = (N + NT - 1) / NT;
    constexpr int GB = (int)(128 / sizeof(C<T>));   // 128 bytes of loads per thread in flight
    constexpr int G = NPT < GB ? NPT : GB;
#pragma unroll
    for (int i0 = 0; i0 < NPT; i0 += G) {
        C<T> v[G];
#pragma unroll
        for (int i = 0; i < G; i++) {
            const int idx = threadIdx.x + (i0 + i) * NT;
            v[i] = zero<T>();
            if (i0 + i < NPT && (N % NT == 0 || idx < N)) {
                const int e = idx % L, p = idx / L;
                if (f0 + p < npen) v[i] = op.load(fld, s, e, f0 + p);
            }
        }
#pragma unroll
        for (int i = 0; i < G; i++) {
            const int idx = threadIdx.x + (i0 + i) * NT;
            if (i0 + i < NPT && (N % NT == 0 || idx < N)) {
                const int e = idx % L, p = idx / L;
                tile[e * PS + p] = v[i];
            }
        }
    }
}

// Index of element e of row s (rows of n elements of stride k) at kx, and of
// element s of the e-th such row.  The register path of the FP64 passes walks e in
// compile-time steps from one base; the staged path takes one product per entry
// (the other way round each was 5% slower).
template <typename T>
__device__ __forceinline__ int64_t row_at(int s, int e, int n, int k, int kx) {
    if constexpr (std::is_same<T, double>::value) return (int64_t)s * n * k + kx + e * k;
    else return ((int64_t)s * n + e) * k + kx;
}
template <typename T>
__device__ __forceinline__ int64_t pencil_at(int e, int s, int n, int k, int kx) {
    if constexpr (std::is_same<T, double>::value) return (int64_t)s * k + kx + (int64_t)e * (n * k);
    else return ((int64_t)e * n + s) * k + kx;
}

// How an Op of real rows maps to the FP64 transforms: 1 = c2r (packed half
// spectra in), 2 = r2c (half spectra out), 0 = complex pencils.
template <class Op> struct RealRows { static constexpr int kind = 0; };

template <class Op, class = void> struct HasPut : std::false_type {};
template <class Op>
struct HasPut<Op, std::void_t<decltype(&Op::put)>> : std::true_type {};

// Shared memory: the tile, the staged twiddles and (FP64) the pencils' scaling words.
template <typename T, class S>
constexpr size_t pass_smem() {
    constexpr int words = S::SKD ? fx_group_words<S>() : FX_WORDS * S::P;
    return S::template smem_bytes<T>() + (std::is_same<T, double>::value ? sizeof(unsigned) * words : 0);
}

// FP64: fixed-point transforms (fft_fixed.cuh).
template <class S, bool INV, bool LD_E, bool ST_E, bool PRUNE, class Op>
__device__ __forceinline__ void fx_pass_body(const Op& op, C<double>* tile, const int4* tw, unsigned* words, int fld, int s,
                                             int f0, int npen) {
    constexpr int L = S::L, P = S::P, PS = S::PS, NT = S::NT;
    constexpr int RR = RealRows<Op>::kind;
    if constexpr (RR != 0) {               // one thread group per pair of rows
        constexpr int TPP = S::TPP;
        const int p = threadIdx.x / TPP, jt = threadIdx.x % TPP, f = f0 + p;
        __syncthreads();
        if (f >= npen) return;
        if constexpr (RR == 1) {
            fx_group_c2r<S, PRUNE>(tile, tw, p, jt, op.Kx, words + 6 * p,
                                   [&](int k, C<double>& A, C<double>& B) { op.load_pair(fld, k, f, A, B); });
            for (int e = jt; e < L; e += TPP) op.put(fld, s, e, f, tile[S::off(e) + p]);
        } else {
            fx_group_r2c<S, PRUNE>(tile, tw, p, jt, op.Kx, op.sexp, op.smul, words + 6 * p,
                                   [&](int e) { return op.load(fld, s, e, f); },
                                   [&](int k, C<double> c) { op.put_row(fld, 2 * f, k, c); },
                                   [&](int k, C<double> c) { if (2 * f + 1 < op.nrows) op.put_row(fld, 2 * f + 1, k, c); });
        }
    } else {
        const int f = f0 + threadIdx.x % P;
        const auto ld = [&](int e) { return f < npen ? op.load(fld, s, e, f) : mk<double>(0., 0.); };
        const auto st = [&](int e, C<double> c) { if (f < npen) op.put(fld, s, e, f, c); };
        if constexpr (LD_E) {
            load_tile<double, L, P, PS, NT>(op, tile, fld, s, f0, npen);
            __syncthreads();
        }
        pencil_fx<S, INV, PRUNE, LD_E ? FX_IN_TILE : FX_IN_GLOBAL, ST_E ? FX_OUT_TILE : FX_OUT_GLOBAL>(tile, tw, words, ld, st);
        if constexpr (ST_E) {
            const int nst = op.nstore();
            for (int idx = threadIdx.x; idx < nst * P; idx += NT) {
                const int e = idx % nst, p = idx / nst;
                if (f0 + p < npen) op.put(fld, s, e, f0 + p, tile[e * PS + p]);
            }
        }
    }
}

template <typename T, class S, bool INV, bool LD_E, bool ST_E, int MB, class Op>
__global__ void __launch_bounds__(S::NT, MB) k_pass(const Op op, int nfield) {
    extern __shared__ __align__(16) unsigned char dd_smem[];
    constexpr int L = S::L, P = S::P, PS = S::PS, NT = S::NT;
    C<T>* tile = reinterpret_cast<C<T>*>(dd_smem);
    const int fld = blockIdx.x % nfield;
    const int f0 = (blockIdx.x / nfield) * P;
    const int s = blockIdx.y + 65535 * blockIdx.z;
    const int npen = op.npencil();
    if constexpr (std::is_same<T, double>::value) {
        int4* tw = reinterpret_cast<int4*>(tile + S::span);
        unsigned* words = reinterpret_cast<unsigned*>(tw + L);
        fx_stage_twiddles<L, INV>(tw, op.tw);
        if constexpr (RealRows<Op>::kind == 0)
            // columns beyond the last pencil hold zeros; the (doubled) high word of 1.0
            // keeps them out of the pre-scaled branch (64^3 rotating step 270.9 us, 272.6 without)
            for (int i = threadIdx.x; i < FX_WORDS * P; i += NT) words[i] = i < P && f0 + i >= npen ? 0x7fe00000u : 0u;
        grid_wait();
        if constexpr (HasKept<Op>::value) {
            if (op.kept() == kept23(L)) {
                fx_pass_body<S, INV, LD_E, ST_E, true>(op, tile, tw, words, fld, s, f0, npen);
                return;
            }
        }
        fx_pass_body<S, INV, LD_E, ST_E, false>(op, tile, tw, words, fld, s, f0, npen);
    } else {
        C<T>* tw = tile + L * PS;
        load_twiddles<T, L>(tw, op.tw);
        grid_wait();
        constexpr bool DIN = !LD_E, DOUT = !ST_E;
        if constexpr (LD_E) {
            load_tile<T, L, P, PS, NT>(op, tile, fld, s, f0, npen);
            __syncthreads();
        }
        const int f = f0 + threadIdx.x % P;
        const auto ld = [&](int e) { return f < npen ? op.load(fld, s, e, f) : zero<T>(); };
        const auto st = [&](int e, const C<T>& c) {
            if constexpr (HasPut<Op>::value) { if (f < npen) op.put(fld, s, e, f, c); }
        };
        pass_fft<T, S, INV, DIN, DOUT>(op, tile, tw, ld, st);
        if constexpr (ST_E) {
            const int nst = op.nstore();
            for (int idx = threadIdx.x; idx < nst * P; idx += NT) {
                const int e = idx % nst, p = idx / nst;
                if (f0 + p >= npen) continue;
                if constexpr (HasPut<Op>::value) op.put(fld, s, e, f0 + p, tile[e * PS + p]);
                else op.store(fld, s, e, f0 + p, tile + p, PS);
            }
        }
    }
}

// MB: resident blocks per SM that the registers have to allow (0: no demand).
template <typename T, class S, bool INV, bool LD_E, bool ST_E, int MB = 0, class Op>
int launch_pass_sched(const Op& op, int npencil, int nslow, int nfield, cudaStream_t st, const char* tag = "s") {
    constexpr size_t smem = pass_smem<T, S>();
    auto kern = k_pass<T, S, INV, LD_E, ST_E, MB, Op>;
    static std::atomic<unsigned long long> configured{0};  // per instantiation and device
    DD_TRY(ensure_smem((const void*)kern, smem, configured));
    if (npencil <= 0 || nslow <= 0 || nfield <= 0) return DD_OK;
    if (nslow > 65535 && nslow % 65535 != 0) {
        set_error("pass: slow extent %d must be <= 65535 or a multiple of it", nslow);
        return DD_ERR_UNSUPPORTED;
    }
    dim3 grid(cdiv(npencil, S::P) * nfield, nslow > 65535 ? 65535 : nslow, nslow > 65535 ? nslow / 65535 : 1);
    static const std::string label = std::string(Op::name) + "_" + std::to_string(S::L) + tag + PrecName<T>::s;
    DD_KT(label.c_str(), st, launch(kern, grid, S::NT, smem, st, op, nfield));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

// Schedule of the FP32 passes over y and z: DefSched with fewer pencils per tile
// at the lengths whose usual rows keep few modes (11, 16, 32 and 43; 32 or 64 pencils
// did up to 75% of the work for padding) and whose 256-thread blocks left SMs idle:
// FP32 hydro steps of 48^3 136 -> 131 us, 96^3 404 -> 376, 128^3 369 -> 339, MHD 128^3
// 639 -> 596.  No gain at 64 points; at 256, 22 and 29 pencils were slower than 16.
template <typename T, int L> struct NarrowSched { using S = DefSched<L>; };
template <> struct NarrowSched<float, 32> { using S = Sched<32, 16, 64, 8, 4, 1>; };
template <> struct NarrowSched<float, 48> { using S = Sched<48, 16, 64, 4, 4, 3>; };
template <> struct NarrowSched<float, 96> { using S = Sched<96, 16, 64, 8, 4, 3>; };
template <> struct NarrowSched<float, 128> { using S = Sched<128, 16, 128, 16, 8, 1>; };

// The pass with the default schedule of its length.  An explicit one (pencils
// per tile, threads, radix sequence) gives a small single-run grid enough
// blocks to fill the GPU: a 128-point y pass of 43 kx pencils is 6 tiles of the
// default 8 pencils (FP32: 3 of 16), but 11 tiles of 4.
template <typename T, int L, bool INV, bool LD_E, bool ST_E, class Op>
int launch_pass(const Op& op, int npencil, int nslow, int nfield, cudaStream_t st) {
    if constexpr (std::is_same<T, double>::value && RealRows<Op>::kind != 0) {
        // 128 threads: no barriers between groups, and a block's shared memory is
        // free sooner (192x128x256 there and back 504 us with 256, 497 with 128); 256
        // at 512 points (64x128x512: 362 against 383)
        constexpr int TPP = FxRowTPP<L>::v, P = TPP == 64 ? 4 : TPP >= 2 ? 128 / TPP : 64;
        return launch_pass_sched<T, FxR<L, INV, P>, INV, LD_E, ST_E, 1024 / (P * TPP)>(op, npencil, nslow, nfield, st, "");
    } else if constexpr (std::is_same<T, double>::value)
        return launch_pass_sched<T, FxS<L, INV>, INV, LD_E, ST_E, FxCfg<L>::MB>(op, npencil, nslow, nfield, st, "");
    else {   // FP32 inverse passes at 256 points: 5 blocks (48 registers) gain 4% on 4, forward ones spill
        using S = std::conditional_t<LD_E || ST_E, DefSched<L>, typename NarrowSched<T, L>::S>;
        return launch_pass_sched<T, S, INV, LD_E, ST_E, (std::is_same<T, float>::value && L == 256 && INV ? 5 : 0)>(
            op, npencil, nslow, nfield, st, "");
    }
}

// Small-tile schedules for single-run 2D grids: 4 pencils of 16 threads, and at
// 256 and 512 points 2 pencils of the usual threads and radices (a 512-point y pass of
// 171 kx pencils of 3 fields is 66 tiles of 8, or 258 of 2, for 152 SMs: a 512^2
// convection step takes 181 us, 195 with 8; a 512^2 hydro step 138, 146 with 8).  The
// lengths 48, 96 and 192 keep the wide tiles: graphs of single steps of 48^2, 96^2 and
// 192^2 take 794, 813 and 816 us in FP64 (most of it phi functions without tables), 793,
// 811 and 812 with tiles of 4, 2 and 2, but 807, 832 and 837 against 800, 820 and 837 in FP32.
template <typename T, int L, bool INV> struct SmallSched { using S = Sched<L, 2, 2 * DefSched<L>::TPP, DefSched<L>::R1, DefSched<L>::R2, DefSched<L>::R3>; };
template <int L, bool INV> struct SmallSched<double, L, INV> { using S = FxS<L, INV, 2>; };
template <typename T, bool INV> struct SmallSched<T, 64, INV> { using S = Sched<64, 4, 64, 4, 4, 4>; };
template <typename T, bool INV> struct SmallSched<T, 128, INV> { using S = Sched<128, 4, 64, 8, 4, 4>; };
template <bool INV> struct SmallSched<double, 64, INV> { using S = Sched<64, 4, 64, 4, 4, 4>; };
template <bool INV> struct SmallSched<double, 128, INV> { using S = Sched<128, 4, 64, 8, 4, 4>; };

// Launch a pass with the small-tile schedule when one exists for length L;
// returns 1 (not launched) otherwise.
template <typename T, bool INV, bool LD_E, bool ST_E, class Op>
int launch_pass_small(int L, const Op& op, int npencil, int nslow, int nfield, cudaStream_t st) {
#define DD_SMALL(N) \
    if (L == N) return launch_pass_sched<T, typename SmallSched<T, N, INV>::S, INV, LD_E, ST_E>(op, npencil, nslow, nfield, st);
    DD_SMALL(64)
    DD_SMALL(128)
    DD_SMALL(256)
    DD_SMALL(512)
#undef DD_SMALL
    return 1;
}

// Tile variants of the default schedule for the 2D y passes of 64..512-point
// grids, chosen per plan by the ensemble autotuner (dd_plan_set_schedule):
// the same radix sequence as the default (so every pencil's arithmetic, and
// its result, is identical) on fewer pencils per block: variant 1 the
// smallest tile (2-4 pencils), variant 2 a middle one (4-8 pencils).  The FP64
// default has 8 pencils itself, so that at 64 and 128 points variant 2 is the
// default; 2 pencils in its place are never faster than 4 and slower for many
// runs (a step of 64 runs of 128^2 240 us, 217 with 4 or 8 pencils).  A single run's
// default is a small tile already (SmallSched): at 256 and 512 points FP64 variant 1.
// The ensemble autotuner leaves these equal ones out.
constexpr int kYSchedVariants = 3;
template <int L, int V> struct YVariant;
template <> struct YVariant<64, 1>  { using S = Sched<64, 4, 32, 8, 8, 1>; };
template <> struct YVariant<64, 2>  { using S = Sched<64, 8, 64, 8, 8, 1>; };
template <> struct YVariant<128, 1> { using S = Sched<128, 4, 32, 16, 8, 1>; };
template <> struct YVariant<128, 2> { using S = Sched<128, 8, 64, 16, 8, 1>; };
template <> struct YVariant<256, 1> { using S = Sched<256, 4, 64, 16, 16, 1>; };
template <> struct YVariant<256, 2> { using S = Sched<256, 8, 128, 16, 16, 1>; };
template <> struct YVariant<512, 1> { using S = Sched<512, 2, 64, 8, 8, 8>; };
template <> struct YVariant<512, 2> { using S = Sched<512, 4, 128, 8, 8, 8>; };
template <typename T, int L, int V, bool INV>
struct YSchedOf { using S = typename YVariant<L, V>::S; };
template <int L, int V, bool INV>
struct YSchedOf<double, L, V, INV> {
    static constexpr int P = L <= 128 ? 4 * V : 2 * V;
    using S = FxS<L, INV, P>;
};

// Launch a pass with tile variant v (1 or 2) of length L; returns 1 (not
// launched) when no variant exists.
template <typename T, bool INV, bool LD_E, bool ST_E, class Op>
int launch_pass_variant(int L, int v, const Op& op, int npencil, int nslow, int nfield, cudaStream_t st) {
#define DD_YV(N, VV) \
    if (L == N && v == VV) \
        return launch_pass_sched<T, typename YSchedOf<T, N, VV, INV>::S, INV, LD_E, ST_E>(op, npencil, nslow, nfield, st);
    DD_YV(64, 1) DD_YV(64, 2) DD_YV(128, 1) DD_YV(128, 2) DD_YV(256, 1) DD_YV(256, 2) DD_YV(512, 1) DD_YV(512, 2)
#undef DD_YV
    return 1;
}

// ============================================================ 3D operators
// Inverse along kz: K[ky][kz][kx] (kept entries) -> W1[kyc][z][kxc].
template <typename T, typename KT>
struct OpZInv3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "z_inv";
    static constexpr int lmin = 8, lmax = 512;
    using KV = typename Vec2<KT>::type;
    Geo3 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.Mz; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Nz; }
    __device__ C<T> load(int fld, int kyc, int e, int kx) const {
        if (!kept_full(e, g.Nz, g.Mz)) return zero<T>();
        const int ky = compact_to_full(kyc, g.Ny, g.Ky);
        const KV v = ((const KV*)in.p[fld])[row_at<T>(ky, e, g.Nz, g.Nh, kx)];
        return mk<T>((T)v.x, (T)v.y);
    }
    __device__ void put(int fld, int kyc, int e, int kx, const C<T>& c) const {
        stc<T>((V*)out.p[fld] + row_at<T>(kyc, e, g.Nz, g.Kx, kx), c);
    }
};

// Inverse along ky: W1[kyc][z][kxc] -> W2[z][y][kxc].
template <typename T>
struct OpYInv3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "y_inv";
    static constexpr int lmin = 8, lmax = 512;
    Geo3 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.My; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Ny; }
    __device__ C<T> load(int fld, int z, int e, int kx) const {
        if (!kept_full(e, g.Ny, g.My)) return zero<T>();
        const int kyc = full_to_compact(e, g.Ny, g.Ky);
        return ldc<T>((const V*)in.p[fld] + pencil_at<T>(kyc, z, g.Nz, g.Kx, kx));
    }
    __device__ void put(int fld, int z, int e, int kx, const C<T>& c) const {
        stc<T>((V*)out.p[fld] + row_at<T>(z, e, g.Ny, g.Kx, kx), c);
    }
};

// Hermitian packing of two half-spectrum rows A, B (kx < Kx) into one full
// complex sequence Z = A + iB whose inverse DFT is a + ib.  The imaginary
// parts at kx = 0 and kx = N/2 are dropped, as a c2r transform does.
template <typename T, typename V>
__device__ __forceinline__ C<T> pack_rows(const V* ra, const V* rb, int e, int N, int K) {
    const int kx = e <= N / 2 ? e : N - e;
    if (kx >= K) return zero<T>();
    C<T> A = ldc<T>(ra + kx), B = ldc<T>(rb + kx);
    if (kx == 0 || 2 * kx == N) { A.y = T(0); B.y = T(0); }
    if (e > N / 2) { A.y = -A.y; B.y = -B.y; }
    return mk<T>(A.x - B.y, A.y + B.x);
}

// Separation of the forward DFT Z of a + ib into the half spectra A (a), B (b)
// at bin k, times s, from z = Z[k] and zn = Z[N - k] (Z[0] at k = 0).
template <typename T>
__device__ __forceinline__ void unpack_pair(C<T> z, C<T> zn, T s, C<T>& A, C<T>& B) {
    const T h = T(0.5) * s;
    A = mk<T>((z.x + zn.x) * h, (z.y - zn.y) * h);
    B = mk<T>((z.y + zn.y) * h, (zn.x - z.x) * h);
}

// The same with Z read from a tile column of row stride PS.
template <typename T>
__device__ __forceinline__ void unpack_rows(const C<T>* col, int PS, int k, int N, T s, C<T>& A, C<T>& B) {
    unpack_pair<T>(col[k * PS], col[(k == 0 ? 0 : N - k) * PS], s, A, B);
}

// c2r along x: W2 rows [r][kxc] (r = z*Ny + y) -> x rows; pencil f = row pair.
template <typename T, typename XT>
struct OpXc2r3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "x_c2r";
    static constexpr int lmin = 8, lmax = 512;
    int nrows, Nx, Kx; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return Kx - 1; }
    __device__ int npencil() const { return (nrows + 1) / 2; }
    __device__ int nstore() const { return Nx; }
    __device__ C<T> load(int fld, int, int e, int f) const {
        const V* W = (const V*)in.p[fld];
        const int ra = 2 * f, rb = min(2 * f + 1, nrows - 1);
        C<T> z = pack_rows<T>(W + (int64_t)ra * Kx, W + (int64_t)rb * Kx, e, Nx, Kx);
        if (rb == ra) z.y = T(0);
        return z;
    }
    // the half spectra of pencil f's two rows at kx = k
    __device__ void load_pair(int fld, int k, int f, C<T>& A, C<T>& B) const {
        const V* W = (const V*)in.p[fld] + (int64_t)(2 * f) * Kx + k;
        A = ldc<T>(W);
        if (2 * f + 1 < nrows) B = ldc<T>(W + Kx);
    }
    __device__ void put(int fld, int, int e, int f, const C<T>& v) const {
        XT* x = (XT*)out.p[fld];
        x[(int64_t)(2 * f) * Nx + e] = (XT)v.x;
        if (2 * f + 1 < nrows) x[(int64_t)(2 * f + 1) * Nx + e] = (XT)v.y;
    }
};

// r2c along x: x rows -> W2 rows [r][kxc], scaled by s (the 1/N of the
// reference's forward transform).
template <typename T, typename XT>
struct OpXr2c3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "x_r2c";
    static constexpr int lmin = 8, lmax = 512;
    int nrows, Nx, Kx; T s; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    int sexp = 0; double smul = 1.0;       // s = 2^sexp smul (fx_split_scale; FP64 only)
    __device__ int kept() const { return Kx - 1; }
    __device__ int npencil() const { return (nrows + 1) / 2; }
    __device__ int nstore() const { return Kx; }
    __device__ C<T> load(int fld, int, int e, int f) const {
        const XT* x = (const XT*)in.p[fld];
        const T a = (T)x[(int64_t)(2 * f) * Nx + e];
        const T b = (2 * f + 1 < nrows) ? (T)x[(int64_t)(2 * f + 1) * Nx + e] : T(0);
        return mk<T>(a, b);
    }
    __device__ void store(int fld, int, int k, int f, const C<T>* col, int PS) const {
        C<T> A, B;
        unpack_rows<T>(col, PS, k, Nx, s, A, B);
        V* W = (V*)out.p[fld];
        stc<T>(W + (int64_t)(2 * f) * Kx + k, A);
        if (2 * f + 1 < nrows) stc<T>(W + (int64_t)(2 * f + 1) * Kx + k, B);
    }
    __device__ void put_row(int fld, int row, int k, C<T> c) const { stc<T>((V*)out.p[fld] + (int64_t)row * Kx + k, c); }
};
template <typename XT> struct RealRows<OpXc2r3<double, XT>> { static constexpr int kind = 1; };
template <typename XT> struct RealRows<OpXr2c3<double, XT>> { static constexpr int kind = 2; };

// Forward along y: W2[z][y][kxc] -> W1[kyc][z][kxc] (kept ky only).
template <typename T>
struct OpYFwd3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "y_fwd";
    static constexpr int lmin = 8, lmax = 512;
    Geo3 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.My; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Ny; }
    __device__ C<T> load(int fld, int z, int e, int kx) const {
        return ldc<T>((const V*)in.p[fld] + row_at<T>(z, e, g.Ny, g.Kx, kx));
    }
    __device__ void put(int fld, int z, int e, int kx, const C<T>& c) const {
        if (!kept_full(e, g.Ny, g.My)) return;
        const int kyc = full_to_compact(e, g.Ny, g.Ky);
        stc<T>((V*)out.p[fld] + pencil_at<T>(kyc, z, g.Nz, g.Kx, kx), c);
    }
};

// Forward along z: W1[kyc][z][kxc] -> K[ky][kz][kx] (kept ky, kx < Kx); the
// non-kept kz entries of those columns are written as zeros.
template <typename T, typename KT>
struct OpZFwd3 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "z_fwd";
    static constexpr int lmin = 8, lmax = 512;
    using KV = typename Vec2<KT>::type;
    Geo3 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.Mz; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Nz; }
    __device__ C<T> load(int fld, int kyc, int e, int kx) const {
        return ldc<T>((const V*)in.p[fld] + row_at<T>(kyc, e, g.Nz, g.Kx, kx));
    }
    __device__ void put(int fld, int kyc, int e, int kx, const C<T>& c) const {
        const int ky = compact_to_full(kyc, g.Ny, g.Ky);
        KV v;
        if (kept_full(e, g.Nz, g.Mz)) {  v.x = (KT)c.x; v.y = (KT)c.y; }
        else { v.x = KT(0); v.y = KT(0); }
        ((KV*)out.p[fld])[row_at<T>(ky, e, g.Nz, g.Nh, kx)] = v;
    }
};

// ============================================================ 2D operators
// Inverse along ky: K[kx][ky] (kept) -> W[y][kxc]; pencil = kx row.
template <typename T, typename KT>
struct OpYInv2 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "y_inv2d";
    static constexpr int lmin = 8, lmax = 512;
    using KV = typename Vec2<KT>::type;
    Geo2 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.My; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Ny; }
    __device__ C<T> load(int fld, int, int e, int kx) const {
        if (!kept_full(e, g.Ny, g.My)) return zero<T>();
        const KV v = ((const KV*)in.p[fld])[(int64_t)kx * g.Ny + e];
        return mk<T>((T)v.x, (T)v.y);
    }
    __device__ void put(int fld, int, int e, int kx, const C<T>& c) const {
        stc<T>((V*)out.p[fld] + row_at<T>(0, e, 0, g.Kx, kx), c);
    }
};

// Forward along y: W[y][kxc] -> K[kx][ky] (all ky; zeros where not kept).
template <typename T, typename KT>
struct OpYFwd2 {
    using V = typename Vec2<T>::type;
    static constexpr const char* name = "y_fwd2d";
    static constexpr int lmin = 8, lmax = 512;
    using KV = typename Vec2<KT>::type;
    Geo2 g; CPtrs in; Ptrs out; const typename TwVec<T>::type* tw;
    __device__ int kept() const { return g.My; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Ny; }
    __device__ C<T> load(int fld, int, int e, int kx) const {
        return ldc<T>((const V*)in.p[fld] + row_at<T>(0, e, 0, g.Kx, kx));
    }
    __device__ void put(int fld, int, int e, int kx, const C<T>& c) const {
        KV v;
        if (kept_full(e, g.Ny, g.My)) {  v.x = (KT)c.x; v.y = (KT)c.y; }
        else { v.x = KT(0); v.y = KT(0); }
        ((KV*)out.p[fld])[(int64_t)kx * g.Ny + e] = v;
    }
};

}  // namespace dd
