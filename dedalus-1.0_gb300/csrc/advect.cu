// 3D right-hand sides in the advective form of the reference, with rotation and
// buoyancy, on a static Fourier basis:
//   du = P[-(u.grad)u - 2 Omega x u + g alpha T e_dir],  dT = -(u.grad)T - beta u_dir
// (physics.py:527-599, 664-712).  One call runs what generic.py otherwise issues
// as one kernel per numpy operation (about 170 launches per 3D Boussinesq RHS,
// host-bound at 64^3: 1.65 ms): five transform passes over all fields at once, with
// the gradients formed while loading and the products inside the x pass, and one
// pointwise kernel.  Products, sums and pointwise terms keep the reference's order
// with one rounding per operation; modes outside the kept set carry only the
// linear terms.  FP64.
#include "rhs3d_impl.cuh"

namespace dd {

// Inverse along kz of u (fields 0..2) and of d_i Y_c (field 3 + 3 c + i; Y = u, then
// the scalar), i k_i formed as it is loaded (representations.py:419-425).
struct OpZInvAdv3 {
    using V = double2;
    static constexpr const char* name = "z_inv_grad";
    static constexpr int lmin = 16, lmax = 512;
    Geo3 g; CPtrs u; Ptrs out; const int4* tw;
    const double* kx; const double* ky; const double* kz;
    __device__ int kept() const { return g.Mz; }
    __device__ int npencil() const { return g.Kx; }
    __device__ int nstore() const { return g.Nz; }
    __device__ C<double> load(int fld, int kyc, int e, int ix) const {
        if (!kept_full(e, g.Nz, g.Mz)) return zero<double>();
        const int ky_i = compact_to_full(kyc, g.Ny, g.Ky);
        const int c = fld < 3 ? fld : (fld - 3) / 3, i = fld < 3 ? 3 : (fld - 3) % 3;
        double2 v = ((const double2*)u.p[c])[row_at<double>(ky_i, e, g.Nz, g.Nh, ix)];
        if (i < 3) v = ideriv(v, i == 0 ? kx[ix] : i == 1 ? ky[ky_i] : kz[e]);
        return mk<double>(v.x, v.y);
    }
    __device__ void put(int fld, int kyc, int e, int ix, const C<double>& c) const {
        stc<double>((V*)out.p[fld] + row_at<double>(kyc, e, g.Nz, g.Kx, ix), c);
    }
};

// (u.grad) Y_c = ((d_x Y u_x) + d_y Y u_y) + d_z Y u_z for NS components.
template <int NS>
struct ProdAdv3 {
    static constexpr int NI = 3 + 3 * NS, NO = NS;
    static constexpr int lmin = 16, lmax = 512;
    __device__ void operator()(const double* in, double* out, int) const {
#pragma unroll
        for (int c = 0; c < NS; c++) {
            const double* d = in + 3 + 3 * c;
            out[c] = radd(radd(rmul(d[0], in[0]), rmul(d[1], in[1])), rmul(d[2], in[2]));
        }
    }
};

struct AdvArgs {
    Geo3 g;
    const double* kx; const double* ky; const double* kz;
    CPtrs adv;              // (u.grad) Y, compact
    CPtrs y;                // u, T
    Ptrs d;                 // du, dT
    double2* ms;            // work fields of the operator sequence as it leaves them, or null
    double2* mv[3];
    int rotation, ns, dir;
    double om[3], gg, alpha_t, beta;
};

// All modes of the full layout, one per thread, bound by the FP64 pipe.  128-thread
// blocks: 64^3 is 6.9 per SM, where 3.5 of 256 threads leave half a wave idle (27 us
// at 64^3; 31 with those and a predicated buoyancy addition per axis).
// a.ms, a.mv: what the sequence leaves in its work fields.  Without a scalar the
// pressure term and Omega x u (without rotation the kept u), with one
// beta u_dir and the kept u.
__global__ void __launch_bounds__(128) k_advect_tail3(AdvArgs a) {
    grid_wait();
    const Geo3& g = a.g;
    const int64_t n = g.kcount();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int ix = (int)(i % g.Nh);
        const int r = (int)(i / g.Nh);
        const int kz_i = r % g.Nz, ky_i = r / g.Nz;
        const bool kept = ix < g.Kx && kept_full(ky_i, g.Ny, g.My) && kept_full(kz_i, g.Nz, g.Mz);
        double2 N[4];
#pragma unroll
        for (int c = 0; c < 4; c++) N[c] = make_double2(0., 0.);
        if (kept) {
            const int64_t j =
                ((int64_t)full_to_compact(ky_i, g.Ny, g.Ky) * g.Kz + full_to_compact(kz_i, g.Nz, g.Kz)) * g.Kx + ix;
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (c < a.ns) {
                    const double2 v = ((const double2*)a.adv.p[c])[j];
                    N[c] = make_double2(-v.x, -v.y);
                }
        }
        double2 u[3];
#pragma unroll
        for (int c = 0; c < 3; c++) u[c] = ((const double2*)a.y.p[c])[i];
        if (a.rotation) {       // physics.py:266-307, 548-551: N -= 2 Omega x u
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int p = (c + 1) % 3, q = (c + 2) % 3;
                const double2 m = make_double2(radd(rmul(u[q].x, a.om[p]), rmul(u[p].x, -a.om[q])),
                                               radd(rmul(u[q].y, a.om[p]), rmul(u[p].y, -a.om[q])));
                N[c] = make_double2(radd(N[c].x, rmul(m.x, -2.)), radd(N[c].y, rmul(m.y, -2.)));
                if (a.ms && a.ns == 3) a.mv[c][i] = m;
            }
        }
        if (a.ms && (a.ns == 4 || !a.rotation)) {
#pragma unroll
            for (int c = 0; c < 3; c++) a.mv[c][i] = kept ? u[c] : make_double2(0., 0.);
        }
        if (a.ns == 4) {        // physics.py:688-708
            const double2 T = ((const double2*)a.y.p[3])[i];
            const double2 b = make_double2(rmul(rmul(T.x, a.gg), a.alpha_t), rmul(rmul(T.y, a.gg), a.alpha_t));
            // one addition and selects: a predicated one per axis takes the FP64 pipe three times
            const double2 ud = a.dir == 0 ? u[0] : a.dir == 1 ? u[1] : u[2];
            double2 nd = a.dir == 0 ? N[0] : a.dir == 1 ? N[1] : N[2];
            nd = make_double2(radd(nd.x, b.x), radd(nd.y, b.y));
            if (a.dir == 0) N[0] = nd;
            else if (a.dir == 1) N[1] = nd;
            else N[2] = nd;
            const double2 bu = make_double2(rmul(ud.x, a.beta), rmul(ud.y, a.beta));
            ((double2*)a.d.p[3])[i] = make_double2(rsub(N[3].x, bu.x), rsub(N[3].y, bu.y));
            if (a.ms) a.ms[i] = bu;
        }
        // pressure projection (physics.py:588-599, 407-416)
        const double kxv = a.kx[ix], kyv = a.ky[ky_i], kzv = a.kz[kz_i];
        const double k2 = radd(radd(rmul(kyv, kyv), rmul(kzv, kzv)), rmul(kxv, kxv));
        const double s = rdiv(1., k2 == 0. ? 1. : k2);
        const double2 dx = ideriv(N[0], kxv), dy = ideriv(N[1], kyv), dz = ideriv(N[2], kzv);
        const double2 dv = make_double2(radd(radd(dx.x, dy.x), dz.x), radd(radd(dx.y, dy.y), dz.y));
        const double2 ph = make_double2(-rmul(dv.x, s), -rmul(dv.y, s));
        if (a.ms && a.ns == 3) a.ms[i] = ph;
        const double2 gr[3] = {ideriv(ph, kxv), ideriv(ph, kyv), ideriv(ph, kzv)};
#pragma unroll
        for (int c = 0; c < 3; c++)
            ((double2*)a.d.p[c])[i] = make_double2(rsub(N[c].x, gr[c].x), rsub(N[c].y, gr[c].y));
    }
}

template <int NS>
static Work3 adv_work(const Geo3& g, void* base) {
    return Work3{(size_t)g.w1count(), (size_t)g.w2count(), (size_t)g.Ky * g.Kz * g.Kx, 3 + 3 * NS, NS, 0, (char*)base};
}

template <int NS>
static int advect_rhs3d(const dd_plan* p, AdvArgs& a, void* work, size_t wb, cudaStream_t st) {
    const Geo3& g = p->g3;
    constexpr int NI = 3 + 3 * NS;
    static_assert(NI <= DD_MAXF, "too many transform fields for Ptrs");
    const size_t need = Work3::bytes<double>(g, NI, NS, 0, false);
    DD_CHECK_ARG(wb >= need, "workspace too small: %zu < %zu", wb, need);
    const Work3 w = adv_work<NS>(g, work);
    Ptrs w1{}, w2{}, nc{};
    CPtrs w1c{}, w2c{};
    for (int f = 0; f < NI; f++) {
        w1c.p[f] = w1.p[f] = w.W1<double>(f);
        w2c.p[f] = w2.p[f] = w.W2<double>(f);
    }
    for (int c = 0; c < NS; c++) a.adv.p[c] = nc.p[c] = w.NC<double>(c);
    OpZInvAdv3 z{g, a.y, w1, p->tw64_z, p->kx, p->ky, p->kz};
    DD_TRY((launch_pass_len<double, true, false, false>(g.Nz, z, g.Kx, g.Ky, NI, st)));
    OpYInv3<double> y{g, w1c, w2, p->tw64_y};
    DD_TRY((launch_pass_len<double, true, false, false>(g.Ny, y, g.Kx, g.Nz, NI, st)));
    // products overwrite fields 0..NS-1 of W2 row by row (each block reads its rows first)
    DD_TRY((launch_x_prod_len<double>("x_advect", g.Nx, g.Nz * g.Ny, g.Kx, w2c, w2, 1, 0, 0, p->tw64_x, p->inv_n,
                                      ProdAdv3<NS>{}, st)));
    OpYFwd3<double> yf{g, w2c, w1, p->tw64_y};
    DD_TRY((launch_pass_len<double, false, false, false>(g.Ny, yf, g.Kx, g.Nz, NS, st)));
    OpZFwdCompact3<double> zf{g, w1c, nc, p->tw64_z};
    DD_TRY((launch_pass_len<double, false, false, false>(g.Nz, zf, g.Kx, g.Ky, NS, st)));
    const int64_t n = g.kcount();
    DD_KT("advect_tail3", st, launch(k_advect_tail3, (unsigned)(n > 152 * 32 * 128 ? 152 * 32 : (n + 127) / 128), 128, 0, st, a));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

}  // namespace dd

using namespace dd;

extern "C" {

int dd_advect_workspace_size(const dd_plan* p, int nscalar, size_t* bytes) {
    DD_CHECK_ARG(p && bytes, "dd_advect_workspace_size: null pointer");
    DD_CHECK_SUPPORTED(p->ndim == 3, "dd_advect_rhs3d: the plan must be 3D");
    DD_CHECK_ARG(nscalar == 0 || nscalar == 1, "dd_advect_rhs3d: nscalar must be 0 or 1");
    *bytes = Work3::bytes<double>(p->g3, nscalar ? 15 : 12, 3 + nscalar, 0, false);
    return DD_OK;
}

int dd_advect_rhs3d_aux(const dd_plan* p, int nscalar, const double* omega, const double* params, const void* const* state,
                        void* const* deriv, void* const* aux, void* work, size_t work_bytes, void* stream) {
    DD_CHECK_ARG(p && state && deriv && work, "dd_advect_rhs3d: null pointer");
    DD_CHECK_SUPPORTED(p->ndim == 3, "dd_advect_rhs3d: the plan must be 3D");
    DD_CHECK_ARG(nscalar == 0 || nscalar == 1, "dd_advect_rhs3d: nscalar must be 0 or 1");
    DD_CHECK_ARG(!nscalar || params, "dd_advect_rhs3d: a scalar needs its parameters");
    AdvArgs a{};
    a.g = p->g3;
    a.kx = p->kx; a.ky = p->ky; a.kz = p->kz;
    a.rotation = omega != nullptr;
    for (int c = 0; c < 3; c++) a.om[c] = omega ? omega[c] : 0.;
    a.ns = 3 + nscalar;
    if (nscalar) {
        a.gg = params[0]; a.alpha_t = params[1]; a.beta = params[2];
        a.dir = (int)params[3];
        DD_CHECK_ARG(a.dir >= 0 && a.dir < 3, "dd_advect_rhs3d: direction %d out of range", a.dir);
    }
    for (int c = 0; c < a.ns; c++) {
        DD_CHECK_ARG(state[c] && deriv[c], "dd_advect_rhs3d: null component pointer %d", c);
        a.y.p[c] = state[c];
        a.d.p[c] = deriv[c];
    }
    if (aux) {
        for (int c = 0; c < 4; c++) DD_CHECK_ARG(aux[c], "dd_advect_rhs3d: null work field %d", c);
        a.ms = (double2*)aux[0];
        for (int c = 0; c < 3; c++) a.mv[c] = (double2*)aux[1 + c];
    }
    const cudaStream_t st = (cudaStream_t)stream;
    return nscalar ? advect_rhs3d<4>(p, a, work, work_bytes, st) : advect_rhs3d<3>(p, a, work, work_bytes, st);
}

int dd_advect_rhs3d(const dd_plan* p, int nscalar, const double* omega, const double* params, const void* const* state,
                    void* const* deriv, void* work, size_t work_bytes, void* stream) {
    return dd_advect_rhs3d_aux(p, nscalar, omega, params, state, deriv, nullptr, work, work_bytes, stream);
}

}  // extern "C"
