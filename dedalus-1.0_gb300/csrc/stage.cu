// Stage-update kernels with the reference's Cython signatures
// (forward_step_cy_3d.pyx:17-124, forward_step_cy_2d.pyx:21-120) and the
// phi-function table used by the fused timesteppers.
#include "dd_common.cuh"
#include "etd.cuh"
#include "geometry.cuh"

namespace dd {

__global__ void k_euler(const double2* __restrict__ s, double2* o, const double2* __restrict__ d,
                        double dt, int64_t n) {
    grid_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 a = s[i], b = d[i];
        double2 r;
        r.x = radd(a.x, rmul(dt, b.x));
        r.y = radd(a.y, rmul(dt, b.y));
        o[i] = r;
    }
}

template <int NDIM>
__global__ void k_etd1(const double2* s, double2* o, const double2* __restrict__ d,
                       const double* __restrict__ intf, double dt, int64_t n) {
    grid_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double Z = rmul(intf[i], dt);
        double f0 = 1., f1 = 1., f2 = 0.5;
        if (Z != 0.) etd_phis<NDIM>(Z, f0, f1, f2);
        o[i] = etd1_entry(s[i], d[i], Z, f0, f1, dt);
    }
}

template <int NDIM>
__global__ void k_etd2rk1(const double2* s, double2* o, const double2* __restrict__ d1,
                          const double2* __restrict__ d2, const double* __restrict__ intf,
                          double dt, int64_t n) {
    grid_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double Z = rmul(intf[i], dt);
        double f0 = 1., f1 = 1., f2 = 0.5;
        if (Z != 0.) etd_phis<NDIM>(Z, f0, f1, f2);
        o[i] = etd2rk1_entry(s[i], d1[i], d2[i], Z, f2, dt);
    }
}

template <int NDIM>
__global__ void k_etd2rk2(const double2* s, double2* o, const double2* __restrict__ d1,
                          const double2* __restrict__ d2, const double* __restrict__ intf,
                          double dt, int64_t n) {
    grid_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double Z = rmul(intf[i], dt);
        double f0 = 1., f1 = 1., f2 = 0.5;
        if (Z != 0.) etd_phis<NDIM>(Z, f0, f1, f2);
        o[i] = etd2rk2_entry(s[i], d1[i], d2[i], Z, f0, f1, f2, dt);
    }
}

// One stage update of up to ETD_FIELDS fields: SCHEME 0 etd1, 1 etd2rk1, 2 etd2rk2.
// Bound by the FP64 pipe (exp and a polynomial or two divisions per entry, 43-48 us
// per field of 64^3), so a thread takes one entry of all fields and evaluates the
// phi functions anew only where the factor differs from the field before (the
// components of u share theirs): the 8 updates of a 64^3 rotating Boussinesq
// RK2trap step took 365 us of 515 as one launch per field, and take 107 of 270 as
// two launches.  Blocks of 128 threads: 64^3 is
// 6.9 of them per SM, where 3.5 of 256 leave half a wave idle.
constexpr int ETD_FIELDS = 6;
struct EtdFields {
    int nf;
    const double2* s[ETD_FIELDS];
    double2* o[ETD_FIELDS];
    const double2* d1[ETD_FIELDS];
    const double2* d2[ETD_FIELDS];
    const double* intf[ETD_FIELDS];
};

template <int NDIM, int SCHEME>
__global__ void __launch_bounds__(128) k_etd_fields(EtdFields a, double dt, int64_t n) {
    grid_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double Zp = 0., f0 = 1., f1 = 1., f2 = 0.5;
#pragma unroll 1
        for (int f = 0; f < a.nf; f++) {
            const double Z = rmul(pick_ptr<ETD_FIELDS>(a.intf, f)[i], dt);
            const double2 s = pick_ptr<ETD_FIELDS>(a.s, f)[i], d1 = pick_ptr<ETD_FIELDS>(a.d1, f)[i];
            if (Z != Zp) {
                if (Z != 0.) etd_phis<NDIM>(Z, f0, f1, f2);
                Zp = Z;
            }
            double2* o = pick_ptr<ETD_FIELDS>(a.o, f);
            if (SCHEME == 0) o[i] = etd1_entry(s, d1, Z, f0, f1, dt);
            else if (SCHEME == 1) o[i] = etd2rk1_entry(s, d1, pick_ptr<ETD_FIELDS>(a.d2, f)[i], Z, f2, dt);
            else o[i] = etd2rk2_entry(s, d1, pick_ptr<ETD_FIELDS>(a.d2, f)[i], Z, f0, f1, f2, dt);
        }
    }
}

template <int NDIM>
static void launch_etd_fields(int scheme, const EtdFields& a, double dt, int64_t n, cudaStream_t st) {
    const int64_t nb = (n + 127) / 128;
    const unsigned b = (unsigned)(nb > 152 * 64 ? 152 * 64 : nb);
    if (scheme == 0) DD_KT("etd1_fields", st, launch(k_etd_fields<NDIM, 0>, b, 128, 0, st, a, dt, n));
    else if (scheme == 1) DD_KT("etd2rk1_fields", st, launch(k_etd_fields<NDIM, 1>, b, 128, 0, st, a, dt, n));
    else DD_KT("etd2rk2_fields", st, launch(k_etd_fields<NDIM, 2>, b, 128, 0, st, a, dt, n));
}

// table[q] = {Z, f0, f1, f2} for integer squared wavenumber q with
// Z = -(nu * q**vo) * h, i.e. the reference's intfactor * dt for k2 == q.
template <int NDIM>
__global__ void k_phi_table(double nu, int vo, double h, int qmax, double4* tab) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > qmax) return;
    const double k2 = (double)q;
    double k2v = (vo == 1) ? k2 : (vo == 2 ? rmul(k2, k2) : pow(k2, (double)vo));
    const double IF = rmul(nu, k2v);
    const double Z = rmul(-IF, h);
    double f0 = 1., f1 = 1., f2 = 0.5;
    if (Z != 0.) etd_phis<NDIM>(Z, f0, f1, f2);
    tab[q] = make_double4(Z, f0, f1, f2);
}

static unsigned ew_blocks(int64_t n) {
    int64_t b = (n + 255) / 256;
    if (b > 152 * 32) b = 152 * 32;
    if (b < 1) b = 1;
    return (unsigned)b;
}

}  // namespace dd

using namespace dd;

extern "C" {

int dd_euler(const void* start, void* output, const void* deriv, double dt, int64_t n, void* stream) {
    DD_CHECK_ARG(start && output && deriv, "dd_euler: null pointer");
    DD_CHECK_ARG(n >= 0, "dd_euler: negative size");
    if (n == 0) return DD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    DD_KT("euler", st, launch(k_euler, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output,
                                                             (const double2*)deriv, dt, n));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

int dd_etd1(int ndim, const void* start, void* output, const void* deriv, const double* intfactor,
            double dt, int64_t n, void* stream) {
    DD_CHECK_ARG(start && output && deriv && intfactor, "dd_etd1: null pointer");
    DD_CHECK_ARG(ndim == 2 || ndim == 3, "dd_etd1: ndim must be 2 or 3");
    DD_CHECK_ARG(n >= 0, "dd_etd1: negative size");
    if (n == 0) return DD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (ndim == 2)
        DD_KT("etd12", st, launch(k_etd1<2>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv, intfactor, dt, n));
    else
        DD_KT("etd13", st, launch(k_etd1<3>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv, intfactor, dt, n));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

int dd_etd2rk1(int ndim, const void* start, void* output, const void* deriv1, const void* deriv2,
               const double* intfactor, double dt, int64_t n, void* stream) {
    DD_CHECK_ARG(start && output && deriv1 && deriv2 && intfactor, "dd_etd2rk1: null pointer");
    DD_CHECK_ARG(ndim == 2 || ndim == 3, "dd_etd2rk1: ndim must be 2 or 3");
    DD_CHECK_ARG(n >= 0, "dd_etd2rk1: negative size");
    if (n == 0) return DD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (ndim == 2)
        DD_KT("etd2rk12", st, launch(k_etd2rk1<2>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv1,
                                                   (const double2*)deriv2, intfactor, dt, n));
    else
        DD_KT("etd2rk13", st, launch(k_etd2rk1<3>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv1,
                                                   (const double2*)deriv2, intfactor, dt, n));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

int dd_etd2rk2(int ndim, const void* start, void* output, const void* deriv1, const void* deriv2,
               const double* intfactor, double dt, int64_t n, void* stream) {
    DD_CHECK_ARG(start && output && deriv1 && deriv2 && intfactor, "dd_etd2rk2: null pointer");
    DD_CHECK_ARG(ndim == 2 || ndim == 3, "dd_etd2rk2: ndim must be 2 or 3");
    DD_CHECK_ARG(n >= 0, "dd_etd2rk2: negative size");
    if (n == 0) return DD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (ndim == 2)
        DD_KT("etd2rk22", st, launch(k_etd2rk2<2>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv1,
                                                   (const double2*)deriv2, intfactor, dt, n));
    else
        DD_KT("etd2rk23", st, launch(k_etd2rk2<3>, ew_blocks(n), 256, 0, st, (const double2*)start, (double2*)output, (const double2*)deriv1,
                                                   (const double2*)deriv2, intfactor, dt, n));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

int dd_etd_fields(int ndim, int scheme, int nf, const void* const* start, void* const* output,
                  const void* const* deriv1, const void* const* deriv2, const void* const* intfactor, double dt,
                  int64_t n, void* stream) {
    DD_CHECK_ARG(start && output && deriv1 && intfactor, "dd_etd_fields: null pointer");
    DD_CHECK_ARG(ndim == 2 || ndim == 3, "dd_etd_fields: ndim must be 2 or 3");
    DD_CHECK_ARG(scheme >= 0 && scheme <= 2, "dd_etd_fields: scheme must be 0, 1 or 2");
    DD_CHECK_ARG(scheme == 0 || deriv2, "dd_etd_fields: null pointer");
    DD_CHECK_ARG(nf >= 0 && n >= 0, "dd_etd_fields: negative size");
    for (int f = 0; f < nf; f++)
        DD_CHECK_ARG(start[f] && output[f] && deriv1[f] && intfactor[f] && (scheme == 0 || deriv2[f]),
                     "dd_etd_fields: null pointer of field %d", f);
    if (n == 0) return DD_OK;
    for (int f0 = 0; f0 < nf; f0 += ETD_FIELDS) {
        EtdFields a{};
        a.nf = nf - f0 < ETD_FIELDS ? nf - f0 : ETD_FIELDS;
        for (int f = 0; f < a.nf; f++) {
            a.s[f] = (const double2*)start[f0 + f];
            a.o[f] = (double2*)output[f0 + f];
            a.d1[f] = (const double2*)deriv1[f0 + f];
            a.d2[f] = scheme == 0 ? nullptr : (const double2*)deriv2[f0 + f];
            a.intf[f] = (const double*)intfactor[f0 + f];
        }
        if (ndim == 2) launch_etd_fields<2>(scheme, a, dt, n, (cudaStream_t)stream);
        else launch_etd_fields<3>(scheme, a, dt, n, (cudaStream_t)stream);
        DD_LAUNCH_CHECK();
    }
    return DD_OK;
}

int dd_phi_table(int ndim, double nu, int viscosity_order, double h, int qmax, void* table, void* stream) {
    DD_CHECK_ARG(table, "dd_phi_table: null pointer");
    DD_CHECK_ARG(ndim == 2 || ndim == 3, "dd_phi_table: ndim must be 2 or 3");
    DD_CHECK_ARG(qmax >= 0, "dd_phi_table: qmax must be >= 0");
    DD_CHECK_ARG(viscosity_order >= 1, "dd_phi_table: viscosity_order must be >= 1");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned nb = (unsigned)((qmax + 256) / 256);
    if (ndim == 2) DD_KT("phi_table2", st, k_phi_table<2><<<nb, 256, 0, st>>>(nu, viscosity_order, h, qmax, (double4*)table));
    else           DD_KT("phi_table3", st, k_phi_table<3><<<nb, 256, 0, st>>>(nu, viscosity_order, h, qmax, (double4*)table));
    DD_LAUNCH_CHECK();
    return DD_OK;
}

}  // extern "C"
