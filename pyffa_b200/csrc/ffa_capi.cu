// ffa_capi.cu -- extern "C" entry points of libffa_cuda.so (see include/ffa_cuda.h).
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <new>
#include <vector>

#include "ffa_internal.cuh"

using namespace ffa;

namespace {

cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// the columns every kernel reads; an empty bunch (n = 0) may leave them NULL
bool state_ok(const ffa_state_soa *st, int64_t n)
{
    if (!st) return false;
    if (n == 0) return true;
    return st->r && st->vr && st->z && st->vz && st->fi && st->f5 && st->rf && st->esc_r && st->esc_z &&
           st->esc_fi && st->inj && st->surv;
}

// ---------------------------------------------------------------- kernels

__global__ void inject_kernel(ffa_state_soa st, int64_t n, int64_t step)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (st.inj_step[i] == step) {
        st.inj[i] = 1;
        st.surv[i] = 1;
    }
}

// AoS rows of 16 doubles -> SoA.  Flags are stored as bytes: a column value
// equal to 1.0 maps to 1; the reference only ever stores 0 or 1 there.
__global__ void aos_to_soa_kernel(const double *__restrict__ aos, int64_t n, ffa_state_soa st)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *row = aos + i * 16;
    st.r[i] = row[0];
    st.vr[i] = row[1];
    st.z[i] = row[2];
    st.vz[i] = row[3];
    st.fi[i] = row[4];
    st.f5[i] = row[5];
    st.inj[i] = row[7] == 1.0 ? 1 : (row[7] != 0.0 ? 2 : 0);
    st.surv[i] = row[8] == 1.0 ? 1 : (row[8] != 0.0 ? 2 : 0);
    st.rf[i] = row[9];
    st.esc_r[i] = row[10];
    st.esc_z[i] = row[11];
    st.esc_fi[i] = row[12];
}

__global__ void soa_to_aos_kernel(ffa_state_soa st, int64_t n, double *__restrict__ aos)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double *row = aos + i * 16;
    row[0] = st.r[i];
    row[1] = st.vr[i];
    row[2] = st.z[i];
    row[3] = st.vz[i];
    row[4] = st.fi[i];
    row[5] = st.f5[i];
    row[7] = st.inj[i] == 2 ? row[7] : (double)st.inj[i];
    row[8] = st.surv[i] == 2 ? row[8] : (double)st.surv[i];
    row[9] = st.rf[i];
    row[10] = st.esc_r[i];
    row[11] = st.esc_z[i];
    row[12] = st.esc_fi[i];
}

__global__ void mean_fi_kernel(const double *__restrict__ fi, int64_t n, double *out, int64_t *count)
{
    __shared__ double ssum[32];
    __shared__ long long scnt[32];
    double s = 0.0;
    long long c = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double v = fi[i];
        if (!isnan(v)) {
            s += v;
            ++c;
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, off);
        c += __shfl_down_sync(0xffffffffu, c, off);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { ssum[w] = s; scnt[w] = c; }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        s = l < nw ? ssum[l] : 0.0;
        c = l < nw ? scnt[l] : 0;
        for (int off = 16; off > 0; off >>= 1) {
            s += __shfl_down_sync(0xffffffffu, s, off);
            c += __shfl_down_sync(0xffffffffu, c, off);
        }
        if (l == 0) {
            atomicAdd(out, s);
            atomicAdd((unsigned long long *)count, (unsigned long long)c);
        }
    }
}

unsigned blocks_for(int64_t n, int tb) { return (unsigned)((n + tb - 1) / tb); }

// ------------------------------------------- one-dimensional field tables
//
// Taylor coefficients of the logistic sigma(u0 + s x) in x, by the recurrence of
// sigma' = sigma (1 - sigma):
//   (n + 1) c_(n+1) = s (c_n - sum_i c_i c_(n-i)).
// Orders 0 to 2 in long double; from order 3, where a cell's terms (|s| <= 0.04,
// |x| <= 1/2) are below 2e-7 of F, double rounds by less than 1e-22.
constexpr int FL_SERIES = 12;

struct Series {
    long double l[3];
    double c[FL_SERIES];
    bool flat;                          // orders above 0 vanish
};

void logistic_series(long double u0, long double s, Series &t)
{
    t.flat = u0 > 46.0L || u0 < -645.0L;                // 1 in long double; the tail's end, clear of denormal numbers
    if (t.flat) {
        t.l[0] = u0 > 0.0L ? 1.0L : 0.0L;
        return;
    }
    const long double c0 = 1.0L / (1.0L + expl(-u0));
    t.l[0] = c0;
    t.l[1] = s * (c0 - c0 * c0);
    t.l[2] = s * (t.l[1] - 2.0L * c0 * t.l[1]) / 2.0L;
    for (int n = 0; n < 3; ++n) t.c[n] = (double)t.l[n];
    if (u0 < -50.0L) {                  // the exponential tail: the products are lost beside c_n
        for (int n = 2; n + 1 < FL_SERIES; ++n) t.c[n + 1] = (double)s * t.c[n] * (1.0 / (n + 1));
        return;
    }
    const double d = (double)(1.0L - 2.0L * c0), sd = (double)s;
    for (int n = 2; n + 1 < FL_SERIES; ++n) {
        double q = 0.0;                 // the pairs i, n - i twice, the latest last
        for (int i = (n - 1) / 2; i >= 1; --i) q += t.c[i] * t.c[n - i];
        q = d * t.c[n] - 2.0 * q;
        if (n % 2 == 0) q -= t.c[n / 2] * t.c[n / 2];
        t.c[n + 1] = sd * q * (1.0 / (n + 1));
    }
}

// Adds y a b to the orders l (0 to 2) and c (3 on)
void add_product(double y, const Series &a, const Series &b, long double l[3], double c[FL_SERIES])
{
    if (a.flat && b.flat) {
        l[0] += (long double)y * (a.l[0] * b.l[0]);
        return;
    }
    if (a.flat || b.flat) {             // by exactly 0 or 1
        const Series &f = a.flat ? a : b, &v = a.flat ? b : a;
        if (f.l[0] == 0.0L) return;
        for (int n = 0; n < 3; ++n) l[n] += (long double)y * v.l[n];
        for (int n = 3; n < FL_SERIES; ++n) c[n] += y * v.c[n];
        return;
    }
    for (int n = 0; n < 3; ++n) {
        long double q = 0.0L;
        for (int i = 0; i <= n; ++i) q += a.l[i] * b.l[n - i];
        l[n] += (long double)y * q;
    }
    for (int n = 3; n < FL_SERIES; ++n) {
        double q = 0.0;
        for (int i = 0; i <= n; ++i) q += a.c[i] * b.c[n - i];
        c[n] += y * q;
    }
}

// Lowers a series on |x| <= 1/2 from FL_SERIES to 8 terms: each top term is
// replaced by the lower powers of its Chebyshev polynomial T_n(2 x)
// (Lanczos' economisation), which spreads its size / 2^(n-1) evenly over the
// cell instead of leaving all of it at the edges.
struct Economise {
    long double T[FL_SERIES][FL_SERIES];        // T_n(2 x), coefficient of x^a over that of x^n
    Economise() : T{{0}}
    {
        T[0][0] = 1.0L;
        T[1][1] = 2.0L;
        for (int n = 2; n < FL_SERIES; ++n)
            for (int a = 0; a <= n; ++a) T[n][a] = (a ? 4.0L * T[n - 1][a - 1] : 0.0L) - T[n - 2][a];
        for (int n = FL_SERIES - 1; n >= 8; --n)
            for (int a = 0; a <= n; ++a) T[n][a] /= T[n][n];
    }
    void operator()(long double c[FL_SERIES]) const
    {
        for (int n = FL_SERIES - 1; n >= 8; --n)
            for (int a = n - 2; a >= 0; a -= 2) c[a] -= c[n] * T[n][a];
    }
};

// The flutter and power tables of FieldK (formed in long double, stored as
// double: flutter cells, then power entries).
// Flutter cells: h = 2^-m with k h <= 0.04 for the sharpest fringe k = 16 / W:
// the degree-7 fit then misses F by less than 1e-19 and F' by less than 1e-17
// of k, below their rounding.  At most 2^17 cells (8 MB); a sharper fringe
// (W below about 3e-3 of a 30 degree sector) keeps the sigmoids.
// Power entries: spacing 2^-p with the first omitted binomial term below
// 2^-57, over the map's radii and a quarter of their span on each side.
// A map pays for them once, but a study of many lattices pays each time: all
// orders of every cell in long double took 7.2 ms for the benchmark's
// lattice and 45 ms with fringes of a sixth of its sharper one, on the host; this
// form 3.3 and 11 ms with the upload.
void field_tables(FieldK &k, std::vector<double> &tab)
{
    double kmax = 0.0;
    for (int j = 0; j < k.n_seg; ++j) kmax = fmax(kmax, fabs(k.seg_k[j]));
    k.fl_n = 1;
    k.fl_direct = 1;
    k.fl_scale = 1.0;
    tab.assign(8, 0.0);
    if (kmax > 0.0 && isfinite(kmax)) {
        int m = 0;
        while (m < 40 && ldexp(kmax, -m) > 0.04) ++m;
        const double cells = k.period * ldexp(1.0, m);
        if (cells <= 131072.0) {
            const int n = (int)ceil(cells);
            k.fl_n = n + 2;
            k.fl_direct = 0;
            k.fl_scale = ldexp(1.0, m);
            tab.resize(8 * (size_t)k.fl_n);
            const long double h = ldexpl(1.0L, -m);
            const Economise economise;
            Series a, b;
            for (int j = 0; j < k.fl_n; ++j) {
                const long double mid = ((long double)(j - 1) + 0.5L) * h;
                long double sum[FL_SERIES] = {0};
                double high[FL_SERIES] = {0};
                for (int g = 0; g < k.n_seg; ++g) {
                    const long double ks = k.seg_k[g];
                    logistic_series(ks * (mid - (long double)k.seg_x0[g]), ks * h, a);
                    logistic_series(-ks * (mid - (long double)k.seg_x1[g]), -ks * h, b);
                    add_product(k.seg_y[g], a, b, sum, high);
                }
                for (int n1 = 3; n1 < FL_SERIES; ++n1) sum[n1] = high[n1];
                economise(sum);
                for (int a1 = 0; a1 < 8; ++a1) tab[8 * (size_t)j + a1] = (double)sum[a1];
            }
        }
    }
    k.pw_n = 0;                                      // no r is inside: the entry is loaded, not used
    k.pw_j0 = 0;
    k.pw_scale = k.pw_h = 1.0;
    if (k.k != 0.0 && k.r_size > 1 && k.r_step > 0.0) {
        const double span = k.r_step * (double)(k.r_size - 1);
        const double lo = fmax(k.r_min - 0.25 * span, 0.25 * k.r_min), hi = k.r_min + 1.25 * span;
        const double e = k.km1, c5 = fabs(e * (e - 1) * (e - 2) * (e - 3) * (e - 4) / 120.0);
        if (lo > 0.0 && hi < 1e6) {
            int p = 0;
            while (p < 24 && c5 * pow(ldexp(0.5, -p) / lo, 5) > ldexp(1.0, -57)) ++p;
            const double j0 = floor(lo * ldexp(1.0, p)), j1 = ceil(hi * ldexp(1.0, p));
            if (j0 >= 1.0 && j1 - j0 < 65536.0 && j1 < 2147483647.0) {
                k.pw_j0 = (int)j0;
                k.pw_n = (int)(j1 - j0) + 1;
                k.pw_scale = ldexp(1.0, p);
                k.pw_h = ldexp(1.0, -p);
                k.pw_c[0] = e;
                k.pw_c[1] = e * (e - 1) / 2;
                k.pw_c[2] = e * (e - 1) * (e - 2) / 6;
                k.pw_c[3] = e * (e - 1) * (e - 2) * (e - 3) / 24;
                for (int j = 0; j < k.pw_n; ++j) {
                    const long double r = (long double)(k.pw_j0 + j) * (long double)k.pw_h;
                    tab.push_back((double)((long double)k.B0 * powl(r, (long double)e)));
                    tab.push_back((double)(1.0L / r));
                }
            }
        }
    }
    if (k.pw_n == 0) tab.insert(tab.end(), 2, 0.0);
    if (k.k == 0.0) {                                // no power: every r is inside a one-entry table of zeros
        k.pw_n = 1;
        k.pw_scale = 0.0;
    }
}

// The tables' device copy, made outside the caller's streams: a mid-plane map
// asks nothing of them, so it can be made while one is captured (allocations are
// then refused unless the thread's capture mode is relaxed) and waits for none.
cudaError_t upload_tables(const double *tab, size_t bytes, double **out)
{
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    cudaStream_t s = nullptr;
    e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(out, bytes);
    if (e == cudaSuccess) e = cudaMemcpyAsync(*out, tab, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (s) cudaStreamDestroy(s);
    cudaThreadExchangeStreamCaptureMode(&mode);
    return e;
}

}  // namespace

extern "C" {

int ffa_fieldmap_create(const ffa_field_desc *d, void *stream, ffa_fieldmap **out)
{
    if (!d || !out) return FFA_ERR_INVALID;
    *out = nullptr;
    if (d->nsectors <= 0 || d->n_spoly < 0 || d->n_spoly > FFA_MAX_POLY || d->n_spolyp < 0 ||
        d->n_spolyp > FFA_MAX_POLY || d->n_convex < 0 || d->n_convex > FFA_MAX_SEG || d->max_order < 0)
        return FFA_ERR_INVALID;
    if (d->max_order > FFA_MAX_ORDER) return FFA_ERR_UNSUPPORTED;
    if (d->max_order > 0 && (d->r_size < 2 || d->fi_size < 2 || !d->bz_stack || !d->bfi_stack || !d->br_stack ||
                             !(d->r_step > 0) || !(d->fi_step > 0)))
        return FFA_ERR_INVALID;
    for (int j = 0; j < d->n_convex; ++j)
        if (!(d->convex[5 * j + 2] != 0.0)) return FFA_ERR_INVALID;
    // the push kernels index the node table with 32-bit offsets (12 values per
    // node at most): larger tables are refused
    if (d->max_order > 0 && (double)d->r_size * (double)d->fi_size * 12.0 >= 2147483647.0)
        return FFA_ERR_UNSUPPORTED;

    ffa_fieldmap *fm = (ffa_fieldmap *)calloc(1, sizeof(ffa_fieldmap));
    if (!fm) return FFA_ERR_NOMEM;
    FieldK &k = fm->k;
    k.nsectors = d->nsectors;
    k.n_spoly = d->n_spoly;
    k.n_spolyp = d->n_spolyp;
    k.n_seg = d->n_convex;
    k.max_order = d->max_order;
    const int nv = 3 * d->max_order;
    k.npad = nv <= 4 ? 4 : (nv <= 8 ? 8 : 12);
    k.B0 = d->B0;
    k.k = d->k;
    k.km1 = d->k - 1.0;
    k.period = 2.0 * PI / (double)d->nsectors;
    k.inv_period = 1.0 / k.period;
    memcpy(k.spoly, d->spoly, sizeof(k.spoly));
    memcpy(k.spolyp, d->spolyp, sizeof(k.spolyp));
    for (int j = 0; j < d->n_convex; ++j) {
        const double *cp = d->convex + 5 * j;
        k.seg_x0[j] = cp[0];
        k.seg_x1[j] = cp[1];
        k.seg_k[j] = 16.0 / cp[2];
        k.seg_y[j] = cp[4] * fabs(cp[3]);
    }
    k.r_min = d->r_min;
    k.r_step = d->r_step;
    k.fi_min = d->fi_min;
    k.fi_step = d->fi_step;
    k.r_size = d->r_size;
    k.fi_size = d->fi_size;
    k.spiral_zero = 1;
    for (int a = 0; a < d->n_spoly; ++a) if (d->spoly[a] != 0.0) k.spiral_zero = 0;
    for (int a = 0; a < d->n_spolyp; ++a) if (d->spolyp[a] != 0.0) k.spiral_zero = 0;
    k.r_ref = (d->r_size > 1 && d->r_step > 0) ? d->r_min + 0.5 * d->r_step * (double)(d->r_size - 1) : 1.0;
    k.inv_r_ref = 1.0 / k.r_ref;
    k.inv_r_step = d->r_step > 0 ? 1.0 / d->r_step : 0.0;
    k.inv_fi_step = d->fi_step > 0 ? 1.0 / d->fi_step : 0.0;
    k.c1 = d->k == 0.0 ? d->B0 : d->B0 * pow(k.r_ref, d->k - 1.0);
    k.kc1 = d->k * k.c1;
    k.B0f = (float)k.B0;
    k.c1f = (float)k.c1;
    k.kc1f = (float)k.kc1;
    k.km1f = (float)k.km1;
    for (int j = 0; j < d->n_convex; ++j) {
        k.seg_x0f[j] = (float)k.seg_x0[j];
        k.seg_x1f[j] = (float)k.seg_x1[j];
        k.seg_kf[j] = (float)k.seg_k[j];
        k.seg_yf[j] = (float)k.seg_y[j];
        k.seg_ykf[j] = (float)(k.seg_y[j] * k.seg_k[j]);
    }
    for (int j = 0; j < d->n_convex; ++j) k.seg_yk[j] = k.seg_y[j] * k.seg_k[j];
    {
        std::vector<double> tab;
        try {
            field_tables(k, tab);
        } catch (const std::bad_alloc &) {          // nothing is thrown through the C entry
            free(fm);
            return FFA_ERR_NOMEM;
        }
        k.unusual = k.fl_direct || k.k == 0.0;
        const cudaError_t e = upload_tables(tab.data(), sizeof(double) * tab.size(), &fm->tables);
        // a mid-plane map can be described where there is no device to push on
        // (FFA_ERR_CUDA from the calls that would read its tables)
        const bool absent = e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver;
        if (e != cudaSuccess && !(absent && d->max_order == 0)) {
            ffa_fieldmap_destroy(fm);
            return e == cudaErrorMemoryAllocation || absent ? FFA_ERR_NOMEM : FFA_ERR_CUDA;
        }
        k.fl_tab = fm->tables;
        k.pw_tab = fm->tables ? reinterpret_cast<const double2 *>(fm->tables + 8 * (size_t)k.fl_n) : nullptr;
    }
    if (d->max_order > 0) {
        const int64_t plane = d->r_size * d->fi_size;
        int per = 0;
        for (int a = 0; a < 12; a += 4) per += map_plane_width(d->max_order, a);
        k.plane = plane;
        if (cudaMalloc(&fm->nodes64, sizeof(double) * plane * per) != cudaSuccess ||
            cudaMalloc(&fm->nodes32, sizeof(float) * plane * k.npad) != cudaSuccess) {
            ffa_fieldmap_destroy(fm);
            return FFA_ERR_NOMEM;
        }
        if (launch_pack_nodes(*d, k.npad, fm->nodes64, fm->nodes32, as_stream(stream)) != cudaSuccess) {
            ffa_fieldmap_destroy(fm);
            return FFA_ERR_CUDA;
        }
    }
    k.nodes64 = fm->nodes64;
    k.nodes32 = fm->nodes32;
    *out = fm;
    return FFA_OK;
}

int ffa_fieldmap_set_harmonics(ffa_fieldmap *fm, int32_t n, const double *m, const double *amp,
                               const double *phase, const double *rmin, const double *rmax)
{
    if (!fm || n < 0) return FFA_ERR_INVALID;
    if (n > FFA_MAX_HARMONICS) return FFA_ERR_UNSUPPORTED;
    if (n > 0 && (!m || !amp || !phase || !rmin || !rmax)) return FFA_ERR_INVALID;
    double rows[5 * FFA_MAX_HARMONICS] = {0};
    for (int k = 0; k < n; ++k) {
        if (m[k] != floor(m[k]) || !isfinite(amp[k]) || !isfinite(phase[k])) return FFA_ERR_INVALID;
        rows[5 * k] = m[k];
        rows[5 * k + 1] = amp[k];
        rows[5 * k + 2] = phase[k];
        rows[5 * k + 3] = rmin[k];
        rows[5 * k + 4] = rmax[k];
    }
    if (n > 0) {
        if (!fm->harm && cudaMalloc(&fm->harm, sizeof(rows)) != cudaSuccess) return FFA_ERR_NOMEM;
        FFA_CHECK_CUDA(cudaMemcpy(fm->harm, rows, sizeof(rows), cudaMemcpyHostToDevice));
    }
    fm->k.harm = fm->harm;
    fm->k.n_harm = n;
    return FFA_OK;
}

int ffa_fieldmap_destroy(ffa_fieldmap *fm)
{
    if (!fm) return FFA_OK;
    if (fm->nodes64) cudaFree(fm->nodes64);
    if (fm->nodes32) cudaFree(fm->nodes32);
    if (fm->tables) cudaFree(fm->tables);
    if (fm->harm) cudaFree(fm->harm);
    free(fm);
    return FFA_OK;
}

int ffa_inject(ffa_state_soa *st, int64_t n, int64_t step, void *stream)
{
    if (n < 0 || !state_ok(st, n) || (n > 0 && !st->inj_step)) return FFA_ERR_INVALID;
    if (n == 0) return FFA_OK;
    inject_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(*st, n, step);
    FFA_CHECK_CUDA(cudaGetLastError());
    return FFA_OK;
}

static int push_impl(const ffa_fieldmap *fm, const ffa_rf_desc *rf, const ffa_aperture *ap, const ffa_consts *cs,
                     const ffa_step_table *tab, ffa_state_soa *st, int64_t n, int64_t step0, int32_t nsteps,
                     double dt, int32_t sc_step, int32_t flags, void *stream, int64_t *status,
                     const ffa_crossing *xing)
{
    if (!fm || !rf || !ap || !cs || !tab || n < 0 || !state_ok(st, n) || nsteps < 0 || step0 < 0)
        return FFA_ERR_INVALID;
    if (!tab->drf || !tab->acc || step0 + nsteps > tab->nsteps) return FFA_ERR_INVALID;
    if (rf->ngaps < 1 || rf->ngaps > FFA_MAX_GAPS) return FFA_ERR_INVALID;
    if (rf->spiral_nodes &&
        (rf->spiral_nr < 2 || rf->spiral_nphi < 2 || !(rf->spiral_dr > 0.0) || !(rf->spiral_dphi > 0.0) ||
         (int64_t)rf->spiral_nr * rf->spiral_nphi >= ((int64_t)1 << 31)))
        return FFA_ERR_INVALID;
    if (sc_step < 0) return FFA_ERR_INVALID;
    if (sc_step > 0 && st->sc_pre &&
        (!st->sc_pp || !st->e_pre_r || !st->e_pre_z || !st->e_pre_fi || !st->e_pp_r || !st->e_pp_z || !st->e_pp_fi))
        return FFA_ERR_INVALID;
    if (flags & ~(FFA_RK4 | FFA_FP32C | FFA_FP32 | FFA_RF_PHYSICAL_SUM | FFA_SHAPE_MASK)) return FFA_ERR_INVALID;
    if ((flags & FFA_FP32) && ((flags & (FFA_RK4 | FFA_FP32C)) || (sc_step > 0 && st->sc_pre) ||
                               fm->k.n_harm > 0))
        return FFA_ERR_UNSUPPORTED;
    const int tb_sel = (flags >> FFA_SHAPE_TB_SHIFT) & 3, nreg_sel = (flags >> FFA_SHAPE_NREG_SHIFT) & 3;
    if ((flags & FFA_RK4) && (tb_sel | nreg_sel)) return FFA_ERR_UNSUPPORTED;
    if (nreg_sel && (!(flags & FFA_FP32C) || (sc_step > 0 && st->sc_pre) || fm->k.n_harm > 0))
        return FFA_ERR_UNSUPPORTED;
    if (n == 0 || nsteps == 0) return FFA_OK;
    if (!fm->tables) return FFA_ERR_CUDA;            // made without a device

    PushK p;
    memset(&p, 0, sizeof(p));
    p.f = fm->k;
    p.rf.enable = rf->enable;
    p.rf.ngaps = rf->ngaps;
    p.rf.physical_sum = (flags & FFA_RF_PHYSICAL_SUM) ? 1 : 0;
    memcpy(p.rf.poly_x, rf->poly_x, sizeof(p.rf.poly_x));
    memcpy(p.rf.poly_y, rf->poly_y, sizeof(p.rf.poly_y));
    memcpy(p.rf.box, rf->box, sizeof(p.rf.box));
    memcpy(p.rf.theta_n, rf->theta_n, sizeof(p.rf.theta_n));
    memcpy(p.rf.rf_shift, rf->rf_shift, sizeof(p.rf.rf_shift));
    for (int g = 0; g < rf->ngaps; ++g) {
        // angular extent of the gap rectangle: a convex polygon that does not
        // contain the origin subtends the angles spanned by its vertices
        double cx = 0.0, cy = 0.0;
        for (int j = 0; j < 4; ++j) { cx += rf->poly_x[g][j]; cy += rf->poly_y[g][j]; }
        const double c0 = atan2(cy, cx);
        double half = 0.0;
        for (int j = 0; j < 4; ++j) {
            double d = atan2(rf->poly_y[g][j], rf->poly_x[g][j]) - c0;
            d -= 2.0 * PI * rint(d / (2.0 * PI));
            half = fmax(half, fabs(d));
        }
        p.rf.win_center[g] = c0;
        p.rf.win_half[g] = half < 1.0 ? half + 1e-9 : 4.0;  // wide gaps: no shortcut
    }
    if (rf->spiral_nodes) {
        p.rf.sp = rf->spiral_nodes;
        p.rf.sp_nr = rf->spiral_nr;
        p.rf.sp_nphi = rf->spiral_nphi;
        p.rf.sp_r0 = rf->spiral_r0;
        p.rf.sp_dr = rf->spiral_dr;
        p.rf.sp_phi0 = rf->spiral_phi0;
        p.rf.sp_dphi = rf->spiral_dphi;
        // phi_max and the window centre as shift_to_nearest_window forms them
        // (src/FFAG_MathTools.py:1072-1073, 1131)
        p.rf.sp_phimax = rf->spiral_phi0 + rf->spiral_dphi * (double)(rf->spiral_nphi - 1);
        p.rf.sp_phic = 0.5 * (rf->spiral_phi0 + p.rf.sp_phimax);
        memcpy(p.rf.gap_az, rf->gap_azimuth, sizeof(p.rf.gap_az));
    }
    p.rf.single = rf->enable && !rf->spiral_nodes && !p.rf.physical_sum ? rf->ngaps - 1 : -1;
    p.ap = *ap;
    if (!ap->enable) {
        p.ap.rmin = p.ap.zmin = -INFINITY;
        p.ap.rmax = p.ap.zmax = INFINITY;
    }
    p.cs = *cs;
    p.st = *st;
    if (sc_step == 0) p.st.sc_pre = nullptr;
    p.drf = tab->drf;
    p.acc = tab->acc;
    p.n = n;
    p.step0 = step0;
    p.nsteps = nsteps;
    p.sc_step = sc_step;
    p.dt = dt;
    {
        const double q = cs->q, c = cs->c, m = cs->m0;
        p.hq = 0.5 * dt * q;
        p.inv_mmcc = 1.0 / (m * m * c * c);
        p.inv_cc = 1.0 / (c * c);
        p.inv_m = 1.0 / m;
        p.hqm = p.hq * p.inv_m;
        p.inv_sc = sc_step > 0 ? 1.0 / (double)sc_step : 0.0;
    }
    p.status = status;
    if (xing) {
        if (xing->ntargets < 1 || xing->ntargets > FFA_MAX_CROSSING_TARGETS) return FFA_ERR_INVALID;
        if (xing->fit_sums) {
            // the fit reads f5 as d(phi)/dt, the Boris state; one target
            if (!xing->fit_instance || !xing->fit_centre || !xing->fit_scale || !xing->fit_last ||
                !xing->fit_has || xing->ntargets != 1)
                return FFA_ERR_INVALID;
            if (flags & FFA_RK4) return FFA_ERR_UNSUPPORTED;
        } else if (!xing->buf || !xing->count || xing->capacity < 0) {
            return FFA_ERR_INVALID;
        }
        for (int t = 0; t < xing->ntargets; ++t)
            if (!(xing->target[t] >= 0.0) || !(xing->target[t] < 2.0 * ffa::PI)) return FFA_ERR_INVALID;
        p.xing = *xing;
    }
    cudaError_t e;
    if (flags & FFA_RK4) e = launch_rk4_f64(p, as_stream(stream), (flags & FFA_FP32C) != 0);
    else if (flags & FFA_FP32) e = launch_boris_f32(p, as_stream(stream), 32 << tb_sel);
    else if (flags & FFA_FP32C) e = launch_boris_f32c(p, as_stream(stream), 32 << tb_sel, nreg_sel);
    else e = launch_boris_f64(p, as_stream(stream), 32 << tb_sel);
    return e == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}

int ffa_push_occupancy(int32_t flags, int32_t max_order, int32_t crossing, int32_t *blocks_per_sm,
                       int32_t *threads_per_block)
{
    if (!blocks_per_sm || !threads_per_block || max_order < 0 || max_order > FFA_MAX_ORDER) return FFA_ERR_INVALID;
    if (flags & ~(FFA_RK4 | FFA_FP32C | FFA_RF_PHYSICAL_SUM | FFA_SHAPE_MASK)) return FFA_ERR_INVALID;
    const int tb_sel = (flags >> FFA_SHAPE_TB_SHIFT) & 3, nreg_sel = (flags >> FFA_SHAPE_NREG_SHIFT) & 3;
    if ((flags & FFA_RK4) && (tb_sel | nreg_sel)) return FFA_ERR_UNSUPPORTED;
    if (nreg_sel && !(flags & FFA_FP32C)) return FFA_ERR_UNSUPPORTED;
    const int tb = (flags & FFA_RK4) ? ffa::RK4_TB : (32 << tb_sel);
    int blocks = 0;
    if (push_occupancy((flags & FFA_RK4) != 0, (flags & FFA_FP32C) != 0, max_order, crossing != 0, tb, nreg_sel,
                       &blocks) != cudaSuccess)
        return FFA_ERR_CUDA;
    *blocks_per_sm = blocks;
    *threads_per_block = tb;
    return FFA_OK;
}

int ffa_theta_track(const ffa_fieldmap *fm, const ffa_theta_track_desc *d, void *stream)
{
    if (!fm || !d || d->m < 0 || d->n_points < 2 || !(d->t_end > 0.0) || !d->x0 || !d->x1)
        return FFA_ERR_INVALID;
    if (d->time_mode != 0 && d->time_mode != 1) return FFA_ERR_INVALID;
    if (d->traj && d->traj_cols != 2 && d->traj_cols != 7) return FFA_ERR_INVALID;
    if (d->m == 0) return FFA_OK;
    if (!fm->tables) return FFA_ERR_CUDA;            // made without a device
    return launch_theta_track(fm->k, *d, as_stream(stream)) == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}

int ffa_push(const ffa_fieldmap *fm, const ffa_rf_desc *rf, const ffa_aperture *ap, const ffa_consts *cs,
             const ffa_step_table *tab, ffa_state_soa *st, int64_t n, int64_t step0, int32_t nsteps, double dt,
             int32_t sc_step, int32_t flags, void *stream, int64_t *status)
{
    return push_impl(fm, rf, ap, cs, tab, st, n, step0, nsteps, dt, sc_step, flags, stream, status, nullptr);
}

int ffa_push_crossing(const ffa_fieldmap *fm, const ffa_rf_desc *rf, const ffa_aperture *ap, const ffa_consts *cs,
                      const ffa_step_table *tab, ffa_state_soa *st, int64_t n, int64_t step0, int32_t nsteps,
                      double dt, int32_t sc_step, int32_t flags, void *stream, int64_t *status,
                      const ffa_crossing *xing)
{
    if (!xing) return FFA_ERR_INVALID;
    return push_impl(fm, rf, ap, cs, tab, st, n, step0, nsteps, dt, sc_step, flags, stream, status, xing);
}

int ffa_aos_to_soa(const double *aos, int64_t n, ffa_state_soa *st, void *stream)
{
    if (n < 0 || !state_ok(st, n) || (n > 0 && !aos)) return FFA_ERR_INVALID;
    if (n == 0) return FFA_OK;
    aos_to_soa_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(aos, n, *st);
    FFA_CHECK_CUDA(cudaGetLastError());
    return FFA_OK;
}

int ffa_soa_to_aos(const ffa_state_soa *st, int64_t n, double *aos, void *stream)
{
    if (n < 0 || !state_ok(st, n) || (n > 0 && !aos)) return FFA_ERR_INVALID;
    if (n == 0) return FFA_OK;
    soa_to_aos_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(*st, n, aos);
    FFA_CHECK_CUDA(cudaGetLastError());
    return FFA_OK;
}

int ffa_mean_fi(const ffa_state_soa *st, int64_t n, double *out, int64_t *count, void *stream)
{
    if (!st || (n > 0 && !st->fi) || !out || !count || n < 0) return FFA_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    FFA_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double), s));
    FFA_CHECK_CUDA(cudaMemsetAsync(count, 0, sizeof(int64_t), s));
    if (n == 0) return FFA_OK;
    unsigned nb = blocks_for(n, 256);
    if (nb > 1184) nb = 1184;
    mean_fi_kernel<<<nb, 256, 0, s>>>(st->fi, n, out, count);
    FFA_CHECK_CUDA(cudaGetLastError());
    return FFA_OK;
}

}  // extern "C"
