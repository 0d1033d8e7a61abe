// ffa_push.cu -- fused multi-step particle pushers for sm_100a.
//
// One thread owns one particle for the whole launch: the state lives in
// registers across `nsteps` time steps, so HBM sees one read and one write of
// the structure-of-arrays state per launch.  Per step the thread does what the
// reference does in ~8 full-array passes:
//   fast_mod_parallel        src/FFAG_MathTools.py:1553-1557
//   GetBfields_Njit          src/FFAG_Field.py:1333-1426
//   Bmap_add_all_orders      src/FFAG_MathTools.py:1139-1188
//   emap_kernel (per gap)    src/FFAG_Utils.py:984-1036
//   cylindrical_to_cartesian src/FFAG_MathTools.py:1969-2014
//   boris_push_cartesian_njit src/FFAG_MathTools.py:1877-1966
//   convert_cartesian_to_cylindrical src/FFAG_MathTools.py:2017-2060
// (RK4: FunctionForAccelerationBunch_dt src/FFAG_track.py:1743-1801 four times,
//  RK4_equations_of_motion_njit and RK4_Post_Step_njit
//  src/FFAG_MathTools.py:2205-2299.)
//
// The Boris step is taken in the particle's own frame (r-hat, fi-hat, z-hat)
// instead of the fixed Cartesian frame.  The Boris update commutes with
// rotations, so this is the reference's step up to rounding: the reference
// rotates x, v, E, B into Cartesian axes, pushes, and rotates back with the
// azimuth change atan2(y', x') - atan2(y, x); here the azimuth change is
// atan2 of the displacement in the local frame.  It saves one atan2 and two
// sin/cos pairs per step and is the more accurate of the two.  Particles that
// are skipped (not injected or lost) take the reference's exact Cartesian
// round trip, which perturbs r, vr and dfi/dt by rounding every step.
// The float64 kernels form the reference's values, not its expressions: the
// mid-plane field from tables, divisions and square roots from ffa_math.cuh, the
// momentum (Boris) and what depends on the energy (RK4) carried from step to
// step.  Each differs from the reference's expression by about an ulp.  The FP32C
// kernels and the rare branches keep its evaluation order; the compiler may fuse
// a multiply and an add into one FMA (at most an ulp per operation).
#include <float.h>

#include "ffa_internal.cuh"
#include "ffa_math.cuh"

namespace ffa {

// ----------------------------------------------------------- field (fp64)

// 32-byte read-only global loads (sm_100): four doubles, eight floats; the
// address must be 32-byte aligned
__device__ __forceinline__ void ldg_v4(const double *p, double t[4])
{
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(t[0]), "=d"(t[1]), "=d"(t[2]), "=d"(t[3]) : "l"(p));
}

__device__ __forceinline__ void ldg_v2(const double *p, double t[2])
{
    asm("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(t[0]), "=d"(t[1]) : "l"(p));
}

__device__ __forceinline__ void ldg_v8(const float *p, float t[8])
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(t[0]), "=f"(t[1]), "=f"(t[2]), "=f"(t[3]), "=f"(t[4]), "=f"(t[5]), "=f"(t[6]), "=f"(t[7])
        : "l"(p));
}

// 1.5 * 2^52: adding it rounds a double below 2^51 in magnitude to the nearest
// integer, which then sits in the low word (the high word is INT_HI for
// integers 0 .. 2^32 - 1)
constexpr double INT_MAGIC = 6755399441055744.0;
constexpr int INT_HI = 0x43380000;

// Flutter sum and its azimuth derivative from the magnets' sigmoids, for
// lattices without a flutter table (fringes sharper than the table's limit).
__device__ __noinline__ double2 flutter_direct(const FieldK &f, double fs)
{
    double F = 0.0, Fp = 0.0;
    for (int j = 0; j < f.n_seg; ++j) {
        const double ks = f.seg_k[j];
        // Past 37.5 the exponential is below 2^-54, so 1 + e rounds to 1 and
        // the sigmoid is exactly 1 (its derivative exactly 0): the branch
        // skips only exponentials that cannot change the result.
        const double a1 = ks * (fs - f.seg_x0[j]);
        const double a2 = ks * (fs - f.seg_x1[j]);
        double s1 = 1.0, s2 = 1.0, s1p = 0.0, s2p = 0.0;
        if (a1 < 37.5) {
            s1 = 1.0 / (1.0 + exp(-a1));
            s1p = ks * s1 * (1.0 - s1);
        }
        if (a2 > -37.5) {
            s2 = 1.0 / (1.0 + exp(a2));
            s2p = -ks * s2 * (1.0 - s2);
        }
        const double y = f.seg_y[j];
        F += y * s1 * s2;
        Fp += y * (s1p * s2 + s1 * s2p);
    }
    return make_double2(F, Fp);
}

// B0 r^(k-1) for radii outside the power table
__device__ __noinline__ double power_direct(const FieldK &f, double r) { return f.B0 * exp(f.km1 * log(r)); }

// One flutter cell and the position in it
struct FlutterCell {
    double c[8], x;
};

// Cell j covers [j, j + 1) cells of azimuth; one guard cell on each side
// takes a reduction that rounded just outside the sector.
__device__ __forceinline__ FlutterCell flutter_fetch(const FieldK &f, double fs)
{
    FlutterCell t;
    const double q = fma(fs, f.fl_scale, -0.5), qi = q + INT_MAGIC;
    const int j = min(max(__double2loint(qi) + 1, 0), f.fl_n - 1);
    t.x = q - (qi - INT_MAGIC);
    ldg_v4(f.fl_tab + 8 * j, t.c);
    ldg_v4(f.fl_tab + 8 * j + 4, t.c + 4);
    return t;
}

__device__ __forceinline__ void flutter_eval(const FieldK &f, const FlutterCell &t, double &F, double &Fp)
{
    F = t.c[7];
    Fp = 0.0;
#pragma unroll
    for (int a = 6; a >= 0; --a) {
        Fp = (a == 6) ? F : fma(Fp, t.x, F);
        F = fma(F, t.x, t.c[a]);
    }
    Fp *= f.fl_scale;
}

// One power entry (B0 r_j^(k-1), 1 / r_j), r - r_j, and whether r is inside
// the table
struct PowerEntry {
    double2 e;
    double d;
    bool in;
};

__device__ __forceinline__ PowerEntry power_fetch(const FieldK &f, double r)
{
    PowerEntry t;
    const double pi = fma(r, f.pw_scale, INT_MAGIC);
    const int k = __double2loint(pi) - f.pw_j0;
    t.in = __double2hiint(pi) == INT_HI && (unsigned)k < (unsigned)f.pw_n;
    t.d = fma(INT_MAGIC - pi, f.pw_h, r);
    t.e = __ldg(f.pw_tab + (t.in ? k : 0));
    return t;
}

// B0 r^(k-1)
__device__ __forceinline__ double power_eval(const FieldK &f, const PowerEntry &t, double r)
{
    const double u = t.d * t.e.y;
    const double P = fma(u, fma(u, fma(u, f.pw_c[3], f.pw_c[2]), f.pw_c[1]), f.pw_c[0]);
    double G = fma(t.e.x * u, P, t.e.x);
    if (!t.in) G = power_direct(f, r);
    return G;
}

struct Tables {
    FlutterCell fl;
    PowerEntry pw;
    double fs, spiral_p;
};

// The table entries of a point, loaded unconditionally (a map without a table
// has one dummy entry), so that these loads and the map's are in flight
// together.
__device__ __forceinline__ Tables tables_fetch(const FieldK &f, double ri, double fim)
{
    // theta' = (fi mod P) - s(r), reduced mod P again.  Without a spiral
    // (all-zero coefficients evaluate to exactly 0) the callers' fim is
    // reduced already: the second reduction would only map a fim within an
    // ulp of P to about 0 (a step lands there with probability ~1e-16), so
    // it is skipped with the polynomials.
    Tables t;
    t.spiral_p = 0.0;
    t.fs = fim;
    if (!f.spiral_zero) {
        double spiral = 0.0;
        for (int a = 0; a < f.n_spoly; ++a) spiral = spiral * ri + f.spoly[a];
        for (int a = 0; a < f.n_spolyp; ++a) t.spiral_p = t.spiral_p * ri + f.spolyp[a];
        t.fs = fim - spiral;
        t.fs -= f.period * floor(t.fs * f.inv_period);
    }
    t.fl = flutter_fetch(f, t.fs);
    t.pw = power_fetch(f, ri);
    return t;
}

// F, F', B0 r^k and k B0 r^(k-1) from the entries of a point
__device__ __forceinline__ void tables_eval(const FieldK &f, const Tables &t, double ri, double &F, double &Fp,
                                            double &B0r, double &kG)
{
    flutter_eval(f, t.fl, F, Fp);
    const double G = power_eval(f, t.pw, ri);
    B0r = G * ri;
    kG = f.k * G;
    if (f.unusual) {                     // no flutter table, or a field index of 0
        if (f.fl_direct) {
            const double2 v = flutter_direct(f, t.fs);
            F = v.x;
            Fp = v.y;
        }
        if (f.k == 0.0) {                // B0 at every radius, also at r <= 0
            B0r = f.B0;
            kG = 0.0;
        }
    }
}

// Bilinear lookup of the z-Taylor coefficients: int() truncation, index
// clamped to [0, n-2], weights not clamped (linear extrapolation).
// Node indices are 32-bit (the largest table offset, NX * NY * 12 values, is
// below 2^31): the truncation saturates outside the int range, where the
// clamp applies anyway, and a NaN coordinate truncates to node 0.
__device__ __forceinline__ int trunc_index(double q) { return __double2int_rz(q); }

// The cell of (x, y) in the z-Taylor map and the position in it
struct Cell {
    int node;            // i * fi_size + j
    double tx, ty;
};

__device__ __forceinline__ Cell map_cell(const FieldK &f, double x, double y, int &clamped)
{
    // cell index and weights from (x - x_min) times 1 / step: within an ulp
    // of the reference's quotient; where that moves the index across a node
    // line, the bilinear interpolant is continuous there, so the field
    // changes by rounding only
    const double qx = (x - f.r_min) * f.inv_r_step;
    const double qy = (y - f.fi_min) * f.inv_fi_step;
    const int nr = (int)f.r_size, nf = (int)f.fi_size;
    const int i0 = trunc_index(qx), j0 = trunc_index(qy);
    const int i = min(max(i0, 0), nr - 2), j = min(max(j0, 0), nf - 2);
    clamped += (i != i0) + (j != j0);
    return {i * nf + j, qx - (double)i, qy - (double)j};
}

// The sums of the z-Taylor terms: hz = sum_n bz_n z^(2n), and hf, hr =
// sum_n (bfi_n, br_n) z^(2n), which the caller multiplies by z.
//
// A warp load costs the L1 data pipe one cycle per distinct 128-byte line it
// touches, and at least its bytes / 128 (measured: 8.5 cycles for a 32-byte load
// of one line, 16 for 16 lines, 32 for 32), and large bunches are bound by
// that pipe.  So the table is split into planes of one load each (FieldK):
// four nodes of a row share a line, where whole 64-byte nodes put two loads
// on every line of two.  Order 2, 1e5 particles, 720 steps: 1.74 ms with whole
// nodes, 1.54 ms in planes; 1e6 particles, 60 steps with space charge (128
// registers): 1.90 and 1.69 ms.
template <int MAXO>
__device__ __forceinline__ void z_taylor64(const FieldK &f, const Cell &cell, double z, double &hz, double &hf,
                                           double &hr)
{
    constexpr int NV = 3 * MAXO;
    const double tx = cell.tx, ty = cell.ty;
    const double w[4] = {(1.0 - tx) * (1.0 - ty), (1.0 - tx) * ty, tx * (1.0 - ty), tx * ty};
    const int nf = (int)f.fi_size;
    // accumulate node by node in the reference's order w00, w01, w10, w11
    double acc[NV];
#pragma unroll
    for (int a = 0; a < NV; a += 4) {
        constexpr int LAST = NV % 4 == 3 ? 4 : NV % 4;
        const int W = NV - a >= 4 || LAST == 0 ? 4 : LAST;
        const double *pl = f.nodes64 + a * f.plane + (int64_t)cell.node * W;
        const double *nd[4] = {pl, pl + W, pl + nf * W, pl + nf * W + W};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double t[4];
            if (W == 4) ldg_v4(nd[k], t);
            else if (W == 2) ldg_v2(nd[k], t);
            else t[0] = __ldg(nd[k]);
#pragma unroll
            for (int b = 0; b < W; ++b)
                if (a + b < NV) acc[a + b] = (k == 0) ? w[0] * t[b] : acc[a + b] + w[k] * t[b];
        }
    }
    const double z2 = z * z;
    hz = acc[NV - 3];
    hf = acc[NV - 2];
    hr = acc[NV - 1];
#pragma unroll
    for (int n = MAXO - 2; n >= 0; --n) {
        hz = fma(hz, z2, acc[3 * n]);
        hf = fma(hf, z2, acc[3 * n + 1]);
        hr = fma(hr, z2, acc[3 * n + 2]);
    }
    hz *= z2;
    hf *= z2;
    hr *= z2;
}

// The field at (r, fim, z): the mid-plane field with its z-linear terms from
// the two one-dimensional tables, and the z-Taylor terms from the map.  ir =
// 1 / r to an ulp.  The cell coordinates of the tables are exact (power-of-two
// cells), so their evaluation adds a few ulp, as the exponentials and the
// 16-term series about the map centre did before; without their branches and
// divisions, and with every load issued before the first use, the field is one
// stretch of code whose chains overlap.  Measured (720 steps, z-Taylor order 2,
// RF): 1e5 particles Boris 2.47 -> 2.07 ms, RK4 11.3 -> 9.6 ms; 1280
// azimuth-domain tracks of 523 steps: 2.46 -> 1.43 ms.
template <int MAXO>
__device__ __forceinline__ void field64(const FieldK &f, double r, double ir, double fim, double z, double &Bz,
                                        double &Br, double &Bfi, int &clamped)
{
    double hz = 0.0, hf = 0.0, hr = 0.0;
    Cell cell;
    if constexpr (MAXO >= 1) cell = map_cell(f, r, fim, clamped);
    const Tables t = tables_fetch(f, r, fim);
    if constexpr (MAXO >= 1) z_taylor64<MAXO>(f, cell, z, hz, hf, hr);
    double F, Fp, B0r, kG;
    tables_eval(f, t, r, F, Fp, B0r, kG);
    const double B0Fp = B0r * Fp;
    Bz = fma(B0r, F, hz);
    Bfi = fma(B0Fp, ir, hf) * z;
    Br = (fma(kG, F, hr) - B0Fp * t.spiral_p) * z;
}

// bharmonics_kernel_1d (src/FFAG_Field.py:1541-1587) for one particle: the
// Bz sum of the field-error harmonics (rows m, amp, phase, rmin, rmax of the
// device table h) whose radial band holds r, fi the unwrapped azimuth; the
// caller adds it to Bz after the map as the reference does, Br and Bfi take
// nothing.  Compiled only into the kernel variants launched for a map with
// harmonics, so the others keep their registers.
__device__ __forceinline__ double harmonics_bz(const double *h, int n, double r, double fi)
{
    if (!(r > 0.0)) return 0.0;
    double b = 0.0;
    for (int k = 0; k < n; ++k) {
        const double *row = h + 5 * k;
        if (row[3] <= r && r <= row[4]) b += row[1] * cos(row[0] * fi + row[2]);
    }
    return b;
}

// One gap of emap_kernel: inside test on (x, y) = r (cos fi, sin fi).
__device__ __forceinline__ bool gap_inside(const RFK &rf, int g, double x, double y)
{
    if (x < rf.box[g][0] || x > rf.box[g][1] || y < rf.box[g][2] || y > rf.box[g][3]) return false;
    double prev = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double x0 = rf.poly_x[g][j], y0 = rf.poly_y[g][j];
        const double x1 = rf.poly_x[g][(j + 1) & 3], y1 = rf.poly_y[g][(j + 1) & 3];
        const double cross = (x1 - x0) * (y - y0) - (y1 - y0) * (x - x0);
        if (j == 0) prev = cross;
        else if (cross * prev < 0.0) return false;
    }
    return true;
}

__device__ __forceinline__ bool in_window(const RFK &rf, int g, double fi)
{
    double d = fi - rf.win_center[g];
    d -= (2.0 * PI) * rint(d * (0.5 / PI));   // a flip of rint at a half turn leaves |d| ~ pi, outside
    return fabs(d) <= rf.win_half[g];
}

// Spiral gaps (interpolate_spiral_emap_unique_gap_kernel, src/FFAG_MathTools.py:
// 1042-1114, with shift_to_nearest_window :1118-1135 and
// Bilinear_interp_2D_vect_uniform_3fields :940-1039): the first gap whose
// window holds the particle, the bilinear map value, the RF factor.  The
// roundings are the reference's, one operation at a time (no contraction).
__device__ __forceinline__ double3 rf_spiral64(const RFK &rf, double acc, double r, double fi, double z, double rfph)
{
    const double tw = 2.0 * PI;
    int hit = -1;
    double phl = 0.0;
    for (int g = 0; g < rf.ngaps; ++g) {
        const double d = fi - rf.gap_az[g];
        const double k = rint((rf.sp_phic - d) / tw);
        const double l = __dadd_rn(d, __dmul_rn(k, tw));
        if (l >= rf.sp_phi0 && l <= rf.sp_phimax) {
            hit = g;
            phl = l;
            break;
        }
    }
    if (hit < 0) return make_double3(0.0, 0.0, 0.0);
    int i = (int)floor((r - rf.sp_r0) / rf.sp_dr);
    int j = (int)floor((phl - rf.sp_phi0) / rf.sp_dphi);
    i = i < 0 ? 0 : (i >= rf.sp_nr - 1 ? rf.sp_nr - 2 : i);
    j = j < 0 ? 0 : (j >= rf.sp_nphi - 1 ? rf.sp_nphi - 2 : j);
    const double tx = (r - __dadd_rn(rf.sp_r0, __dmul_rn((double)i, rf.sp_dr))) / rf.sp_dr;
    const double ty = (phl - __dadd_rn(rf.sp_phi0, __dmul_rn((double)j, rf.sp_dphi))) / rf.sp_dphi;
    const double w00 = (1.0 - tx) * (1.0 - ty), w01 = (1.0 - tx) * ty, w10 = tx * (1.0 - ty), w11 = tx * ty;
    // node (i, j): Er, Ez/z as one 16-byte load, Ephi in the next
    const double2 *nd = reinterpret_cast<const double2 *>(rf.sp);
    const int64_t b0 = 2 * ((int64_t)i * rf.sp_nphi + j), b1 = b0 + 2 * (int64_t)rf.sp_nphi;
    const double2 a00 = __ldg(nd + b0), a01 = __ldg(nd + b0 + 2), a10 = __ldg(nd + b1), a11 = __ldg(nd + b1 + 2);
    const double f00 = __ldg(rf.sp + 2 * b0 + 2), f01 = __ldg(rf.sp + 2 * b0 + 6);
    const double f10 = __ldg(rf.sp + 2 * b1 + 2), f11 = __ldg(rf.sp + 2 * b1 + 6);
    const double er = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(w00, a00.x), __dmul_rn(w01, a01.x)),
                                          __dmul_rn(w10, a10.x)), __dmul_rn(w11, a11.x));
    const double ez = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(w00, a00.y), __dmul_rn(w01, a01.y)),
                                          __dmul_rn(w10, a10.y)), __dmul_rn(w11, a11.y));
    const double ef = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(w00, f00), __dmul_rn(w01, f01)),
                                          __dmul_rn(w10, f10)), __dmul_rn(w11, f11));
    const double s = sin(rfph + rf.rf_shift[hit]);
    return make_double3((acc * er) * s, ((acc * ez) * z) * s, (acc * ef) * s);   // Er, Ez, Efi
}

// Er, Efi of fixed gap g at a particle inside its angular window
__device__ __forceinline__ double2 gap_field(const RFK &rf, int g, double acc, double r, double fi, double rfph)
{
    double sf, cf;
    sincos(fi, &sf, &cf);
    if (!gap_inside(rf, g, r * cf, r * sf)) return make_double2(0.0, 0.0);
    double sd, cd;
    sincos(rf.theta_n[g] - fi, &sd, &cd);
    const double s = sin(rfph + rf.rf_shift[g]);
    return make_double2((acc * cd) * s, (acc * sd) * s);
}

// The FP64 kernels call their rare branches out of line (a few steps of a turn
// come there), which keeps the usual step short.  The FP32C kernels, at 80
// registers with spills, have no registers to spare around a call and keep
// them inline: with the calls FP32C RK4 took 7 % and FP32C Boris with space
// charge 14 % longer (5.48 against 5.11 ms per 360 steps of 1e5 particles,
// 1.94 against 1.71 ms per 60 steps of 1e6).
__device__ __noinline__ double2 gap_field64(const RFK &rf, int g, double acc, double r, double fi, double rfph)
{
    return gap_field(rf, g, acc, r, fi, rfph);
}

// RF field (cylindrical r, z, fi components) times sin(RF phase +
// rf_shift[gap]).  Fixed gaps, reference semantics: every gap's emap_kernel
// call overwrites the field, so only the last gap contributes (no Ez);
// physical_sum adds all gaps.  Spiral gaps: rf_spiral64.
__device__ __forceinline__ void rf_field64(const RFK &rf, double acc, double r, double fi, double z, double rfph,
                                           double &Er, double &Ez, double &Efi)
{
    Er = 0.0;
    Ez = 0.0;
    Efi = 0.0;
    if (!rf.enable) return;
    if (rf.sp) {
        const double3 e = rf_spiral64(rf, acc, r, fi, z, rfph);
        Er = e.x;
        Ez = e.y;
        Efi = e.z;
        return;
    }
    const int g0 = rf.physical_sum ? 0 : rf.ngaps - 1;
    for (int g = g0; g < rf.ngaps; ++g) {
        if (!in_window(rf, g, fi)) continue;
        const double2 e = gap_field(rf, g, acc, r, fi, rfph);
        Er += e.x;
        Efi += e.y;
    }
}

// The RF field of the FP64 kernels at a point: false (and no field) outside
// the gaps.  With the reference's semantics on fixed gaps (rf.single >= 0,
// the one gap that acts) the angular window decides inline and only the few
// steps inside it call gap_field64.
__device__ __noinline__ double3 rf_general64(const RFK &rf, double acc, double r, double fi, double z, double rfph)
{
    double Er, Ez, Efi;
    rf_field64(rf, acc, r, fi, z, rfph, Er, Ez, Efi);
    return make_double3(Er, Ez, Efi);
}

__device__ __forceinline__ bool rf_hit64(const RFK &rf, const double *acc, double r, double fi, double z, double rfph,
                                         double3 &e)
{
    if (rf.single >= 0) {
        if (!in_window(rf, rf.single, fi)) return false;
        const double2 g = gap_field64(rf, rf.single, __ldg(acc), r, fi, rfph);
        e = make_double3(g.x, 0.0, g.y);
        return g.x != 0.0 || g.y != 0.0;
    }
    if (!rf.enable) return false;
    e = rf_general64(rf, __ldg(acc), r, fi, z, rfph);
    return e.x != 0.0 || e.y != 0.0 || e.z != 0.0;
}

__device__ __forceinline__ double3 atan_rotation(double y, double x)
{
    const double a = atan2(y, x);
    double s, c;
    sincos(a, &s, &c);
    return make_double3(a, s, c);
}

__device__ __noinline__ double3 wide_rotation(double y, double x) { return atan_rotation(y, x); }

// Azimuth change of one step and its sine / cosine, from the new position's
// unit vector in the local frame: sin and cos of the step angle are y / r and
// x / r (r^-1 is at hand from the drift); a step turns the particle by about
// 2 pi / (steps per turn), and for |sin| < 0.02 the angle is the arcsine series
//   asin(s) = s (1 + s^2/6 + 3 s^4/40 + 5 s^6/112 + 35 s^8/1152)
// (truncation < 3e-19 relative): no division and no sin/cos series.
template <bool INLINE = false>
__device__ __forceinline__ void step_rotation(double y, double x, double ir, double &a, double &s, double &c)
{
    const double s0 = y * ir;
    if (x > 0.0 && fabs(s0) < 0.02) {
        const double s2 = s0 * s0;
        a = s0 * (1.0 + s2 * (1.0 / 6 + s2 * (3.0 / 40 + s2 * (5.0 / 112 + s2 * (35.0 / 1152)))));
        s = s0;
        c = x * ir;
    } else {
        const double3 w = INLINE ? atan_rotation(y, x) : wide_rotation(y, x);
        a = w.x;
        s = w.y;
        c = w.z;
    }
}

__device__ __forceinline__ void status_add(int64_t *status, int lost, int bad, int oob)
{
    if (!status) return;
    const unsigned mask = __activemask();
    for (int off = 16; off > 0; off >>= 1) {
        lost += __shfl_down_sync(mask, lost, off);
        bad += __shfl_down_sync(mask, bad, off);
        oob += __shfl_down_sync(mask, oob, off);
    }
    if ((threadIdx.x & 31) == __ffs(mask) - 1) {
        if (lost) atomicAdd((unsigned long long *)&status[FFA_STATUS_LOST], (unsigned long long)lost);
        if (bad) atomicAdd((unsigned long long *)&status[FFA_STATUS_NAN], (unsigned long long)bad);
        if (oob) atomicAdd((unsigned long long *)&status[FFA_STATUS_OUT_OF_MAP], (unsigned long long)oob);
    }
}

// Azimuth-crossing test of detect_azimuth_crossing (src/FFAG_MathTools.py:
// 1633-1695) on the step's pre / post azimuth, and the record append.  The
// reductions mod 2 pi are a - 2 pi floor(a / 2 pi) with no fused multiply-add,
// as in fast_mod_parallel (src/FFAG_MathTools.py:1554-1557); the targets come in
// already reduced to [0, 2 pi).
__device__ __forceinline__ double mod_2pi(double a)
{
    const double tw = 2.0 * PI;
    return __dsub_rn(a, __dmul_rn(tw, floor(a / tw)));
}

// sin and cos of a small angle (|d| below a push step's azimuth advance, a
// few 1e-3 rad) by their Taylor series to d^9 / 9! and d^8 / 8!: truncation
// below 1e-22 for |d| < 0.02.
__device__ __forceinline__ void sincos_small(double d, double &s, double &c)
{
    const double d2 = d * d;
    s = d * (1.0 - d2 * (1.0 / 6 - d2 * (1.0 / 120 - d2 * (1.0 / 5040 - d2 * (1.0 / 362880)))));
    c = 1.0 - d2 * (0.5 - d2 * (1.0 / 24 - d2 * (1.0 / 720 - d2 * (1.0 / 40320))));
}

// One-turn-map sums at a crossing (the fit_sums form of ffa_crossing).  d0
// and d1: the step's start and end azimuth relative to the target (d0 <= 0
// <= d1, reduced mod 2 pi).
__device__ __forceinline__ void fit_accumulate(const ffa_crossing &xc, int64_t i, double dt, double d0, double d1,
                                               const double pre[7], const double post[7])
{
    // Cartesian state in the frame whose x axis points at the target azimuth
    double s0, c0, s1, c1;
    sincos_small(d0, s0, c0);
    sincos_small(d1, s1, c1);
    const double r0 = pre[0], vf0 = r0 * pre[5], r1 = post[0], vf1 = r1 * post[5];
    const double X0 = r0 * c0, Y0 = r0 * s0, VX0 = pre[1] * c0 - vf0 * s0, VY0 = pre[1] * s0 + vf0 * c0;
    const double X1 = r1 * c1, Y1 = r1 * s1, VX1 = post[1] * c1 - vf1 * s1, VY1 = post[1] * s1 + vf1 * c1;
    double tau = Y0 / (Y0 - Y1);
    for (int it = 0; it < 3; ++it) {
        const double t2 = tau * tau, t3 = t2 * tau;
        const double y = (2 * t3 - 3 * t2 + 1) * Y0 + (t3 - 2 * t2 + tau) * VY0 * dt + (3 * t2 - 2 * t3) * Y1 +
                         (t3 - t2) * VY1 * dt;
        const double dy = (6 * t2 - 6 * tau) * Y0 + (3 * t2 - 4 * tau + 1) * VY0 * dt + (6 * tau - 6 * t2) * Y1 +
                          (3 * t2 - 2 * tau) * VY1 * dt;
        tau = tau - y / dy;
    }
    const double t2 = tau * tau, t3 = t2 * tau;
    const double h00 = 2 * t3 - 3 * t2 + 1, h10 = t3 - 2 * t2 + tau, h01 = 3 * t2 - 2 * t3, h11 = t3 - t2;
    const int k = xc.fit_instance[i];
    const double *ce = xc.fit_centre + 4 * k, *sc = xc.fit_scale + 4 * k;
    double u[4];
    u[0] = h00 * X0 + h10 * VX0 * dt + h01 * X1 + h11 * VX1 * dt;
    u[1] = VX0 + tau * (VX1 - VX0);
    u[2] = h00 * pre[2] + h10 * pre[3] * dt + h01 * post[2] + h11 * post[3] * dt;
    u[3] = pre[3] + tau * (post[3] - pre[3]);
    for (int c = 0; c < 4; ++c) u[c] = (u[c] - ce[c]) * sc[c];
    double *acc = xc.fit_sums + (int64_t)k * FFA_FIT_SUMS;
    double *w = xc.fit_last + 4 * i;
    if (xc.fit_has[i]) {
        for (int pl = 0; pl < 2; ++pl) {
            const double f0 = w[2 * pl], f1 = w[2 * pl + 1], a = u[2 * pl], b = u[2 * pl + 1];
            double *q = acc + 12 * pl;
            atomicAdd(q + 0, f0 * f0);
            atomicAdd(q + 1, f0 * f1);
            atomicAdd(q + 2, f0);
            atomicAdd(q + 3, f1 * f1);
            atomicAdd(q + 4, f1);
            atomicAdd(q + 5, 1.0);
            atomicAdd(q + 6, a * f0);
            atomicAdd(q + 7, a * f1);
            atomicAdd(q + 8, a);
            atomicAdd(q + 9, b * f0);
            atomicAdd(q + 10, b * f1);
            atomicAdd(q + 11, b);
        }
    }
    atomicAdd(acc + 24, 1.0);
    for (int c = 0; c < 4; ++c) w[c] = u[c];
    xc.fit_has[i] = 1;
}

__device__ __forceinline__ void xing_check(const ffa_crossing &xc, int64_t i, int64_t gs, const double pre[7],
                                           const double post[7], int surv_after, int inj, double esr, double esz,
                                           double esf, double dt)
{
    const double tw = 2.0 * PI;
    const double a = mod_2pi(pre[4]), b = mod_2pi(post[4]);
    for (int t = 0; t < xc.ntargets; ++t) {
        const double target = xc.target[t];
        bool hit;
        double ratio = 0.0;
        if (b >= a) {
            hit = a <= target && target <= b;
            if (hit && b - a > 1e-12) ratio = (target - a) / (b - a);
        } else {
            hit = (target >= a && target < tw) || (target >= 0 && target <= b);
            if (hit) {
                const double span = (b + tw) - a;
                if (span > 1e-12) ratio = ((target <= b ? target + tw : target) - a) / span;
            }
        }
        if (!hit) continue;
        if (xc.fit_sums) {
            double d0 = a - target, d1 = b - target;
            if (b < a) {
                if (target >= a) d1 += tw;
                else d0 -= tw;
            }
            fit_accumulate(xc, i, dt, d0, d1, pre, post);
            continue;
        }
        const unsigned long long k = atomicAdd((unsigned long long *)xc.count, 1ull);
        if ((int64_t)k >= xc.capacity) continue;
        double *rec = xc.buf + (int64_t)k * FFA_CROSSING_RECORD;
        rec[0] = (double)t;
        rec[1] = (double)i;
        rec[2] = (double)gs;
        rec[3] = ratio;
        for (int c = 0; c < 7; ++c) { rec[4 + c] = pre[c]; rec[11 + c] = post[c]; }
        rec[18] = (double)surv_after;
        rec[19] = (double)inj;
        rec[20] = esr; rec[21] = esz; rec[22] = esf;
    }
}

// Position of step gs in its space-charge interval (0 in the first interval)
__device__ __forceinline__ int sc_phase(const PushK &p, int64_t gs)
{
    return gs >= p.sc_step ? (int)(gs % p.sc_step) : 0;
}

// Linear extrapolation of the space-charge field between updates
// (src/FFAG_track.py:449-478).
struct SCExtrap {
    bool pre = false, pp = false;
    double epr = 0, epz = 0, epf = 0, eqr = 0, eqz = 0, eqf = 0;
    __device__ void load(const ffa_state_soa &S, int64_t i)
    {
        pre = S.sc_pre[i] != 0;
        pp = S.sc_pp[i] != 0;
        if (pre) {
            epr = S.e_pre_r[i]; epz = S.e_pre_z[i]; epf = S.e_pre_fi[i];
            if (pp) { eqr = S.e_pp_r[i]; eqz = S.e_pp_z[i]; eqf = S.e_pp_fi[i]; }
        }
    }
    // ph: the step's position gs mod sc_step in its interval (0 in the first)
    __device__ void apply(int ph, double inv_sc, double &esr, double &esz, double &esf) const
    {
        if (pre) blend((double)ph * inv_sc, esr, esz, esf);
    }
    // FP32C: the fraction formed anew from the step number
    __device__ void apply(const PushK &p, int64_t gs, double &esr, double &esz, double &esf) const
    {
        if (pre) blend(gs >= p.sc_step ? (double)(gs % p.sc_step) / (double)p.sc_step : 0.0, esr, esz, esf);
    }
    __device__ void blend(double sf, double &esr, double &esz, double &esf) const
    {
        if (pp) {
            esr = epr + sf * (epr - eqr);
            esz = epz + sf * (epz - eqz);
            esf = epf + sf * (epf - eqf);
        } else {
            esr = epr; esz = epz; esf = epf;
        }
    }
};

// ------------------------------------------------- field, float32 kernels
//
// The FP32C Boris pusher spends float32 arithmetic only where float64 is
// expensive: the exponentials of the fringe sigmoids and of the power law
// (expf / log1pf, accurately rounded library functions) and the bilinear
// lookup of the z-Taylor nodes (float32 table).  The constants these values
// are combined with, the products with r and z, and the whole Boris push stay
// float64, so float32 rounding enters the field as an error of relative size
// ~1e-7 that changes from step to step, never as a fixed scale error of the
// bending (a fixed bias of the bending shifts the revolution time and, with
// the RF on, the synchronous phase).
template <int MAXO>
__device__ __forceinline__ void field_mixed(const FieldK &f, double r, double ir, double fim, double z,
                                            double &Bz, double &Br, double &Bfi, int &clamped)
{
    // the table lookup first, so its loads are in flight during the rest
    double hz = 0.0, hf = 0.0, hr = 0.0;
    if constexpr (MAXO >= 1) {
        const double qx = (r - f.r_min) * f.inv_r_step;
        const double qy = (fim - f.fi_min) * f.inv_fi_step;
        const int nr = (int)f.r_size, nf = (int)f.fi_size;
        int i = trunc_index(qx), jj = trunc_index(qy);
        if (i < 0) { i = 0; ++clamped; } else if (i >= nr - 1) { i = nr - 2; ++clamped; }
        if (jj < 0) { jj = 0; ++clamped; } else if (jj >= nf - 1) { jj = nf - 2; ++clamped; }
        const float tx = (float)(qx - (double)i), ty = (float)(qy - (double)jj);
        const float w[4] = {(1.0f - tx) * (1.0f - ty), (1.0f - tx) * ty, tx * (1.0f - ty), tx * ty};
        constexpr int NP = (3 * MAXO <= 4) ? 4 : ((3 * MAXO <= 8) ? 8 : 12);
        constexpr int NV = 3 * MAXO;
        const float *nd[4];
        nd[0] = f.nodes32 + (i * nf + jj) * NP;
        nd[1] = nd[0] + NP;
        nd[2] = nd[0] + nf * NP;
        nd[3] = nd[2] + NP;
        float acc[NV];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if constexpr (NP == 8) {   // 32-byte nodes: one 32-byte load each
                float tv[8];
                ldg_v8(nd[k], tv);
#pragma unroll
                for (int b = 0; b < NV; ++b) acc[b] = (k == 0) ? w[0] * tv[b] : acc[b] + w[k] * tv[b];
            } else {
#pragma unroll
                for (int a = 0; a < NV; a += 4) {
                    const float4 t = __ldg(reinterpret_cast<const float4 *>(nd[k] + a));
                    const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (a + b < NV) acc[a + b] = (k == 0) ? w[0] * tv[b] : acc[a + b] + w[k] * tv[b];
                }
            }
        }
        const double z2 = z * z;
        double ze = z2, zo = z2 * z;
#pragma unroll
        for (int n = 0; n < MAXO; ++n) {
            hz += (double)acc[3 * n] * ze;
            hf += (double)acc[3 * n + 1] * zo;
            hr += (double)acc[3 * n + 2] * zo;
            ze *= z2;
            zo *= z2;
        }
    }

    double spiral = 0.0, spiral_p = 0.0;
    if (!f.spiral_zero) {
        for (int a = 0; a < f.n_spoly; ++a) spiral = spiral * r + f.spoly[a];
        for (int a = 0; a < f.n_spolyp; ++a) spiral_p = spiral_p * r + f.spolyp[a];
    }
    double B0r, B0r_p;
    if (f.k == 0.0) {
        B0r = f.B0;
        B0r_p = 0.0;
    } else {
        // (r / r_ref)^(k-1) with r / r_ref = 1 + eps, eps formed in float64
        const float eps = (float)((r - f.r_ref) * f.inv_r_ref);
        const double g = (double)expf((float)(f.km1 * (double)log1pf(eps)));
        B0r_p = f.kc1 * g;
        B0r = f.c1 * g * r;
    }
    double fs = fim;
    if (!f.spiral_zero) {   // as in tables_fetch
        fs = fim - spiral;
        fs -= f.period * floor(fs * f.inv_period);
    }
    double F = 0.0, Fp = 0.0;
    for (int j = 0; j < f.n_seg; ++j) {
        const float a1 = (float)(f.seg_k[j] * (fs - f.seg_x0[j]));
        const float a2 = (float)(f.seg_k[j] * (fs - f.seg_x1[j]));
        // exponents capped at 80 so e stays finite: past it s < 2e-35, which
        // is 0 in every sum below, and e * s would otherwise be inf * 0.
        // Where a sigmoid is saturated at 1 (e < 4e-11) its exponential is
        // skipped and e taken as 0.
        float e1 = 0.0f, e2 = 0.0f;
        if (a1 < 24.0f) e1 = expf(fminf(-a1, 80.0f));
        if (a2 > -24.0f) e2 = expf(fminf(a2, 80.0f));
        const float s1 = __frcp_rn(1.0f + e1), s2 = __frcp_rn(1.0f + e2);
        const float ss = s1 * s2;
        // s1' s2 + s1 s2' = k s1 s2 ((1 - s1) - (1 - s2)) with 1 - s = e s:
        // no cancellation where a sigmoid saturates
        const float dd = e1 * s1 - e2 * s2;
        F += f.seg_y[j] * (double)ss;
        Fp += f.seg_yk[j] * (double)(ss * dd);
    }
    Bz = B0r * F + hz;
    Bfi = B0r * Fp * ir * z + hf;
    Br = (B0r_p * F - B0r * Fp * spiral_p) * z + hr;
}

// ------------------------------------------------------------ Boris fp64

// One-warp blocks; at 80 registers a launch holds the most warps that run
// without heavy spills.  The register file is split over
// the SM's four schedulers (16384 registers each): 80 x 32 = 2560 registers
// per warp gives 6 warps per scheduler, 24 per SM, 3552 on 148 SMs, so the
// 3125 warps of a 1e5-particle bunch are resident in one wave.  At 88
// registers it is 5 per scheduler (2960 warps): the last 165 warps then run
// all their steps as a second, nearly empty wave (measured: 5.09 ms per
// 720-step turn at 88 registers, 3.81 ms at 80).

// The FP64 step carries u = gamma v and 1 / gamma instead of the velocities.
// The reference forms gamma from |v| at the start of every step and again
// after each half kick; but a step without an electric field turns u and
// leaves gamma as it is, and u is known from the step before.  So a
// particle's 1 / gamma is recomputed only after a kick (an RF gap, space
// charge); the velocities are formed where they are read: at the end of the
// launch, at a crossing, and when a particle leaves flight (not injected or
// lost particles keep velocities, which the reference's Cartesian round trip
// perturbs).  A live step is then one stretch of code without branches but the
// rare ones (gap window, wide steps), so its independent chains overlap.
// Large bunches are bound by the L1 data pipe (z_taylor64), small ones by one
// step's chain: the node loads from L2 (about 300 cycles) and some 110
// dependent FP64 operations of 8 cycles.  720 steps, with the tables of field64
// and the planes of z_taylor64: 1e5 particles, order 2, RF 2.47 -> 1.42 ms; 1e4
// particles, order 4, 1.88 -> 0.77 ms; 1e6 particles, 60 steps with space
// charge 2.05 -> 1.69 ms.
template <int MAXO, bool SC, bool XING, int NREG, bool HARM = false>
__global__ void __maxnreg__(NREG) boris_f64_kernel(const __grid_constant__ PushK p)
{
    const int64_t t_ = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t_ >= p.n) return;
    const int64_t i = p.st.order ? (int64_t)__ldg(p.st.order + t_) : t_;   // the particle this thread advances
    const FieldK &f = p.f;
    const ffa_state_soa &S = p.st;
    // (a, b, c): in flight u_r, u_fi, u_z; otherwise vr, dfi/dt, vz
    double r = S.r[i], a = S.vr[i], z = S.z[i], c = S.vz[i], fi = S.fi[i], b = S.f5[i];
    double rfph = S.rf[i];
    int inj = S.inj[i], surv = S.surv[i];
    // the launch's step at which the particle is injected (none: -1)
    const int64_t injs = (S.inj_step ? (int64_t)S.inj_step[i] : -1) - p.step0;
    const int inj_at = injs >= 0 && injs < p.nsteps ? (int)injs : -1;
    double esr = S.esc_r[i], esz = S.esc_z[i], esf = S.esc_fi[i];
    const bool esc = SC || esr != 0.0 || esz != 0.0 || esf != 0.0;   // also for NaN
    SCExtrap ex;
    int ph = 0;
    if (SC) {
        ex.load(S, i);
        ph = sc_phase(p, p.step0);
    }
    double ir = 1.0 / r, ig = 0.0;           // 1 / r and 1 / gamma, carried
    auto take_off = [&]() {
        const double vf = r * b, x = 1 - (a * a + vf * vf + c * c) * p.inv_cc, g = rsqrt(x);
        a *= g;
        b = g * vf;
        c *= g;
        ig = x * g;
    };
    auto land = [&]() {
        a *= ig;
        b = r > 1e-12 ? b * ig * ir : 0.0;
        c *= ig;
    };
    // the turn of u about -B by the angle of the step (Boris)
    auto turn = [&](double Bz, double Br, double Bfi) {
        const double cb = -p.hqm * ig;
        const double tx = cb * Br, ty = cb * Bfi, tz = cb * Bz;
        const double pa = a + (b * tz - c * ty);
        const double pb = b + (c * tx - a * tz);
        const double pc = c + (a * ty - b * tx);
        const double sb = 2.0 * rcp64(1.0 + (tx * tx + ty * ty + tz * tz));
        const double sx = sb * tx, sy = sb * ty, sz = sb * tz;
        a += (pb * sz - pc * sy);
        b += (pc * sx - pa * sz);
        c += (pa * sy - pb * sx);
    };
    auto kick = [&](const double3 &e) {      // half the step's electric kick (e: r, z, fi)
        a = fma(p.hqm, e.x, a);
        b = fma(p.hqm, e.z, b);
        c = fma(p.hqm, e.y, c);
        ig = rsqrt64(fma(a * a + b * b + c * c, p.inv_cc, 1.0));
    };
    bool live = inj == 1 && surv == 1;
    if (live) take_off();
    int lost = 0, oob = 0;
    const double *drf = p.drf + p.step0;

    for (int s = 0; s < p.nsteps; ++s) {
        if (s == inj_at) {
            inj = 1;
            surv = 1;
            if (!live) take_off();
            live = true;
        }
        if (SC) {
            ex.apply(ph, p.inv_sc, esr, esz, esf);
            const int64_t gs = p.step0 + s;
            ph = (gs + 1 <= p.sc_step || ph + 1 == p.sc_step) ? 0 : ph + 1;   // sc_phase of the next step
        }
        double pre[7];
        const int surv0 = surv;
        if constexpr (XING) {
            pre[0] = r; pre[2] = z; pre[4] = fi; pre[6] = rfph;
            pre[1] = live ? a * ig : a;
            pre[3] = live ? c * ig : c;
            pre[5] = live ? (r > 1e-12 ? b * ig * ir : 0.0) : b;
        }
        if (live) {
            // fi mod the sector; a multiply by 1 / period instead of the
            // division can move floor() only where fi / period is within an
            // ulp of an integer, i.e. between two equal values of the
            // periodic field (0 and the period)
            const double fim = fi - f.period * floor(fi * f.inv_period);
            double Bz, Br, Bfi;
            field64<MAXO>(f, r, ir, fim, z, Bz, Br, Bfi, oob);
            if constexpr (HARM) Bz += harmonics_bz(f.harm, f.n_harm, r, fi);
            if (r > p.ap.rmax || r < p.ap.rmin || z > p.ap.zmax || z < p.ap.zmin) {   // infinite when off
                surv = 0;
                ++lost;
            }
            double3 e = make_double3(0.0, 0.0, 0.0);
            const bool hit = rf_hit64(p.rf, p.acc + p.step0 + s, r, fi, z, rfph, e);
            if (esc || hit) {
                if (esc) {
                    if (!SC) { esr = S.esc_r[i]; esz = S.esc_z[i]; esf = S.esc_fi[i]; }   // not held over the loop
                    e.x += esr;
                    e.y += esz;
                    e.z += esf;
                }
                kick(e);
                turn(Bz, Br, Bfi);
                kick(e);
            } else {
                turn(Bz, Br, Bfi);
            }
            // drift, in the frame x along r-hat, y along fi-hat
            const double dtg = p.dt * ig;
            const double xn = fma(a, dtg, r), yn = b * dtg;
            z = fma(c, dtg, z);
            const double rr2 = xn * xn + yn * yn;
            ir = rsqrt64(rr2);
            r = rr2 * ir;
            double dfi, sn, cn;
            step_rotation(yn, xn, ir, dfi, sn, cn);
            fi = fi + dfi;
            const double an = a * cn + b * sn;
            b = b * cn - a * sn;
            a = an;
            if (surv == 0) {
                land();
                live = false;
            }
        } else {
            // skipped particle: the reference's Cartesian round trip
            double sinFi, cosFi;
            sincos(fi, &sinFi, &cosFi);
            const double x = r * cosFi, y = r * sinFi;
            const double vx = a * cosFi - r * b * sinFi;
            const double vy = a * sinFi + r * b * cosFi;
            const double rn = sqrt(x * x + y * y);
            a = vx * cosFi + vy * sinFi;
            const double vfi = -vx * sinFi + vy * cosFi;
            b = rn > 1e-12 ? vfi / rn : 0.0;
            r = rn;
            ir = 1.0 / rn;
        }
        rfph += __ldg(drf + s);
        if constexpr (XING) {
            if (surv0 == 1) {
                const double post[7] = {r, live ? a * ig : a, z, live ? c * ig : c, fi,
                                        live ? (r > 1e-12 ? b * ig * ir : 0.0) : b, rfph};
                if (!SC) { esr = S.esc_r[i]; esz = S.esc_z[i]; esf = S.esc_fi[i]; }
                xing_check(p.xing, i, p.step0 + s, pre, post, surv, inj, esr, esz, esf, p.dt);
            }
        }
    }
    if (live) land();
    S.r[i] = r; S.vr[i] = a; S.z[i] = z; S.vz[i] = c; S.fi[i] = fi; S.f5[i] = b;
    S.rf[i] = rfph;
    if (SC) { S.esc_r[i] = esr; S.esc_z[i] = esz; S.esc_fi[i] = esf; }
    S.inj[i] = (uint8_t)inj;
    S.surv[i] = (uint8_t)surv;
    status_add(p.status, lost, !(isfinite(r) && isfinite(fi) && isfinite(z)), oob);
}

// The FP32C step: the float32 field under the reference's velocity form of the
// push, as all its stored results were made.  NREG: the register cap.  80 is
// the default launch shape; the compensated
// float32 pusher without space charge is also built with 72, 64 and 56
// (more resident warps, more spills) for the launch-shape autotuner.  The
// cap changes register allocation only, not the arithmetic.
template <int MAXO, bool SC, bool XING, int NREG = 80, bool HARM = false>
__global__ void __maxnreg__(NREG) boris_f32c_kernel(const __grid_constant__ PushK p)
{
    const int64_t t_ = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t_ >= p.n) return;
    const int64_t i = p.st.order ? (int64_t)__ldg(p.st.order + t_) : t_;   // the particle this thread advances
    const FieldK &f = p.f;
    const ffa_state_soa &S = p.st;
    double r = S.r[i], rdot = S.vr[i], z = S.z[i], zdot = S.vz[i], fi = S.fi[i], fidot = S.f5[i];
    double rfph = S.rf[i];
    double esr = S.esc_r[i], esz = S.esc_z[i], esf = S.esc_fi[i];
    int inj = S.inj[i], surv = S.surv[i];
    const int32_t injs = S.inj_step ? S.inj_step[i] : -1;
    SCExtrap ex;
    if (SC) ex.load(S, i);
    const double m = p.cs.m0, dt = p.dt;
    const double hq = p.hq, hqm = p.hqm, inv_m = p.inv_m, inv_cc = p.inv_cc, inv_mmcc = p.inv_mmcc;
    double ir = 1.0 / r;                     // 1 / r, carried from the previous step
    int lost = 0, oob = 0;

    for (int s = 0; s < p.nsteps; ++s) {
        const int64_t gs = p.step0 + s;
        if (injs == gs) { inj = 1; surv = 1; }
        if (SC) ex.apply(p, gs, esr, esz, esf);
        const double drf = __ldg(p.drf + gs);
        double pre[7];
        const int surv0 = surv;
        if constexpr (XING) {
            pre[0] = r; pre[1] = rdot; pre[2] = z; pre[3] = zdot; pre[4] = fi; pre[5] = fidot; pre[6] = rfph;
        }
        if ((inj == 1) && (surv == 1)) {
            const double acc = __ldg(p.acc + gs);
            // fi mod the sector; a multiply by 1 / period instead of the
            // division can move floor() only where fi / period is within an
            // ulp of an integer, i.e. between two equal values of the
            // periodic field (0 and the period)
            const double fim = fi - f.period * floor(fi * f.inv_period);
            double Bz, Br, Bfi;
            field_mixed<MAXO>(f, r, ir, fim, z, Bz, Br, Bfi, oob);
            if constexpr (HARM) Bz += harmonics_bz(f.harm, f.n_harm, r, fi);
            double Er, Ez, Efi;
            rf_field64(p.rf, acc, r, fi, z, rfph, Er, Ez, Efi);
            Ez += esz;
            Er += esr;
            Efi += esf;
            if (p.ap.enable && (r > p.ap.rmax || r < p.ap.rmin || z > p.ap.zmax || z < p.ap.zmin)) {
                surv = 0;
                ++lost;
            }
            // local frame: x along r-hat, y along fi-hat; B enters negated
            const double vx = rdot, vy = r * fidot, vz = zdot;
            const double Bx = -Br, By = -Bfi, Bzc = -Bz;
            const double v2 = vx * vx + vy * vy + vz * vz;
            const double gamma = rsqrt(1 - v2 * inv_cc);
            double px = gamma * m * vx, py = gamma * m * vy, pz = gamma * m * vz;
            px += hq * Er;
            py += hq * Efi;
            pz += hq * Ez;
            const double p2 = px * px + py * py + pz * pz;
            const double cb = hqm * rsqrt(1 + p2 * inv_mmcc);
            const double tx = cb * Bx, ty = cb * By, tz = cb * Bzc;
            const double pxp = px + (py * tz - pz * ty);
            const double pyp = py + (pz * tx - px * tz);
            const double pzp = pz + (px * ty - py * tx);
            const double t2 = tx * tx + ty * ty + tz * tz;
            const double sb = 2.0 / (1.0 + t2);
            const double sx = sb * tx, sy = sb * ty, sz = sb * tz;
            px += (pyp * sz - pzp * sy);
            py += (pzp * sx - pxp * sz);
            pz += (pxp * sy - pyp * sx);
            px += hq * Er;
            py += hq * Efi;
            pz += hq * Ez;
            const double p2n = px * px + py * py + pz * pz;
            const double igm = inv_m * rsqrt(1 + p2n * inv_mmcc);
            const double vxn = px * igm, vyn = py * igm, vzn = pz * igm;
            const double xn = r + vxn * dt, yn = vyn * dt;
            z = z + vzn * dt;
            zdot = vzn;
            const double rr2 = xn * xn + yn * yn;
            const double irn = rsqrt(rr2);
            const double rn = rr2 * irn;
            double dfi, sn, cn;
            step_rotation<true>(yn, xn, irn, dfi, sn, cn);
            fi = fi + dfi;
            rdot = vxn * cn + vyn * sn;
            const double vfi = -vxn * sn + vyn * cn;
            fidot = rn > 1e-12 ? vfi * irn : 0.0;
            r = rn;
            ir = irn;
        } else {
            // skipped particle: the reference's Cartesian round trip
            double sinFi, cosFi;
            sincos(fi, &sinFi, &cosFi);
            const double x = r * cosFi, y = r * sinFi;
            const double vx = rdot * cosFi - r * fidot * sinFi;
            const double vy = rdot * sinFi + r * fidot * cosFi;
            const double rn = sqrt(x * x + y * y);
            rdot = vx * cosFi + vy * sinFi;
            const double vfi = -vx * sinFi + vy * cosFi;
            fidot = rn > 1e-12 ? vfi / rn : 0.0;
            r = rn;
            ir = 1.0 / rn;
        }
        rfph += drf;
        if constexpr (XING) {
            if (surv0 == 1) {
                const double post[7] = {r, rdot, z, zdot, fi, fidot, rfph};
                xing_check(p.xing, i, gs, pre, post, surv, inj, esr, esz, esf, p.dt);
            }
        }
    }
    S.r[i] = r; S.vr[i] = rdot; S.z[i] = z; S.vz[i] = zdot; S.fi[i] = fi; S.f5[i] = fidot;
    S.rf[i] = rfph;
    S.esc_r[i] = esr; S.esc_z[i] = esz; S.esc_fi[i] = esf;
    S.inj[i] = (uint8_t)inj;
    S.surv[i] = (uint8_t)surv;
    status_add(p.status, lost, !(isfinite(r) && isfinite(fi) && isfinite(z)), oob);
}

// ------------------------------------------------------ Boris, float32 push
//
// The float32 pusher: field and Boris update in float32, the positions (r,
// fi, z) and the RF phase accumulated in float64 from float32 increments.
// It carries the normalised momentum u = gamma v / c across the launch
// (float32) and converts from and to the float64 state once per launch.
// Each step the radius increment comes from
//   r' - r = (2 r dx + dx^2 + dy^2) / (r' + r)
// (dx, dy the local-frame displacement, formed in float32, so the increment
// keeps float32's relative accuracy instead of the radius), the azimuth
// increment from the arcsine series of dy / r'.  The RF gap test runs in
// float64 inside the gap's angular window.  Velocities keep float32
// precision: their rounding (~6e-8 of |u| per step) walks over a run, which
// is what limits this pusher's accuracy.  Not built with space charge,
// crossing capture of the steps' states is.

template <int MAXO>
__device__ __forceinline__ void field_f32(const FieldK &f, double r, double fim, float z, float &Bz, float &Br,
                                          float &Bfi, int &clamped)
{
    float hz = 0.0f, hf = 0.0f, hr = 0.0f;
    if constexpr (MAXO >= 1) {
        const double qx = (r - f.r_min) * f.inv_r_step;
        const double qy = (fim - f.fi_min) * f.inv_fi_step;
        const int nr = (int)f.r_size, nf = (int)f.fi_size;
        int i = trunc_index(qx), jj = trunc_index(qy);
        if (i < 0) { i = 0; ++clamped; } else if (i >= nr - 1) { i = nr - 2; ++clamped; }
        if (jj < 0) { jj = 0; ++clamped; } else if (jj >= nf - 1) { jj = nf - 2; ++clamped; }
        const float tx = (float)(qx - (double)i), ty = (float)(qy - (double)jj);
        const float w[4] = {(1.0f - tx) * (1.0f - ty), (1.0f - tx) * ty, tx * (1.0f - ty), tx * ty};
        constexpr int NP = (3 * MAXO <= 4) ? 4 : ((3 * MAXO <= 8) ? 8 : 12);
        constexpr int NV = 3 * MAXO;
        const float *nd[4];
        nd[0] = f.nodes32 + (i * nf + jj) * NP;
        nd[1] = nd[0] + NP;
        nd[2] = nd[0] + nf * NP;
        nd[3] = nd[2] + NP;
        float acc[NV];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if constexpr (NP == 8) {   // 32-byte nodes: one 32-byte load each
                float tv[8];
                ldg_v8(nd[k], tv);
#pragma unroll
                for (int b = 0; b < NV; ++b) acc[b] = (k == 0) ? w[0] * tv[b] : acc[b] + w[k] * tv[b];
            } else {
#pragma unroll
                for (int a = 0; a < NV; a += 4) {
                    const float4 t = __ldg(reinterpret_cast<const float4 *>(nd[k] + a));
                    const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (a + b < NV) acc[a + b] = (k == 0) ? w[0] * tv[b] : acc[a + b] + w[k] * tv[b];
                }
            }
        }
        const float z2 = z * z;
        float ze = z2, zo = z2 * z;
#pragma unroll
        for (int n = 0; n < MAXO; ++n) {
            hz += acc[3 * n] * ze;
            hf += acc[3 * n + 1] * zo;
            hr += acc[3 * n + 2] * zo;
            ze *= z2;
            zo *= z2;
        }
    }
    float spiral_p = 0.0f;
    double fs = fim;
    if (!f.spiral_zero) {   // as in tables_fetch, in float64 (spiral lattices only)
        double spiral = 0.0, sp = 0.0;
        for (int a = 0; a < f.n_spoly; ++a) spiral = spiral * r + f.spoly[a];
        for (int a = 0; a < f.n_spolyp; ++a) sp = sp * r + f.spolyp[a];
        spiral_p = (float)sp;
        fs = fim - spiral;
        fs -= f.period * floor(fs * f.inv_period);
    }
    const float rf = (float)r;
    float B0r, B0r_p;
    if (f.k == 0.0) {
        B0r = f.B0f;
        B0r_p = 0.0f;
    } else {
        const float eps = (float)((r - f.r_ref) * f.inv_r_ref);
        const float g = expf(f.km1f * log1pf(eps));
        B0r_p = f.kc1f * g;
        B0r = f.c1f * g * rf;
    }
    const float fsf = (float)fs;
    float F = 0.0f, Fp = 0.0f;
    for (int j = 0; j < f.n_seg; ++j) {
        const float a1 = f.seg_kf[j] * (fsf - f.seg_x0f[j]);
        const float a2 = f.seg_kf[j] * (fsf - f.seg_x1f[j]);
        float e1 = 0.0f, e2 = 0.0f;   // as in field_mixed
        if (a1 < 24.0f) e1 = expf(fminf(-a1, 80.0f));
        if (a2 > -24.0f) e2 = expf(fminf(a2, 80.0f));
        const float s1 = __frcp_rn(1.0f + e1), s2 = __frcp_rn(1.0f + e2);
        const float ss = s1 * s2;
        const float dd = e1 * s1 - e2 * s2;
        F += f.seg_yf[j] * ss;
        Fp += f.seg_ykf[j] * (ss * dd);
    }
    Bz = B0r * F + hz;
    Bfi = B0r * Fp * __frcp_rn(rf) * z + hf;
    Br = (B0r_p * F - B0r * Fp * spiral_p) * z + hr;
}

template <int MAXO, bool XING>
__global__ void __launch_bounds__(128) boris_f32_kernel(const __grid_constant__ PushK p)
{
    const int64_t t_ = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t_ >= p.n) return;
    const int64_t i = p.st.order ? (int64_t)__ldg(p.st.order + t_) : t_;   // the particle this thread advances
    const FieldK &f = p.f;
    const ffa_state_soa &S = p.st;
    const double c = p.cs.c;
    double r = S.r[i], z = S.z[i], fi = S.fi[i], rfph = S.rf[i];
    float ux, uy, uz;
    {
        const double vr = S.vr[i], vf = r * S.f5[i], vz = S.vz[i];
        const double g = 1.0 / sqrt(1.0 - (vr * vr + vf * vf + vz * vz) * p.inv_cc);
        ux = (float)(g * vr / c);
        uy = (float)(g * vf / c);
        uz = (float)(g * vz / c);
    }
    const double esr = S.esc_r[i], esz = S.esc_z[i], esf = S.esc_fi[i];
    int inj = S.inj[i], surv = S.surv[i];
    const int32_t injs = S.inj_step ? S.inj_step[i] : -1;
    const float aE = (float)(p.hq / (p.cs.m0 * c));   // q dt / (2 m c): E [V/m] -> du
    const float aB = (float)p.hqm;                     // q dt / (2 m): B [T] -> gamma t
    const float cdt = (float)(c * p.dt);
    const float esrf = (float)esr, eszf = (float)esz, esff = (float)esf;
    int lost = 0, oob = 0;
    // vr, vz and dfi/dt of the current momentum in float64 (crossing records)
    auto vstate = [&](double rr, double out[3]) {
        const double ig = 1.0 / sqrt(1.0 + (double)ux * ux + (double)uy * uy + (double)uz * uz);
        out[0] = (double)ux * ig * c;
        out[1] = (double)uz * ig * c;
        out[2] = (double)uy * ig * c / rr;
    };

    for (int s = 0; s < p.nsteps; ++s) {
        const int64_t gs = p.step0 + s;
        if (injs == gs) { inj = 1; surv = 1; }
        const double drf = __ldg(p.drf + gs);
        double pre[7];
        const int surv0 = surv;
        if constexpr (XING) {
            double v[3];
            vstate(r, v);
            pre[0] = r; pre[1] = v[0]; pre[2] = z; pre[3] = v[1]; pre[4] = fi; pre[5] = v[2]; pre[6] = rfph;
        }
        if ((inj == 1) && (surv == 1)) {
            const double acc = __ldg(p.acc + gs);
            const double fim = fi - f.period * floor(fi * f.inv_period);
            float Bz, Br, Bfi;
            field_f32<MAXO>(f, r, fim, (float)z, Bz, Br, Bfi, oob);
            double Erd, Ezd, Efid;
            rf_field64(p.rf, acc, r, fi, z, rfph, Erd, Ezd, Efid);
            const float Er = (float)Erd + esrf, Efi = (float)Efid + esff, Ez = (float)Ezd + eszf;
            if (p.ap.enable && (r > p.ap.rmax || r < p.ap.rmin || z > p.ap.zmax || z < p.ap.zmin)) {
                surv = 0;
                ++lost;
            }
            // local frame, B negated as in the float64 pusher
            const float Bx = -Br, By = -Bfi, Bzc = -Bz;
            ux += aE * Er;
            uy += aE * Efi;
            uz += aE * Ez;
            const float cb = aB * rsqrtf(1.0f + ux * ux + uy * uy + uz * uz);
            const float tx = cb * Bx, ty = cb * By, tz = cb * Bzc;
            const float upx = ux + (uy * tz - uz * ty);
            const float upy = uy + (uz * tx - ux * tz);
            const float upz = uz + (ux * ty - uy * tx);
            const float sb = 2.0f * __frcp_rn(1.0f + tx * tx + ty * ty + tz * tz);
            const float sx = sb * tx, sy = sb * ty, sz = sb * tz;
            ux += (upy * sz - upz * sy);
            uy += (upz * sx - upx * sz);
            uz += (upx * sy - upy * sx);
            ux += aE * Er;
            uy += aE * Efi;
            uz += aE * Ez;
            const float k = cdt * rsqrtf(1.0f + ux * ux + uy * uy + uz * uz);
            const float dx = ux * k, dy = uy * k, dz = uz * k;
            const float rf = (float)r;
            const float xn = rf + dx;
            const float rn2 = xn * xn + dy * dy;
            const float irn = rsqrtf(rn2);
            const float rn = rn2 * irn;
            const float dr = (2.0f * rf * dx + dx * dx + dy * dy) * __frcp_rn(rn + rf);
            const float sn = dy * irn, cn = xn * irn;
            const float s2 = sn * sn;
            const float dfi = sn * (1.0f + s2 * (1.0f / 6 + s2 * (3.0f / 40 + s2 * (5.0f / 112))));
            r += (double)dr;
            fi += (double)dfi;
            z += (double)dz;
            const float nux = ux * cn + uy * sn;
            uy = -ux * sn + uy * cn;
            ux = nux;
        }
        rfph += drf;
        if constexpr (XING) {
            if (surv0 == 1) {
                double v[3];
                vstate(r, v);
                const double post[7] = {r, v[0], z, v[1], fi, v[2], rfph};
                xing_check(p.xing, i, gs, pre, post, surv, inj, esr, esz, esf, p.dt);
            }
        }
    }
    const double ig = 1.0 / sqrt(1.0 + (double)ux * ux + (double)uy * uy + (double)uz * uz);
    S.r[i] = r; S.z[i] = z; S.fi[i] = fi; S.rf[i] = rfph;
    S.vr[i] = (double)ux * ig * c;
    S.vz[i] = (double)uz * ig * c;
    S.f5[i] = (double)uy * ig * c / r;
    S.inj[i] = (uint8_t)inj;
    S.surv[i] = (uint8_t)surv;
    status_add(p.status, lost, !(isfinite(r) && isfinite(fi) && isfinite(z)), oob);
}

// -------------------------------------------------------------- RK4 fp64

struct Y7 {
    double r, vr, z, vz, fi, E, rf;
};

// The FP64 stage: RK4_equations_of_motion_njit for one live particle.  What
// depends on the energy alone (v^2, q c^2 / E) is carried and formed anew only
// where the stage's energy differs from the last one, i.e. in an electric
// field; one reciprocal (1 / r) and one inverse square root are left of the
// seven divisions and square roots of the reference's form.  The stages are
// one loop, so the right-hand side is in the code once (four inlined copies
// miss the instruction cache); stage k is evaluated at y + a h d(k-1) with
// a = 1/2, 1/2, 1 and the derivatives are summed as d1 + 2 d2 + 2 d3 + d4.
// Bound as the Boris step (boris_f64_kernel): the node loads' latency and the
// chain behind them, four times a step.  1e5 particles, 720 steps, order 2, RF:
// 9.2 -> 5.6 ms (11.3 ms before field64).
template <int MAXO, bool SC, bool XING, int NREG, bool HARM = false>
__global__ void __maxnreg__(NREG) rk4_f64_kernel(const __grid_constant__ PushK p)
{
    const int64_t t_ = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t_ >= p.n) return;
    const int64_t i = p.st.order ? (int64_t)__ldg(p.st.order + t_) : t_;   // the particle this thread advances
    const FieldK &f = p.f;
    const ffa_state_soa &S = p.st;
    double r = S.r[i], vr = S.vr[i], z = S.z[i], vz = S.vz[i], fi = S.fi[i], E = S.f5[i], rf = S.rf[i];
    double esr = S.esc_r[i], esz = S.esc_z[i], esf = S.esc_fi[i];
    const bool esc = SC || esr != 0.0 || esz != 0.0 || esf != 0.0;   // also for NaN
    int inj = S.inj[i], surv = S.surv[i];
    const int32_t injs = S.inj_step ? S.inj_step[i] : -1;
    SCExtrap ex;
    if (SC) ex.load(S, i);
    const double h = p.dt, h6 = p.dt * (1.0 / 6.0), c2 = p.cs.c * p.cs.c, q = p.cs.q;
    double Ev = __longlong_as_double(0x7FF8000000000000ll), v2 = 0.0, qc2E = 0.0;   // the energy these two belong to (none yet)
    int oob = 0;
    for (int s = 0; s < p.nsteps; ++s) {
        const int64_t gs = p.step0 + s;
        if (injs == gs) { inj = 1; surv = 1; }
        if (SC) ex.apply(sc_phase(p, gs), p.inv_sc, esr, esz, esf);
        const double *rate = p.drf + 4 * gs;
        double pre[7];
        if constexpr (XING) {
            pre[0] = r; pre[1] = vr; pre[2] = z; pre[3] = vz; pre[4] = fi; pre[5] = E; pre[6] = rf;
        }
        const double drf = h6 * (__ldg(rate) + 2 * __ldg(rate + 1) + 2 * __ldg(rate + 2) + __ldg(rate + 3));
        if (inj == 1 && surv == 1) {
            double sr = 0.0, svr = 0.0, sz = 0.0, svz = 0.0, sfi = 0.0, sE = 0.0;
            double yr = r, yvr = vr, yz = z, yvz = vz, yfi = fi, yE = E, yrf = rf;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const double fim = yfi - f.period * floor(yfi * f.inv_period);
                const double ir = rcp64(yr);
                double Bz, Br, Bfi;
                field64<MAXO>(f, yr, ir, fim, yz, Bz, Br, Bfi, oob);
                if constexpr (HARM) Bz += harmonics_bz(f.harm, f.n_harm, yr, yfi);
                if (yE != Ev) {
                    // ig = E0 / E, the product corrected by its residual: at low
                    // energies its rounding is divided by beta^2 in v2
                    const double iE = 1.0 / yE, ig0 = p.cs.E0 * iE, ig = fma(fma(-ig0, yE, p.cs.E0), iE, ig0);
                    Ev = yE;
                    v2 = (1.0 - ig * ig) * c2;
                    qc2E = q * c2 * iE;
                }
                const double vp2 = v2 - yvr * yvr - yvz * yvz;
                // rsqrt64 wants a normal argument: a particle at rest, or moving
                // in r and z alone, has vp2 == 0 and vp = 0 (negative: NaN).
                // The smallest normal number changes no other sum; a select on
                // vp2 == 0 cost 1.7 % (1e5 particles, 720 steps: 5.70 against 5.60 ms)
                const double vp = vp2 * rsqrt64(vp2 + DBL_MIN);
                const double w = vp * ir;                        // d(fi)/dt
                double dvr = vp * w + qc2E * (yvz * Bfi - vp * Bz);
                double dvz = qc2E * (vp * Br - yvr * Bfi);
                double dE = 0.0;
                double3 e = make_double3(0.0, 0.0, 0.0);
                const bool hit = rf_hit64(p.rf, p.acc + 4 * gs + k, yr, yfi, yz, yrf, e);
                if (esc || hit) {
                    if (esc) {
                        if (!SC) { esr = S.esc_r[i]; esz = S.esc_z[i]; esf = S.esc_fi[i]; }   // not held over the loop
                        e.x += esr;
                        e.y += esz;
                        e.z += esf;
                    }
                    const double P = yvr * e.x + vp * e.z + yvz * e.y, c = q / yE * P;
                    dvr += qc2E * e.x - yvr * c;
                    dvz += qc2E * e.y - yvz * c;
                    dE = q * P;
                }
                const double wk = (k == 1 || k == 2) ? 2.0 : 1.0, ah = k == 2 ? h : 0.5 * h;
                sr = fma(wk, yvr, sr);
                svr = fma(wk, dvr, svr);
                sz = fma(wk, yvz, sz);
                svz = fma(wk, dvz, svz);
                sfi = fma(wk, w, sfi);
                sE = fma(wk, dE, sE);
                yr = fma(ah, yvr, r);
                yz = fma(ah, yvz, z);
                yvr = fma(ah, dvr, vr);
                yvz = fma(ah, dvz, vz);
                yfi = fma(ah, w, fi);
                yE = fma(ah, dE, E);
                yrf = fma(ah, __ldg(rate + k), rf);
            }
            r = fma(h6, sr, r);
            vr = fma(h6, svr, vr);
            z = fma(h6, sz, z);
            vz = fma(h6, svz, vz);
            fi = fma(h6, sfi, fi);
            E = fma(h6, sE, E);
        }
        rf += drf;
        if constexpr (XING) {
            if (surv == 1) {
                const double post[7] = {r, vr, z, vz, fi, E, rf};
                if (!SC) { esr = S.esc_r[i]; esz = S.esc_z[i]; esf = S.esc_fi[i]; }
                xing_check(p.xing, i, gs, pre, post, surv, inj, esr, esz, esf, p.dt);
            }
        }
    }
    S.r[i] = r; S.vr[i] = vr; S.z[i] = z; S.vz[i] = vz; S.fi[i] = fi; S.f5[i] = E;
    S.rf[i] = rf;
    if (SC) { S.esc_r[i] = esr; S.esc_z[i] = esz; S.esc_fi[i] = esf; }
    S.inj[i] = (uint8_t)inj;
    S.surv[i] = (uint8_t)surv;
    status_add(p.status, 0, !(isfinite(r) && isfinite(fi) && isfinite(z)), oob);
}

// RK4_equations_of_motion_njit for one live particle at stage state y.
// FP32C: the field of the FP32C Boris pusher (field_mixed: float32 flutter
// exponentials and map lookup, float64 products with r and z); the
// equations of motion and the RK4 stages stay float64.
template <int MAXO, bool HARM>
__device__ __forceinline__ void rk4_rhs_f32c(const PushK &p, const Y7 &y, double rate, double acc,
                                          double esr, double esz, double esf, Y7 &d, int &oob)
{
    const FieldK &f = p.f;
    const double q = p.cs.q, c = p.cs.c, E0 = p.cs.E0;
    const double fim = y.fi - f.period * floor(y.fi / f.period);
    double Bz, Br, Bfi;
    field_mixed<MAXO>(f, y.r, 1.0 / y.r, fim, y.z, Bz, Br, Bfi, oob);
    if constexpr (HARM) Bz += harmonics_bz(f.harm, f.n_harm, y.r, y.fi);
    double Er, Ez, Efi;
    rf_field64(p.rf, acc, y.r, y.fi, y.z, y.rf, Er, Ez, Efi);
    Ez += esz;
    Er += esr;
    Efi += esf;
    const double ig = E0 / y.E;
    const double beta2 = 1.0 - ig * ig;
    const double v2 = beta2 * (c * c);
    const double vperp2 = v2 - y.vr * y.vr - y.vz * y.vz;
    const double fidot = sqrt(vperp2) / y.r;
    const double Edv = y.vr * Er + (y.r * fidot) * Efi + y.vz * Ez;
    const double qc2E = q * (c * c) / y.E;
    d.r = y.vr;
    d.vr = y.r * fidot * fidot + qc2E * (Er - y.r * fidot * Bz + y.vz * Bfi) - q * y.vr / y.E * Edv;
    d.z = y.vz;
    d.vz = qc2E * (Ez + y.r * fidot * Br - y.vr * Bfi) - q * y.vz / y.E * Edv;
    d.fi = fidot;
    d.E = q * Edv;
    d.rf = rate;
}

// FP32C: one-warp blocks (RK4_TB), at most 80 registers (24 warps per SM, spills
// to L1): the 3125 warps of a 1e5-particle bunch are resident in one wave.
// Uncapped the kernel takes 130 registers, 12 warps per SM, 1.76 waves
// (measured on c1: 14.8 ms per 720-step turn uncapped; at 80 registers
// 12.4 ms in 128-thread blocks, 12.3 ms in 32-thread blocks; 11.3 ms with
// the stages as one loop, whose loop body the instruction cache holds).

template <int MAXO, bool SC, bool XING, bool HARM = false>
__global__ void __maxnreg__(80) rk4_f32c_kernel(const __grid_constant__ PushK p)
{
    const int64_t t_ = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t_ >= p.n) return;
    const int64_t i = p.st.order ? (int64_t)__ldg(p.st.order + t_) : t_;   // the particle this thread advances
    const ffa_state_soa &S = p.st;
    Y7 y{S.r[i], S.vr[i], S.z[i], S.vz[i], S.fi[i], S.f5[i], S.rf[i]};
    double esr = S.esc_r[i], esz = S.esc_z[i], esf = S.esc_fi[i];
    int inj = S.inj[i], surv = S.surv[i];
    const int32_t injs = S.inj_step ? S.inj_step[i] : -1;
    SCExtrap ex;
    if (SC) ex.load(S, i);
    const double h = p.dt;
    int oob = 0;
    for (int s = 0; s < p.nsteps; ++s) {
        const int64_t gs = p.step0 + s;
        if (injs == gs) { inj = 1; surv = 1; }
        if (SC) ex.apply(p, gs, esr, esz, esf);
        const double *rate = p.drf + 4 * gs;
        const double *acc = p.acc + 4 * gs;
        const double k1rf = h * __ldg(rate + 0), k2rf = h * __ldg(rate + 1);
        const double k3rf = h * __ldg(rate + 2), k4rf = h * __ldg(rate + 3);
        const double drf = (k1rf + 2 * k2rf + 2 * k3rf + k4rf) / 6;
        Y7 y0;
        if constexpr (XING) y0 = y;
        if (!((inj == 1) && (surv == 1))) {
            y.rf += drf;
            if constexpr (XING) {
                if (surv == 1) {
                    const double pre[7] = {y0.r, y0.vr, y0.z, y0.vz, y0.fi, y0.E, y0.rf};
                    const double post[7] = {y.r, y.vr, y.z, y.vz, y.fi, y.E, y.rf};
                    xing_check(p.xing, i, gs, pre, post, surv, inj, esr, esz, esf, p.dt);
                }
            }
            continue;
        }
        // the four stages as one loop, so the right-hand side is in the code
        // once: stage k is evaluated at y + a K(k-1) with a = 1/2, 1/2, 1, and
        // the increments are summed as K1 + 2 K2 + 2 K3 + K4, in that order
        Y7 d, K, S, ys = y;
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            rk4_rhs_f32c<MAXO, HARM>(p, ys, __ldg(rate + k), __ldg(acc + k), esr, esz, esf, d, oob);
            K = {h * d.r, h * d.vr, h * d.z, h * d.vz, h * d.fi, h * d.E, h * d.rf};
            if (k == 0) {
                S = K;
            } else if (k < 3) {
                S = {S.r + 2 * K.r, S.vr + 2 * K.vr, S.z + 2 * K.z, S.vz + 2 * K.vz, S.fi + 2 * K.fi,
                     S.E + 2 * K.E, S.rf + 2 * K.rf};
            } else {
                S = {S.r + K.r, S.vr + K.vr, S.z + K.z, S.vz + K.vz, S.fi + K.fi, S.E + K.E, S.rf + K.rf};
            }
            const double a = k == 2 ? 1.0 : 0.5;
            ys = {y.r + a * K.r, y.vr + a * K.vr, y.z + a * K.z, y.vz + a * K.vz, y.fi + a * K.fi,
                  y.E + a * K.E, y.rf + a * K.rf};
        }
        y.r += S.r / 6;
        y.vr += S.vr / 6;
        y.z += S.z / 6;
        y.vz += S.vz / 6;
        y.fi += S.fi / 6;
        y.E += S.E / 6;
        y.rf += S.rf / 6;
        if constexpr (XING) {
            const double pre[7] = {y0.r, y0.vr, y0.z, y0.vz, y0.fi, y0.E, y0.rf};
            const double post[7] = {y.r, y.vr, y.z, y.vz, y.fi, y.E, y.rf};
            xing_check(p.xing, i, gs, pre, post, surv, inj, esr, esz, esf, p.dt);
        }
    }
    S.r[i] = y.r; S.vr[i] = y.vr; S.z[i] = y.z; S.vz[i] = y.vz; S.fi[i] = y.fi; S.f5[i] = y.E;
    S.rf[i] = y.rf;
    S.esc_r[i] = esr; S.esc_z[i] = esz; S.esc_fi[i] = esf;
    S.inj[i] = (uint8_t)inj;
    S.surv[i] = (uint8_t)surv;
    status_add(p.status, 0, !(isfinite(y.r) && isfinite(y.fi) && isfinite(y.z)), oob);
}

// ------------------------------------------------- closed-orbit tracks

// An azimuth t >= 0 reduced mod 2 pi and then mod the sector, as the
// reference's fmod pair does; a multiple that rounding puts off by one leaves
// a value just outside the sector, where the field is the same.  Every
// track of a launch has the same t, so this is off their chains.
__device__ __forceinline__ double sector_azimuth(const FieldK &f, double t)
{
    const double tw = 2.0 * PI;
    const double fi = fma(-tw, floor(t * (0.5 / PI)), t);
    return fma(-f.period, floor(fi * f.inv_period), fi);
}

// d/dtheta of (r, pr, z, pz) at fixed momentum P (FunctionForSEO,
// src/FFAG_track.py:1698-1740), qP = q / P, from the flutter F, F', B0r = B0
// r^k and kG = k B0 r^(k-1).  The field enters only times r, which cancels the
// 1 / r of Bfi.
__device__ __forceinline__ void seo_rhs(const double x[4], double qP, double F, double Fp, double B0r, double kG,
                                        double spiral_p, double d[4])
{
    const double r = x[0], pr = x[1], z = x[2], pz = x[3];
    const double pf2 = 1.0 - pr * pr - pz * pz, ipf = rsqrt64(pf2);
    const double rBz = B0r * r * F, rBfi = B0r * Fp * z;
    const double rBr = r * fma(kG, F, -B0r * Fp * spiral_p) * z;
    const double ur = pr * ipf, uz = pz * ipf;
    d[0] = r * ur;
    d[1] = fma(pf2, ipf, qP * (uz * rBfi - rBz));
    d[2] = r * uz;
    d[3] = qP * (rBr - ur * rBfi);
}

// One thread per track; a scan has a few thousand of them, so the launch is
// one step's chain long whatever the chip could hold: power-table load
// (about 40 cycles from L1), field, inverse square root, stage update.  One
// warp per block, so that the warps spread over the SMs.  Without a spiral
// (PLAIN) the flutter depends on the azimuth alone, which is known ahead: two
// evaluations a step instead of four, their cells loaded a step before.
// 1280 tracks of 523 steps: 1.37 -> 0.40 ms (2.5 ms before field64);
// 100000 tracks of 128 steps: 1.40 -> 0.29 ms.
template <bool PLAIN>
__global__ void __launch_bounds__(32) theta_track_kernel(const __grid_constant__ FieldK f,
                                                         const __grid_constant__ ffa_theta_track_desc d)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.m) return;
    double x[4] = {d.x0[5 * i], d.x0[5 * i + 1], d.x0[5 * i + 2], d.x0[5 * i + 3]};
    const double qP = d.q / d.x0[5 * i + 4];
    const double h = d.t_end / (double)(d.n_points - 1);
    const int nc = d.traj_cols;
    double *tr = d.traj ? d.traj + (int64_t)i * d.n_points * nc : nullptr;
    double t = 0.0;
    // row of point s: the state and, for 7 columns, the field there
    auto record = [&](int s, double ts) {
        double *row = tr + (int64_t)s * nc;
        row[0] = x[0];
        row[1] = x[1];
        if (nc == 7) {
            row[2] = x[2];
            row[3] = x[3];
            int clamped = 0;
            field64<0>(f, x[0], 1.0 / x[0], sector_azimuth(f, ts), x[2], row[4], row[5], row[6], clamped);
        }
    };
    if (tr) record(0, 0.0);
    auto start = [&](int s) { return d.time_mode == 0 ? (double)s * h : t; };
    // PLAIN: the flutter at the step's start, and the cells of its middle and
    // end (the next step's start)
    double F0 = 0.0, Fp0 = 0.0;
    FlutterCell mid, end;
    if constexpr (PLAIN) {
        flutter_eval(f, flutter_fetch(f, sector_azimuth(f, 0.0)), F0, Fp0);
        mid = flutter_fetch(f, sector_azimuth(f, 0.5 * h));
        end = flutter_fetch(f, sector_azimuth(f, h));
    }
    for (int s = 0; s < d.n_points - 1; ++s) {
        t = start(s);
        double F1 = 0.0, Fp1 = 0.0, F2 = 0.0, Fp2 = 0.0;
        if constexpr (PLAIN) {
            flutter_eval(f, mid, F1, Fp1);
            flutter_eval(f, end, F2, Fp2);
            const double tn = d.time_mode == 0 ? (double)(s + 1) * h : t + h;
            mid = flutter_fetch(f, sector_azimuth(f, tn + 0.5 * h));
            end = flutter_fetch(f, sector_azimuth(f, tn + h));
        }
        auto rhs = [&](double ts, const double *y, double F, double Fp, double *k) {
            if constexpr (PLAIN) {
                const double G = power_eval(f, power_fetch(f, y[0]), y[0]);
                seo_rhs(y, qP, F, Fp, G * y[0], f.k * G, 0.0, k);
            } else {
                const Tables tab = tables_fetch(f, y[0], sector_azimuth(f, ts));
                double B0r, kG;
                tables_eval(f, tab, y[0], F, Fp, B0r, kG);
                seo_rhs(y, qP, F, Fp, B0r, kG, tab.spiral_p, k);
            }
        };
        double y[4], k[4], S[4];
        rhs(t, x, F0, Fp0, k);
#pragma unroll
        for (int c = 0; c < 4; ++c) { S[c] = k[c]; y[c] = fma(0.5 * h, k[c], x[c]); }
        rhs(t + 0.5 * h, y, F1, Fp1, k);
#pragma unroll
        for (int c = 0; c < 4; ++c) { S[c] = fma(2.0, k[c], S[c]); y[c] = fma(0.5 * h, k[c], x[c]); }
        rhs(t + 0.5 * h, y, F1, Fp1, k);
#pragma unroll
        for (int c = 0; c < 4; ++c) { S[c] = fma(2.0, k[c], S[c]); y[c] = fma(h, k[c], x[c]); }
        rhs(t + h, y, F2, Fp2, k);
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = fma(h * (1.0 / 6.0), S[c] + k[c], x[c]);
        F0 = F2;
        Fp0 = Fp2;
        if (d.time_mode != 0) t = t + h;
        if (tr) record(s + 1, d.time_mode != 0 ? t : (double)(s + 1) * h);
    }
    for (int c = 0; c < 4; ++c) d.x1[4 * i + c] = x[c];
}

cudaError_t launch_theta_track(const FieldK &f, const ffa_theta_track_desc &d, cudaStream_t s)
{
    const unsigned g = (unsigned)((d.m + 31) / 32);
    if (f.spiral_zero && !f.unusual) theta_track_kernel<true><<<g, 32, 0, s>>>(f, d);
    else theta_track_kernel<false><<<g, 32, 0, s>>>(f, d);
    return cudaGetLastError();
}

// ------------------------------------------------------------ node packing

__global__ void pack_nodes_kernel(const double *__restrict__ bz, const double *__restrict__ bfi,
                                  const double *__restrict__ br, int64_t plane, int max_order,
                                  int npad, double *__restrict__ n64, float *__restrict__ n32)
{
    const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= plane) return;
    for (int v = 0; v < npad; ++v) {
        double val = 0.0;
        const int n = v / 3 + 1, comp = v % 3;
        if (n <= max_order) {
            const double *src = comp == 0 ? bz : (comp == 1 ? bfi : br);
            val = src[(int64_t)n * plane + node];
        }
        const int a = v & ~3, w = map_plane_width(max_order, a);
        if (v - a < w) n64[a * plane + node * w + (v - a)] = val;
        n32[node * npad + v] = (float)val;
    }
}

cudaError_t launch_pack_nodes(const ffa_field_desc &d, int npad, double *n64, float *n32, cudaStream_t s)
{
    const int64_t plane = d.r_size * d.fi_size;
    const int tb = 256;
    pack_nodes_kernel<<<(unsigned)((plane + tb - 1) / tb), tb, 0, s>>>(d.bz_stack, d.bfi_stack, d.br_stack,
                                                                        plane, d.max_order, npad, n64, n32);
    return cudaGetLastError();
}

// Register cap of a float64 Boris launch of n particles.  More registers
// keep more of a step's loads and chains in flight per warp, fewer hold more
// warps; 80, 128 and 255 leave 24, 16 and 8 warps per SM.  What decides is how
// many waves the warps make (us per 180 steps, z-Taylor order 2, RF, 148 SMs):
//   particles     10000  56800  75000  100000  113600  150000  200000  300000  1000000
//   80 registers    246    268    281     357     355     570     623     908     2739
//   128 registers   197    218    252     421     434     480     657     929     3001
//   255 registers   198    219    405     417     425     605       -    1162     3608
// so 128 up to 16 warps per SM, 80 while that is one wave, 128 again while that
// is two, and 80 beyond (order 0, 120 steps, 1e6 particles: 1338 us with 128,
// 1113 with 80; order 1 1754 and 1486).  Orders 3 and 4 stay at 128 there (order
// 4, 300000 particles: 830 us, with 80 901; 1e6: 2745 and 2700).  From order 3 a
// step's node loads alone need more than 128 (order 4, 10000 particles, 720
// steps: 935 us with 128, 791 us with 255).
// Field-error harmonics follow the same rule (order 2, 120 steps: 100000
// particles 550 us with 128, 358 with 80; 1e6, 30 steps: 966 and 796).
// With space charge the endpoints' registers make 80 spill: only for the bunches
// that it keeps in one wave (60 steps, order 2 / 4: 77000 particles 217 / 292 us
// with 128, 194 / 267 with 80; 113000 231 / 338 and 226 / 314; 1e6 1627 us with
// 128, 1898 with 80).
// Launches that look for crossings hold more values over a step and gain from
// the one wave up to 20 warps per SM (order 2, 120 steps: 90000 particles 473 us
// with 128, 461 with 80; 100000 480 and 502; 113000 496 and 533), with harmonics
// up to 24 (113000: 740 and 656).
static int boris_cap(const PushK &p, bool sc, int max_order)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t warps = (p.n + 31) / 32;
    if (!sc && max_order >= 3 && warps <= (int64_t)8 * sms) return 255;
    if (warps <= (int64_t)16 * sms) return 128;
    if (warps <= (int64_t)(xing_on(p) && !sc && p.f.n_harm == 0 ? 20 : 24) * sms) return 80;
    if (sc) return 128;
    return max_order >= 3 || xing_on(p) || warps <= (int64_t)32 * sms ? 128 : 80;
}

template <int MAXO, bool SC, int NREG, bool HARM>
static void boris_shaped(const PushK &p, cudaStream_t s, int tb)
{
    const unsigned g = (unsigned)((p.n + tb - 1) / tb);
    if (xing_on(p)) boris_f64_kernel<MAXO, SC, true, NREG, HARM><<<g, tb, 0, s>>>(p);
    else boris_f64_kernel<MAXO, SC, false, NREG, HARM><<<g, tb, 0, s>>>(p);
}

// Field-error harmonics select their own kernel variants (HARM), so that
// the harmonic sum costs the common case nothing.
template <int MAXO, bool SC>
static void boris_launch(const PushK &p, cudaStream_t s, int tb, int)
{
    const int cap = boris_cap(p, SC, MAXO);
    if (p.f.n_harm > 0) {
        if (cap == 80) return boris_shaped<MAXO, SC, 80, true>(p, s, tb);
        return boris_shaped<MAXO, SC, 128, true>(p, s, tb);
    }
    if (cap == 80) return boris_shaped<MAXO, SC, 80, false>(p, s, tb);
    if constexpr (!SC) {
        if constexpr (MAXO >= 3) {
            if (cap == 255) return boris_shaped<MAXO, SC, 255, false>(p, s, tb);
        }
    }
    boris_shaped<MAXO, SC, 128, false>(p, s, tb);
}

// Register cap of a float64 RK4 launch of n particles: 255, 168 or 128 leave 8,
// 12 or 16 warps per SM, and a wave of them takes about 0.69, 0.83 and 1 of
// the time (with space charge 0.60, 0.72 and 1); the cap with the least total
// over its waves.  Measured (us per 180 steps, z-Taylor order 2, RF, 148 SMs):
//   particles     10000  37800  56800  75000  100000  150000  200000  1000000
//   128 registers   605    652    741    846    1448    1619    2278    10379
//   168 registers   570    624    704   1269    1308    1912    2516    11481
//   255 registers   528    583   1113   1156    1657    2236    3220    14586
// (80 registers spill the stages: 806 and 1718 us at 10000 and 100000)
static int rk4_cap(const PushK &p, bool sc)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t warps = (p.n + 31) / 32;
    const int cap[3] = {128, 168, 255}, per_sm[3] = {16, 12, 8}, cost[2][3] = {{100, 83, 69}, {100, 72, 60}};
    int best = 0;
    int64_t least = INT64_MAX;
    for (int v = 0; v < 3; ++v) {
        const int64_t room = (int64_t)per_sm[v] * sms, t = (warps + room - 1) / room * cost[sc][v];
        if (t < least) { least = t; best = v; }
    }
    return cap[best];
}

template <int MAXO, bool SC, int NREG, bool HARM>
static void rk4_shaped(const PushK &p, cudaStream_t s)
{
    const unsigned g = (unsigned)((p.n + RK4_TB - 1) / RK4_TB);
    if (xing_on(p)) rk4_f64_kernel<MAXO, SC, true, NREG, HARM><<<g, RK4_TB, 0, s>>>(p);
    else rk4_f64_kernel<MAXO, SC, false, NREG, HARM><<<g, RK4_TB, 0, s>>>(p);
}

template <int MAXO, bool SC>
static void rk4_launch(const PushK &p, cudaStream_t s, bool f32)
{
    if (f32) {
        const unsigned g = (unsigned)((p.n + RK4_TB - 1) / RK4_TB);
        const bool x = xing_on(p);
        if (p.f.n_harm > 0) {
            if (x) rk4_f32c_kernel<MAXO, SC, true, true><<<g, RK4_TB, 0, s>>>(p);
            else rk4_f32c_kernel<MAXO, SC, false, true><<<g, RK4_TB, 0, s>>>(p);
        } else {
            if (x) rk4_f32c_kernel<MAXO, SC, true><<<g, RK4_TB, 0, s>>>(p);
            else rk4_f32c_kernel<MAXO, SC, false><<<g, RK4_TB, 0, s>>>(p);
        }
        return;
    }
    if (p.f.n_harm > 0) return rk4_shaped<MAXO, SC, 128, true>(p, s);
    switch (rk4_cap(p, SC)) {
    case 255: return rk4_shaped<MAXO, SC, 255, false>(p, s);
    case 168: return rk4_shaped<MAXO, SC, 168, false>(p, s);
    default: return rk4_shaped<MAXO, SC, 128, false>(p, s);
    }
}

#define FFA_DISPATCH(FN, p, ...)                                                       \
    do {                                                                               \
        const bool sc_ = (p).st.sc_pre != nullptr && (p).sc_step > 0;                  \
        switch ((p).f.max_order) {                                                     \
        case 0: sc_ ? FN<0, true>(p, __VA_ARGS__) : FN<0, false>(p, __VA_ARGS__); break; \
        case 1: sc_ ? FN<1, true>(p, __VA_ARGS__) : FN<1, false>(p, __VA_ARGS__); break; \
        case 2: sc_ ? FN<2, true>(p, __VA_ARGS__) : FN<2, false>(p, __VA_ARGS__); break; \
        case 3: sc_ ? FN<3, true>(p, __VA_ARGS__) : FN<3, false>(p, __VA_ARGS__); break; \
        default: sc_ ? FN<4, true>(p, __VA_ARGS__) : FN<4, false>(p, __VA_ARGS__); break; \
        }                                                                              \
    } while (0)

cudaError_t launch_boris_f64(const PushK &p, cudaStream_t s, int tb)
{
    FFA_DISPATCH(boris_launch, p, s, tb, 0);
    return cudaGetLastError();
}

cudaError_t launch_rk4_f64(const PushK &p, cudaStream_t s, bool f32)
{
    FFA_DISPATCH(rk4_launch, p, s, f32);
    return cudaGetLastError();
}

template <int MAXO, bool XING, int NREG>
static void boris32_shaped(const PushK &p, cudaStream_t s, int tb)
{
    boris_f32c_kernel<MAXO, false, XING, NREG><<<(unsigned)((p.n + tb - 1) / tb), tb, 0, s>>>(p);
}

template <int MAXO, bool SC>
static void boris32_launch(const PushK &p, cudaStream_t s, int tb, int nreg_sel)
{
    if constexpr (!SC) {
        if (nreg_sel != 0) {   // the caller has checked: no space charge, no harmonics
            const bool x = xing_on(p);
            switch (nreg_sel) {
            case 1: x ? boris32_shaped<MAXO, true, 72>(p, s, tb) : boris32_shaped<MAXO, false, 72>(p, s, tb); break;
            case 2: x ? boris32_shaped<MAXO, true, 64>(p, s, tb) : boris32_shaped<MAXO, false, 64>(p, s, tb); break;
            default: x ? boris32_shaped<MAXO, true, 56>(p, s, tb) : boris32_shaped<MAXO, false, 56>(p, s, tb); break;
            }
            return;
        }
    }
    const unsigned g = (unsigned)((p.n + tb - 1) / tb);
    const bool x = xing_on(p);
    if (p.f.n_harm > 0) {
        if (x) boris_f32c_kernel<MAXO, SC, true, 80, true><<<g, tb, 0, s>>>(p);
        else boris_f32c_kernel<MAXO, SC, false, 80, true><<<g, tb, 0, s>>>(p);
    } else {
        if (x) boris_f32c_kernel<MAXO, SC, true><<<g, tb, 0, s>>>(p);
        else boris_f32c_kernel<MAXO, SC, false><<<g, tb, 0, s>>>(p);
    }
}

cudaError_t launch_boris_f32c(const PushK &p, cudaStream_t s, int tb, int nreg_sel)
{
    FFA_DISPATCH(boris32_launch, p, s, tb, nreg_sel);
    return cudaGetLastError();
}

template <int MAXO, bool SC>
static void boris_f32_launch(const PushK &p, cudaStream_t s, int tb, int)
{
    const unsigned g = (unsigned)((p.n + tb - 1) / tb);
    if (xing_on(p)) boris_f32_kernel<MAXO, true><<<g, tb, 0, s>>>(p);
    else boris_f32_kernel<MAXO, false><<<g, tb, 0, s>>>(p);
}

cudaError_t launch_boris_f32(const PushK &p, cudaStream_t s, int tb)
{
    switch (p.f.max_order) {
    case 0: boris_f32_launch<0, false>(p, s, tb, 0); break;
    case 1: boris_f32_launch<1, false>(p, s, tb, 0); break;
    case 2: boris_f32_launch<2, false>(p, s, tb, 0); break;
    case 3: boris_f32_launch<3, false>(p, s, tb, 0); break;
    default: boris_f32_launch<4, false>(p, s, tb, 0); break;
    }
    return cudaGetLastError();
}

// Resident blocks per SM of a push kernel (no space charge), from the runtime.
template <int MAXO, bool X>
static const void *push_kernel_fn(bool rk4, bool f32, int nreg_sel)
{
    if (rk4) return f32 ? (const void *)rk4_f32c_kernel<MAXO, false, X> : (const void *)rk4_f64_kernel<MAXO, false, X, 128>;
    if (!f32) return (const void *)boris_f64_kernel<MAXO, false, X, 80>;
    switch (nreg_sel) {
    case 0: return (const void *)boris_f32c_kernel<MAXO, false, X, 80>;
    case 1: return (const void *)boris_f32c_kernel<MAXO, false, X, 72>;
    case 2: return (const void *)boris_f32c_kernel<MAXO, false, X, 64>;
    default: return (const void *)boris_f32c_kernel<MAXO, false, X, 56>;
    }
}

cudaError_t push_occupancy(bool rk4, bool f32, int max_order, bool xing, int tb, int nreg_sel, int *blocks)
{
    const void *fn;
    switch (max_order) {
    case 0: fn = xing ? push_kernel_fn<0, true>(rk4, f32, nreg_sel) : push_kernel_fn<0, false>(rk4, f32, nreg_sel); break;
    case 1: fn = xing ? push_kernel_fn<1, true>(rk4, f32, nreg_sel) : push_kernel_fn<1, false>(rk4, f32, nreg_sel); break;
    case 2: fn = xing ? push_kernel_fn<2, true>(rk4, f32, nreg_sel) : push_kernel_fn<2, false>(rk4, f32, nreg_sel); break;
    case 3: fn = xing ? push_kernel_fn<3, true>(rk4, f32, nreg_sel) : push_kernel_fn<3, false>(rk4, f32, nreg_sel); break;
    default: fn = xing ? push_kernel_fn<4, true>(rk4, f32, nreg_sel) : push_kernel_fn<4, false>(rk4, f32, nreg_sel); break;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, fn, tb, 0);
}

}  // namespace ffa
