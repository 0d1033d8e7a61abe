// ffa_internal.cuh -- shared device-side definitions of libffa_cuda.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/ffa_cuda.h"

#define FFA_CHECK_CUDA(call)                         \
    do {                                             \
        cudaError_t e_ = (call);                     \
        if (e_ != cudaSuccess) return FFA_ERR_CUDA;  \
    } while (0)

namespace ffa {

constexpr double PI = 3.141592653589793;

// The kernels of a space-charge update and of a training step follow one another
// by programmatic dependent launch: each starts as the blocks of its predecessor
// exit, and waits (chain_wait, no effect on an ordinary launch) before it touches
// what its predecessors write or read.  The first kernel of a chain is an ordinary
// launch, so everything before the chain is complete.  In the update and in the
// step's last two kernels every thread waits; the step's tile kernel says itself
// which of its threads need not.
// Letting a successor start earlier (griddepcontrol.launch_dependents) cost
// 10-20 us of a 145 us update: its waiting blocks take the room of the running ones.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A launch that may begin while the kernel before it in the stream still runs
// (its kernel calls chain_wait).  It hides the 1-2 us between launches: 100003
// particles, 32 x 64 x 64 cells 52 -> 44 us.
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// Values per node in the plane of the float64 z-Taylor table that starts at
// value a (0, 4, 8): four, or the one or two values left (three are padded)
inline __host__ __device__ int map_plane_width(int max_order, int a)
{
    const int left = 3 * max_order - a;
    return left >= 3 ? 4 : (left > 0 ? left : 0);
}

// Kernel-side view of the field (analytic parameters precomputed once and the
// packed z-Taylor table).  A node (i, j) of the r x fi grid has, for
// n = 1..max_order, the values (bz_n, bfi_n, br_n).  The float32 table keeps a
// node's values together, padded to `npad` (4, 8, 12).  The float64 table is
// split into planes of up to four values per node (map_plane_width), each
// over all nodes: value a + b of a node, a = 0, 4, 8, is at
// a * plane + node * width + b with `plane` the number of nodes.
struct FieldK {
    int32_t nsectors, n_spoly, n_spolyp, n_seg, max_order, npad;
    // B0, k, k - 1; pad4 keeps what follows where 16-byte parameter loads reach
    // it (without: 10,000 particles, order 4, 720 steps 770 -> 800 us)
    double B0, k, km1, pad4;
    double period;                // 2 pi / nsectors
    double inv_period;            // nsectors / (2 pi)
    double spoly[FFA_MAX_POLY];
    double spolyp[FFA_MAX_POLY];
    double seg_x0[FFA_MAX_SEG], seg_x1[FFA_MAX_SEG];
    double seg_k[FFA_MAX_SEG];    // 16 / W0
    double seg_y[FFA_MAX_SEG];    // y02 * |y01|
    double r_min, r_step, fi_min, fi_step;
    int64_t r_size, fi_size, plane;
    const double *nodes64;
    const float *nodes32;
    // float32 field: B0 r^(k-1) = c1 * (1 + eps)^(k-1), eps = (r - r_ref) / r_ref
    int32_t spiral_zero;          // s(r) == 0: skip the spiral polynomials
    int32_t pad1;
    double r_ref, inv_r_ref, inv_r_step, inv_fi_step;
    double c1, kc1;               // B0 r_ref^(k-1), k * c1
    double seg_yk[FFA_MAX_SEG];   // seg_y * seg_k
    // Flutter table: F = sum_j y_j s1_j s2_j over one sector as degree-7
    // polynomials (8 coefficients, lowest first, in x = q - j - 1/2,
    // q = fs * fl_scale) over fl_n cells of 1 / fl_scale = 2^-m rad, a guard
    // cell before and after the sector; fl_direct: no table (one dummy cell),
    // the sigmoids are evaluated
    int32_t fl_n, fl_direct;
    int32_t unusual, pad3;   // fl_direct, or k == 0
    double fl_scale;
    const double *fl_tab;
    // Power table: (B0 r_j^(k-1), 1 / r_j) at r_j = (pw_j0 + j) pw_h,
    // pw_h = 1 / pw_scale = 2^-p m, and the binomial coefficients 1 .. 4 of
    // the exponent k - 1; without a table one dummy entry that no r reaches
    // (k = 0: that every r reaches, pw_scale = 0)
    int32_t pw_j0, pw_n;
    double pw_scale, pw_h;
    const double2 *pw_tab;
    double pw_c[4];
    // field-error harmonics: Bz += sum_k amp cos(m fi + phase) over the n_harm
    // rows (m, amp, phase, rmin, rmax) of the device table `harm` with
    // rmin <= r <= rmax (fi unwrapped)
    int32_t n_harm, pad2;
    const double *harm;
    // float32 copies for the float32 pusher
    float B0f, c1f, kc1f, km1f;
    float seg_x0f[FFA_MAX_SEG], seg_x1f[FFA_MAX_SEG], seg_kf[FFA_MAX_SEG], seg_yf[FFA_MAX_SEG], seg_ykf[FFA_MAX_SEG];
};

struct RFK {
    int32_t enable, ngaps, physical_sum;
    int32_t single;       // the one fixed gap that acts (the last), -1: none, or spiral gaps or the sum of all
    double poly_x[FFA_MAX_GAPS][4];
    double poly_y[FFA_MAX_GAPS][4];
    double box[FFA_MAX_GAPS][4];
    double theta_n[FFA_MAX_GAPS];
    double rf_shift[FFA_MAX_GAPS];
    // Angular window of each gap rectangle as seen from the origin: every
    // point of the rectangle lies within win_half of win_center, so a
    // particle outside the window is outside the gap without the Cartesian
    // test (win_half = pi disables the shortcut).
    double win_center[FFA_MAX_GAPS];
    double win_half[FFA_MAX_GAPS];
    // spiral gaps (sp != NULL): the shared (r, phi) map, its axes, the
    // middle and end of the phi axis, and each gap's azimuth
    const double *sp;
    int32_t sp_nr, sp_nphi;
    double sp_r0, sp_dr, sp_phi0, sp_dphi, sp_phimax, sp_phic;
    double gap_az[FFA_MAX_GAPS];
};

struct PushK {
    FieldK f;
    RFK rf;
    ffa_aperture ap;
    ffa_consts cs;
    ffa_state_soa st;
    const double *drf;
    const double *acc;
    int64_t n, step0;
    int32_t nsteps, sc_step;
    double dt;
    int64_t *status;
    ffa_crossing xing;  // buf and fit_sums both NULL: no crossing capture
    // Boris constants, formed on the host so the kernel reads them from the
    // parameter bank instead of holding them in registers
    double hq;          // (0.5 dt) q
    double hqm;         // hq / m
    double inv_m;       // 1 / m
    double inv_cc;      // 1 / c^2
    double inv_mmcc;    // 1 / (m^2 c^2)
    double inv_sc;      // 1 / sc_step (0 without space charge)
};

inline __host__ __device__ bool xing_on(const PushK &p)
{
    return p.xing.buf != nullptr || p.xing.fit_sums != nullptr;
}

}  // namespace ffa

struct ffa_fieldmap {
    ffa::FieldK k;
    double *nodes64;
    float *nodes32;
    double *tables;       // device: flutter cells, then the power table
    double *harm;         // device, FFA_MAX_HARMONICS rows of 5
};

// Launchers implemented in ffa_push.cu
namespace ffa {
// tb: threads per block; nreg_sel: register cap 80, 72, 64, 56 (0..3)
cudaError_t launch_boris_f64(const PushK &p, cudaStream_t s, int tb);
// RK4 (f32: the FP32C field) in blocks of RK4_TB threads
constexpr int RK4_TB = 32;
cudaError_t launch_rk4_f64(const PushK &p, cudaStream_t s, bool f32);
cudaError_t launch_boris_f32c(const PushK &p, cudaStream_t s, int tb, int nreg_sel);
cudaError_t launch_boris_f32(const PushK &p, cudaStream_t s, int tb);
cudaError_t push_occupancy(bool rk4, bool f32, int max_order, bool xing, int tb, int nreg_sel, int *blocks);
cudaError_t launch_theta_track(const FieldK &f, const ffa_theta_track_desc &d, cudaStream_t s);
cudaError_t launch_pack_nodes(const ffa_field_desc &d, int npad, double *n64, float *n32, cudaStream_t s);
}  // namespace ffa
