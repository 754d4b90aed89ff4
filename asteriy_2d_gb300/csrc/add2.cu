// add2.cu - the drop-in for the reference's first-order planar step add2
// (kernel.cu:1928-2291), as its own kernel.
//
// add2 is not a special case of the face-once step: it evaluates each cell's
// four faces from that cell, and its flux selection is not symmetric.  The
// face on the cell's right and its r faces take HLLC inside the region
// (x + dx/2, resp. x, in (region_lo, region_hi)) and HLL outside, but the
// face on its left takes HLL inside the region (x - dx/2 in it) and HLLC
// outside (kernel.cu:2057-2085).  So inside the region the face between two
// cells is HLLC for the cell on its left and HLL for the cell on its right:
// the scheme is not conservative there.  This kernel evaluates every face
// of a 32x16 tile once (both fluxes on the z faces, from one sound speed) and
// gives each cell the flux its own rule picks.  It is bound by the FP64 pipe:
// at 32000x400, 13.1 ms per step with one thread per cell, its four faces
// and an atomic on *T by every cell (12.8 M of them to one address), 9.6 ms
// of it with the short FP64 fluxes; this form 4.72 ms.
//
// Per cell (kernel.cu:1928-2291): neighbours with add2's boundary rules
// (right side outflow at n = N-1; left side the fixed inflow state at
// n = 0, its density perturbed by 1 + 0.01 sin(2 pi TT) for y < 0.5 while
// TT < 3 when method != 0; reflecting r = 0 and r = y_max); the four face
// fluxes (HLL or HLLC per the rule above, each in the cell's outward frame);
// dt candidate krit*rad/S per face; the planar update with the body force
// Q2 = -+amp*rho in v_r for body_lo < x < body_hi (r >= / < body_rsplit);
// the density and pressure floors.  *T is lowered to the cells' smallest dt
// candidate by an exact atomic minimum (the reference's write races), one
// per tile: krit*rad/S falls with S, so the tile's largest wave speeds give
// its smallest candidate.
#include <cuda_runtime.h>

#include "../../include/asteriy_gb300.h"
#include "launch.cuh"

using namespace ast;

namespace {

struct Add2Params {
    int N, M;
    double x_min, dx, y_min, dy;
    double krit_dx, krit_dy, dt_cap, p_floor;
    double region_lo, region_hi;
    int body_force;
    double body_lo, body_hi, body_rsplit, body_amp;
    double in_rho, in_p, in_vz, in_vr;   // the inflow state at n = 0 (the z_lo side's FIXED values)
    int perturb;                         // method != 0: the time-dependent inflow density
    Gas<double> g;
};

__device__ __forceinline__ bool in_region(const Add2Params& P, double xf)
{
    return xf > P.region_lo && xf < P.region_hi;
}

// the tile, and the flux components of its faces
constexpr int kAZ = 32, kAR = 16, kWarps = kThreads / 32, kCells = kAR / kWarps;
static_assert(kAZ == 32 && kAR % kWarps == 0, "a warp per row, whole rows per warp");
struct Add2Smem {
    double zr[4][kAR][kAZ + 1];   // z faces as their lower cell uses them (its right face)
    double r[4][kAR + 1][kAZ];    // r faces
    double smax[2][kWarps];
};

struct Cell {
    double rho, p, vz, vr;
};
__device__ __forceinline__ Cell load_cell(const double2* __restrict__ s, const double2* __restrict__ u, long long k)
{
    const double2 a = s[k], b = u[k];
    return Cell{a.x, a.y, b.x, b.y};
}

// the density of the inflow state of row m at n = 0 (kernel.cu:2004-2024)
__device__ __forceinline__ double inflow_rho(const Add2Params& P, double y, const double* TT_p)
{
    const double TT = *TT_p;
    if (y < 0.5 && TT < 3.0 && P.perturb) return P.in_rho * (1.0 + 0.01 * sin(TT * 3.14159265358979323846 * 2.0));
    return P.in_rho;
}

// z face at the left of column n (0 <= n <= N): its flux as its lower cell's
// right face in `right` and as its upper cell's left face in `left`
__device__ __forceinline__ double add2_zface(const Add2Params& P, const double2* s, const double2* u,
                                             const double* TT_p, int n, int m, double y, double right[4],
                                             double left[4])
{
    const long long k = (long long)m * P.N + n;
    Cell l, h;
    if (n < P.N) h = load_cell(s, u, k);
    if (n > 0) l = load_cell(s, u, k - 1);
    else l = Cell{inflow_rho(P, y, TT_p), P.in_p, P.in_vz, P.in_vr};
    if (n == P.N) h = l;   // outflow copy at n = N-1 (kernel.cu:1971-2001)
    const Gas<double>& g = P.g;
    double A[4], B[4], S;   // HLL, HLLC
    if (face_tame(l.rho, l.p, l.vz, l.vr, h.rho, h.p, h.vz, h.vr)) {
        const double c = sound_max(g, l.rho, l.p, h.rho, h.p);
        S = flux_hll_of(g, c, l.rho, l.p, l.vz, l.vr, h.rho, h.p, h.vz, h.vr, A);
        flux_hllc_of(g, c, l.rho, l.p, l.vz, l.vr, h.rho, h.p, h.vz, h.vr, B);
    } else {
        S = flux_hll_wild(g, l.rho, l.p, l.vz, l.vr, h.rho, h.p, h.vz, h.vr).get(A);
        S = fmax(S, flux_hllc_wild(g, l.rho, l.p, l.vz, l.vr, h.rho, h.p, h.vz, h.vr).get(B));
    }
    // HLLC inside the region for the lower cell, HLL inside for the upper
    // one (kernel.cu:2078-2085), each by its own cell's face position
    const double hdx = P.dx / 2.0;
    const bool cr = in_region(P, __dadd_rn(P.x_min, __dmul_rn((double)(n - 1), P.dx)) + hdx);
    const bool cl = !in_region(P, __dadd_rn(P.x_min, __dmul_rn((double)n, P.dx)) - hdx);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        right[q] = cr ? B[q] : A[q];
        left[q] = cl ? B[q] : A[q];
    }
    return S;
}

// r face below row m (0 <= m <= M), reflecting at both ends (kernel.cu:2026-2054)
__device__ __forceinline__ double add2_rface(const Add2Params& P, const double2* s, const double2* u, int n, int m,
                                             bool hllc, double F[4])
{
    const long long k = (long long)m * P.N + n;
    Cell l, h;
    if (m < P.M) h = load_cell(s, u, k);
    if (m > 0) l = load_cell(s, u, k - P.N);
    if (m == 0) { l = h; l.vr = -h.vr; }
    if (m == P.M) { h = l; h.vr = -l.vr; }
    double G[4];
    const double S = hllc ? flux_hllc(P.g, l.rho, l.p, l.vr, l.vz, h.rho, h.p, h.vr, h.vz, G)
                          : flux_hll(P.g, l.rho, l.p, l.vr, l.vz, h.rho, h.p, h.vr, h.vz, G);
    F[0] = G[0]; F[1] = G[2]; F[2] = G[1]; F[3] = G[3];   // mass, mom_z, mom_r, energy
    return S;
}

// the larger of a wave-speed maximum and S; a NaN leaves it (as the minimum
// of the dt candidates left a NaN out)
__device__ __forceinline__ double raised(double a, double S) { return is_nan(S) ? a : larger_speed(a, S); }

__global__ void __launch_bounds__(kThreads, 2)
    add2_kernel(const double2* __restrict__ s, const double2* __restrict__ u, double2* s2, double2* u2, double* T,
                const double* T_do_p, const double* TT_p, Add2Params P)
{
    __shared__ Add2Smem sm;
    const unsigned tiles_z = (unsigned)(P.N + kAZ - 1) / kAZ;
    const int n0 = (int)(blockIdx.x % tiles_z) * kAZ, m0 = (int)(blockIdx.x / tiles_z) * kAR, tid = threadIdx.x;
    const int col = tid & 31, w = tid >> 5, n = n0 + col;
    // cell centres as the reference forms them (separate products and sums)
    const double x = __dadd_rn(P.x_min, __dmul_rn((double)n, P.dx));
    auto row_y = [&](int m) { return __dadd_rn(P.y_min, __dmul_rn((double)m, P.dy)); };
    const bool rhllc = in_region(P, x);
    double left[kCells][4], sz = 0.0, sr = 0.0;
    // each thread the left and the bottom face of its cells
#pragma unroll
    for (int it = 0; it < kCells; it++) {
        const int row = w + it * kWarps, m = m0 + row;
        if (n <= P.N && m < P.M) {
            double right[4];
            sz = raised(sz, add2_zface(P, s, u, TT_p, n, m, row_y(m), right, left[it]));
#pragma unroll
            for (int q = 0; q < 4; q++) sm.zr[q][row][col] = right[q];
        }
        if (n < P.N && m <= P.M) {
            double F[4];
            sr = raised(sr, add2_rface(P, s, u, n, m, rhllc, F));
#pragma unroll
            for (int q = 0; q < 4; q++) sm.r[q][row][col] = F[q];
        }
    }
    // the tile's top row of r faces, and the last z face of each row
    if (w == 0) {
        const int m = m0 + kAR;
        if (n < P.N && m <= P.M) {
            double F[4];
            sr = raised(sr, add2_rface(P, s, u, n, m, rhllc, F));
#pragma unroll
            for (int q = 0; q < 4; q++) sm.r[q][kAR][col] = F[q];
        }
    } else if (w == 1 && col < kAR) {
        const int m = m0 + col;
        if (n0 + kAZ <= P.N && m < P.M) {
            double right[4], l[4];
            sz = raised(sz, add2_zface(P, s, u, TT_p, n0 + kAZ, m, row_y(m), right, l));
#pragma unroll
            for (int q = 0; q < 4; q++) sm.zr[q][col][kAZ] = right[q];
        }
    }
    sz = warp_max(sz);
    sr = warp_max(sr);
    if (col == 0) {
        sm.smax[0][w] = sz;
        sm.smax[1][w] = sr;
    }
    __syncthreads();
    if (tid == 0) {
        // dt candidate: min over faces of krit*rad/S = krit*rad/max S
        for (int i = 1; i < kWarps; i++) {
            sz = larger_speed(sz, sm.smax[0][i]);
            sr = larger_speed(sr, sm.smax[1][i]);
        }
        double tmin = P.dt_cap;
        if (sz > 0.0) tmin = fmin(tmin, P.krit_dx / sz);
        if (sr > 0.0) tmin = fmin(tmin, P.krit_dy / sr);
        atomicMin((unsigned long long*)T, (unsigned long long)__double_as_longlong(tmin));
    }

    // the planar update (kernel.cu:2201-2290)
    const double T_do = *T_do_p;
    const double ntz = -T_do / P.dx, zr = P.dx / P.dy;
    const bool body = P.body_force && x > P.body_lo && x < P.body_hi;
#pragma unroll
    for (int it = 0; it < kCells; it++) {
        const int row = w + it * kWarps, m = m0 + row;
        if (n >= P.N || m >= P.M) continue;
        const long long k = (long long)m * P.N + n;
        const Cell c = load_cell(s, u, k);
        const double in[4] = {c.rho, c.p, c.vz, c.vr};
        double f[4][4], o[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            f[q][0] = sm.zr[q][row][col + 1];
            f[q][1] = left[it][q];
            f[q][2] = sm.r[q][row][col];
            f[q][3] = sm.r[q][row + 1][col];
        }
        double Q2 = 0.0;
        if (body) Q2 = (row_y(m) >= P.body_rsplit) ? -P.body_amp * c.rho : P.body_amp * c.rho;
        int nrho = 0, np = 0;
        unsigned status = 0;
        update_cell64(P.g, P.p_floor, false, in, f, T_do, ntz, zr, 0.0, body, Q2, false, 0.0, 0.0, nrho, np, status, o);
        s2[k] = make_double2(o[0], o[1]);
        u2[k] = make_double2(o[2], o[3]);
    }
}

}  // namespace

extern "C" int ast_add2_raw(const double* s, const double* u, double* s2, double* u2, double* T, const double* T_do,
                            const double* TT, int method, int step, const ast_config* cfg, void* stream)
{
    (void)step;
    if (!s || !u || !s2 || !u2 || !T || !T_do || !TT || !cfg) return set_error(AST_ERR_INVALID, "null argument");
    int rc = ast_config_check(cfg);
    if (rc != AST_OK) return rc;
    if (cfg->precision != AST_PREC_FP64 || cfg->recon != AST_RECON_NONE || cfg->geom != AST_GEOM_PLANAR ||
        cfg->bc[AST_Z_LO].kind != AST_BC_FIXED)
        return set_error(AST_ERR_INVALID, "add2 is FP64, first order, planar, with a fixed z_lo inflow");
    Add2Params P;
    P.N = cfg->N;
    P.M = cfg->M;
    P.x_min = cfg->x_min;
    P.dx = (cfg->x_max - cfg->x_min) / (cfg->N - 1);
    P.dy = cfg->y_max / cfg->M;
    P.y_min = cfg->y_max / (2.0 * cfg->M);
    P.krit_dx = cfg->cfl * P.dx;
    P.krit_dy = cfg->cfl * P.dy;
    P.dt_cap = cfg->dt_cap;
    P.p_floor = cfg->p_floor;
    P.region_lo = cfg->region_select ? cfg->region_lo : 1e300;
    P.region_hi = cfg->region_select ? cfg->region_hi : -1e300;
    P.body_force = cfg->body_force;
    P.body_lo = cfg->body_lo;
    P.body_hi = cfg->body_hi;
    P.body_rsplit = cfg->body_rsplit;
    P.body_amp = cfg->body_amp;
    P.in_rho = cfg->bc[AST_Z_LO].rho;
    P.in_p = cfg->bc[AST_Z_LO].p;
    P.in_vz = cfg->bc[AST_Z_LO].vz;
    P.in_vr = cfg->bc[AST_Z_LO].vr;
    P.perturb = method != 0;
    P.g = make_gas<double>(cfg->gamma, cfg->riemann_tol, cfg->riemann_max_iter);
    const long long tiles = (long long)((P.N + kAZ - 1) / kAZ) * ((P.M + kAR - 1) / kAR);
    add2_kernel<<<(unsigned)tiles, kThreads, 0, (cudaStream_t)stream>>>((const double2*)s, (const double2*)u, (double2*)s2,
                                                             (double2*)u2, T, T_do, TT, P);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AST_OK : cuda_fail(e, "add2 kernel launch");
}
