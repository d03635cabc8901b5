// k_bc.cu - the per-iteration boundary conditions of the atmosphere on sm_100a
// (athad_boundary_conditions): BC_Atm::bcRadius, TurbulenceAtm::apply_wall_bc,
// BC_Atm::bcTheta, BC_Atm::bcPhi, BC_Atm::bcScalarSurfSur and BC_Atm::bcSolidGround, in the
// order of their call site (cAtmosphereModel.cpp:1439-1446), for flat terrain (every cell is
// air, so of the last two only bcSolidGround's value limits over every cell change anything).
//
// Three launches, one per direction, because each reads the boundary cells the previous
// one wrote (the corners): radial columns (one thread per (j, k) and field), polar rows (one
// thread per (i, k) and field), seam rows (one thread per (i, j) and field); then the value
// limits, cell by cell.  A field's conditions read that field only (and 2-D inputs), so the
// fields run side by side, blockIdx.z apart; one thread taking all 43 to 50 fields in turn
// waited for one field's loads after another's stores: radial 61, polar 44, seam 61 us at
// 41x181x361, now 26, 6 and 28; the limits 88, now 56 with all loads before the first store.  Every formula is a copy or
// a short sum evaluated in the reference's order; the file is compiled without fused
// multiply-add, so the results are bit-identical to the reference's.
//
// Fields: those of the reference's lists that the context holds (the right-hand side's
// CoriolisForce and BuoyancyForce, the heat diagnostics Q_Latent and Q_Sensible and the
// radiation flux included).  The reference's other arrays in the same lists, the outputs of
// ThermoAtm::forces and precipitableWater, are not held.  c43 and c13 are `const int` members
// initialised from 4.0/3.0 and 1.0/3.0 (cAtmosphereModel.h:158), i.e. 1 and 0.
#include "kernels.cuh"

namespace athad {

namespace {

template <int N>
constexpr int count(const int (&)[N]) { return N; }

__constant__ int kBothCubic[] = {                       // BC_Atm.h:567-574, Pattern A
    ATHAD_S_C_C, ATHAD_S_V, ATHAD_S_C, ATHAD_S_I, ATHAD_S_R, ATHAD_S_S, ATHAD_S_G,
    ATHAD_Q_V_U, ATHAD_Q_C_U, ATHAD_U_U, ATHAD_V_U, ATHAD_W_U,
    ATHAD_MC_S, ATHAD_MC_S_U, ATHAD_MC_S_D, ATHAD_M_U, ATHAD_M_D, ATHAD_Q_LATENT, ATHAD_Q_SENSIBLE,
    ATHAD_CORIOLIS_FORCE, ATHAD_BUOYANCY_FORCE};
__constant__ int kCubicBotVnTop[] = {                   // :599-603, Pattern C
    ATHAD_CLOUD, ATHAD_ICE, ATHAD_GR, ATHAD_CO2,
    ATHAD_C_U, ATHAD_E_DD, ATHAD_E_L, ATHAD_E_P, ATHAD_G_P,
    ATHAD_TKE, ATHAD_DIS, ATHAD_NUE, ATHAD_PROD, ATHAD_TKE_SOURCE, ATHAD_DIS_SOURCE};
__constant__ int kHydro[] = {ATHAD_P_STAT, ATHAD_R_HUMID, ATHAD_R_DRY};  // :656-665, Pattern D
__constant__ int kTheta[] = {                           // :760-776
    ATHAD_T, ATHAD_RADIATION, ATHAD_P_STAT, ATHAD_R_HUMID, ATHAD_R_DRY, ATHAD_U, ATHAD_V, ATHAD_W, ATHAD_C,
    ATHAD_CLOUD, ATHAD_ICE, ATHAD_GR, ATHAD_CO2, ATHAD_TKE, ATHAD_DIS, ATHAD_NUE, ATHAD_PROD,
    ATHAD_TKE_SOURCE, ATHAD_DIS_SOURCE,
    ATHAD_S_C_C, ATHAD_S_V, ATHAD_S_C, ATHAD_S_I, ATHAD_S_R, ATHAD_S_S, ATHAD_S_G,
    ATHAD_Q_V_U, ATHAD_Q_C_U, ATHAD_U_U, ATHAD_V_U, ATHAD_W_U, ATHAD_MC_S, ATHAD_MC_S_U,
    ATHAD_MC_S_D, ATHAD_C_U, ATHAD_E_DD, ATHAD_E_L, ATHAD_E_P, ATHAD_G_P, ATHAD_Q_LATENT,
    ATHAD_Q_SENSIBLE, ATHAD_CORIOLIS_FORCE, ATHAD_BUOYANCY_FORCE};
__constant__ int kPhiAvg[] = {                          // :806-817
    ATHAD_T, ATHAD_RADIATION, ATHAD_P_STAT, ATHAD_R_HUMID, ATHAD_R_DRY, ATHAD_U, ATHAD_V, ATHAD_W, ATHAD_C,
    ATHAD_CLOUD, ATHAD_ICE, ATHAD_GR, ATHAD_CO2,
    ATHAD_S_C_C, ATHAD_S_V, ATHAD_S_C, ATHAD_S_I, ATHAD_S_R, ATHAD_S_S, ATHAD_S_G,
    ATHAD_Q_V_U, ATHAD_Q_C_U, ATHAD_U_U, ATHAD_V_U, ATHAD_W_U, ATHAD_MC_S, ATHAD_MC_S_U,
    ATHAD_MC_S_D, ATHAD_C_U, ATHAD_E_DD, ATHAD_E_L, ATHAD_E_P, ATHAD_G_P, ATHAD_Q_LATENT,
    ATHAD_Q_SENSIBLE, ATHAD_CORIOLIS_FORCE, ATHAD_BUOYANCY_FORCE};
__constant__ int kPhiExtrap[] = {ATHAD_TKE, ATHAD_DIS, ATHAD_NUE, ATHAD_PROD, ATHAD_TKE_SOURCE,
                                 ATHAD_DIS_SOURCE};    // :822-825

// the field's place q in a list of lists: the list and the field there
constexpr int kNBothCubic = count(kBothCubic), kNHydro = count(kHydro), kNCubicBotVnTop = count(kCubicBotVnTop);
// the fields whose radial conditions are their own: the lid temperature, the velocities and
// their level n, P_conv
__constant__ int kRadialOwn[] = {ATHAD_T, ATHAD_U, ATHAD_UN, ATHAD_V, ATHAD_W, ATHAD_VN, ATHAD_WN, ATHAD_P_CONV};
constexpr int kNRadius = kNBothCubic + kNHydro + kNCubicBotVnTop + count(kRadialOwn);

// bcRadius (BC_Atm.h:556-746) and apply_wall_bc (TurbulenceAtm.h:109-147), one radial
// column of one field per thread
__global__ void __launch_bounds__(128) bc_radius_kernel(BcArgs a)
{
    const Dims& d = a.d;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (k >= d.km) return;
    const int iml = d.im - 1;
    const long long s = d.plane;
    const long long c0 = idx3(d, 0, j, k), cl = idx3(d, iml, j, k);
    const long long c2 = (long long)j * d.pitch + k;
    int q = blockIdx.z;
    if (q < kNBothCubic) {                                                             // :629-633
        const int f = kBothCubic[q];
        double* x = a.F[f];
        const double v = x[c0 + 3 * s] - 3.0 * x[c0 + 2 * s] + 3.0 * x[c0 + s];
        // the lid reads level 0 on a grid of four levels
        const double x1 = x[cl - s], x2 = x[cl - 2 * s], x3 = (iml == 3) ? v : x[cl - 3 * s];
        x[c0] = ((f == ATHAD_Q_V_U || f == ATHAD_Q_C_U) && v < 0.0) ? 0.0 : v;          // :734-735
        x[cl] = x3 - 3.0 * x2 + 3.0 * x1;
        return;
    }
    q -= kNBothCubic;
    if (q < kNHydro) {                                                                 // :656-665
        double* x = a.F[kHydro[q]];
        const double v = x[c0 + 3 * s] - 3.0 * x[c0 + 2 * s] + 3.0 * x[c0 + s];
        const double x1 = x[cl - s], x2 = x[cl - 2 * s];
        x[c0] = v;
        x[cl] = (x1 > 0.0 && x2 > 0.0) ? (x1 * x1 / x2) : x1;
        return;
    }
    q -= kNHydro;
    if (q < kNCubicBotVnTop) {                                                         // :727-731
        const int f = kCubicBotVnTop[q];
        double* x = a.F[f];
        double v = x[c0 + 3 * s] - 3.0 * x[c0 + 2 * s] + 3.0 * x[c0 + s];
        const double top = 1.0 * x[cl - s] - 0.0 * x[cl - 2 * s];
        if (a.wall_bc) {   // apply_wall_bc: the wall values of tke, nue and dis
            const double vs = a.vel_star[c2];
            if (f == ATHAD_TKE) v = vs * vs / a.tke_wall_den;
            if (f == ATHAD_NUE) v = 0.0;
            if (f == ATHAD_DIS && a.set_dis_wall) v = a.dis_wall;
        }
        x[c0] = v;
        x[cl] = top;
        return;
    }
    q -= kNCubicBotVnTop;
    const int f = kRadialOwn[q];
    double* x = a.F[f];
    if (f == ATHAD_T) {
        x[cl] = a.t_top_init[c2];                                                      // :613-614
    } else if (f == ATHAD_U || f == ATHAD_UN) {
        x[cl] = 0.0; x[c0] = 0.0;                                                      // :704-705, 723-724
    } else {
        if (f == ATHAD_V || f == ATHAD_W || f == ATHAD_P_CONV) {                       // :671-675
            x[c0] = 1.0 * x[c0 + s] - 0.0 * x[c0 + 2 * s];
            if (f == ATHAD_P_CONV) { x[cl] = x[cl - s]; return; }
        }
        x[cl] = 0.0;                                                                   // :685-690
        x[cl - s] *= (1.0 / 3.0);
        x[cl - 2 * s] *= (2.0 / 3.0);
    }
}

// bcTheta (BC_Atm.h:750-796): pole copies, one (i, k) of one field per thread
__global__ void __launch_bounds__(128) bc_theta_kernel(BcArgs a)
{
    const Dims& d = a.d;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (k >= d.km) return;
    const long long n0 = idx3(d, i, 0, k), nl = idx3(d, i, d.jm - 1, k);
    double* x = a.F[kTheta[blockIdx.z]];
    const double v0 = x[n0 + d.pitch], vl = x[nl - d.pitch];
    x[n0] = v0;
    x[nl] = vl;
}

// one 1-2-1 pass over the three seam cells {km-2, 0 = km-1, 1} of a row (BC_Atm.h:869-906)
__device__ __forceinline__ void smooth_seam(double* x, int km)
{
    const double c = 0.25;
    const double f_km2 = x[km - 2], f_0 = x[0], f_1 = x[1];
    const double w_km2 = x[km - 3], e_km2 = f_0;
    const double w_0 = f_km2, e_0 = f_1;
    const double w_1 = f_0, e_1 = x[2];
    x[km - 2] = f_km2 + c * (w_km2 - 2.0 * f_km2 + e_km2);
    const double m = f_0 + c * (w_0 - 2.0 * f_0 + e_0);
    x[0] = m;
    x[km - 1] = m;
    x[1] = f_1 + c * (w_1 - 2.0 * f_1 + e_1);
}

// the level n of the velocities: smoothed, not averaged
__constant__ int kPhiSmooth[] = {ATHAD_UN, ATHAD_VN, ATHAD_WN};
constexpr int kNPhiAvg = count(kPhiAvg), kNPhiExtrap = count(kPhiExtrap);
constexpr int kNPhi = kNPhiAvg + kNPhiExtrap + count(kPhiSmooth);

// bcPhi (BC_Atm.h:803-918), one (i, j) row of one field per thread: seam average or
// zero-gradient, then the two smoothing passes of the velocities (each row's passes read only
// that row, so running them right after the row's own averaging is the reference's order)
__global__ void __launch_bounds__(128) bc_phi_kernel(BcArgs a)
{
    const Dims& d = a.d;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= d.jm) return;
    const long long r = idx3(d, i, j, 0);
    const int km = d.km;
    const int q = blockIdx.z;
    int f;
    if (q < kNPhiAvg + kNPhiExtrap) {
        f = q < kNPhiAvg ? kPhiAvg[q] : kPhiExtrap[q - kNPhiAvg];
        double* x = a.F[f] + r;
        const double v0 = 1.0 * x[1] - 0.0 * x[2];
        const double vend = 1.0 * x[km - 2] - 0.0 * x[km - 3];
        const double m = (v0 + vend) * 0.5;
        x[0] = q < kNPhiAvg ? m : v0;
        x[km - 1] = q < kNPhiAvg ? m : vend;
        if (f != ATHAD_U && f != ATHAD_V && f != ATHAD_W) return;
    } else {
        f = kPhiSmooth[q - kNPhiAvg - kNPhiExtrap];
    }
    for (int pass = 0; pass < 2; pass++) smooth_seam(a.F[f] + r, km);
}

// bcScalarSurfSur and bcSolidGround (BC_Atm.h:1026-1123, 23-547) with flat terrain: their
// land branches and the surface copies x[0] := x[i_mount = 0] change nothing, which leaves
// bcSolidGround's value limits over every cell (:470-545), one (i, j) row per block row
// a limit stores only where it changes the value (bit for bit: -0.0 stays -0.0), so the
// common case reads the fields and writes nothing
__device__ __forceinline__ void store_if_changed(double* p, double old_v, double new_v)
{
    if (__double_as_longlong(old_v) != __double_as_longlong(new_v)) *p = new_v;
}

__global__ void __launch_bounds__(128) bc_limits_kernel(BcArgs a)
{
    const Dims& d = a.d;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.km) return;
    const long long c = (long long)blockIdx.y * d.pitch + k;
    double* const* F = a.F;
    const double prod_max = 1.0e4, dis_max = 1.0e6, vm = a.vel_max_nd;
    // c, cloud, ice; tke, dis; the clamped fields; the velocities and their level n: all
    // loaded before the first store
    const int field[17] = {ATHAD_C, ATHAD_CLOUD, ATHAD_ICE, ATHAD_TKE, ATHAD_DIS, ATHAD_TKEN, ATHAD_DISN, ATHAD_NUE,
                           ATHAD_PROD, ATHAD_TKE_SOURCE, ATHAD_DIS_SOURCE,
                           ATHAD_U, ATHAD_UN, ATHAD_V, ATHAD_VN, ATHAD_W, ATHAD_WN};
    const double lo[11] = {0.0, 0.0, 0.0, 0.0, 1.0e-10, 0.0, 1.0e-10, 0.0, 0.0, -prod_max, -prod_max};
    const double hi[11] = {0.0, 0.0, 0.0, a.tke_max_nd, dis_max, a.tke_max_nd, dis_max, a.nue_max, prod_max, prod_max,
                           prod_max};
    double v[17];
#pragma unroll
    for (int q = 0; q < 17; q++) v[q] = F[field[q]][c];
#pragma unroll
    for (int q = 0; q < 17; q++) {
        double w = v[q];
        if (q < 3) {
            if (w < 0.0) w = 0.0;
        } else if (q < 11) {
            // tke and dis: a negative value becomes 0 first, which the clamp keeps, or 1e-10
            if (q < 5 && w < 0.0) w = 0.0;
            w = safe_clamp(w, lo[q], hi[q]);
        } else {
            w = !is_finite_bits(w) ? 0.0 : (w < -vm) ? -vm : (w > vm) ? vm : w;
        }
        store_if_changed(F[field[q]] + c, v[q], w);
    }
}

}  // namespace

void launch_boundary_conditions(const BcArgs& a, cudaStream_t st)
{
    const Dims& d = a.d;
    bc_radius_kernel<<<dim3((d.km + 127) / 128, d.jm, kNRadius), 128, 0, st>>>(a);
    bc_theta_kernel<<<dim3((d.km + 127) / 128, d.im, count(kTheta)), 128, 0, st>>>(a);
    bc_phi_kernel<<<dim3((d.jm + 127) / 128, d.im, kNPhi), 128, 0, st>>>(a);
    bc_limits_kernel<<<dim3((d.km + 127) / 128, d.im * d.jm), 128, 0, st>>>(a);
}

}  // namespace athad
