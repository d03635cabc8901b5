// k_rad.cu - MultiLayerRadiation::run (MultiLayerRadiation.h:56-388) of the ATHAD_COND
// atmosphere on sm_100a, and the radiative heating of radiation mode 2
// (cAtmosphereModel.cpp:864-879), flat terrain.
//
// The layer emissivities come from the column mass with pressure broadening and the cloud
// liquid/ice paths; then the cloud short-wave albedo bump, four grey upward/downward sweeps
// that set each air layer to its radiative equilibrium, a final sweep, and the linearised
// surface energy balance.
//
// A CTA of eight warps takes 32 columns.  All warps form the emissivities, each its share of
// the levels, into shared memory; one warp runs the sweeps, one column per thread, from
// there; all warps write the results.  The emission sigma T^4 of a layer in equilibrium is
// the flux it absorbs, 0.5 (up + down), so the sweeps keep that flux instead of T: the
// temperatures are formed once at the end (two square roots per layer) instead of in every
// sweep (a division, two square roots and two fourth powers per layer and sweep).
// Before, one thread per column kept T and both fluxes in global memory: 593 us for the
// columns alone at 61x181x361, 17 of 21 cycles per issue waiting for loads, with two more
// passes over t for the blend.  Radiation mode 2 with the blend folded in: 629 -> 188 us.
// Compiled without fused multiply-add; exp is CUDA's.
#include "kernels.cuh"
#include "thermo.cuh"

namespace athad {

namespace {

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }

// T^4 as two squarings and x^(1/4) as two square roots, where the reference calls
// pow(T, 4.0) and pow(x, 0.25): each within two ulps of the exact power (sqrt is correctly
// rounded), at a few instructions instead of a logarithm and an exponential
__device__ __forceinline__ double pow4(double T) { const double t2 = T * T; return t2 * t2; }
__device__ __forceinline__ double root4(double x) { return sqrt(sqrt(x)); }

constexpr int kWarps = 8;        // warps per CTA
constexpr int kChunk = 4;        // levels whose operands a sweep loads at a time

// Where a column's values stand: [level][32 columns] in shared memory, or, for columns too
// tall for it, in the fields (emissivity) and scratch fields, a plane apart.
struct Column {
    double* e;       // emissivity
    double* f;       // emitted flux sigma T^4; the sign bit marks a layer no sweep has set
    double* up;      // upward flux
    long long s;     // distance between levels
};

// the four relaxation sweeps and the final one (:205-262) of one column; returns the
// downward flux at the lowest layer.  Level i's absorbed flux is formed in the downward
// sweep, where the flux from above is the running one; the values of kChunk levels are
// loaded before the first of them is stored.
__device__ __forceinline__ double sweeps(const Column& C, int i_trop, double up0)
{
    double dd = 0.0;
    for (int it = 0; it <= 4; it++) {
        double u = up0;
        for (int i0 = 1; i0 <= i_trop; i0 += kChunk) {
            double e[kChunk], f[kChunk], o[kChunk];
#pragma unroll
            for (int q = 0; q < kChunk; q++) {
                const long long at = (long long)min(i0 + q, i_trop) * C.s;
                e[q] = C.e[at]; f[q] = fabs(C.f[at]);
            }
#pragma unroll
            for (int q = 0; q < kChunk; q++) { u = u * (1.0 - e[q]) + e[q] * f[q]; o[q] = u; }
#pragma unroll
            for (int q = 0; q < kChunk; q++)
                if (i0 + q <= i_trop) C.up[(long long)(i0 + q) * C.s] = o[q];
        }
        dd = 0.0;
        for (int i0 = i_trop; i0 >= 1; i0 -= kChunk) {
            double e[kChunk], f[kChunk], below[kChunk];
#pragma unroll
            for (int q = 0; q < kChunk; q++) {
                const int i = max(i0 - q, 1);
                e[q] = C.e[(long long)i * C.s];
                f[q] = C.f[(long long)i * C.s];
                below[q] = (i == 1) ? up0 : C.up[(long long)(i - 1) * C.s];
            }
#pragma unroll
            for (int q = 0; q < kChunk; q++) {
                if (i0 - q < 1) break;
                const double emit = 0.5 * (below[q] + dd);
                if (it < 4 && emit > 0.0 && is_finite_bits(emit)) C.f[(long long)(i0 - q) * C.s] = emit;
                dd = dd * (1.0 - e[q]) + e[q] * fabs(f[q]);
            }
        }
    }
    return dd;
}

// BLEND: radiation mode 2, t := t (1 - omega) + t_RE omega, instead of t := t_RE.
// SHARED: the columns in shared memory (3 im doubles each).
template <bool BLEND, bool SHARED>
__global__ void __launch_bounds__(32 * kWarps) mlr_columns_kernel(RadArgs a, double omega)
{
    extern __shared__ double column_mem[];
    __shared__ double lwp_part[kWarps][32], iwp_part[kWarps][32];
    const Dims& d = a.d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    const int j = blockIdx.y;
    const bool mine = k < d.km;
    const long long sI = d.plane;
    const long long c0 = idx3(d, 0, j, mine ? k : 0);
    const int im = d.im, i_trop = im - 1;
    const double t_0 = a.t_0, sigma = a.sigma;
    Column C;
    if (SHARED) {
        C = {column_mem + lane, column_mem + 32 * im + lane, column_mem + 64 * im + lane, 32};
    } else {
        C = {a.epsilon + c0, a.T + c0, a.radiation + c0, sI};
    }
    // emissivities and condensate paths (:130-190), level i by warp i mod kWarps
    const double p_ref = 1.0e5, inv_g = 1.0 / a.g;
    double lwp = 0.0, iwp = 0.0;
    if (mine) {
        for (int i = warp; i <= i_trop; i += kWarps) {
            const long long c = c0 + i * sI;
            const double ps = a.p_stat[c];
            double dp_Pa = (i < i_trop) ? (ps - a.p_stat[c + sI]) * 100.0 : ps * 100.0;
            if (dp_Pa < 0.0) dp_Pa = 0.0;
            const double q_v = dmax(0.0, a.c[c]);
            const double q_c = dmax(0.0, a.co2[c]);
            const double q_b = dmax(0.0, 1.0 - q_v - q_c);
            const double u_col = dp_Pa * inv_g;
            const double broad = ps * 100.0 / p_ref;
            const double tau_gas = (a.kappa_H2O * q_v + a.kappa_CO2 * q_c + a.kappa_bg * q_b) * u_col * broad;
            const double dz = (i < i_trop) ? a.step_f[i] : a.step_f[i - 1];
            const double T_i = a.t[c] * t_0;
            const double R_i = thermo::R_of(q_v, q_c, a.R_bg);
            const double rho_i = (T_i > 0.0) ? (ps * 100.0) / (R_i * T_i) : 0.0;
            const double LWP_i = dmax(0.0, a.cloud[c]) * rho_i * dz * 1000.0;
            const double IWP_i = dmax(0.0, a.ice[c]) * rho_i * dz * 1000.0;
            lwp += LWP_i;
            iwp += IWP_i;
            const double tau = tau_gas + 0.12 * LWP_i + 0.055 * IWP_i;
            const double e = (tau > 700.0) ? 1.0 : (1.0 - exp(-tau));
            if (SHARED) a.epsilon[c] = e;
            C.e[i * C.s] = e;
            C.f[i * C.s] = -fabs(sigma * pow4(T_i));
            if (i == 0) a.epsilon_2D[(long long)j * d.pitch + k] = e;
        }
    }
    lwp_part[warp][lane] = lwp;
    iwp_part[warp][lane] = iwp;
    __syncthreads();
    if (warp == 0 && mine) {
        double lwp_col = 0.0, iwp_col = 0.0;
        for (int w = 0; w < kWarps; w++) { lwp_col += lwp_part[w][lane]; iwp_col += iwp_part[w][lane]; }
        // short-wave insolation: pole-to-equator parabola, mirrored (:99-114)
        const int j_max = d.jm - 1, j_half = j_max / 2;
        const int jj = (j > j_half) ? j_max - j : j;
        const double x = (double)jj / (double)j_half;
        const double sw = (a.rad_pole_short - a.rad_equator_short) * (x * x - 2.0 * x) + a.rad_pole_short;
        double albedo = a.albedo_surface;
        {
            const double cwp_sw = lwp_col + 0.50 * iwp_col;
            const double tau = cwp_sw / 100.0;
            const double refl = tau / (tau + 2.0);
            if (a.albedo_cloud > albedo) albedo = albedo + (a.albedo_cloud - albedo) * refl;
        }
        a.albedo[(long long)j * d.pitch + k] = albedo;
        const double t_s = a.t[c0], T_s0 = t_s * t_0;
        const double up0 = sigma * pow4(T_s0);
        const double L_down = sweeps(C, i_trop, up0);
        // the surface energy balance (:268-284)
        const double SW_abs = (1.0 - albedo) * sw;
        const double f1 = C.f[C.s];
        const double T_air1 = signbit(f1) ? a.t[c0 + sI] * t_0 : root4(f1 / sigma);
        const double c_H = 15.0;
        const double dsigT4 = 4.0 * sigma * T_s0 * T_s0 * T_s0;
        const double T_s = (SW_abs + a.geothermal_flux + L_down - sigma * pow4(T_s0)
                           + dsigT4 * T_s0 + c_H * T_air1) / (dsigT4 + c_H);
        const double t_re = T_s / t_0;
        a.t[c0] = BLEND ? t_s * (1.0 - omega) + t_re * omega : t_re;
        a.radiation[c0] = sigma * pow4(T_s);
    }
    __syncthreads();
    if (!mine) return;
    for (int i = 1 + warp; i <= i_trop; i += kWarps) {
        const long long c = c0 + i * sI;
        const double f = C.f[i * C.s], t = a.t[c];
        const double T = signbit(f) ? t * t_0 : root4(f / sigma);
        const double t_re = T / t_0;
        a.t[c] = BLEND ? t * (1.0 - omega) + t_re * omega : t_re;
        if (SHARED) a.radiation[c] = C.up[i * C.s];
    }
}

// cAtmosphereModel::planetaryShortWave's row sums (cAtmosphereModel.cpp:244-246): one CTA
// stages its row in shared memory and one thread adds the longitudes in order, so the host
// finishes the budget bit for bit.  (A thread adding its row from global memory: 37 us at
// 181x361, one dependent load after another.)
__global__ void __launch_bounds__(128) albedo_rows_kernel(Dims d, const double* __restrict__ albedo,
                                                         double* __restrict__ out)
{
    constexpr int kPart = 1024;
    __shared__ double part[kPart];
    const double* row = albedo + (long long)blockIdx.x * d.pitch;
    double s = 0.0;
    for (int k0 = 0; k0 < d.km; k0 += kPart) {
        const int n = min(kPart, d.km - k0);
        __syncthreads();
        for (int k = threadIdx.x; k < n; k += blockDim.x) part[k] = row[k0 + k];
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll 8
            for (int k = 0; k < n; k++) s += part[k];
        }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

template <bool BLEND>
void launch_columns(const RadArgs& a, double omega, cudaStream_t st)
{
    const dim3 grid((a.d.km + 31) / 32, a.d.jm);
    const size_t mem = 3 * 32 * sizeof(double) * (size_t)a.d.im;
    // Columns of up to 288 layers fit the 227 KB of a CTA (with the path sums), and of up to 145
    // two CTAs fit an SM.  Above that one CTA is left on an SM, seven of its warps wait for the
    // eighth, and the columns in the fields, of which many CTAs run on an SM, are faster unless
    // the SMs have no second CTA to run.  Shared memory and fields, us per call: 181 x 361
    // columns 189 and 329 (61 layers), 774 and 893 (140), 1502 and 992 (150), 2849 and 2486
    // (288); 91 x 181 42 and 86, 197 and 258, 402 and 279, 761 and 671; 30 x 61 (60 CTAs) 37 and
    // 56, 79 and 142, 84 and 150, 156 and 375.
    constexpr size_t kMost = 3 * 32 * sizeof(double) * 288, kTwoPerSM = 3 * 32 * sizeof(double) * 145;
    const bool few = (size_t)grid.x * grid.y <= 148;
    if (mem <= (few ? kMost : kTwoPerSM)) {
        // the kernel's limit is the process's: every caller sets the same one, so that a thread
        // with lower columns cannot lower it between another's call and its launch
        if (mem > 40960)
            cudaFuncSetAttribute(mlr_columns_kernel<BLEND, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
        mlr_columns_kernel<BLEND, true><<<grid, 32 * kWarps, mem, st>>>(a, omega);
    } else {
        mlr_columns_kernel<BLEND, false><<<grid, 32 * kWarps, 0, st>>>(a, omega);
    }
}

}  // namespace

void launch_albedo_rows(const Dims& d, const double* albedo, double* out, cudaStream_t st)
{
    albedo_rows_kernel<<<d.jm, 128, 0, st>>>(d, albedo, out);
}

void launch_multilayer_radiation(const RadArgs& a, cudaStream_t st) { launch_columns<false>(a, 0.0, st); }

void launch_radiative_heating(const RadArgs& a, double omega, cudaStream_t st) { launch_columns<true>(a, omega, st); }

}  // namespace athad
