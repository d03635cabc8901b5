// k_rk4m.cu - the mixed-precision RK4 step (athad_params.precision = MIXED) on sm_100a.
//
// Same time step as k_rk4.cu (RungeKutta_Atm_Turb.cpp:44-273 with the right-hand side of
// RHS_Atm_Turb.cpp:31-1080, flat terrain, Jacobi stages), with this split of precision:
//   * FP32: the right-hand-side arithmetic, the three intermediate stage states, the RK4
//     accumulator K = k1 + 2k2 + 2k3, a FP32 copy of the time level n for stages 2-3, and
//     the per-cell forcing, packed once per step by stage 1 (below);
//   * FP64: the prognostic fields themselves (time level n and the result), the final
//     combination y = y_n + dt/6 (K + k4) of stage 4, the stage-1 state y_n + dt/2 k1,
//     the level-mean temperature and the mean-density profile.
// The model's other modules keep reading and writing the FP64 fields; only the RK4
// step's private buffers are FP32.
//
// Private buffers: four fields of a cell side by side in a float4 (rk4m_field_group), so a
// stencil point of four fields is one 16-byte load and one address instead of four.  Stage
// state: (u, v, w, p_dyn), (tke, dis, t, c), (cloud, ice, gr, co2).  The accumulator and the
// FP32 level n have the same groups; their fourth place of group 0 carries nue and MC_v's
// source.  Separate FP32 arrays per field made stages 2 and 3 issue-limited: 140 M warp
// instructions and 205 us each at 41x181x361, now 113 M and 135 us, the step 1042 -> 848 us
// (809 with prefetch_tile, 785 with each stage's own registers); the results are the same bits.
//
// Forcing packing: the reference's RHS reads 15 per-cell forcing fields (p_dyn, nue, t_eq,
// p_stat, r_humid, S_c..S_v, MC_t..MC_w) in every stage.  Stage 1 reads them in FP64 and
// writes 11 FP32 values that the later stages read instead: p_dyn (with the stage state),
// nue, t_eq, the Held-Suarez relaxation rate k_T L/u_0, and the combined source terms of t,
// c, cloud, ice, gr, v and w, each formed in FP64 from the same operands as the reference's
// terms (stage 4, which does not read the FP32 level n, forms v's again).
//
// Memory traffic per grid point and step (algorithmic, 4-byte FP32 and 8-byte FP64
// fields): stage 1 reads 11 state + 11 level-n + 15 forcing FP64 and writes 12 stage + 12 K
// + 12 level-n + 8 forcing FP32 = 472 B; stages 2-3 read 12 stage + 12 level-n + 12 K + 8
// forcing FP32 and write 12 stage + 12 K FP32 = 272 B each; stage 4 reads 12 stage + 12 K +
// 8 forcing FP32 and 11 level-n and MC_v FP64 and writes 11 FP64 results + 3 FP64 aux =
// 336 B; with the level mean (8 B), 1360 B against 2096 B for the FP64 step.
//
// Mirror symmetry: the same expression structure as the FP64 kernel (second differences
// sum the two neighbours first; mirror-exact FP32 tables rounded from the FP64 ones);
// negation commutes with every IEEE operation including fused multiply-add, so a mirrored
// state still gives a bit-for-bit mirrored result.
#include "kernels.cuh"

namespace athad {

namespace {

__device__ __forceinline__ float fmaxs(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float fmins(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float fclamps(float v, float lo, float hi) { return (v < lo) ? lo : (hi < v) ? hi : v; }
__device__ __forceinline__ float fminmod(float a, float b)
{
    return (a * b <= 0.0f) ? 0.0f : (fabsf(a) < fabsf(b) ? a : b);
}

struct StarF {
    float c, ip, im, jp, jm, kp, km;
};
// the stars of one cell group's four values
struct Star4 {
    float4 c, ip, im, jp, jm, kp, km;
};

// The field at place q of group G (rk4m_field_group, rk4m_field_place); 11 = p_dyn
__host__ __device__ constexpr int group_field(int G, int q)
{
    return G == 0 ? (q < 3 ? 1 + q : 11) : G == 1 ? (q == 0 ? 9 : q == 1 ? 10 : q == 2 ? 0 : 4) : 5 + q;
}

__device__ __forceinline__ Star4 load_star4(const float4* __restrict__ p, int sI, int sJ)
{
    Star4 s;
    s.c = __ldg(p);
    s.ip = __ldg(p + sI); s.im = __ldg(p - sI);
    s.jp = __ldg(p + sJ); s.jm = __ldg(p - sJ);
    s.kp = __ldg(p + 1);  s.km = __ldg(p - 1);
    return s;
}
// the star of one FP64 field, rounded to FP32
__device__ __forceinline__ StarF load_star64(const double* __restrict__ p, int sI, int sJ)
{
    StarF s;
    s.c = (float)__ldg(p);
    s.ip = (float)__ldg(p + sI); s.im = (float)__ldg(p - sI);
    s.jp = (float)__ldg(p + sJ); s.jm = (float)__ldg(p - sJ);
    s.kp = (float)__ldg(p + 1);  s.km = (float)__ldg(p - 1);
    return s;
}
template <int Q> __device__ __forceinline__ float comp(const float4& v)
{
    return Q == 0 ? v.x : Q == 1 ? v.y : Q == 2 ? v.z : v.w;
}
template <int Q> __device__ __forceinline__ StarF comp(const Star4& s)
{
    return {comp<Q>(s.c), comp<Q>(s.ip), comp<Q>(s.im), comp<Q>(s.jp), comp<Q>(s.jm), comp<Q>(s.kp), comp<Q>(s.km)};
}

// The stars of one group: stage 1 reads the FP64 fields, the others the grouped buffer
struct Group {
    StarF s[4];
};
template <int STAGE, int G>
__device__ __forceinline__ Group load_group(const RK4MArgs& a, long long c, int sI, int sJ)
{
    Group g;
    if (STAGE == 1) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int n = group_field(G, q);
            g.s[q] = load_star64((n == 11 ? a.p_dyn : a.Y[n]) + c, sI, sJ);
        }
    } else {
        const Star4 s = load_star4(a.Yin[G] + c, sI, sJ);
        g.s[0] = comp<0>(s); g.s[1] = comp<1>(s); g.s[2] = comp<2>(s); g.s[3] = comp<3>(s);
    }
    return g;
}

__device__ __forceinline__ float d1r(const StarF& s, const RK4MArgs& a) { return (s.ip - s.im) * a.inv_2dr; }
__device__ __forceinline__ float d1t(const StarF& s, const RK4MArgs& a) { return (s.jp - s.jm) * a.inv_2dthe; }
__device__ __forceinline__ float d1p(const StarF& s, const RK4MArgs& a) { return (s.kp - s.km) * a.inv_2dphi; }
__device__ __forceinline__ float d2r(const StarF& s, const RK4MArgs& a) { return (s.ip - 2.0f * s.c + s.im) * a.inv_dr2; }
__device__ __forceinline__ float d2t(const StarF& s, const RK4MArgs& a) { return ((s.jp + s.jm) - 2.0f * s.c) * a.inv_dthe2; }
__device__ __forceinline__ float d2p(const StarF& s, const RK4MArgs& a) { return (s.kp - 2.0f * s.c + s.km) * a.inv_dphi2; }
__device__ __forceinline__ float ar(const StarF& s, const RK4MArgs& a) { return fminmod(s.c - s.im, s.ip - s.c) * a.inv_dr; }
__device__ __forceinline__ float at(const StarF& s, const RK4MArgs& a) { return fminmod(s.c - s.jm, s.jp - s.c) * a.inv_dthe; }
__device__ __forceinline__ float ap(const StarF& s, const RK4MArgs& a) { return fminmod(s.c - s.km, s.kp - s.c) * a.inv_dphi; }

// the clamps of RungeKutta_Atm_Turb.cpp:176-263 on the stage's value of field n
__device__ __forceinline__ double clamp_field(const RK4MArgs& a, int n, double y)
{
    if (n >= 4 && n <= 7) return smax(0.0, y);
    if (n == 9) return safe_clamp(y, 0.0, (double)a.tke_max_nd);
    if (n == 10) return smax(1.0e-10, y);
    return y;
}
__device__ __forceinline__ float clamp_field(const RK4MArgs& a, int n, float y)
{
    if (n >= 4 && n <= 7) return fmaxs(0.0f, y);
    if (n == 9) return isfinite(y) ? fclamps(y, 0.0f, a.tke_max_nd) : 0.0f;
    if (n == 10) return fmaxs(1.0e-10f, y);
    return y;
}

// Stage update of group G from its right-hand sides kn.  acc and yn are the group's
// accumulator and FP32 time level n (stages 2-4, 2-3; loaded by the caller).  In group 0 the
// fourth places carry p_dyn (stage buffers), nue (accumulator) and MC_v's source (level n).
template <int STAGE, int G>
__device__ __forceinline__ void update_group(const RK4MArgs& a, long long c, const float (&kn)[4], const float4& acc4,
                                             const float4& yn4, float p, float nue, float mv)
{
    const float acc[4] = {acc4.x, acc4.y, acc4.z, acc4.w};
    const float ynf[4] = {yn4.x, yn4.y, yn4.z, yn4.w};
    float y_out[4], k_out[4], n_out[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int n = group_field(G, q);
        if (n == 11) {
            y_out[q] = p; k_out[q] = nue; n_out[q] = mv;
            continue;
        }
        if (STAGE == 1) {
            const double yn = __ldg(a.Yn[n] + c);
            n_out[q] = (float)yn;
            k_out[q] = kn[q];
            y_out[q] = (float)clamp_field(a, n, yn + (double)kn[q] * a.half_dt);
        } else if (STAGE < 4) {
            k_out[q] = acc[q] + 2.0f * kn[q];
            y_out[q] = clamp_field(a, n, ynf[q] + kn[q] * ((STAGE == 3) ? a.dt_f : a.half_dt_f));
        } else {
            const double yn = __ldg(a.Yn[n] + c);
            const float kk = acc[q] + kn[q];
            const double y = clamp_field(a, n, yn + (double)kk * a.dt_sixth);
            a.Y[n][c] = y;
            if (a.store_n) a.Yn_store[n][c] = y;   // storeIntermediateData3D fused
        }
    }
    if (STAGE < 4) {
        a.Yout[G][c] = make_float4(y_out[0], y_out[1], y_out[2], y_out[3]);
        a.K[G][c] = make_float4(k_out[0], k_out[1], k_out[2], k_out[3]);
    }
    if (STAGE == 1) a.Yn32[G][c] = make_float4(n_out[0], n_out[1], n_out[2], n_out[3]);
}

}  // namespace

// Asks the L2 for the rows that a tile's cells read once (and for its centre rows), BY rows
// of bx cells from (i, j0, k0): one bulk prefetch per field and row, issued by the threads of
// the CTA before they start.  A cell's loads are spread over its arithmetic because they
// have to go through registers; the prefetch puts the tile's whole traffic in flight at
// once.  The FP64 fields of stage 1 are t..MC_w in the slab's order, one fstride apart.
// The pitch is a multiple of 32, so every row piece starts and ends on 16 bytes.
// 41x181x361: 848 -> 809 us per step.  Prefetching another CTA's tile (300 or more CTAs
// ahead) is slower, 847-985 us: the SM that will read it may be on the other die.
template <int STAGE>
__device__ __forceinline__ void prefetch_tile(const RK4MArgs& a, int i, int j0, int k0, int bx, int by, int tid,
                                              int nthreads)
{
    static_assert(ATHAD_T == 0 && ATHAD_P_DYN == 22 && ATHAD_MC_W == 36, "stage 1 prefetches fields 0..36");
    constexpr int kRows = (STAGE == 1) ? 37 : (STAGE == 4) ? 20 : 11;
    const unsigned n = (unsigned)min(bx, a.d.pitch - k0);
    for (int q = tid; q < kRows * by; q += nthreads) {
        const int f = q % kRows, j = j0 + q / kRows;
        if (j >= a.d.jm) break;
        const long long c0 = idx3(a.d, i, j, k0);
        const void* p;
        unsigned bytes = n * 16;
        if (STAGE == 1) { p = a.Y[0] + f * a.d.fstride + c0; bytes = n * 8; }
        else if (f < 3) p = a.Yin[f] + c0;
        else if (f < 6) p = a.K[f - 3] + c0;
        else if (f < 8) p = a.F[f - 6] + c0;
        else if (STAGE < 4) p = a.Yn32[f - 8] + c0;
        else { p = (f < 19 ? a.Yn[f - 8] : a.MC_v) + c0; bytes = n * 8; }
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
    }
}

// One cell of one stage.
template <int STAGE>
__device__ __forceinline__ void rk4m_cell(const RK4MArgs& a, int i, int j, int k, float buoy_pref)
{
    const Dims& d = a.d;
    const long long c = idx3(d, i, j, k);
    if (STAGE == 4 && a.store_n) {   // the copy's precipitation fluxes (UtilsAtm.h:41-42)
        a.rain_n[c] = __ldg(a.rain + c);
        a.rain_n[c + d.fstride] = __ldg(a.rain + c + d.fstride);
    }
    const bool interior = (i > 0 && i < d.im - 1 && j > 0 && j < d.jm - 1 && k > 0 && k < d.km - 1);
    if (!interior) {
        if (STAGE == 1) {   // boundary values into both stage buffers; p_dyn for the stencil
#pragma unroll
            for (int G = 0; G < 3; G++) {
                float v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int n = group_field(G, q);
                    v[q] = (float)__ldg((n == 11 ? a.p_dyn : a.Y[n]) + c);
                }
                const float4 v4 = make_float4(v[0], v[1], v[2], v[3]);
                a.Yout[G][c] = v4;
                a.Ybnd[G][c] = v4;
            }
        }
        if (STAGE == 4 && a.store_n) {   // the time-level copy of the cells RK4 leaves alone
#pragma unroll
            for (int n = 0; n < 11; n++) a.Yn_store[n][c] = __ldg(a.Y[n] + c);
        }
        return;
    }
    const int sI = (int)d.plane, sJ = d.pitch;
    const GeoF* G = a.geo + (i * d.jm + j);
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // group 0's accumulator and level n carry nue and MC_v's source; F[0] the w and t forcing
    const float4 acc0 = (STAGE == 1) ? zero4 : a.K[0][c];
    const float4 yn0 = (STAGE == 2 || STAGE == 3) ? __ldg(a.Yn32[0] + c) : zero4;
    float4 F0 = (STAGE == 1) ? zero4 : __ldg(a.F[0] + c);
    const Group g0 = load_group<STAGE, 0>(a, c, sI, sJ);
    const StarF &U = g0.s[0], &V = g0.s[1], &W = g0.s[2], &P = g0.s[3];
    const float exp_rm = G->exp_rm, inv_rm = G->inv_rm, inv_rmsinthe = G->inv_rmsinthe;

    const float u_ijk = U.c, v_ijk = V.c, w_ijk = W.c;
    const float nue_ijk = (STAGE == 1) ? (float)__ldg(a.nue + c) : acc0.w;
    const float u_exp = u_ijk * exp_rm, v_invrm = v_ijk * inv_rm, w_invrs = w_ijk * inv_rmsinthe;
    const float diffusion_vel_re = (a.inv_re + nue_ijk) * a.diffusion_ramp;

    // group 1's centre values, which the production and the buoyancy need; its stars are
    // loaded after group 0 is done, so that only one group's stars are held at a time
    const float4 y1 = (STAGE == 1) ? make_float4((float)__ldg(a.Y[9] + c), (float)__ldg(a.Y[10] + c),
                                                 (float)__ldg(a.Y[0] + c), 0.0f) : __ldg(a.Yin[1] + c);
    // ---- turbulence production (RHS_Atm_Turb.cpp:528-561) ----
    float prod;
    {
        const float dudr_s = d1r(U, a) * exp_rm, dvdr_s = d1r(V, a) * exp_rm, dwdr_s = d1r(W, a) * exp_rm;
        const float dudthe_s = d1t(U, a) * inv_rm, dvdthe_s = d1t(V, a) * inv_rm, dwdthe_s = d1t(W, a) * inv_rm;
        const float dudphi_s = d1p(U, a) * inv_rmsinthe, dvdphi_s = d1p(V, a) * inv_rmsinthe,
                    dwdphi_s = d1p(W, a) * inv_rmsinthe;
        const float tke_ijk = y1.x, dis_ijk = y1.y;
        const float dis_here = fmaxs(dis_ijk, 1.0e-10f);
        const float tke_here = fmaxs(tke_ijk, 0.0f);
        float cnue = (a.turb_model == ATHAD_TURB_K_EPSILON) ? 0.028f * tke_here * tke_here / dis_here
                                                           : tke_here / dis_here;
        cnue = fmins(cnue, a.nue_max);
        const float der = 0.66667f * (dudr_s + dvdthe_s + dwdphi_s);
        prod = fmaxs(0.0f,
              (cnue * (2.0f * dudr_s - der) - 0.66667f * tke_ijk) * dudr_s
            + (cnue * (dudthe_s + dvdr_s)) * dudthe_s
            + (cnue * (dudphi_s + dwdr_s)) * dudphi_s
            + (cnue * (2.0f * dvdthe_s - der) - 0.66667f * tke_ijk) * dvdthe_s
            + (cnue * (dvdr_s + dudthe_s)) * dvdr_s
            + (cnue * (dvdphi_s + dwdthe_s)) * dvdphi_s
            + (cnue * (2.0f * dwdphi_s - der) - 0.66667f * tke_ijk) * dwdphi_s
            + (cnue * (dwdr_s + dudphi_s)) * dwdr_s
            + (cnue * (dwdthe_s + dvdphi_s)) * dwdthe_s);
    }

    // ---- momentum (RHS_Atm_Turb.cpp:816-828, 870-884, 1001-1057, 1077-1079) ----
    float pressure_t;
    {
        const float exp_2_rm = G->exp_2_rm, inv_rm2 = G->inv_rm2, inv_rm2sinthe2 = G->inv_rm2sinthe2;
        const float inv_rm2sinthe = G->inv_rm2sinthe;
        const float cos_rm2sin = G->costhe_inv_rm2sinthe, two_over_rm_exp = G->two_over_rm_exp;
        const float sinthe = G->sinthe, costhe = G->costhe, v_metric = G->v_metric;
        const float dpdr = (P.ip - P.im) * a.inv_2dr;
        const float dpdthe = (P.jp - P.jm) * a.inv_2dthe;
        const float dpdphi = (P.kp - P.km) * a.inv_2dphi;
        const float dpdr_exp = dpdr * exp_rm, dpdthe_invrm = dpdthe * inv_rm, dpdphi_invrs = dpdphi * inv_rmsinthe;
        const float nontrad = a.nontrad ? 1.0f : 0.0f;
        const float cotanthe = a.curvature ? costhe / sinthe : 0.0f;
        float drag_profile = 1.0f - (float)i / 5.0f;
        if (drag_profile < 0.0f) drag_profile = 0.0f;
        const float surf_drag = a.drag_pref * drag_profile;
        float dudthe, dudphi, dvdphi;
        float k0[4];
        k0[3] = 0.0f;
        // stages 1 and 4 form MC_v's source from the FP64 field, 2 and 3 read stage 1's
        const float mcv = (STAGE == 1 || STAGE == 4) ? (float)(a.coeff_MC_vel * __ldg(a.MC_v + c)) : yn0.w;
        {   // u
            dudthe = d1t(U, a);
            dudphi = d1p(U, a);
            float tr_u = u_exp * ar(U, a) + v_invrm * at(U, a) + w_invrs * ap(U, a);
            if (a.curvature) tr_u += -(v_ijk * v_ijk + w_ijk * w_ijk) * inv_rm;
            const float diffusion_u = (d2r(U, a) * exp_2_rm + 2.0f * u_ijk * inv_rm2
                + d2t(U, a) * inv_rm2 + 4.0f * d1r(U, a) * inv_rm * exp_rm
                + dudthe * cos_rm2sin + d2p(U, a) * inv_rm2sinthe2) * diffusion_vel_re;
            const float t_ijk = y1.z;
            const float coriolis_rad = nontrad * 2.0f * sinthe * w_ijk;
            const float rhs_u = -dpdr_exp - tr_u + diffusion_u
                + buoy_pref * (t_ijk - (float)__ldg(a.t_ref + i))
                + a.force_nd * coriolis_rad;
            k0[0] = rhs_u;
            if (STAGE == 4) a.aux_u[c] = (double)rhs_u + (double)dpdr_exp;
        }
        {   // v
            dvdphi = d1p(V, a);
            float tr_v = u_exp * ar(V, a) + v_invrm * at(V, a) + w_invrs * ap(V, a);
            if (a.curvature) tr_v += (u_ijk * v_ijk - w_ijk * w_ijk * cotanthe) * inv_rm;
            const float part_v = d2r(V, a) * exp_2_rm + d1r(V, a) * two_over_rm_exp
                + d2t(V, a) * inv_rm2 + d1t(V, a) * cos_rm2sin
                - v_metric * v_ijk + d2p(V, a) * inv_rm2sinthe2
                + 2.0f * dudthe * inv_rm2;
            const float dwdphi = (W.kp - W.km) * a.inv_2dphi;
            const float diffusion_v = (part_v - dwdphi * 2.0f * costhe * inv_rm2sinthe2) * diffusion_vel_re;
            const float coriolis_the = 2.0f * costhe * w_ijk;
            const float rhs_v = -dpdthe_invrm - tr_v + diffusion_v
                + a.force_nd * coriolis_the + mcv - surf_drag * v_ijk;
            k0[1] = rhs_v;
            if (STAGE == 4) a.aux_v[c] = (double)rhs_v + (double)dpdthe_invrm;
        }
        {   // w
            float tr_w = u_exp * ar(W, a) + v_invrm * at(W, a) + w_invrs * ap(W, a);
            if (a.curvature) tr_w += (w_ijk * u_ijk + v_ijk * w_ijk * cotanthe) * inv_rm;
            const float diffusion_w = (d2r(W, a) * exp_2_rm + d1r(W, a) * two_over_rm_exp
                + d2t(W, a) * inv_rm2 + d1t(W, a) * cos_rm2sin
                - v_metric * w_ijk + d2p(W, a) * inv_rm2sinthe2
                + 2.0f * dudphi * inv_rm2sinthe
                + dvdphi * 2.0f * costhe * inv_rm2sinthe2) * diffusion_vel_re;
            const float coriolis_phi = -2.0f * (costhe * v_ijk + nontrad * sinthe * u_ijk);
            if (STAGE == 1) F0.x = (float)(a.coeff_MC_vel * __ldg(a.MC_w + c));
            const float mcw = F0.x;
            const float rhs_w = -dpdphi_invrs - tr_w + diffusion_w
                + a.force_nd * coriolis_phi + mcw - surf_drag * w_ijk;
            k0[2] = rhs_w;
            if (STAGE == 4) a.aux_w[c] = (double)rhs_w + (double)dpdphi_invrs;
        }
        update_group<STAGE, 0>(a, c, k0, acc0, yn0, P.c, nue_ijk, mcv);
        pressure_t = a.coeff_energy_p * (u_exp * dpdr + v_invrm * dpdthe + w_invrs * dpdphi);
    }

    const Group g1 = load_group<STAGE, 1>(a, c, sI, sJ);
    const StarF &TK = g1.s[0], &DI = g1.s[1], &T = g1.s[2];
    float k1[4];
    // ---- tke and omega/epsilon (RHS_Atm_Turb.cpp:563-721, 835-836, 936-942, 1074-1075) ----
    {
        const float exp_2_rm = G->exp_2_rm, inv_rm2 = G->inv_rm2, inv_rm2sinthe2 = G->inv_rm2sinthe2;
        const float cos_rm2sin = G->costhe_inv_rm2sinthe, two_over_rm_exp = G->two_over_rm_exp;
        const float tke_ijk = TK.c, dis_ijk = DI.c;
        const float dtkedr = d1r(TK, a), dtkedthe = d1t(TK, a), dtkedphi = d1p(TK, a);
        const float ddisdr = d1r(DI, a), ddisdthe = d1t(DI, a), ddisdphi = d1p(DI, a);
        const float tke_s = fmaxs(tke_ijk, 1.0e-10f), dis_s = fmaxs(dis_ijk, 1.0e-10f);
        const float dis_src_max = 20.0f * dis_s * dis_s, tke_src_max = 20.0f * tke_s * dis_s;
        const float cross = dtkedr * ddisdr + dtkedthe * inv_rm * ddisdthe * inv_rm
                          + dtkedphi * inv_rmsinthe * ddisdphi * inv_rmsinthe;
        float diffusion_tke_re, diffusion_dis_re, tke_source, dis_source;
        if (a.turb_model == ATHAD_TURB_K_EPSILON) {
            diffusion_tke_re = a.inv_re + nue_ijk / 1.0f;
            diffusion_dis_re = a.inv_re + nue_ijk / 1.3f;
            const float P_k = prod, Y_k = dis_s;
            const float P_w = 1.35f * (dis_s / tke_s) * P_k;
            const float Y_w = 1.80f * dis_s * dis_s / tke_s;
            tke_source = fclamps(P_k - Y_k, -tke_src_max, tke_src_max);
            dis_source = fclamps(P_w - Y_w, -dis_src_max, dis_src_max);
        } else if (a.turb_model == ATHAD_TURB_K_OMEGA) {
            diffusion_tke_re = a.inv_re + 0.6f * nue_ijk;
            diffusion_dis_re = a.inv_re + 0.5f * nue_ijk;
            const float P_k = fmins(prod, 20.0f * 0.09f * tke_s * dis_s);
            const float Y_k = 0.09f * tke_s * dis_s;
            const float P_w = 0.52f * (dis_s / tke_s) * P_k;
            const float Y_w = 0.0708f * dis_s * dis_s;
            const float sig_d = (cross <= 0.0f) ? 0.0f : 0.125f;
            const float D_w = sig_d * cross / dis_s;
            tke_source = fclamps(P_k - Y_k, -tke_src_max, tke_src_max);
            dis_source = fclamps(P_w - Y_w + D_w, -dis_src_max, dis_src_max);
        } else {   // k-omega SST; wall distance as the FP64 kernel
            const float bet_star = 0.09f, sig_w2 = 1.168f;
            float d_j = (float)j;
            if (a.wall_mode == ATHAD_WALL_MIRROR) { const int jr = d.jm - 1 - j; if (jr < j) d_j = (float)jr; }
            float d_close = (float)i;
            if (d_j <= d_close) d_close = d_j;
            if ((float)k <= d_close) d_close = (float)k;
            const float CD_kw = fmaxs((2.0f * sig_w2) / dis_ijk * cross, 1.0e-20f);
            const float arg1 = fmins(fmaxs(
                sqrtf(tke_ijk) / (bet_star * dis_ijk * d_close),
                (500.0f * a.nue_air_nd) / (d_close * d_close * dis_ijk)),
                (4.0f * sig_w2 * tke_ijk) / (CD_kw * d_close * d_close));
            const float a2 = arg1 * arg1;
            const float F1 = tanhf(a2 * a2);
            const float bk = F1 * 1.176f + (1.0f - F1) * 1.0f;
            const float bw = F1 * 2.0f + (1.0f - F1) * sig_w2;
            diffusion_tke_re = a.inv_re + nue_ijk / bk;
            diffusion_dis_re = a.inv_re + nue_ijk / bw;
            const float P_k = fmins(prod, 20.0f * bet_star * tke_s * dis_s);
            const float Y_k = bet_star * tke_s * dis_s;
            const float P_w = (F1 * 0.413f + (1.0f - F1) * 0.2f) * P_k * dis_s / tke_s;
            const float Y_w = (F1 * 0.0333f + (1.0f - F1) * 0.0368f) * dis_s * dis_s;
            const float D_w = 2.0f * (1.0f - F1) * sig_w2 / dis_s * cross;
            tke_source = fclamps(P_k - Y_k, -tke_src_max, tke_src_max);
            dis_source = fclamps(P_w - Y_w + D_w, -dis_src_max, dis_src_max);
        }
        diffusion_tke_re *= a.diffusion_ramp;
        diffusion_dis_re *= a.diffusion_ramp;
        const float tr_tke = u_exp * dtkedr + v_invrm * dtkedthe + w_invrs * dtkedphi;
        const float tr_dis = u_exp * ddisdr + v_invrm * ddisdthe + w_invrs * ddisdphi;
        const float diffusion_tke = (d2r(TK, a) * exp_2_rm + dtkedr * two_over_rm_exp
            + d2t(TK, a) * inv_rm2 + dtkedthe * cos_rm2sin + d2p(TK, a) * inv_rm2sinthe2) * diffusion_tke_re;
        const float diffusion_dis = (d2r(DI, a) * exp_2_rm + ddisdr * two_over_rm_exp
            + d2t(DI, a) * inv_rm2 + ddisdthe * cos_rm2sin + d2p(DI, a) * inv_rm2sinthe2) * diffusion_dis_re;
        k1[0] = -tr_tke + diffusion_tke + tke_source;
        k1[1] = -tr_dis + diffusion_dis + dis_source;
        if (STAGE == 4 && a.write_diag) {
            a.prod[c] = prod;
            a.tke_source[c] = tke_source;
            a.dis_source[c] = dis_source;
        }
    }

    {
        const float exp_2_rm = G->exp_2_rm, inv_rm2 = G->inv_rm2, inv_rm2sinthe2 = G->inv_rm2sinthe2;
        const float cos_rm2sin = G->costhe_inv_rm2sinthe, two_over_rm_exp = G->two_over_rm_exp;
        // ---- temperature (RHS_Atm_Turb.cpp:752, 829, 866-868, 963-992) ----
        {
            const float t_ijk = T.c;
            const float tr_t = u_exp * ar(T, a) + v_invrm * at(T, a) + w_invrs * ap(T, a);
            const float diffusion_t_re = (a.inv_re + nue_ijk) * a.inv_pr_turb * a.diffusion_ramp;
            const float diffusion_t = (d2r(T, a) * exp_2_rm + d1r(T, a) * two_over_rm_exp
                + d2t(T, a) * inv_rm2 + d1t(T, a) * cos_rm2sin + d2p(T, a) * inv_rm2sinthe2) * diffusion_t_re;
            if (STAGE == 1) {
                const double r_h = __ldg(a.r_humid + c);
                const double q_t = a.coeff_MC_t * __ldg(a.MC_t + c)
                    + a.coeff_energy * (__ldg(a.S_c + c) + __ldg(a.S_r + c)) * a.lv * r_h
                    + a.coeff_energy * (__ldg(a.S_i + c) + __ldg(a.S_s + c) + __ldg(a.S_g + c)) * a.ls * r_h;
                const double k_a = 1.0 / (4.0 * 86400.0), k_s = 1.0 / (0.4 * 86400.0), sigma_b = 0.7;
                const double p_surf = __ldg(a.p_stat + idx3(d, 0, j, k));
                const double sigma = (p_surf > 0.0) ? __ldg(a.p_stat + c) / p_surf : 0.0;
                double bl = (sigma - sigma_b) / (1.0 - sigma_b);
                if (bl < 0.0) bl = 0.0;
                F0.y = (float)q_t;
                F0.z = (float)((k_a + (k_s - k_a) * bl * (double)G->cos4lat) * a.L_atm_over_u0);
                F0.w = (float)__ldg(a.t_eq + c);
                a.F[0][c] = F0;
            }
            const float qt = F0.y, kTf = F0.z, teqf = F0.w;
            k1[2] = pressure_t - tr_t + diffusion_t + qt - kTf * (t_ijk - teqf);
        }
    }
    // ---- moisture and tracers (RHS_Atm_Turb.cpp:830-834, 911-934, 1059-1072) ----
    {
        const float exp_2_rm = G->exp_2_rm, inv_rm2 = G->inv_rm2, inv_rm2sinthe2 = G->inv_rm2sinthe2;
        const float cos_rm2sin = G->costhe_inv_rm2sinthe, two_over_rm_exp = G->two_over_rm_exp;
        const float dlnrho_dr_i = a.tracer_diff_flux ? (float)__ldg(a.dlnrho + i) * exp_2_rm : 0.0f;
        float F1[4];   // the sources of c, cloud, ice, gr
        if (STAGE == 1) {
            const double r_h = __ldg(a.r_humid + c);
            F1[0] = (float)(__ldg(a.S_v + c) * r_h + a.coeff_MC_q * __ldg(a.MC_q + c));
            F1[1] = (float)(__ldg(a.S_c + c) * r_h);
            F1[2] = (float)(__ldg(a.S_i + c) * r_h);
            F1[3] = (float)(__ldg(a.S_g + c) * r_h);
            a.F[1][c] = make_float4(F1[0], F1[1], F1[2], F1[3]);
        } else {
            const float4 f = __ldg(a.F[1] + c);
            F1[0] = f.x; F1[1] = f.y; F1[2] = f.z; F1[3] = f.w;
        }
        auto tracer = [&](int n, const StarF& Q, float src) {
            const float coef = (n == 8) ? a.diff_co2_re_inv : a.diff_prec_re_inv;
            const float tr = (n <= 6) ? (u_exp * ar(Q, a) + v_invrm * at(Q, a) + w_invrs * ap(Q, a))
                                      : (u_exp * d1r(Q, a) + v_invrm * d1t(Q, a) + w_invrs * d1p(Q, a));
            const float q1r = d1r(Q, a);
            const float dif = (d2r(Q, a) * exp_2_rm + q1r * two_over_rm_exp
                + d2t(Q, a) * inv_rm2 + d1t(Q, a) * cos_rm2sin
                + d2p(Q, a) * inv_rm2sinthe2
                + q1r * dlnrho_dr_i) * coef;
            return -tr + dif + src;
        };
        k1[3] = tracer(4, g1.s[3], F1[0]);
        const float4 acc1 = (STAGE == 1) ? zero4 : a.K[1][c];
        const float4 yn1 = (STAGE == 2 || STAGE == 3) ? __ldg(a.Yn32[1] + c) : zero4;
        update_group<STAGE, 1>(a, c, k1, acc1, yn1, 0.0f, 0.0f, 0.0f);
        const Group g2 = load_group<STAGE, 2>(a, c, sI, sJ);
        const float4 acc2 = (STAGE == 1) ? zero4 : a.K[2][c];
        const float4 yn2 = (STAGE == 2 || STAGE == 3) ? __ldg(a.Yn32[2] + c) : zero4;
        const float k2[4] = {tracer(5, g2.s[0], F1[1]), tracer(6, g2.s[1], F1[2]), tracer(7, g2.s[2], F1[3]),
                             tracer(8, g2.s[3], 0.0f)};
        update_group<STAGE, 2>(a, c, k2, acc2, yn2, 0.0f, 0.0f, 0.0f);
    }
}

// CTAs of 128 threads per SM that the registers are sized for: stage 1 (FP64 stars, most
// values live) 5 (96 registers), 2 and 3 7 (72), 4 6 (80).  One group's stars are 28
// registers, so few values spill at any of these.  41x181x361 / 27x117x245 per step with
// (S1, S2-3, S4): (5,7,6) 785 / 248 us, (5,8,6) 781 / 250, (4,7,6) 801 / 252, (5,7,7)
// 791 / 249, (6,7,7) 805 / 255, (7,7,7) 810 / 258, (7,9,7) 834 / 274, (7,7,9) 852 / 272.
#ifndef ATHAD_RK4M_MIN_BLOCKS
#define ATHAD_RK4M_MIN_BLOCKS 7
#endif
#ifndef ATHAD_RK4M_MIN_BLOCKS_S1
#define ATHAD_RK4M_MIN_BLOCKS_S1 5
#endif
#ifndef ATHAD_RK4M_MIN_BLOCKS_S4
#define ATHAD_RK4M_MIN_BLOCKS_S4 6
#endif

// MEMBER: a batch's member on a lane of its own; its buoyancy prefactor changes from
// iteration to iteration of a captured graph, so it is read from the member's step record.
// BX longitudes x BY rows of one level per CTA: 128 x 1 for a single grid (41x181x361: 785 us,
// 64 x 2 804, 32 x 4 832, 32 x 8 901).
template <int STAGE, int BX, int BY, bool MEMBER>
__global__ void __launch_bounds__(BX * BY,
    (STAGE == 1 ? ATHAD_RK4M_MIN_BLOCKS_S1 : STAGE == 4 ? ATHAD_RK4M_MIN_BLOCKS_S4 : ATHAD_RK4M_MIN_BLOCKS) * 128 / (BX * BY))
rk4m_stage_kernel(const RK4MArgs a, const BatchStep* step)
{
    pdl_trigger();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    // the even stages walk the radial planes from the top down, so that each stage starts
    // on the planes its predecessor wrote last (1.036 -> 1.030 ms per step at 41x181x361;
    // a stage's cells are independent, so the order changes no result)
#if ATHAD_RK4_SERPENTINE
    int i = (STAGE % 2 == 0) ? a.d.im - 1 - (int)blockIdx.z : (int)blockIdx.z;
#else
    int i = blockIdx.z;
#endif
    pdl_wait(k, i);   // i alone addresses t_ref, which the launch before stage 1 writes
    prefetch_tile<STAGE>(a, i, blockIdx.y * BY, blockIdx.x * BX, BX, BY, threadIdx.y * BX + threadIdx.x, BX * BY);
    if (k >= a.d.km || j >= a.d.jm) return;
    rk4m_cell<STAGE>(a, i, j, k, MEMBER ? step->buoy_pref : a.buoy_pref);
}

template <int BX, int BY, bool MEMBER>
static void launch_stage(int stage, const RK4MArgs& a, const BatchStep* step, cudaStream_t st)
{
    const dim3 block(BX, BY, 1);
    const dim3 grid((a.d.km + BX - 1) / BX, (a.d.jm + BY - 1) / BY, a.d.im);
    switch (stage) {
        case 1: launch_dependent(rk4m_stage_kernel<1, BX, BY, MEMBER>, grid, block, 0, st, a, step); break;
        case 2: launch_dependent(rk4m_stage_kernel<2, BX, BY, MEMBER>, grid, block, 0, st, a, step); break;
        case 3: launch_dependent(rk4m_stage_kernel<3, BX, BY, MEMBER>, grid, block, 0, st, a, step); break;
        default: launch_dependent(rk4m_stage_kernel<4, BX, BY, MEMBER>, grid, block, 0, st, a, step); break;
    }
}

void launch_rk4m_stage(int stage, const RK4MArgs& a, cudaStream_t st)
{
    launch_stage<128, 1, false>(stage, a, nullptr, st);
}

// The tile shapes a batch's autotuner chooses from.
int batch_shape_count() { return 6; }

void launch_rk4m_member_stage(int stage, int shape, const RK4MArgs& a, const BatchStep* step, cudaStream_t st)
{
    switch (shape) {
        case 0: launch_stage<128, 1, true>(stage, a, step, st); break;
        case 1: launch_stage<64, 2, true>(stage, a, step, st); break;
        case 2: launch_stage<32, 4, true>(stage, a, step, st); break;
        case 3: launch_stage<32, 8, true>(stage, a, step, st); break;
        case 4: launch_stage<64, 4, true>(stage, a, step, st); break;
        default: launch_stage<128, 2, true>(stage, a, step, st); break;
    }
}

}  // namespace athad
