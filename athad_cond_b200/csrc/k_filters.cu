// k_filters.cu - the smoothing filters of the model iteration on sm_100a, flat terrain
// (every cell is fluid; the orographic, steep-massif and coastal filters flag nothing):
//
//   athad_post_rk4_filters (cAtmosphereModel.cpp:1507-1520)
//     AtomUtils::polar_zonal_filter of u, v, w (lib/Utils.cpp:542-611): per row j a
//       number of periodic 1-2-1 passes along k that grows toward the poles;
//     AtomUtils::radial_shapiro_filter of u (:831-873): two 1-2-1 passes along i;
//     AtomUtils::radial_shapiro_filter_ho of v, w (:884-940): two 4th-order passes along
//       i, the 1-2-1 where i+-2 is outside the column;
//   athad_damp_wiggles (:429-531): one 1-2-1 pass along k (periodic), j (clamped) and i
//     (clamped), the moist iteration's de-checkerboarding of t, ice, c, cloud
//     (cAtmosphereModel.cpp:1225-1228).
//
// Every pass of the reference works from a snapshot of the field.  Along k a CTA holds
// its row in shared memory and iterates its passes there; along i a thread walks its
// column with the snapshot values it still needs in registers.  Compiled without fused
// multiply-add: bit-identical to the reference.
#include "kernels.cuh"

namespace athad {

namespace {

// periodic 1-2-1 passes along k of one row per CTA; passes[j] of them (zero: untouched)
__global__ void __launch_bounds__(128) zonal_rows_kernel(FilterArgs a, int nfields)
{
    extern __shared__ double row[];          // two buffers of km
    const Dims& d = a.d;
    const int j = blockIdx.x, i = blockIdx.y, q = blockIdx.z;
    if (q >= nfields) return;
    const int np = a.polar_passes[j];
    if (np == 0) return;
    double* x = a.field[q] + idx3(d, i, j, 0);
    double* b0 = row;
    double* b1 = row + d.km;
    for (int k = threadIdx.x; k < d.km; k += blockDim.x) b0[k] = x[k];
    __syncthreads();
    for (int pass = 0; pass < np; pass++) {
        for (int k = threadIdx.x; k < d.km; k += blockDim.x) {
            const int km1 = (k == 0) ? d.km - 1 : k - 1;
            const int kp1 = (k == d.km - 1) ? 0 : k + 1;
            b1[k] = b0[k] + 0.25 * (b0[km1] - 2.0 * b0[k] + b0[kp1]);
        }
        __syncthreads();
        double* t = b0; b0 = b1; b1 = t;
    }
    for (int k = threadIdx.x; k < d.km; k += blockDim.x) x[k] = b0[k];
}

// two passes along i of one column per thread: field 0 (u) 1-2-1, fields 1-2 (v, w) the
// 4th-order Shapiro filter; rows 0 and im-1 untouched
__global__ void __launch_bounds__(128) radial_columns_kernel(FilterArgs a)
{
    const Dims& d = a.d;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, q = blockIdx.z;
    if (k >= d.km) return;
    double* x = a.field[q] + idx3(d, 0, j, k);
    const long long s = d.plane;
    const int im = d.im;
    for (int pass = 0; pass < 2; pass++) {
        // snapshot window o[i-2 .. i+2] of the values before this pass
        double om2 = 0.0, om1 = x[0], o0 = x[s], op1 = (im > 2) ? x[2 * s] : 0.0;
        for (int i = 1; i < im - 1; i++) {
            const double op2 = (i + 2 <= im - 1) ? x[(i + 2) * s] : 0.0;
            double v;
            if (q != 0 && i - 2 >= 0 && i + 2 <= im - 1) {
                const double d4 = op2 - 4.0 * op1 + 6.0 * o0 - 4.0 * om1 + om2;
                v = o0 - 0.0625 * d4;
            } else {
                v = o0 + 0.25 * (om1 - 2.0 * o0 + op1);
            }
            x[i * s] = v;
            om2 = om1; om1 = o0; o0 = op1; op1 = op2;
        }
    }
}

// damp_wiggles in two launches.  The first forms the zonal and the meridional pass into the
// scratch field, the second the radial one back into the field (a pass reads its neighbours
// before the pass, so neither can run in place); a thread takes two longitudes and walks
// kWalk rows (levels), keeping the three values that the pass combines, so each value is
// loaded about once: 14 + 9 us per field at 41x181x361.  A CTA per row for the zonal pass and
// one cell per thread for the other two (nine loads each) took 22 + 17.
// The meridional pass adds the two neighbours first, so the result at row jm-1-j is bit for
// bit the result at row j of the mirrored field; the reference's left-to-right
// (v[j-1] - 2 v[j]) + v[j+1] rounds the mirrored rows differently (an ulp at most).
// The fields of one launch lie side by side in its grid: a field alone ends each launch with
// SMs that wait for the last CTAs, and a small one does not fill the GPU.  The 23 fields of a
// moist iteration, one at a time and up to eleven: 21x91x181 262 and 73 us, 41x181x361 483
// and 396, 61x181x361 607 and 575.  Limiting a launch to what the L2 holds with its scratch
// is no better (41x181x361, four fields: 417).
constexpr int kWalk = 8;

// the zonal pass (periodic) of the longitudes k, k + 1 of one row; k is even, and the second
// value is not used where k + 1 = km
__device__ __forceinline__ double2 zonal_two(const double* __restrict__ row, int k, int km)
{
    const double2 x = *reinterpret_cast<const double2*>(row + k);
    const double west = row[k == 0 ? km - 1 : k - 1];
    const double east = (k + 1 >= km) ? 0.0 : row[k + 2 >= km ? 0 : k + 2];
    const double e0 = (k + 1 >= km) ? row[0] : x.y;
    return make_double2(x.x + 0.25 * (west - 2.0 * x.x + e0), x.y + 0.25 * (x.x - 2.0 * x.y + east));
}

__global__ void __launch_bounds__(128) wiggle_kj_kernel(Dims d, const WiggleFields w)
{
    pdl_trigger();
    int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    pdl_wait(k);
    const int q = blockIdx.z / d.im, i = blockIdx.z - q * d.im;
    const int j0 = blockIdx.y * kWalk;
    if (k >= d.km) return;
    const double* __restrict__ src = w.f[q];
    double* __restrict__ dst = w.scratch[q];
    const int jn = min(j0 + kWalk, d.jm);
    const double* plane = src + idx3(d, i, 0, 0);
    double2 c = zonal_two(plane + (long long)j0 * d.pitch, k, d.km);
    double2 m = (j0 > 0) ? zonal_two(plane + (long long)(j0 - 1) * d.pitch, k, d.km) : c;
#pragma unroll 4
    for (int j = j0; j < jn; j++) {
        const double2 p = (j < d.jm - 1) ? zonal_two(plane + (long long)(j + 1) * d.pitch, k, d.km) : c;
        *reinterpret_cast<double2*>(dst + idx3(d, i, j, k)) =
            make_double2(c.x + 0.25 * ((m.x + p.x) - 2.0 * c.x), c.y + 0.25 * ((m.y + p.y) - 2.0 * c.y));
        m = c; c = p;
    }
}

__global__ void __launch_bounds__(128) wiggle_i_kernel(Dims d, const WiggleFields w)
{
    pdl_trigger();
    int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    pdl_wait(k);
    const int nz = (d.im + kWalk - 1) / kWalk;
    const int q = blockIdx.z / nz, i0 = (blockIdx.z - q * nz) * kWalk;
    const int j = blockIdx.y;
    if (k >= d.km) return;
    const double* __restrict__ src = w.scratch[q];
    double* __restrict__ dst = w.f[q];
    const int in = min(i0 + kWalk, d.im);
    auto two = [&](int i) { return *reinterpret_cast<const double2*>(src + idx3(d, i, j, k)); };
    double2 c = two(i0), m = (i0 > 0) ? two(i0 - 1) : c;
#pragma unroll 4
    for (int i = i0; i < in; i++) {
        const double2 p = (i < d.im - 1) ? two(i + 1) : c;
        const double2 v = make_double2(c.x + 0.25 * (m.x - 2.0 * c.x + p.x), c.y + 0.25 * (m.y - 2.0 * c.y + p.y));
        double* o = dst + idx3(d, i, j, k);
        if (k + 1 < d.km) *reinterpret_cast<double2*>(o) = v;
        else *o = v.x;
        m = c; c = p;
    }
}

}  // namespace

void launch_post_rk4_filters(const FilterArgs& a, cudaStream_t st)
{
    const Dims& d = a.d;
    zonal_rows_kernel<<<dim3(d.jm, d.im, 3), 128, 2 * d.km * sizeof(double), st>>>(a, 3);
    radial_columns_kernel<<<dim3((d.km + 127) / 128, d.jm, 3), 128, 0, st>>>(a);
}

void launch_damp_wiggles(const Dims& d, const WiggleFields& w, cudaStream_t st)
{
    const unsigned kx = ((d.km + 1) / 2 + 127) / 128;
    launch_dependent(wiggle_kj_kernel, dim3(kx, (d.jm + kWalk - 1) / kWalk, d.im * w.n), dim3(128), 0, st, d, w);
    launch_dependent(wiggle_i_kernel, dim3(kx, d.jm, (d.im + kWalk - 1) / kWalk * w.n), dim3(128), 0, st, d, w);
}

}  // namespace athad
