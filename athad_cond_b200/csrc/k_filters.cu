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
// its row in shared memory and iterates its passes there, four at a time; along i a thread
// walks its column with the values that the two passes still need in registers.  Compiled without fused
// multiply-add: bit-identical to the reference.
#include "kernels.cuh"

namespace athad {

namespace {

// P periodic 1-2-1 passes along a row: from src to dst, three consecutive longitudes a thread.
// The values that the passes need on either side are formed again in registers, so P passes
// cost P + 1.5 reads of shared memory per value and one barrier instead of 3 P and P.
template <int P>
__device__ __forceinline__ void zonal_passes(const double* src, double* dst, int km)
{
    for (int k0 = 3 * threadIdx.x; k0 < km; k0 += 3 * blockDim.x) {
        double v[3 + 2 * P];
        const bool inside = k0 >= P && k0 + 2 + P < km;
#pragma unroll
        for (int m = 0; m < 3 + 2 * P; m++) {
            int k = k0 - P + m;
            if (!inside) {
                if (k < 0) k += km;
                if (k >= km) k -= km;
                if (k >= km) k -= km;   // the two values past the row's end on the shortest rows
            }
            v[m] = src[k];
        }
#pragma unroll
        for (int p = 0; p < P; p++)
#pragma unroll
            for (int m = 0; m < 1 + 2 * (P - p); m++) v[m] = v[m + 1] + 0.25 * (v[m] - 2.0 * v[m + 1] + v[m + 2]);
#pragma unroll
        for (int m = 0; m < 3; m++)
            if (k0 + m < km) dst[k0 + m] = v[m];
    }
}

// periodic 1-2-1 passes along k of one row per CTA; passes[j] of them (zero: untouched), up to
// four between barriers.  A pass at a time read three values of shared memory per value and was
// bound by that.
__global__ void __launch_bounds__(128) zonal_rows_kernel(FilterArgs a, int nfields)
{
    extern __shared__ double row[];          // two buffers of km
    const Dims& d = a.d;
    const int j = blockIdx.x, i = blockIdx.y, q = blockIdx.z;
    if (q >= nfields) return;
    int np = a.polar_passes[j];
    if (np == 0) return;
    double* x = a.field[q] + idx3(d, i, j, 0);
    double* b0 = row;
    double* b1 = row + d.km;
    for (int k = threadIdx.x; k < d.km; k += blockDim.x) b0[k] = x[k];
    __syncthreads();
    for (; np > 4; np -= 4) {
        zonal_passes<4>(b0, b1, d.km);
        __syncthreads();
        double* t = b0; b0 = b1; b1 = t;
    }
    switch (np) {
        case 1: zonal_passes<1>(b0, x, d.km); break;
        case 2: zonal_passes<2>(b0, x, d.km); break;
        case 3: zonal_passes<3>(b0, x, d.km); break;
        default: zonal_passes<4>(b0, x, d.km); break;
    }
}

// one pass of a column at level i from the values of i-2 .. i+2 before it; levels 0 and im-1
// stay: 1-2-1 for the field u, the 4th-order Shapiro filter for v and w where i+-2 is inside
__device__ __forceinline__ double radial_pass(const double (&o)[5], int i, int im, bool fourth)
{
    if (i < 1 || i > im - 2) return o[2];
    if (fourth && i >= 2 && i + 2 <= im - 1)
        return o[2] - 0.0625 * (o[4] - 4.0 * o[3] + 6.0 * o[2] - 4.0 * o[1] + o[0]);
    return o[2] + 0.25 * (o[1] - 2.0 * o[2] + o[3]);
}

// Both passes along i of one column per thread, in one walk: the second pass follows the first
// two levels behind, four levels are loaded ahead, and a level is stored when the walk has read
// all that it feeds.  A walk per pass with one load a step waited for memory.  Both kernels, u, v
// and w at 41x181x361: 95 -> 79 us.
__global__ void __launch_bounds__(128) radial_columns_kernel(FilterArgs a)
{
    const Dims& d = a.d;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, q = blockIdx.z;
    if (k >= d.km) return;
    double* x = a.field[q] + idx3(d, 0, j, k);
    const long long s = d.plane;
    const int im = d.im;
    const bool fourth = q != 0;
    constexpr int kAhead = 4;
    double o[5] = {}, y[5] = {}, nx[kAhead];
#pragma unroll
    for (int m = 0; m < kAhead; m++) nx[m] = (m < im) ? x[m * s] : 0.0;
    for (int t0 = 0; t0 < im + 3; t0 += kAhead) {
        double cur[kAhead];
#pragma unroll
        for (int m = 0; m < kAhead; m++) {
            cur[m] = nx[m];
            nx[m] = (t0 + kAhead + m < im) ? x[(t0 + kAhead + m) * s] : 0.0;
        }
#pragma unroll
        for (int m = 0; m < kAhead; m++) {
            const int t = t0 + m;      // o: levels t-4 .. t; y: the first pass's t-6 .. t-2
            o[0] = o[1]; o[1] = o[2]; o[2] = o[3]; o[3] = o[4]; o[4] = cur[m];
            y[0] = y[1]; y[1] = y[2]; y[2] = y[3]; y[3] = y[4]; y[4] = radial_pass(o, t - 2, im, fourth);
            const int i = t - 4;
            if (i >= 1 && i <= im - 2) x[i * s] = radial_pass(y, i, im, fourth);
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
// Rows (levels) per thread: on a small grid a walk is the launch's length.  One field with 2, 4
// and 8: 11x21x41 5.8, 6.7 and 9.7 us (8.1 with the passes as separate cells), 21x91x181 6.3, 7.4
// and 10.6, 41x181x361 20.9, 16.7 and 18.6; eleven fields of 27x99x151 36.9, 27.5 and 26.5, of
// 41x181x361 215, 178 and 176.
constexpr int kWalk = 4;

// the zonal pass (periodic) of the longitudes k, k + 1 of one row; k is even, and the second
// value is not used where k + 1 = km
__device__ __forceinline__ double2 zonal_two(const double* __restrict__ row, int k, int km)
{
    const double2 x = *reinterpret_cast<const double2*>(row + k);
    const double west = row[k == 0 ? km - 1 : k - 1];
    const double east = (k + 1 >= km) ? 0.0 : row[k + 2 >= km ? 0 : k + 2];
    const double e0 = (k + 1 >= km) ? row[k + 1 - km] : x.y;   // row[0], addressed from k (pdl_wait)
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
