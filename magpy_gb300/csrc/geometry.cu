// geometry.cu -- seeded cluster geometry and initial conditions on the device.
//
// The reference builds cluster geometries on the host with numpy's global
// generator: easy axes uniform on the sphere (magpy/initial_conditions.py:4-37,
// uniform_random_axes), chains (magpy/geometry/coordinates.py,
// chain_coordinates) and hand-placed clusters.  For large batched ensembles
// with a different cluster per member this library draws them on the device
// from a counter-based generator (Philox-4x32-10 keyed by the member seed),
// so no host work scales with the ensemble:
//   * radii log-normal, r = median * exp(sigma z), z standard normal;
//   * easy axes uniform on the sphere (z uniform on [-1, 1], azimuth uniform),
//     the initial moments along the easy axes or independently uniform;
//   * locations: random packing in a sphere of radius R sized for a target
//     packing fraction phi of the exclusion spheres (R = r_x (N / phi)^(1/3),
//     r_x = spacing * mean(r) / 2), every pair at least spacing * (r_i + r_j) / 2
//     apart; or a straight chain along z with pitch spacing * mean(r).
// Packing: one CTA per member places particle i by drawing a batch of
// candidates (one per thread) and taking the lowest-numbered valid one, so
// the result depends only on the seed and not on the batch; a member that
// finds no valid candidate among max_rounds x 256 is reported and its
// remaining particles are left at NaN.
//
// What bounds it: an FP64 instruction takes 64 issue cycles of a
// sub-partition here, and a candidate is compared with every placed particle
// (9 FP64 operations a pair).  So a candidate's coordinates and distances are
// formed in FP32 in units of the sphere's radius, with a bound on their
// error that decides all but ~1e-5 of the comparisons; the rest, and the
// location of the candidate that is taken, are FP64, the same bits as with
// FP64 throughout.  Drawing 1000 clusters of 27, a call: 2.14 ms with 256 FP64
// candidates a batch, 0.19 ms with this search, at a packing of 20 %; 67 and 66 ms
// at 45 %, where a few members need thousands of batches (of 100: 990 and 342 ms).
#include <cmath>
#include "common.cuh"
#include "plan.hpp"

namespace magpy {

namespace {

constexpr int64_t GEO_ROUND = 256;  // candidates per round of max_rounds
constexpr int GEO_WIDE = 128;       // threads per member of a small ensemble
// FP32 comparisons are trusted outside GEO_ABS + GEO_REL * (squared exclusion
// distance), in units of R: a candidate's coordinate is off by at most
// 1.8e-7, a placed one by 6e-8, their difference by 3.6e-7, its square summed
// over the axes by 2 * 2 sqrt(3) * 3.6e-7 + 7e-7 = 3.2e-6; the exclusion
// distance squared by 4e-7 of itself.
constexpr float GEO_ABS = 8e-6f, GEO_REL = 2e-6f;
constexpr uint32_t TAG_RADIUS = 0x6e01u, TAG_AXIS = 0x6e02u, TAG_MOMENT = 0x6e03u,
                   TAG_PLACE = 0x6e04u;

// Uniform on (0, 1) from 53 bits of two words.
__device__ inline double u53(uint32_t hi, uint32_t lo)
{
    const uint64_t b = ((uint64_t)(hi >> 5) << 26) | (uint64_t)(lo >> 6);
    return ((double)b + 0.5) * 1.1102230246251565404e-16;  // 2^-53
}

__device__ inline U4 draw(uint64_t seed, uint32_t i, uint32_t j, uint32_t tag)
{
    return philox4x32_10(U4{i, j, tag, 0x9e01u}, (uint32_t)seed, (uint32_t)(seed >> 32));
}

__device__ inline void unit_vector(U4 r, double v[3])
{
    const double z = 2.0 * u53(r.x, r.y) - 1.0;
    const double ph = 6.283185307179586477 * u53(r.z, r.w);
    const double s = sqrt(fmax(0.0, 1.0 - z * z));
    v[0] = s * cos(ph);
    v[1] = s * sin(ph);
    v[2] = z;
}

// Coordinate of a candidate: uniform on (-R, R).
__device__ inline double cand_coord(double R, uint32_t hi, uint32_t lo)
{
    return R * (2.0 * u53(hi, lo) - 1.0);
}

// T: candidates per batch; a divisor of GEO_ROUND.
template <int T>
__global__ void __launch_bounds__(T)
    geometry_kernel(GeoArgs a)
{
    extern __shared__ __align__(16) double gsm[];
    const int n = a.n;
    float4 *near = (float4 *)gsm;            // [n] placed locations / R, exclusion radius / R
    double *pos = (double *)(near + n);      // [n][3] accepted locations
    double *rad = pos + 3 * n;               // [n] radii
    const int64_t e = blockIdx.x;
    const uint64_t seed = (uint64_t)a.seeds[e];
    const int tid = threadIdx.x;

    // radii, axes, moments: one particle per thread
    for (int i = tid; i < n; i += T) {
        const U4 r = draw(seed, (uint32_t)i, 0u, TAG_RADIUS);
        const double z = sqrt(-2.0 * log(u53(r.x, r.y))) * cos(6.283185307179586477 * u53(r.z, r.w));
        const double ri = a.median_radius * exp(a.sigma * z);
        rad[i] = ri;
        double ax[3], m[3];
        unit_vector(draw(seed, (uint32_t)i, 0u, TAG_AXIS), ax);
        if (a.moments_random) unit_vector(draw(seed, (uint32_t)i, 0u, TAG_MOMENT), m);
        else { m[0] = ax[0]; m[1] = ax[1]; m[2] = ax[2]; }
        const int64_t g = e * n + i;
        a.radius[g] = ri;
        for (int c = 0; c < 3; c++) {
            a.axes[3 * g + c] = ax[c];
            a.m0[3 * g + c] = m[c];
        }
    }
    __syncthreads();
    // mean radius (fixed order: the same bits on every launch)
    __shared__ double s_mean;
    if (tid == 0) {
        double s = 0.0;
        for (int i = 0; i < n; i++) s += rad[i];
        s_mean = s / n;
    }
    __syncthreads();
    const double mean_r = s_mean;
    if (a.layout == 1) {  // chain along z
        for (int i = tid; i < n; i += T) {
            const int64_t g = e * n + i;
            a.location[3 * g + 0] = 0.0;
            a.location[3 * g + 1] = 0.0;
            a.location[3 * g + 2] = a.spacing * mean_r * i;
        }
        if (tid == 0) a.status[e] = 0;
        return;
    }
    const double rx = 0.5 * a.spacing * mean_r;
    const double R = rx * cbrt((double)n / a.packing);
    // FP32 comparisons need a radius that FP64 can square and divide by
    const bool fast = R > 1e-100 && R < 1e100;
    const double inv_R = 1.0 / R;
    for (int i = tid; i < n; i += T)
        near[i] = make_float4(0.f, 0.f, 0.f, (float)(0.5 * a.spacing * rad[i] * inv_R));
    __syncthreads();
    __shared__ int s_pick;
    int32_t status = 0;
    int placed = 0;
    for (int i = 0; i < n && status == 0; i++) {
        bool done = false;
        const float ri = near[i].w;
        for (int64_t base = 0; base < a.max_rounds * GEO_ROUND && !done; base += T) {
            const U4 r = draw(seed, (uint32_t)i, (uint32_t)(base + tid), TAG_PLACE);
            const U4 r2 = draw(seed, (uint32_t)i, (uint32_t)(base + tid), TAG_PLACE + 1u);
            const float x = __fmaf_rn((float)r.x, 4.656612873077393e-10f, -1.f);  // 2 u - 1
            const float y = __fmaf_rn((float)r.z, 4.656612873077393e-10f, -1.f);
            const float z = __fmaf_rn((float)r2.x, 4.656612873077393e-10f, -1.f);
            // the comparisons in FP64, as they decide where FP32 cannot
            auto inside = [&]() {
                const double c[3] = {cand_coord(R, r.x, r.y), cand_coord(R, r.z, r.w),
                                     cand_coord(R, r2.x, r2.y)};
                return c[0] * c[0] + c[1] * c[1] + c[2] * c[2] <= R * R;
            };
            auto apart = [&](int j) {
                const double c[3] = {cand_coord(R, r.x, r.y), cand_coord(R, r.z, r.w),
                                     cand_coord(R, r2.x, r2.y)};
                const double d0 = c[0] - pos[3 * j], d1 = c[1] - pos[3 * j + 1],
                             d2 = c[2] - pos[3 * j + 2];
                const double need = a.spacing * 0.5 * (rad[i] + rad[j]);
                return d0 * d0 + d1 * d1 + d2 * d2 >= need * need;
            };
            const float out = __fmaf_rn(z, z, __fmaf_rn(y, y, x * x)) - 1.f;
            bool ok = fast && out < -GEO_ABS ? true : fast && out > GEO_ABS ? false : inside();
            for (int j = 0; j < i && ok; j++) {
                const float4 p = near[j];
                const float d0 = x - p.x, d1 = y - p.y, d2 = z - p.z, need = ri + p.w;
                const float nn = need * need;
                const float over = __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, d0 * d0)) - nn;
                const float tol = __fmaf_rn(GEO_REL, nn, GEO_ABS);
                if (!(fast && over > tol)) ok = !(fast && over < -tol) && apart(j);
            }
            int w;
            if (T == 32) {
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                w = m ? __ffs(m) - 1 : T;
            } else {
                if (tid == 0) s_pick = T;
                __syncthreads();
                if (ok) atomicMin(&s_pick, tid);
                __syncthreads();
                w = s_pick;
            }
            if (w < T) {
                if (tid == w) {
                    const double c[3] = {cand_coord(R, r.x, r.y), cand_coord(R, r.z, r.w),
                                         cand_coord(R, r2.x, r2.y)};
                    for (int k = 0; k < 3; k++) pos[3 * i + k] = c[k];
                    near[i] = make_float4((float)(c[0] * inv_R), (float)(c[1] * inv_R),
                                          (float)(c[2] * inv_R), ri);
                }
                done = true;
            }
            __syncthreads();
        }
        if (!done) status = 1;
        else placed = i + 1;
    }
    for (int i = tid; i < n; i += T) {
        const int64_t g = e * n + i;
        for (int k = 0; k < 3; k++) a.location[3 * g + k] = i < placed ? pos[3 * i + k] : NAN;
    }
    if (tid == 0) a.status[e] = status;
}

}  // namespace

size_t geometry_smem_bytes(int n) { return (size_t)n * (4 * sizeof(double) + sizeof(float4)); }

template <int T>
static cudaError_t launch_geometry_t(const GeoArgs &a, cudaStream_t stream)
{
    const size_t smem = geometry_smem_bytes(a.n);
    if (smem + 64 > 48 * 1024) {  // with the static words
        cudaError_t err = cudaFuncSetAttribute(geometry_kernel<T>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem);
        if (err != cudaSuccess) return err;
    }
    geometry_kernel<T><<<(unsigned)a.E, T, smem, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_geometry(const GeoArgs &a, cudaStream_t stream)
{
    if (a.E == 0) return cudaSuccess;
    // One warp per member wastes the fewest candidates (the first valid one
    // ends a batch); with fewer members than sub-partitions the chip has idle
    // ones, and a wider batch shortens the search of each.
    return a.E >= sub_partitions() ? launch_geometry_t<32>(a, stream) : launch_geometry_t<GEO_WIDE>(a, stream);
}

}  // namespace magpy
