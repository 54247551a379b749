// fw_mi.cu -- sampled Mattes mutual information of the Rigid/Affine stages: the joint Parzen
// histogram, ITK's ComputeResults and the parameter gradient (metric/mi.rs:364-511, 702-768;
// GPU counterpart GpuMiLevel, crates/fastwarp-gpu/src/wgpu_backend/mi.rs:144-491).
//
// Device design:
//  - samples are resident as 16-byte records (x, y, z relative to the cloud centre as float32,
//    fixed bin as u32): one vector load per sample;
//  - the histogram is accumulated in 2^-32 fixed point, two 32-bit words a cell in block-private
//    shared memory, and merged with u64 atomics: integer sums do not depend on order, so a rerun is
//    bit-identical, and the normalising sum is exact (no Kahan sum needed);
//  - ComputeResults (normalisation, marginals, -MI, the per-cell ratio) runs on the device in
//    float64, so value_and_derivative needs a single read-back;
//  - the derivative is linear in the Jacobian, which is affine in the sample point for Euler3D and
//    affine transforms: col_mu(p) = G_mu [p; 1]. The kernel therefore reduces only the twelve
//    moments M_ij = sum_s w_s grad_i(s) [r_s; 1]_j (w_s = sum_k B3'(k - term) ratio[f, k]) and the
//    host contracts them with every parameter's G_mu in float64 -- the same sum as the
//    reference's sum_cell dpdf[cell] * ratio[cell], reordered.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <vector>

#include "fw_internal.cuh"

struct fw_mi_level {
    fw_ctx* ctx;
    fw_image* moving;
    bool own_moving;
    bool own_rec;  // false: the records belong to the caller (a linear chain's sample cache)
    float4* d_rec;
    int64_t n;
    double center[3];
    fw_mi_binning binning;
    unsigned long long* d_hist;  // [T][bins*bins + bins]
    double* d_ratio;             // [bins*bins]
    double* d_out;               // [T][4]: value, num_valid, status, pad
    double* d_mom;               // [12]
    double* d_part;              // block partials
    unsigned int* d_counter;
    unsigned int blocks;
    unsigned int hist_grid;  // resident histogram blocks (one wave)
    size_t hist_smem;
    bool hist_clear;         // the histograms are zero (the next pass may add into them)
    int64_t last_valid;
    size_t rec_bytes;
};

namespace fw {

namespace {

constexpr int MI_THREADS = 256;
constexpr int HIST_THREADS = 512;   // k_mi_hist: two blocks an SM, 32 warps over 8 copies each
constexpr int DENSE_THREADS = 1024; // k_dense_hist: one block an SM
constexpr int MAX_BINS = 32;
constexpr double FIXED = 4294967296.0;  // 2^32

struct MiMap {
    double a[9];   // moving index from relative sample point
    double b[3];
    double h[3][3];  // index offset of +half a spacing along physical axis d (central difference)
    DevGrid m;
    int bins;
    int aligned;     // every h[d] lies along index axis d, upwards
    double mmin, mmax, mbin, mnmin;
    double isp[3];   // 1 / spacing of the moving image
};

__device__ __forceinline__ int clamp_bin(double term, int bins) {
    long long idx = isnan(term) ? 0 : (long long)term;  // truncation toward zero
    return (int)min(max(idx, 2LL), (long long)bins - 3);
}

// The continuous moving index of a sample record.
__device__ __forceinline__ void sample_index(const MiMap& mp, float4 r, double c[3]) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
        c[q] = mp.a[q * 3] * r.x + mp.a[q * 3 + 1] * r.y + mp.a[q * 3 + 2] * r.z + mp.b[q];
}

// The Parzen term and bin of a moving value; false when it is not finite or outside the range.
__device__ __forceinline__ bool sample_term(const MiMap& mp, float v, double& mv, double& term,
                                            int& mbin) {
    mv = (double)v;
    if (!isfinite(v) || mv < mp.mmin || mv > mp.mmax) return false;
    term = mv / mp.mbin - mp.mnmin;
    mbin = clamp_bin(term, mp.bins);
    return true;
}

// The moving sample: index, interpolated value and its Parzen term; false when the sample does
// not contribute (outside the buffer, not finite, or outside the moving range).
__device__ __forceinline__ bool sample_value(const MiMap& mp, const float* __restrict__ img,
                                             float4 r, double c[3], double& mv, double& term,
                                             int& mbin) {
    sample_index(mp, r, c);
    if (!inside_index(c[0], c[1], c[2], mp.m.nx, mp.m.ny, mp.m.nz)) return false;
    return sample_term(mp, lin_at_index(img, mp.m.nx, mp.m.ny, mp.m.nz, c[0], c[1], c[2]), mv, term,
                       mbin);
}

// metric/mi.rs:61-88: the cubic B-spline and its derivative at any argument.
__device__ __noinline__ double bspline3(double u) {
    const double a = fabs(u), s = a * a;
    if (a < 1.0) return (4.0 - 6.0 * s + 3.0 * s * a) / 6.0;
    if (a < 2.0) return (8.0 - 12.0 * a + 6.0 * s - s * a) / 6.0;
    return 0.0;
}

__device__ __noinline__ double bspline3_derivative(double u) {
    if (u >= 0.0 && u < 1.0) return -2.0 * u + 1.5 * u * u;
    if (u > -1.0 && u < 0.0) return -2.0 * u - 1.5 * u * u;
    if (u >= 1.0 && u < 2.0) return -2.0 + 2.0 * u - 0.5 * u * u;
    if (u > -2.0 && u <= -1.0) return 2.0 + 2.0 * u + 0.5 * u * u;
    return 0.0;
}

// The four cubic B-spline weights of a term that lies t = term - bin above its bin, at the bins
// -1, 0, 1, 2 from it, in 2^-32 fixed point (round to nearest: adding 2^52 to a value below 2^32
// leaves its rounded integer in the low bits of the sum). With t in [0, 1] the spline's pieces in
// powers of t and 1 - t need no branch and no division; a binning whose ranges and bin sizes do
// not belong together can put a term further from its clamped bin, which takes the definition.
__device__ __forceinline__ void parzen_taps(double t, unsigned int q[4]) {
    const double s = 1.0 - t, t2 = t * t, s2 = s * s, t3 = t2 * t, s3 = s2 * s;
    double w[4] = {s3 * (1.0 / 6.0), fma(0.5, t3, 2.0 / 3.0 - t2),
                   fma(0.5, s3, 2.0 / 3.0 - s2), t3 * (1.0 / 6.0)};
    if (!(t >= 0.0 && t <= 1.0)) {
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = bspline3((double)(k - 1) - t);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        q[k] = (unsigned int)__double2loint(fma(w[k], FIXED, 4503599627370496.0));
}

// The four derivative weights B3'(k - t), k = -1, 0, 1, 2, in the same way.
__device__ __forceinline__ void parzen_slopes(double t, double d[4]) {
    const double s = 1.0 - t;
    d[0] = 0.5 * s * s;
    d[1] = t * fma(-1.5, t, 2.0);
    d[2] = s * fma(1.5, s, -2.0);
    d[3] = -0.5 * t * t;
    if (!(t >= 0.0 && t <= 1.0)) {
#pragma unroll
        for (int k = 0; k < 4; ++k) d[k] = bspline3_derivative((double)(k - 1) - t);
    }
}

// Block-private histograms in shared memory. A cell's 2^-32 sum is kept as two 32-bit words, the
// sums of its addends' low and high 16 bits, because shared memory adds 32-bit words natively and
// a 64-bit add is a compare-and-swap loop that repeats for every lane on the same cell. A word
// takes 65535 addends without overflow: MI_SEGMENT bounds the samples between two merges into the
// 64-bit global histogram, so the totals are the exact integers they were with 64-bit cells.
// Lane l adds into copy l mod R of the histogram: neighbouring samples see nearly the same
// intensities, and copies keep a warp's lanes off one another's cells. Odd copy strides put a
// cell's copies on different banks.
// A copy: [bins*bins] low words, [bins*bins] high words, [bins] counts (fixed marginal).
constexpr int MI_REP = 8;
constexpr int MI_ADDENDS = 65535;

__host__ __device__ constexpr int mi_copy_words(int bins) { return (2 * bins * bins + bins) | 1; }

__device__ __forceinline__ void mi_add(unsigned int* sh, int nc, int row, int bin,
                                       const unsigned int q[4]) {
    unsigned int* c = sh + row + bin - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        atomicAdd(c + k, q[k] & 0xffffu);
        atomicAdd(c + nc + k, q[k] >> 16);
    }
}

// The sum of `copies` copies of cell s (a joint cell or, from nc on, a count).
__device__ __forceinline__ unsigned long long mi_cell(const unsigned int* sh, int copies,
                                                      int stride, int nc, int s) {
    unsigned long long v = 0ULL;
    if (s < nc) {
        for (int k = 0; k < copies; ++k)
            v += (unsigned long long)sh[k * stride + s] +
                 ((unsigned long long)sh[k * stride + nc + s] << 16);
    } else {
        for (int k = 0; k < copies; ++k) v += sh[k * stride + nc + s];
    }
    return v;
}

size_t mi_hist_smem(int bins) { return sizeof(unsigned int) * MI_REP * (size_t)mi_copy_words(bins); }

// Joint histogram of one transform over a chunk of samples per block, added into `out`. What
// bounds it: the shared-memory adds (nine a sample) and the eight scattered loads of the
// interpolation. 2.13 M samples of a 193 x 229 x 193 image: 73 us with 64-bit cells and
// the branched spline, 37 us now with ComputeResults in its last block (6.6 us as a launch before).
__device__ __forceinline__ void mi_hist_body(const MiMap& mp, const float4* __restrict__ rec,
                                             long long n, const float* __restrict__ img,
                                             unsigned long long* __restrict__ out) {
    const int bins = mp.bins;
    const int nc = bins * bins, cells = nc + bins;
    const int stride = mi_copy_words(bins);
    extern __shared__ unsigned int sh_all[];
    unsigned int* sh = sh_all + (threadIdx.x & (MI_REP - 1)) * stride;
    // samples of a thread between two merges: blockDim.x / MI_REP threads share a copy
    const int segment = MI_ADDENDS * MI_REP / HIST_THREADS;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long first = (long long)blockIdx.x * blockDim.x; first < n; first += step * segment) {
        for (int s = threadIdx.x; s < MI_REP * stride; s += blockDim.x) sh_all[s] = 0u;
        __syncthreads();
        const long long end = min(n, first + step * segment);
        long long i = first + threadIdx.x;
        float4 next = i < end ? __ldg(rec + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (; i < end; i += step) {
            const float4 r = next;
            if (i + step < end) next = __ldg(rec + i + step);
            double c[3], mv, term;
            int mbin;
            if (!sample_value(mp, img, r, c, mv, term, mbin)) continue;
            const int fbin = (int)__float_as_uint(r.w);
            unsigned int q[4];
            parzen_taps(term - (double)mbin, q);
            atomicAdd(&sh[2 * nc + fbin], 1u);
            mi_add(sh, nc, fbin * bins, mbin, q);
        }
        __syncthreads();
        for (int s = threadIdx.x; s < cells; s += blockDim.x) {
            const unsigned long long v = mi_cell(sh_all, MI_REP, stride, nc, s);
            if (v) atomicAdd(&out[s], v);
        }
        __syncthreads();
    }
}

// Whether this block is the last of `total` to get here (its predecessors' writes are visible).
__device__ __forceinline__ bool mi_last_block(unsigned int* counter, unsigned int total) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1u) == total - 1;
        if (last) *counter = 0;
    }
    __syncthreads();
    return last;
}

// ComputeResults (metric/mi.rs:702-768) of histogram h by one block: o[0] = -MI, [1] = valid
// samples, [2] = status (0 ok, 1 no valid sample, 2 zero PDF); ratio[cell] with want_ratio.
__device__ __forceinline__ void mi_finish_body(const unsigned long long* h, int bins,
                                               double moving_bin_size, double* ratio, double* o,
                                               int want_ratio);

// What the last block of a histogram pass does: ComputeResults, then the histogram is zeroed,
// ready for the next evaluation's pass.
struct MiFinish {
    unsigned int* counter;  // one per transform; null: the pass leaves its histogram
    double moving_bin_size;
    double* ratio;
    double* out;
    int want_ratio;
};

__device__ __forceinline__ void mi_hist_finish(const MiFinish& fin, int t, int bins,
                                               unsigned long long* h) {
    if (!fin.counter || !mi_last_block(fin.counter + t, gridDim.x)) return;
    mi_finish_body(h, bins, fin.moving_bin_size, fin.ratio + (size_t)t * bins * bins,
                   fin.out + 4 * t, fin.want_ratio);
    __syncthreads();  // every read of the histogram is done
    for (int s = threadIdx.x; s < bins * bins + bins; s += blockDim.x) h[s] = 0ULL;
}

// Transform blockIdx.y of a batch (maps in device memory).
__global__ void __launch_bounds__(HIST_THREADS, 2) k_mi_hist(const MiMap* __restrict__ maps,
                                                             const float4* __restrict__ rec,
                                                             long long n,
                                                             const float* __restrict__ img,
                                                             unsigned long long* __restrict__ hist,
                                                             MiFinish fin) {
    const MiMap& mp = maps[blockIdx.y];
    unsigned long long* h = hist + (size_t)blockIdx.y * (mp.bins * mp.bins + mp.bins);
    mi_hist_body(mp, rec, n, img, h);
    mi_hist_finish(fin, blockIdx.y, mp.bins, h);
}

// One transform, its map passed with the launch (no copy ahead of it).
__global__ void __launch_bounds__(HIST_THREADS, 2) k_mi_hist1(const __grid_constant__ MiMap mp,
                                                              const float4* __restrict__ rec,
                                                              long long n,
                                                              const float* __restrict__ img,
                                                              unsigned long long* __restrict__ hist,
                                                              MiFinish fin) {
    mi_hist_body(mp, rec, n, img, hist);
    mi_hist_finish(fin, 0, mp.bins, hist);
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ComputeResults for histogram blockIdx.x as a kernel of its own (the dense pair, whose moving
// bin sizes mbin_dev[t] are measured on the device, and pass timing with `moving_bin_size`).
__global__ void __launch_bounds__(1024) k_mi_finish(const unsigned long long* hist, int bins,
                                                    double moving_bin_size,
                                                    const double* __restrict__ mbin_dev,
                                                    double* __restrict__ ratio_all,
                                                    double* __restrict__ out, int want_ratio) {
    if (mbin_dev) moving_bin_size = mbin_dev[blockIdx.x];
    mi_finish_body(hist + (size_t)blockIdx.x * (bins * bins + bins), bins, moving_bin_size,
                   ratio_all + (size_t)blockIdx.x * bins * bins, out + 4 * blockIdx.x, want_ratio);
}

__device__ __forceinline__ void mi_finish_body(const unsigned long long* h, int bins,
                                               double moving_bin_size, double* ratio, double* o,
                                               int want_ratio) {
    __shared__ unsigned long long s_js[32], s_vs[32];
    __shared__ double s_c[32];
    __shared__ double joint[MAX_BINS * MAX_BINS];  // in units of 2^-32 until normalised
    __shared__ double fmarg[MAX_BINS], mmarg[MAX_BINS];
    __shared__ double norm_s;
    __shared__ unsigned long long valid_s;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, nw = blockDim.x >> 5;
    const int nc = bins * bins;
    // exact integer totals: the joint sum and the number of valid samples (warp shuffles, then
    // the first warp over the warps' sums)
    unsigned long long js = 0, vs = 0;
    for (int s = t; s < nc; s += blockDim.x) {
        const unsigned long long v = __ldcg(h + s);
        js += v;
        joint[s] = (double)v;
    }
    for (int s = t; s < bins; s += blockDim.x) vs += __ldcg(h + nc + s);
    js = warp_sum_u64(js);
    vs = warp_sum_u64(vs);
    if (lane == 0) {
        s_js[wp] = js;
        s_vs[wp] = vs;
    }
    __syncthreads();
    if (wp == 0) {
        unsigned long long a = lane < nw ? s_js[lane] : 0ULL, b = lane < nw ? s_vs[lane] : 0ULL;
        a = warp_sum_u64(a);
        b = warp_sum_u64(b);
        if (lane == 0) {
            norm_s = (double)a / FIXED;
            valid_s = b;
        }
    }
    __syncthreads();
    const double pdf_sum = norm_s;
    const unsigned long long num_valid = valid_s;
    if (num_valid == 0 || pdf_sum < DBL_EPSILON) {
        if (t == 0) {
            o[0] = 0.0;
            o[1] = (double)num_valid;
            o[2] = num_valid == 0 ? 1.0 : 2.0;
        }
        return;
    }
    const double norm = 1.0 / pdf_sum;
    if (t < bins) fmarg[t] = (double)__ldcg(h + nc + t) * norm;
    if (t < bins) {
        double s = 0.0;
        for (int row = 0; row < bins; ++row) s += (joint[row * bins + t] / FIXED) * norm;
        mmarg[t] = s;
    }
    __syncthreads();
    const double n_factor = -1.0 / (moving_bin_size * (double)num_valid);
    double contrib = 0.0;
    for (int s = t; s < nc; s += blockDim.x) {
        int f = s / bins, m = s - f * bins;
        double fm = fmarg[f], mm = mmarg[m];
        double jv = (joint[s] / FIXED) * norm;
        double r = 0.0;
        if (fm > DBL_EPSILON && mm > DBL_EPSILON && jv > DBL_EPSILON) {
            double pr = log(jv / mm);
            contrib += jv * (pr - log(fm));
            r = n_factor * pr;
        }
        if (want_ratio) ratio[s] = r;
    }
    // the sum of the cells' terms in a fixed order: each thread's cells, each warp's butterfly,
    // then the first warp's over the warps in order
    contrib = warp_sum_d(contrib);
    if (lane == 0) s_c[wp] = contrib;
    __syncthreads();
    double total = 0.0;
    if (wp == 0) total = warp_sum_d(lane < nw ? s_c[lane] : 0.0);
    if (t == 0) {
        o[0] = -total;
        o[1] = (double)num_valid;
        o[2] = 0.0;
    }
}

// The moving value and the three half-spacing differences v(c + h) - v(c - h) of a sample whose
// probes move up and down one index axis each (MiMap::aligned), from 20 voxels: an axis's probes lie
// a voxel apart, so their corners are the sample's own eight and, per axis, four more on one side.
// The sample's eight and the probes' 48 reads came to two thirds of the gradient pass in L1
// wavefronts (samples four voxels apart in a warp: five lines a load). False where a corner is
// outside the buffer or a weight is zero (whose corner must not be read into the value): the general
// path then takes the sample. Every interpolation in lin_at_axes' order.
__device__ __forceinline__ bool sample_stencil(const MiMap& mp, const float* __restrict__ img,
                                               const double c[3], float& value, float diff[3]) {
    const int nn[3] = {mp.m.nx, mp.m.ny, mp.m.nz};
    int b[3], s[3];        // the sample's lower corner; the lowest of an axis's three positions
    float w[3], w1[3], w2[3];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double c1 = c[d] - mp.h[d][d], c2 = c[d] + mp.h[d][d];
        const double f0 = floor(c[d]), f1 = floor(c1), f2 = floor(c2);
        w[d] = (float)(c[d] - f0);
        w1[d] = (float)(c1 - f1);
        w2[d] = (float)(c2 - f2);
        // in the buffer with both neighbours: before the conversions to int
        ok = ok && f1 >= 0.0 && f2 <= (double)(nn[d] - 2) && f2 == f1 + 1.0 &&
             (f0 == f1 || f0 == f2) && w[d] > 0.0f && w1[d] > 0.0f && w2[d] > 0.0f;
        b[d] = (int)f0;
        s[d] = (int)f1;
    }
    if (!ok) return false;
    const unsigned int sy = (unsigned int)nn[0], sz = sy * (unsigned int)nn[1];
    const unsigned int o = (unsigned int)b[0] + sy * (unsigned int)b[1] + sz * (unsigned int)b[2];
    // the sample's cube v[z][y][x], and each axis's extra face e[axis][.][.]
    float v[2][2][2], e[3][2][2];
    const unsigned int st[3] = {1u, sy, sz};
    unsigned int face[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) face[d] = s[d] < b[d] ? o - st[d] : o + 2u * st[d];
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) v[z][y][x] = __ldg(img + (o + x + y * sy + z * sz));
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            e[0][q][r] = __ldg(img + (face[0] + r * sy + q * sz));  // [z][y]
            e[1][q][r] = __ldg(img + (face[1] + r + q * sz));       // [z][x]
            e[2][q][r] = __ldg(img + (face[2] + r + q * sy));       // [y][x]
        }
    auto lerp = [](float a, float b2, float t) { return fmaf(b2 - a, t, a); };
    // rows along x at the sample's fraction: [z][y], and the extra rows
    float rx[2][2], ry[2], rz[2];
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int y = 0; y < 2; ++y) rx[z][y] = lerp(v[z][y][0], v[z][y][1], w[0]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        ry[q] = lerp(e[1][q][0], e[1][q][1], w[0]);
        rz[q] = lerp(e[2][q][0], e[2][q][1], w[0]);
    }
    value = lerp(lerp(rx[0][0], rx[0][1], w[1]), lerp(rx[1][0], rx[1][1], w[1]), w[2]);
    // axis x: three positions of every row
    {
        const bool low = s[0] < b[0];
        float p[2], q[2];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            float a1[2], a2[2];
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float t0 = low ? e[0][z][y] : v[z][y][0], t1 = low ? v[z][y][0] : v[z][y][1],
                            t2 = low ? v[z][y][1] : e[0][z][y];
                a1[y] = lerp(t0, t1, w1[0]);
                a2[y] = lerp(t1, t2, w2[0]);
            }
            p[z] = lerp(a1[0], a1[1], w[1]);
            q[z] = lerp(a2[0], a2[1], w[1]);
        }
        diff[0] = lerp(q[0], q[1], w[2]) - lerp(p[0], p[1], w[2]);
    }
    // axis y: three rows of each slice
    {
        const bool low = s[1] < b[1];
        float p[2], q[2];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const float t0 = low ? ry[z] : rx[z][0], t1 = low ? rx[z][0] : rx[z][1],
                        t2 = low ? rx[z][1] : ry[z];
            p[z] = lerp(t0, t1, w1[1]);
            q[z] = lerp(t1, t2, w2[1]);
        }
        diff[1] = lerp(q[0], q[1], w[2]) - lerp(p[0], p[1], w[2]);
    }
    // axis z: three slices
    {
        const bool low = s[2] < b[2];
        const float u0 = lerp(rx[0][0], rx[0][1], w[1]), u1 = lerp(rx[1][0], rx[1][1], w[1]),
                    ue = lerp(rz[0], rz[1], w[1]);
        const float t0 = low ? ue : u0, t1 = low ? u0 : u1, t2 = low ? u1 : ue;
        diff[2] = lerp(t1, t2, w2[2]) - lerp(t0, t1, w1[2]);
    }
    return true;
}

// Derivative moments M[i][j] = sum_s w_s grad_i [r; 1]_j with a fixed-order last-block reduction.
// 2.13 M samples of a 193 x 229 x 193 image: 109 us with 56 reads a sample; a line search step of six
// evaluations with one gradient takes 435 us with them and 412 with 20.
__global__ void __launch_bounds__(MI_THREADS, 3) k_mi_deriv(const __grid_constant__ MiMap mp,
                                                         const float4* __restrict__ rec,
                                                         long long n,
                                                         const float* __restrict__ img,
                                                         const double* __restrict__ ratio,
                                                         double* __restrict__ partials,
                                                         unsigned int* __restrict__ counter,
                                                         double* __restrict__ mom) {
    const int bins = mp.bins;
    __shared__ double sratio[MAX_BINS * MAX_BINS];
    for (int s = threadIdx.x; s < bins * bins; s += blockDim.x) sratio[s] = ratio[s];
    __syncthreads();
    double acc[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) acc[q] = 0.0;
    const long long step = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float4 next = i < n ? __ldg(rec + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (; i < n; i += step) {
        const float4 r = next;
        if (i + step < n) next = __ldg(rec + i + step);
        double c[3], mv, term;
        float v, diff[3];
        int mbin;
        sample_index(mp, r, c);
        const bool near = mp.aligned && sample_stencil(mp, img, c, v, diff);
        if (!near) {
            if (!inside_index(c[0], c[1], c[2], mp.m.nx, mp.m.ny, mp.m.nz)) continue;
            v = lin_at_index(img, mp.m.nx, mp.m.ny, mp.m.nz, c[0], c[1], c[2]);
        }
        if (!sample_term(mp, v, mv, term, mbin)) continue;
        const int fbin = (int)__float_as_uint(r.w);
        double w = 0.0, slope[4];
        parzen_slopes(term - (double)mbin, slope);
#pragma unroll
        for (int k = 0; k < 4; ++k) w += slope[k] * sratio[fbin * bins + mbin - 1 + k];
        if (w == 0.0) continue;
        if (!near) {
            // interp.rs:96-120: half-spacing central differences along the physical axes, every
            // probe by itself; an axis with a probe outside the buffer contributes zero
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double c1x = c[0] - mp.h[d][0], c1y = c[1] - mp.h[d][1],
                             c1z = c[2] - mp.h[d][2];
                const double c2x = c[0] + mp.h[d][0], c2y = c[1] + mp.h[d][1],
                             c2z = c[2] + mp.h[d][2];
                const bool ok = inside_index(c1x, c1y, c1z, mp.m.nx, mp.m.ny, mp.m.nz) &&
                                inside_index(c2x, c2y, c2z, mp.m.nx, mp.m.ny, mp.m.nz);
                const float v1 = lin_at_index(img, mp.m.nx, mp.m.ny, mp.m.nz, c1x, c1y, c1z);
                const float v2 = lin_at_index(img, mp.m.nx, mp.m.ny, mp.m.nz, c2x, c2y, c2z);
                diff[d] = ok ? v2 - v1 : 0.0f;
            }
        }
        double g[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) g[d] = (double)diff[d] * mp.isp[d];
        if (!(isfinite(g[0]) && isfinite(g[1]) && isfinite(g[2]))) g[0] = g[1] = g[2] = 0.0;
        const double p[4] = {(double)r.x, (double)r.y, (double)r.z, 1.0};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a * 4 + b] += w * g[a] * p[b];
    }
    __shared__ double red[12][MI_THREADS / 32];
    __shared__ bool last;
#pragma unroll
    for (int q = 0; q < 12; ++q) {
        double v = warp_sum_d(acc[q]);
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        double s = 0.0;
        for (int w = 0; w < MI_THREADS / 32; ++w) s += red[threadIdx.x][w];
        partials[(size_t)blockIdx.x * 12 + threadIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // the whole last block sums the partials of each moment in a fixed order
    __shared__ double fin[MI_THREADS / 32];
    for (int q = 0; q < 12; ++q) {
        const double s = block_sum_fixed(partials + q, gridDim.x, 12, fin);
        if (threadIdx.x == 0) mom[q] = s;
    }
    if (threadIdx.x == 0) *counter = 0;
}

// ---- dense Mattes MI pair of two images on one grid (SyN Mattes channels) -----------------
//
// Backend::mi_value_derivative_pair[_masked] (backend.rs:179-205) as cpu/mod.rs:352-381 runs it:
// MattesMi::evaluate_dense (metric/mi.rs:601-680) twice, (fixed, moving) then (moving, fixed),
// with identity transforms and the masks (when given) on the images' grid. Both directions use
// the same two Parzen terms per voxel (f / s_f - n_f and m / s_m - n_m), so one pass builds both
// joint histograms and one pass writes both derivatives. The intensity ranges (MiBinning::dense,
// mi.rs:276-295: each image over the voxels inside its own mask, non-finite voxels skipped) and
// the bin geometry (MiBinning::from_ranges, mi.rs:238-274) are measured on the device.

struct DenseState {
    unsigned int key[4];    // order-preserving keys: inverted f min, f max, inverted m min, m max
    unsigned int count[2];  // finite voxels inside each image's own mask
    unsigned int done;      // blocks of the range pass that are through
    int status;             // 0 ok; 1 / 2 no finite fixed / moving voxel; 3 / 4 constant
    double fmin, fmax, mmin, mmax;
    double sf, nf, sm, nm;  // bin size and normalised minimum of each image
    double mbin[2];         // moving-axis bin size of direction 0 (m) and 1 (f)
};

__device__ __forceinline__ unsigned int order_key(float v) {
    unsigned int b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float key_value(unsigned int k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// MiBinning::dense's ranges and MiBinning::from_ranges (mi.rs:238-295) from the keys.
__device__ __forceinline__ void dense_setup(DenseState* st, int bins) {
    const unsigned int c0 = __ldcg(&st->count[0]), c1 = __ldcg(&st->count[1]);
    if (c0 == 0 || c1 == 0) {
        st->status = c0 == 0 ? 1 : 2;
        return;
    }
    const double fmin = key_value(~__ldcg(&st->key[0])), fmax = key_value(__ldcg(&st->key[1]));
    const double mmin = key_value(~__ldcg(&st->key[2])), mmax = key_value(__ldcg(&st->key[3]));
    st->fmin = fmin;
    st->fmax = fmax;
    st->mmin = mmin;
    st->mmax = mmax;
    if (fmax - fmin <= DBL_EPSILON || mmax - mmin <= DBL_EPSILON) {
        st->status = fmax - fmin <= DBL_EPSILON ? 3 : 4;
        return;
    }
    const double span = (double)(bins - 4);
    st->sf = (fmax - fmin) / span;
    st->sm = (mmax - mmin) / span;
    st->nf = fmin / st->sf - 2.0;
    st->nm = mmin / st->sm - 2.0;
    st->mbin[0] = st->sm;
    st->mbin[1] = st->sf;
}

// Four voxels l .. l + 3 (l a multiple of 4) of an image: one 16-byte load (images start on 256
// bytes), or single ones at the end of the image.
__device__ __forceinline__ void load4(const float* __restrict__ p, long long l, long long n,
                                      float v[4]) {
    if (l + 3 < n) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p + l));
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = l + k < n ? __ldg(p + l + k) : 0.0f;
    }
}

// The intensity ranges over the voxels inside each image's own mask (a null mask: all), a stream
// of 16-byte loads; the last block turns them into the bins. The state is zero before the pass.
__global__ void __launch_bounds__(256) k_dense_range(const float* __restrict__ f,
                                                     const float* __restrict__ m,
                                                     const float* __restrict__ fm,
                                                     const float* __restrict__ mm, long long n,
                                                     int bins, DenseState* __restrict__ st) {
    unsigned int key[4] = {0u, 0u, 0u, 0u}, cnt[2] = {0u, 0u};
    for (long long l = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); l < n;
         l += 4LL * gridDim.x * blockDim.x) {
        float v[2][4], in[2][4];
        load4(f, l, n, v[0]);
        load4(m, l, n, v[1]);
        if (fm) load4(fm, l, n, in[0]);
        if (mm) load4(mm, l, n, in[1]);
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (l + e < n && (!(q ? mm : fm) || in[q][e] != 0.0f) && isfinite(v[q][e])) {
                    const unsigned int k = order_key(v[q][e]);
                    key[2 * q] = max(key[2 * q], ~k);
                    key[2 * q + 1] = max(key[2 * q + 1], k);
                    ++cnt[q];
                }
    }
    __shared__ unsigned int s_key[4], s_cnt[2];
    if (threadIdx.x < 4) s_key[threadIdx.x] = 0u;
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned int k = __reduce_max_sync(0xffffffffu, key[q]);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_key[q], k);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const unsigned int c = __reduce_add_sync(0xffffffffu, cnt[q]);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_cnt[q], c);
    }
    __syncthreads();
    if (threadIdx.x < 4) atomicMax(&st->key[threadIdx.x], s_key[threadIdx.x]);
    if (threadIdx.x < 2) atomicAdd(&st->count[threadIdx.x], s_cnt[threadIdx.x]);
    if (mi_last_block(&st->done, gridDim.x) && threadIdx.x == 0) dense_setup(st, bins);
}

// The voxel's two Parzen terms and bins; false when it does not contribute (mi.rs:560-595).
__device__ __forceinline__ bool dense_voxel(const DenseState& st, int bins, float a, float b,
                                            bool in, double& tf, double& tm, int& bf, int& bm) {
    if (!in || !isfinite(a) || !isfinite(b)) return false;
    const double fv = a, mv = b;
    // each direction's moving value must lie in its range: m for (f, m), f for (m, f)
    if (mv < st.mmin || mv > st.mmax || fv < st.fmin || fv > st.fmax) return false;
    tf = fv / st.sf - st.nf;
    tm = mv / st.sm - st.nm;
    bf = clamp_bin(tf, bins);
    bm = clamp_bin(tm, bins);
    return true;
}

// Copies of the pair's two histograms per block (lane l into copy l mod MI_REP), as in
// k_mi_hist: [direction][joint low words, high words, counts].
size_t dense_hist_smem(int bins) {
    return sizeof(unsigned int) * MI_REP * (size_t)((2 * mi_copy_words(bins)) | 1);
}

// Both joint histograms: [direction][bins*bins joint + bins fixed marginal] in 2^-32 fixed point.
// Bound by the shared-memory adds (18 a voxel). A thread takes four consecutive voxels by one
// 16-byte load of each image. 193 x 229 x 193: 667 us with 64-bit cells, 90 us.
__global__ void __launch_bounds__(DENSE_THREADS, 1) k_dense_hist(
    const float* __restrict__ f, const float* __restrict__ m, const float* __restrict__ fm,
    const float* __restrict__ mm, long long n, int bins, const DenseState* __restrict__ st,
    unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned int sh_all[];
    const int nc = bins * bins, cells = nc + bins;
    const int half = mi_copy_words(bins), stride = (2 * half) | 1;
    unsigned int* sh = sh_all + (threadIdx.x & (MI_REP - 1)) * stride;
    const DenseState S = *st;
    if (S.status != 0) return;
    const int segment = MI_ADDENDS * MI_REP / (4 * DENSE_THREADS);  // groups of four a thread
    const long long step = 4LL * gridDim.x * blockDim.x;
    for (long long first = 4LL * blockIdx.x * blockDim.x; first < n; first += step * segment) {
        for (int s = threadIdx.x; s < MI_REP * stride; s += blockDim.x) sh_all[s] = 0u;
        __syncthreads();
        const long long end = min(n, first + step * segment);
        for (long long l = first + 4 * threadIdx.x; l < end; l += step) {
            float a[4], b[4], ia[4], ib[4];
            load4(f, l, n, a);
            load4(m, l, n, b);
            if (fm) load4(fm, l, n, ia);
            if (mm) load4(mm, l, n, ib);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                double tf, tm;
                int bf, bm;
                const bool in = l + e < n && (!fm || ia[e] != 0.0f) && (!mm || ib[e] != 0.0f);
                if (!dense_voxel(S, bins, a[e], b[e], in, tf, tm, bf, bm)) continue;
                unsigned int q[4];
                atomicAdd(&sh[2 * nc + bf], 1u);
                atomicAdd(&sh[half + 2 * nc + bm], 1u);
                parzen_taps(tm - (double)bm, q);
                mi_add(sh, nc, bf * bins, bm, q);
                parzen_taps(tf - (double)bf, q);
                mi_add(sh + half, nc, bm * bins, bf, q);
            }
        }
        __syncthreads();
        for (int s = threadIdx.x; s < 2 * cells; s += blockDim.x) {
            const int d = s >= cells;
            const unsigned long long v =
                mi_cell(sh_all + d * half, MI_REP, stride, nc, s - d * cells);
            if (v) atomicAdd(&hist[s], v);
        }
        __syncthreads();
    }
}

struct DenseArgs {
    DevGrid g;
    long long ps;
    int bins;
    int zchunk;
    double isp[3];
};

// One voxel's derivatives from its terms and the images' gradients (mi.rs:655-672).
__device__ __forceinline__ void dense_outputs(double w0, double w1, float gm[3], float gf[3],
                                              float o0[3], float o1[3], double& n0, double& n1) {
    if (!(isfinite(gm[0]) && isfinite(gm[1]) && isfinite(gm[2]))) gm[0] = gm[1] = gm[2] = 0.0f;
    if (!(isfinite(gf[0]) && isfinite(gf[1]) && isfinite(gf[2]))) gf[0] = gf[1] = gf[2] = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        o0[d] = (float)(w0 * (double)gm[d]);
        o1[d] = (float)(w1 * (double)gf[d]);
        n0 += (double)o0[d] * o0[d];
        n1 += (double)o1[d] * o1[d];
    }
}

// Both derivatives: sum_k B3'(k - term) ratio[fixed bin, k] * grad(moving image of the
// direction), zero where the voxel does not contribute; result[0..1] = their sums of squares, and
// the last block publishes the pair's scalars.
//
// A thread takes a column and a chunk of z (consecutive threads consecutive columns, whatever the
// grid's width, then the next chunk) and marches along z. With IDENTITY (an identity direction) a
// column keeps its two images' previous, current and next slices in registers, so a voxel loads one new
// value and the four neighbours of its slice for each image, and decides the face probes of x and y
// once; any other direction takes the exact probes of every voxel. Bound by the f64 spline weights
// and the eight ratio reads from shared memory. The pair's whole call at 193 x 229 x 193: 1420 us with
// a voxel a thread over a 296-block grid (the pass 494) and the histogram of 64-bit cells, 336 with
// columns in tiles of 32 x 8 (the pass 185), 323 now (174); turned 2120, 1390 and 960. At 1 x 1000 x 1000, where
// such a tile has one column in 32: 172, 560 and 107 us.
template <bool IDENTITY>
__global__ void __launch_bounds__(MI_THREADS) k_dense_deriv(
    DenseArgs a, const float* __restrict__ f, const float* __restrict__ m,
    const float* __restrict__ fm, const float* __restrict__ mm, const DenseState* __restrict__ st,
    const double* __restrict__ ratio, float* __restrict__ d0, float* __restrict__ d1,
    double* __restrict__ partials, unsigned int* __restrict__ counter,
    double* __restrict__ result, const double* __restrict__ out, double* __restrict__ publish) {
    __shared__ double sr[2 * MAX_BINS * MAX_BINS];
    const int bins = a.bins, nc = bins * bins;
    for (int s = threadIdx.x; s < 2 * nc; s += blockDim.x) sr[s] = ratio[s];
    __syncthreads();
    const DenseState S = *st;
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    double n0 = 0.0, n1 = 0.0;
    const int sxy = nx * ny;
    const long long t = (long long)blockIdx.x * MI_THREADS + threadIdx.x;
    const long long z0 = t / sxy * a.zchunk;
    if (z0 < nz) {
        const int z1 = (int)min(z0 + a.zchunk, (long long)nz);
        const int col = (int)(t % sxy), y = col / nx, x = col - y * nx;
        // identity grids: whether each face probe is inside, and the neighbours' offsets
        bool okx = true, oky = true;
        float2 lo = make_float2(0.0f, 0.0f), cur = lo, hi = lo;  // (f, m) of slices z - 1, z, z + 1
        auto at = [&](int z) {
            return make_float2(__ldg(f + (long long)z * sxy + col), __ldg(m + (long long)z * sxy + col));
        };
        if (IDENTITY) {
            okx = axis_probe_inside(a.g, x, y, z0, 0, -1.0, nx) &&
                  axis_probe_inside(a.g, x, y, z0, 0, +1.0, nx);
            oky = axis_probe_inside(a.g, x, y, z0, 1, -1.0, ny) &&
                  axis_probe_inside(a.g, x, y, z0, 1, +1.0, ny);
            if (z0 > 0) lo = at(z0 - 1);
            cur = at(z0);
        }
        for (int z = (int)z0; z < z1; ++z) {
            const long long l = (long long)z * sxy + col;
            if (IDENTITY) {
                if (z + 1 < nz) hi = at(z + 1);
            } else {
                cur = at(z);
            }
            const bool in = (!fm || fm[l] != 0.0f) && (!mm || mm[l] != 0.0f);
            double tf, tm;
            int bf, bm;
            float o0[3] = {0.0f, 0.0f, 0.0f}, o1[3] = {0.0f, 0.0f, 0.0f};
            if (S.status == 0 && dense_voxel(S, bins, cur.x, cur.y, in, tf, tm, bf, bm)) {
                double sl[4], w0 = 0.0, w1 = 0.0;
                parzen_slopes(tm - (double)bm, sl);
#pragma unroll
                for (int k = 0; k < 4; ++k) w0 += sl[k] * sr[bf * bins + bm - 1 + k];
                parzen_slopes(tf - (double)bf, sl);
#pragma unroll
                for (int k = 0; k < 4; ++k) w1 += sl[k] * sr[nc + bm * bins + bf - 1 + k];
                float gm[3], gf[3];
                if (IDENTITY) {
                    // interp.rs:96-120 at +-half a spacing: halfway to the neighbours
                    // (the face probes decided by axis_probe_inside)
                    auto diff = [&](int d, bool ok, bool has_lo, bool has_hi, float2 p, float2 q) {
                        const float f2 = has_hi ? fmaf(q.x - cur.x, 0.5f, cur.x) : cur.x;
                        const float f1 = has_lo ? fmaf(cur.x - p.x, 0.5f, p.x) : cur.x;
                        const float m2 = has_hi ? fmaf(q.y - cur.y, 0.5f, cur.y) : cur.y;
                        const float m1 = has_lo ? fmaf(cur.y - p.y, 0.5f, p.y) : cur.y;
                        gf[d] = ok ? (float)((double)(f2 - f1) * a.isp[d]) : 0.0f;
                        gm[d] = ok ? (float)((double)(m2 - m1) * a.isp[d]) : 0.0f;
                    };
                    auto pair = [&](bool has, long long o) {
                        return has ? make_float2(__ldg(f + o), __ldg(m + o)) : cur;
                    };
                    diff(0, okx, x > 0, x < nx - 1, pair(x > 0, l - 1), pair(x < nx - 1, l + 1));
                    diff(1, oky, y > 0, y < ny - 1, pair(y > 0, l - nx), pair(y < ny - 1, l + nx));
                    const bool okz = axis_probe_inside(a.g, x, y, z, 2, -1.0, nz) &&
                                     axis_probe_inside(a.g, x, y, z, 2, +1.0, nz);
                    diff(2, okz, z > 0, z < nz - 1, lo, hi);
                } else {
                    central_difference_exact(m, a.g, x, y, z, gm);
                    central_difference_exact(f, a.g, x, y, z, gf);
                }
                dense_outputs(w0, w1, gm, gf, o0, o1, n0, n1);
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                d0[l + d * a.ps] = o0[d];
                d1[l + d * a.ps] = o1[d];
            }
            if (IDENTITY) {
                lo = cur;
                cur = hi;
            }
        }
    }
    __shared__ double red[2][MI_THREADS / 32];
    n0 = warp_sum_d(n0);
    n1 = warp_sum_d(n1);
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = n0;
        red[1][threadIdx.x >> 5] = n1;
    }
    __syncthreads();
    const unsigned int nblocks = gridDim.x;
    if (threadIdx.x < 2) {
        double s = 0.0;
        for (int w = 0; w < MI_THREADS / 32; ++w) s += red[threadIdx.x][w];
        partials[(size_t)blockIdx.x * 2 + threadIdx.x] = s;
    }
    if (!mi_last_block(counter, nblocks)) return;
    __shared__ double fin[MI_THREADS / 32];
    for (int q = 0; q < 2; ++q) {
        const double s = block_sum_fixed(partials + q, nblocks, 2, fin);
        if (threadIdx.x == 0) result[q] = s;
    }
    // [vF, |dF|^2, |dM|^2, 0, vM, status]: the scalars of the pair where the SyN driver reads them.
    // status: 0 ok, 1 / 2 no finite fixed / moving voxel (inside its mask), 3 / 4 fixed / moving
    // image constant, 5 no voxel contributes, 6 joint PDF zero.
    if (threadIdx.x == 0) {
        int status = S.status;
        for (int dir = 0; dir < 2 && status == 0; ++dir) {
            if (out[4 * dir + 2] == 1.0) status = 5;
            else if (out[4 * dir + 2] == 2.0) status = 6;
        }
        publish[0] = out[0];
        publish[1] = result[0];
        publish[2] = result[1];
        publish[3] = 0.0;
        publish[4] = out[4];
        publish[5] = (double)status;
    }
}

// ---- host: transform maps and Jacobian matrices (transform/param.rs, affine.rs) -------------

void parametric_affine(const fw_linear_transform* t, double M[9], double off[3]) {
    double tr[3];
    if (t->kind == 0) {
        const double* p = t->parameters;
        double cx = std::cos(p[0]), sx = std::sin(p[0]);
        double cy = std::cos(p[1]), sy = std::sin(p[1]);
        double cz = std::cos(p[2]), sz = std::sin(p[2]);
        double rx[9] = {1, 0, 0, 0, cx, -sx, 0, sx, cx};
        double ry[9] = {cy, 0, sy, 0, 1, 0, -sy, 0, cy};
        double rz[9] = {cz, -sz, 0, sz, cz, 0, 0, 0, 1};
        double tmp[9];
        if (t->zyx) {
            mat3_mul(rz, ry, tmp);
            mat3_mul(tmp, rx, M);
        } else {
            mat3_mul(rz, rx, tmp);
            mat3_mul(tmp, ry, M);
        }
        tr[0] = p[3];
        tr[1] = p[4];
        tr[2] = p[5];
    } else {
        for (int k = 0; k < 9; ++k) M[k] = t->parameters[k];
        tr[0] = t->parameters[9];
        tr[1] = t->parameters[10];
        tr[2] = t->parameters[11];
    }
    double mc[3];
    mat3_vec(M, t->center, mc);
    for (int r = 0; r < 3; ++r) off[r] = tr[r] + t->center[r] - mc[r];
}

void linear_map(const fw_linear_transform* t, double Mout[9], double off_out[3]) {
    double M[9], off[3];
    parametric_affine(t, M, off);
    double oc[3], ooff[3];
    mat3_vec(t->outer_matrix, t->outer_center, oc);
    for (int r = 0; r < 3; ++r) ooff[r] = t->outer_translation[r] + t->outer_center[r] - oc[r];
    mat3_mul(t->outer_matrix, M, Mout);
    double mo[3];
    mat3_vec(t->outer_matrix, off, mo);
    for (int r = 0; r < 3; ++r) off_out[r] = mo[r] + ooff[r];
}

// transform/param.rs:188-288, 448-457: Jacobian columns at p (outer matrix applied).
int jacobian_columns(const fw_linear_transform* t, const double p[3], double cols[36]) {
    for (int k = 0; k < 36; ++k) cols[k] = 0.0;
    int np;
    if (t->kind == 0) {
        const double* q = t->parameters;
        double cx = std::cos(q[0]), sx = std::sin(q[0]);
        double cy = std::cos(q[1]), sy = std::sin(q[1]);
        double cz = std::cos(q[2]), sz = std::sin(q[2]);
        double px = p[0] - t->center[0], py = p[1] - t->center[1], pz = p[2] - t->center[2];
        double *o0 = cols, *o1 = cols + 3, *o2 = cols + 6;
        if (t->zyx) {
            o0[0] = (cz * sy * cx + sz * sx) * py + (-cz * sy * sx + sz * cx) * pz;
            o0[1] = (sz * sy * cx - cz * sx) * py + (-sz * sy * sx - cz * cx) * pz;
            o0[2] = (cy * cx) * py + (-cy * sx) * pz;
            o1[0] = (-cz * sy) * px + (cz * cy * sx) * py + (cz * cy * cx) * pz;
            o1[1] = (-sz * sy) * px + (sz * cy * sx) * py + (sz * cy * cx) * pz;
            o1[2] = (-cy) * px + (-sy * sx) * py + (-sy * cx) * pz;
            o2[0] = (-sz * cy) * px + (-sz * sy * sx - cz * cx) * py + (-sz * sy * cx + cz * sx) * pz;
            o2[1] = (cz * cy) * px + (cz * sy * sx - sz * cx) * py + (cz * sy * cx + sz * sx) * pz;
        } else {
            o0[0] = (-sz * cx * sy) * px + (sz * sx) * py + (sz * cx * cy) * pz;
            o0[1] = (cz * cx * sy) * px + (-cz * sx) * py + (-cz * cx * cy) * pz;
            o0[2] = (sx * sy) * px + cx * py + (-sx * cy) * pz;
            o1[0] = (-cz * sy - sz * sx * cy) * px + (cz * cy - sz * sx * sy) * pz;
            o1[1] = (-sz * sy + cz * sx * cy) * px + (sz * cy + cz * sx * sy) * pz;
            o1[2] = (-cx * cy) * px + (-cx * sy) * pz;
            o2[0] = (-sz * cy - cz * sx * sy) * px + (-cz * cx) * py + (-sz * sy + cz * sx * cy) * pz;
            o2[1] = (cz * cy - sz * sx * sy) * px + (-sz * cx) * py + (cz * sy + sz * sx * cy) * pz;
        }
        for (int d = 0; d < 3; ++d) cols[3 * (3 + d) + d] = 1.0;
        np = 6;
    } else {
        for (int r = 0; r < 3; ++r) {
            for (int c = 0; c < 3; ++c) cols[3 * (r * 3 + c) + r] = p[c] - t->center[c];
            cols[3 * (9 + r) + r] = 1.0;
        }
        np = 12;
    }
    for (int k = 0; k < np; ++k) {
        double v[3] = {cols[3 * k], cols[3 * k + 1], cols[3 * k + 2]}, o[3];
        mat3_vec(t->outer_matrix, v, o);
        for (int r = 0; r < 3; ++r) cols[3 * k + r] = o[r];
    }
    return np;
}

MiMap make_map(const fw_mi_level* L, const fw_linear_transform* t) {
    MiMap mp;
    std::memset(&mp, 0, sizeof(mp));
    const HostGrid& g = L->moving->grid;
    double M[9], off[3];
    linear_map(t, M, off);
    // index = inv (M (centre + r) + off - org) = (inv M) r + inv (M centre + off - org)
    mat3_mul(g.inv, M, mp.a);
    double mc[3];
    mat3_vec(M, L->center, mc);
    double v[3] = {mc[0] + off[0] - g.org[0], mc[1] + off[1] - g.org[1], mc[2] + off[2] - g.org[2]};
    mat3_vec(g.inv, v, mp.b);
    for (int d = 0; d < 3; ++d)
        for (int r = 0; r < 3; ++r) mp.h[d][r] = 0.5 * g.sp[d] * g.inv[r * 3 + d];
    mp.aligned = 1;
    for (int d = 0; d < 3; ++d)
        for (int r = 0; r < 3; ++r)
            if (r == d ? !(mp.h[d][r] > 0.0) : mp.h[d][r] != 0.0) mp.aligned = 0;
    for (int d = 0; d < 3; ++d) mp.isp[d] = 1.0 / g.sp[d];
    mp.m = dev_grid(g);
    mp.bins = L->binning.bins;
    mp.mmin = L->binning.moving_min;
    mp.mmax = L->binning.moving_max;
    mp.mbin = L->binning.moving_bin_size;
    mp.mnmin = L->binning.moving_normalized_min;
    return mp;
}

// The histogram kernel's shared memory can exceed the 48 KB default.
int hist_launch_setup(fw_ctx* ctx, size_t smem) {
    (void)ctx;
    FW_CUDA(cudaFuncSetAttribute(k_mi_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    FW_CUDA(cudaFuncSetAttribute(k_mi_hist1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return 0;
}

// One wave of resident histogram blocks (each merges its copies into the global histogram once).
unsigned int hist_blocks(const fw_mi_level* L, size_t smem) {
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mi_hist, HIST_THREADS, smem) != cudaSuccess ||
        occ < 1) {
        cudaGetLastError();
        occ = 1;
    }
    const long long want = (L->n + HIST_THREADS - 1) / HIST_THREADS;
    return (unsigned int)std::max<long long>(1, std::min<long long>(want, (long long)occ * L->ctx->num_sms));
}

// The histogram pass of `count` transforms, ComputeResults in its last block (a launch of its own
// cost 3-4 us more an evaluation). One transform's map goes with the launch; a batch's maps are
// copied ahead. The histograms are zero before the pass (cleared by the previous pass's last
// block, or here after an interrupted evaluation). `map0` (nullable) receives the first transform's map.
int hist_and_finish(fw_mi_level* L, const fw_linear_transform* ts, int count, bool want_ratio,
                    MiMap* map0 = nullptr) {
    fw_ctx* ctx = L->ctx;
    const int bins = L->binning.bins;
    const int cells = bins * bins + bins;
    if (!L->hist_clear) {
        FW_CUDA(cudaMemsetAsync(L->d_hist, 0, sizeof(unsigned long long) * cells * 16, ctx->stream));
        L->hist_clear = true;
    }
    L->hist_clear = false;
    const MiFinish fin{L->d_counter + 1, L->binning.moving_bin_size, L->d_ratio, L->d_out,
                       want_ratio ? 1 : 0};
    if (count == 1) {
        const MiMap mp = make_map(L, &ts[0]);
        if (map0) *map0 = mp;
        k_mi_hist1<<<L->hist_grid, HIST_THREADS, L->hist_smem, ctx->stream>>>(
            mp, L->d_rec, L->n, L->moving->d, L->d_hist, fin);
        FW_TRY(check_launch(ctx, "k_mi_hist1"));
    } else {
        std::vector<MiMap> maps(count);
        for (int t = 0; t < count; ++t) maps[t] = make_map(L, &ts[t]);
        if (map0) *map0 = maps[0];
        FW_TRY(ensure_scratch(ctx, SLOT_PARTIALS + (sizeof(MiMap) * count + 7) / 8 + 16));
        MiMap* d_maps = reinterpret_cast<MiMap*>(ctx->d_scratch + SLOT_PARTIALS);
        FW_CUDA(cudaMemcpyAsync(d_maps, maps.data(), sizeof(MiMap) * count, cudaMemcpyHostToDevice,
                                ctx->stream));
        dim3 grid(L->hist_grid, count);
        k_mi_hist<<<grid, HIST_THREADS, L->hist_smem, ctx->stream>>>(
            d_maps, L->d_rec, L->n, L->moving->d, L->d_hist, fin);
        FW_TRY(check_launch(ctx, "k_mi_hist"));
    }
    L->hist_clear = true;
    return 0;
}

int check_status(fw_mi_level* L, const double* out) {
    L->last_valid = (int64_t)out[1];
    if (out[2] == 1.0) return fail(FW_ERR_INVALID, "mattes: all samples map outside the moving image buffer");
    if (out[2] == 2.0) return fail(FW_ERR_INVALID, "mattes: joint PDF summed to zero");
    return 0;
}

}  // namespace

}  // namespace fw

using namespace fw;

// A level over sample records already on the device (float32 offsets from `center`, the fixed
// bin in w). Takes the moving image when own_moving and the records when own_rec, also on failure.
int fw::mi_level_create(fw_ctx* ctx, fw_image* moving, bool own_moving, float4* d_rec,
                        bool own_rec, int64_t n, const double center[3],
                        const fw_mi_binning* binning, fw_mi_level** out) {
    auto drop = [&] {
        if (own_rec && d_rec) dev_free(ctx, d_rec, sizeof(float4) * (size_t)std::max<int64_t>(n, 0));
        if (own_moving) fw_image_free(moving);
    };
    if (n <= 0) {
        drop();
        return fail(FW_ERR_INVALID, "mattes: no samples inside the fixed image");
    }
    if (binning->bins <= 4 || binning->bins > MAX_BINS) {
        drop();
        return fail(FW_ERR_INVALID, "mattes: bins must be in 5..=32");
    }
    fw_mi_level* L = new fw_mi_level();
    L->ctx = ctx;
    L->moving = moving;
    L->own_moving = own_moving;
    L->own_rec = own_rec;
    L->d_rec = d_rec;
    L->n = n;
    L->binning = *binning;
    for (int a = 0; a < 3; ++a) L->center[a] = center[a];
    L->rec_bytes = sizeof(float4) * (size_t)n;
    const int cells = binning->bins * binning->bins + binning->bins;
    const int max_t = 16;
    // the gradient pass: one wave of resident blocks (a partial second wave would run its tail
    // at a fraction of the occupancy)
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mi_deriv, MI_THREADS, 0) != cudaSuccess ||
        occ < 1) {
        cudaGetLastError();
        occ = 1;
    }
    L->blocks = (unsigned int)std::max<long long>(
        1, std::min<long long>((n + MI_THREADS - 1) / MI_THREADS, (long long)occ * ctx->num_sms));
    int rc = dev_alloc(ctx, sizeof(unsigned long long) * cells * max_t, (void**)&L->d_hist);
    if (!rc) rc = dev_alloc(ctx, sizeof(double) * binning->bins * binning->bins, (void**)&L->d_ratio);
    if (!rc) rc = dev_alloc(ctx, sizeof(double) * 4 * max_t, (void**)&L->d_out);
    if (!rc) rc = dev_alloc(ctx, sizeof(double) * 16, (void**)&L->d_mom);
    if (!rc) rc = dev_alloc(ctx, sizeof(double) * 12 * L->blocks, (void**)&L->d_part);
    if (!rc) rc = dev_alloc(ctx, sizeof(unsigned int) * 32, (void**)&L->d_counter);
    if (!rc) {
        cudaError_t e = cudaMemsetAsync(L->d_counter, 0, sizeof(unsigned int) * 32, ctx->stream);
        if (e == cudaSuccess)
            e = cudaMemsetAsync(L->d_hist, 0, sizeof(unsigned long long) * cells * max_t, ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "mi level setup");
        L->hist_clear = true;
    }
    if (!rc) {
        L->hist_smem = mi_hist_smem(binning->bins);
        rc = hist_launch_setup(ctx, L->hist_smem);
        if (!rc) L->hist_grid = hist_blocks(L, L->hist_smem);
    }
    if (rc) {
        fw_mi_level_free(L);
        return rc;
    }
    *out = L;
    return 0;
}

extern "C" {

static int mi_prepare_common(fw_ctx* ctx, fw_image* moving, bool own, const double* points,
                             const uint32_t* fixed_bin, int64_t n, const fw_mi_binning* binning,
                             fw_mi_level** out) {
    if (n <= 0 || binning->bins <= 4 || binning->bins > MAX_BINS)
        return mi_level_create(ctx, moving, own, nullptr, false, n, nullptr, binning, out);
    // the cloud centre in float64; records hold float32 offsets from it
    double c[3] = {0, 0, 0};
    for (int64_t i = 0; i < n; ++i)
        for (int a = 0; a < 3; ++a) c[a] += points[3 * i + a];
    for (int a = 0; a < 3; ++a) c[a] /= (double)n;
    std::vector<float4> rec((size_t)n);
    for (int64_t i = 0; i < n; ++i) {
        if (fixed_bin[i] >= (uint32_t)binning->bins) {
            if (own) fw_image_free(moving);
            return fail(FW_ERR_INVALID, "mattes: a fixed bin is out of range");
        }
        rec[i].x = (float)(points[3 * i] - c[0]);
        rec[i].y = (float)(points[3 * i + 1] - c[1]);
        rec[i].z = (float)(points[3 * i + 2] - c[2]);
        uint32_t b = fixed_bin[i];
        std::memcpy(&rec[i].w, &b, 4);
    }
    const size_t bytes = sizeof(float4) * (size_t)n;
    float4* d_rec = nullptr;
    int rc = dev_alloc(ctx, bytes, (void**)&d_rec);
    if (!rc) {
        cudaError_t e = cudaMemcpyAsync(d_rec, rec.data(), bytes, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "mi level upload");
        ctx->stats.bytes_uploaded += bytes;
    }
    if (!rc) rc = sync(ctx);
    if (rc) {
        if (d_rec) dev_free(ctx, d_rec, bytes);
        if (own) fw_image_free(moving);
        return rc;
    }
    return mi_level_create(ctx, moving, own, d_rec, true, n, c, binning, out);
}

int fw_mi_level_prepare(fw_ctx* ctx, const fw_grid* moving_grid, const double* moving,
                        const double* points, const uint32_t* fixed_bin, int64_t n,
                        const fw_mi_binning* binning, fw_mi_level** out) {
    FW_CHECK(ctx && moving_grid && moving && points && fixed_bin && binning && out, "null argument");
    fw_image* img;
    FW_TRY(fw_image_upload(ctx, moving_grid, moving, &img));
    return mi_prepare_common(ctx, img, true, points, fixed_bin, n, binning, out);
}

int fw_mi_level_prepare_image(fw_ctx* ctx, const fw_image* moving, const double* points,
                              const uint32_t* fixed_bin, int64_t n,
                              const fw_mi_binning* binning, fw_mi_level** out) {
    FW_CHECK(ctx && moving && points && fixed_bin && binning && out, "null argument");
    return mi_prepare_common(ctx, const_cast<fw_image*>(moving), false, points, fixed_bin, n,
                             binning, out);
}

int fw_mi_level_value(fw_mi_level* L, const fw_linear_transform* t, double* value) {
    FW_CHECK(L && t && value, "null argument");
    FW_TRY(hist_and_finish(L, t, 1, false));
    double out[3];
    FW_TRY(read_back(L->ctx, L->d_out, 3, out));
    FW_TRY(check_status(L, out));
    *value = out[0];
    return 0;
}

int fw_mi_level_values(fw_mi_level* L, const fw_linear_transform* ts, int32_t count,
                       double* values) {
    FW_CHECK(L && ts && values, "null argument");
    FW_CHECK(count >= 1 && count <= 16, "mattes: 1..=16 transforms per batch");
    FW_TRY(hist_and_finish(L, ts, count, false));
    std::vector<double> out(4 * count);
    FW_TRY(read_back(L->ctx, L->d_out, 4 * count, out.data()));
    for (int t = 0; t < count; ++t) {
        FW_TRY(check_status(L, &out[4 * t]));
        values[t] = out[4 * t];
    }
    return 0;
}

int fw_mi_level_value_and_derivative(fw_mi_level* L, const fw_linear_transform* t,
                                     double* value, double* derivative) {
    FW_CHECK(L && t && value && derivative, "null argument");
    fw_ctx* ctx = L->ctx;
    MiMap mp;
    FW_TRY(hist_and_finish(L, t, 1, true, &mp));
    k_mi_deriv<<<L->blocks, MI_THREADS, 0, ctx->stream>>>(mp, L->d_rec, L->n, L->moving->d,
                                                          L->d_ratio, L->d_part, L->d_counter,
                                                          L->d_mom);
    FW_TRY(check_launch(ctx, "k_mi_deriv"));
    // one read-back: status block (value, valid, status) and the twelve moments
    FW_CUDA(cudaMemcpyAsync(ctx->h_pinned, L->d_out, sizeof(double) * 4, cudaMemcpyDeviceToHost, ctx->stream));
    FW_CUDA(cudaMemcpyAsync(ctx->h_pinned + 4, L->d_mom, sizeof(double) * 12, cudaMemcpyDeviceToHost, ctx->stream));
    FW_TRY(sync(ctx));
    double out[4], mom[12];
    std::memcpy(out, ctx->h_pinned, sizeof(out));
    std::memcpy(mom, ctx->h_pinned + 4, sizeof(mom));
    FW_TRY(check_status(L, out));
    *value = out[0];
    // G_mu in relative coordinates: col_mu(c + r) = J(c) + (J(c + e_j) - J(c)) r_j
    double j0[36], je[3][36];
    FW_TRY(0);
    int np = jacobian_columns(t, L->center, j0);
    for (int j = 0; j < 3; ++j) {
        double p[3] = {L->center[0], L->center[1], L->center[2]};
        p[j] += 1.0;
        jacobian_columns(t, p, je[j]);
    }
    for (int mu = 0; mu < np; ++mu) {
        double s = 0.0;
        for (int i = 0; i < 3; ++i) {
            for (int j = 0; j < 3; ++j) s += (je[j][3 * mu + i] - j0[3 * mu + i]) * mom[i * 4 + j];
            s += j0[3 * mu + i] * mom[i * 4 + 3];
        }
        derivative[mu] = s;
    }
    return 0;
}

int fw_mi_level_time(fw_mi_level* L, const fw_linear_transform* t, int32_t reps, double ms[3],
                     double bytes[3]) {
    FW_CHECK(L && t && ms && bytes && reps > 0, "null argument");
    fw_ctx* ctx = L->ctx;
    // one evaluation first: the maps in scratch, the ratio table and the status
    double v = 0.0, d[12];
    FW_TRY(fw_mi_level_value_and_derivative(L, t, &v, d));
    const int bins = L->binning.bins;
    const int cells = bins * bins + bins;
    const MiMap mp = make_map(L, t);
    cudaEvent_t a = nullptr, b = nullptr;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
        if (a) cudaEventDestroy(a);
        return fail(FW_ERR_CUDA, "event creation failed");
    }
    int rc = 0;
    for (int kind = 0; kind < 3 && !rc; ++kind) {
        auto launch = [&]() -> int {
            if (kind == 0) {
                FW_CUDA(cudaMemsetAsync(L->d_hist, 0, sizeof(unsigned long long) * cells,
                                        ctx->stream));
                k_mi_hist1<<<L->hist_grid, HIST_THREADS, L->hist_smem, ctx->stream>>>(
                    mp, L->d_rec, L->n, L->moving->d, L->d_hist, MiFinish{});
                return check_launch(ctx, "k_mi_hist1");
            }
            if (kind == 1) {
                k_mi_finish<<<1, 1024, 0, ctx->stream>>>(L->d_hist, bins, L->binning.moving_bin_size,
                                                         nullptr, L->d_ratio, L->d_out, 1);
                return check_launch(ctx, "k_mi_finish");
            }
            k_mi_deriv<<<L->blocks, MI_THREADS, 0, ctx->stream>>>(mp, L->d_rec, L->n,
                                                                  L->moving->d, L->d_ratio,
                                                                  L->d_part, L->d_counter,
                                                                  L->d_mom);
            return check_launch(ctx, "k_mi_deriv");
        };
        rc = launch();  // warm-up
        if (rc) break;
        cudaEventRecord(a, ctx->stream);
        for (int r = 0; r < reps && !rc; ++r) rc = launch();
        cudaEventRecord(b, ctx->stream);
        if (!rc) rc = sync(ctx);
        float tm = 0.0f;
        if (!rc) cudaEventElapsedTime(&tm, a, b);
        ms[kind] = (double)tm / reps;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    L->hist_clear = false;  // the timed passes leave a histogram behind
    // algorithmic bytes per pass: the 16-byte sample records plus the moving image's gathers,
    // at most the whole image and at most one 8-corner gather per sample (32 bytes)
    const double S = (double)L->n, Nm = (double)L->moving->grid.count();
    const double pass = 16.0 * S + std::min(4.0 * Nm, 32.0 * S);
    bytes[0] = pass + 8.0 * cells;
    bytes[1] = 16.0 * cells;
    bytes[2] = pass + 8.0 * bins * bins;
    return rc;
}

int fw_mi_level_num_valid(const fw_mi_level* L, int64_t* out) {
    FW_CHECK(L && out, "null argument");
    *out = L->last_valid;
    return 0;
}

int fw_mi_level_samples(const fw_mi_level* L, double* points, uint32_t* fixed_bins, int64_t cap,
                        int64_t* n, fw_mi_binning* binning) {
    FW_CHECK(L && n, "null argument");
    *n = L->n;
    if (binning) *binning = L->binning;
    if (cap < L->n || (!points && !fixed_bins)) return 0;
    fw_ctx* ctx = L->ctx;
    std::vector<float4> rec((size_t)L->n);
    FW_CUDA(cudaMemcpyAsync(rec.data(), L->d_rec, L->rec_bytes, cudaMemcpyDeviceToHost, ctx->stream));
    FW_TRY(sync(ctx));
    ctx->stats.bytes_downloaded += L->rec_bytes;
    for (int64_t i = 0; i < L->n; ++i) {
        if (points) {
            points[3 * i] = L->center[0] + (double)rec[i].x;
            points[3 * i + 1] = L->center[1] + (double)rec[i].y;
            points[3 * i + 2] = L->center[2] + (double)rec[i].z;
        }
        if (fixed_bins) std::memcpy(&fixed_bins[i], &rec[i].w, 4);
    }
    return 0;
}

void fw_mi_level_free(fw_mi_level* L) {
    if (!L) return;
    fw_ctx* ctx = L->ctx;
    const int cells = L->binning.bins * L->binning.bins + L->binning.bins;
    if (L->own_rec) dev_free(ctx, L->d_rec, L->rec_bytes);
    dev_free(ctx, L->d_hist, sizeof(unsigned long long) * cells * 16);
    dev_free(ctx, L->d_ratio, sizeof(double) * L->binning.bins * L->binning.bins);
    dev_free(ctx, L->d_out, sizeof(double) * 4 * 16);
    dev_free(ctx, L->d_mom, sizeof(double) * 16);
    dev_free(ctx, L->d_part, sizeof(double) * 12 * L->blocks);
    dev_free(ctx, L->d_counter, sizeof(unsigned int) * 32);
    if (L->own_moving) fw_image_free(L->moving);
    delete L;
}

}  // extern "C"

namespace fw {
void linear_transform_map(const fw_linear_transform* t, double M[9], double off[3]) {
    linear_map(t, M, off);
}

const fw_ctx* mi_level_context(const fw_mi_level* level) { return level ? level->ctx : nullptr; }
}  // namespace fw

// ---- dense Mattes MI pair: host side -----------------------------------------------------------

namespace fw {
namespace {

std::string empty_range_message(const char* role, bool masked) {
    if (masked)
        return std::string("no finite ") + role + "-image voxel lies inside the " + role + " mask";
    return std::string("the ") + role + " image has no finite voxel";
}

// The gradient pass's blocks on `g`: a thread a column and z chunk, the chunks for about eight blocks
// an SM (every block loads the two ratio tables first, 16 KB).
unsigned int dense_deriv_blocks(const HostGrid& g, int num_sms, int* zchunk) {
    const long long cols = g.n[0] * g.n[1];
    const long long want = (8LL * num_sms * MI_THREADS + cols - 1) / cols;
    *zchunk = (int)std::max<long long>(1, (g.n[2] + want - 1) / want);
    const long long chunks = (g.n[2] + *zchunk - 1) / *zchunk;
    return (unsigned int)((cols * chunks + MI_THREADS - 1) / MI_THREADS);
}

}  // namespace
}  // namespace fw

// Device scratch of one dense pair: [state | out 2x4 | norms 2 | counter | hist | ratio | partials].
// The state and the histograms are zeroed by one memset before every pair.
struct fw_dense_mi {
    fw_ctx* ctx = nullptr;
    void* base = nullptr;
    size_t bytes = 0;
    int bins = 0;
    fw::DenseState* st = nullptr;
    double* out = nullptr;
    double* norms = nullptr;
    unsigned long long* hist = nullptr;
    double* ratio = nullptr;
    double* partials = nullptr;
    unsigned int* counter = nullptr;
};

namespace fw {

int dense_mi_create(fw_ctx* ctx, int bins, const HostGrid& g, fw_dense_mi** out) {
    if (bins <= 4) return fail(FW_ERR_INVALID, "mattes: at least five histogram bins are required");
    if (bins > MAX_BINS) return fail(FW_ERR_INVALID, "mattes: bins must be in 5..=32");
    fw_dense_mi* d = new fw_dense_mi();
    d->ctx = ctx;
    d->bins = bins;
    int zchunk = 1;
    const size_t blocks = dense_deriv_blocks(g, ctx->num_sms, &zchunk);
    const size_t cells = (size_t)bins * bins + bins;
    const size_t o_hist = 512, o_ratio = o_hist + 16 * cells,
                 o_part = o_ratio + 16 * (size_t)bins * bins;
    d->bytes = o_part + 16 * blocks;
    static_assert(sizeof(DenseState) <= 256, "the state's place in the scratch");
    int rc = dev_alloc(ctx, d->bytes, &d->base);
    if (rc) {
        delete d;
        return rc;
    }
    char* b = static_cast<char*>(d->base);
    d->st = reinterpret_cast<DenseState*>(b);
    d->out = reinterpret_cast<double*>(b + 256);
    d->norms = reinterpret_cast<double*>(b + 256 + 64);
    d->hist = reinterpret_cast<unsigned long long*>(b + o_hist);
    d->ratio = reinterpret_cast<double*>(b + o_ratio);
    d->partials = reinterpret_cast<double*>(b + o_part);
    d->counter = reinterpret_cast<unsigned int*>(b + 256 + 128);
    cudaError_t e = cudaMemsetAsync(d->base, 0, d->bytes, ctx->stream);
    if (e != cudaSuccess) {
        dense_mi_free(d);
        return cuda_fail(e, "dense MI scratch");
    }
    *out = d;
    return 0;
}

void dense_mi_free(fw_dense_mi* d) {
    if (!d) return;
    if (d->base) dev_free(d->ctx, d->base, d->bytes);
    delete d;
}

int enqueue_dense_mi_pair(fw_ctx* ctx, const fw_image* f, const fw_image* m, const fw_image* fm,
                          const fw_image* mm, fw_field* d_fixed, fw_field* d_moving,
                          fw_dense_mi* sc, double* publish) {
    if (!f->grid.same(m->grid)) return fail(FW_ERR_INVALID, "mattes: the images are not on one grid");
    if ((fm && !fm->grid.same(f->grid)) || (mm && !mm->grid.same(f->grid)))
        return fail(FW_ERR_INVALID, "mattes: a mask is not on the grid of the images");
    const HostGrid& g = f->grid;
    const long long n = g.count();
    const int bins = sc->bins;
    const float* fmp = fm ? fm->d : nullptr;
    const float* mmp = mm ? mm->d : nullptr;
    FW_CUDA(cudaMemsetAsync(sc->base, 0, 512 + 16 * ((size_t)bins * bins + bins), ctx->stream));
    auto blocks_of = [&](int threads, long long most) {
        return (unsigned int)std::max<long long>(1, std::min((n + 4LL * threads - 1) / (4LL * threads), most));
    };
    k_dense_range<<<blocks_of(256, 8LL * ctx->num_sms), 256, 0, ctx->stream>>>(f->d, m->d, fmp, mmp,
                                                                               n, bins, sc->st);
    FW_TRY(check_launch(ctx, "k_dense_range"));
    const size_t sh = dense_hist_smem(bins);
    FW_CUDA(cudaFuncSetAttribute(k_dense_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
    k_dense_hist<<<blocks_of(DENSE_THREADS, ctx->num_sms), DENSE_THREADS, sh, ctx->stream>>>(
        f->d, m->d, fmp, mmp, n, bins, sc->st, sc->hist);
    FW_TRY(check_launch(ctx, "k_dense_hist"));
    k_mi_finish<<<2, 1024, 0, ctx->stream>>>(sc->hist, bins, 0.0, sc->st->mbin, sc->ratio,
                                             sc->out, 1);
    FW_TRY(check_launch(ctx, "k_mi_finish"));
    DenseArgs da;
    std::memset(&da, 0, sizeof(da));
    da.g = dev_grid(g);
    da.ps = d_fixed->ps;
    da.bins = bins;
    bool identity = true;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c)
            if (g.dir[r * 3 + c] != (r == c ? 1.0 : 0.0)) identity = false;
    for (int d = 0; d < 3; ++d) da.isp[d] = 1.0 / g.sp[d];
    const unsigned int grid = dense_deriv_blocks(g, ctx->num_sms, &da.zchunk);
    auto deriv = identity ? k_dense_deriv<true> : k_dense_deriv<false>;
    deriv<<<grid, MI_THREADS, 0, ctx->stream>>>(da, f->d, m->d, fmp, mmp, sc->st, sc->ratio,
                                                d_fixed->d, d_moving->d, sc->partials, sc->counter,
                                                sc->norms, sc->out, publish);
    return check_launch(ctx, "k_dense_deriv");
}

int dense_mi_status(int status, bool masked) {
    switch (status) {
        case 0: return 0;
        case 1: return fail(FW_ERR_INVALID, "mattes: " + empty_range_message("fixed", masked));
        case 2: return fail(FW_ERR_INVALID, "mattes: " + empty_range_message("moving", masked));
        case 3: return fail(FW_ERR_INVALID, "mattes: the fixed image is constant");
        case 4: return fail(FW_ERR_INVALID, "mattes: the moving image is constant");
        case 5:
            return fail(FW_ERR_INVALID, masked ? std::string("mattes: ") + FW_NO_VOXEL_IN_MASKS
                                               : std::string("mattes: all samples map outside the moving image buffer"));
        default: return fail(FW_ERR_INVALID, "mattes: joint PDF summed to zero");
    }
}

namespace {

int dense_pair(fw_ctx* ctx, const fw_image* f, const fw_image* m, const fw_image* fm,
               const fw_image* mm, int bins, double values[2], fw_field** d_fixed,
               fw_field** d_moving, double norms[2]) {
    FW_CHECK(ctx && f && m && values && d_fixed && d_moving, "null argument");
    if (!f->grid.same(m->grid)) return fail(FW_ERR_INVALID, "mattes: the images are not on one grid");
    fw_dense_mi* sc = nullptr;
    FW_TRY(dense_mi_create(ctx, bins, f->grid, &sc));
    fw_field *a = nullptr, *b = nullptr;
    int rc = new_field(ctx, f->grid, &a);
    if (!rc) rc = new_field(ctx, f->grid, &b);
    double* pub = ctx->d_scratch + SLOT_MI;
    if (!rc) rc = enqueue_dense_mi_pair(ctx, f, m, fm, mm, a, b, sc, pub);
    double h[6] = {0, 0, 0, 0, 0, 0};
    if (!rc) rc = read_back(ctx, pub, 6, h);
    if (!rc) rc = dense_mi_status((int)h[5], fm || mm);
    dense_mi_free(sc);
    if (rc) {
        fw_field_free(a);
        fw_field_free(b);
        return rc;
    }
    values[0] = h[0];
    values[1] = h[4];
    if (norms) {
        norms[0] = std::sqrt(h[1]);
        norms[1] = std::sqrt(h[2]);
    }
    *d_fixed = a;
    *d_moving = b;
    return 0;
}

}  // namespace
}  // namespace fw

extern "C" {

int fw_mi_value_derivative_pair(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                                int32_t bins, double values[2], fw_field** d_fixed,
                                fw_field** d_moving) {
    return fw::dense_pair(ctx, fixed, moving, nullptr, nullptr, bins, values, d_fixed, d_moving,
                          nullptr);
}

int fw_mi_value_derivative_pair_masked(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                                       const fw_image* fixed_mask, const fw_image* moving_mask,
                                       int32_t bins, double values[2], fw_field** d_fixed,
                                       fw_field** d_moving) {
    return fw::dense_pair(ctx, fixed, moving, fixed_mask, moving_mask, bins, values, d_fixed,
                          d_moving, nullptr);
}

int fw_mi_value_derivative_pair_with_norms(fw_ctx* ctx, const fw_image* fixed,
                                           const fw_image* moving, int32_t bins, double values[2],
                                           fw_field** d_fixed, fw_field** d_moving,
                                           double norms[2]) {
    FW_CHECK(norms, "null norms");
    return fw::dense_pair(ctx, fixed, moving, nullptr, nullptr, bins, values, d_fixed, d_moving,
                          norms);
}

int fw_mi_value_derivative_pair_masked_with_norms(fw_ctx* ctx, const fw_image* fixed,
                                                  const fw_image* moving,
                                                  const fw_image* fixed_mask,
                                                  const fw_image* moving_mask, int32_t bins,
                                                  double values[2], fw_field** d_fixed,
                                                  fw_field** d_moving, double norms[2]) {
    FW_CHECK(norms, "null norms");
    return fw::dense_pair(ctx, fixed, moving, fixed_mask, moving_mask, bins, values, d_fixed,
                          d_moving, norms);
}

}  // extern "C"
