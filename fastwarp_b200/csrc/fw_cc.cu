// fw_cc.cu -- ANTs neighbourhood cross-correlation, both directions in one pass.
//
// Restates metric/cc.rs:170-321 (CcMetric::evaluate_masked with identity transforms on one grid,
// what cpu/mod.rs:299-331 runs for Backend::cc_value_derivative_pair): the six window sums over a
// clamped (2r+1)^3 box, local CC = sFM^2 / (sFF sMM), value = -mean(localCC), and the derivative
// coefficient * grad(moving) by ITK's half-spacing central difference (interp.rs:96-120).
//
// Kernel design (sm_100a): one CTA owns a TX x TY column tile and marches along z over a chunk
// of slices. The z window comes first, as running sums over the tile's halo columns kept in
// shared memory (entering slice added, leaving slice subtracted); the y and x box passes then run
// on those sums, eight outputs an item by suffix and prefix sums (window_sums). Sums are float64:
// products of float32 voxels are exact in float64, so the centred second moments
// (sum f^2 - (sum f)^2 / n) keep their precision in flat bright regions where float32 cancels. The
// window planes never touch HBM: the kernel reads the two images (the leaving slice and the halo a
// second time, from L2) and writes the two derivative fields.
//
// What bounds it: shared memory (two thirds of its bandwidth) and issue (60 %), at three CTAs of 8
// warps an SM (80 registers a thread, 60 KB of shared memory); the float64 pipe is a fifth busy.
// The pair's whole call at 193 x 229 x 193, r = 4: 400 us with 64 additions an x group and 20 a y
// group, window counters, and the face tests and float64 scaling of the gradients at every voxel;
// 325 us now. Masked, r = 3, 181 x 217 x 165 on a rotated grid with every probe from global memory in
// float64: 458 us; 289 us with the probes' common corners and weights on the raw slices, the faces
// included (328 with every probe of a face's warp from global memory; unmasked 64 x 217 x 165, where
// every warp holds a face, 311 us with all probes from global memory, 386 with them at the faces, 139).
// Measured and dropped: z sums in registers (spills at three CTAs: 521 us), 16 rows a tile with one
// or two voxels a thread (363-424 us), two CTAs an SM without spills (374 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "fw_internal.cuh"

namespace fw {

namespace {

constexpr int TX = 32;
constexpr int CC_TY = 8;         // rows of a tile
constexpr int CC_NT = 256;       // threads of a CTA

// Kinds of grids by their central differences, a kernel each: CC_AXES an identity direction with every
// 1 / spacing a float32 (1, 2, 0.5, 0.8 mm ...); CC_AXES64 one with others (0.9, 0.7 mm), whose
// differences are scaled in float64; CC_ROTATED another direction whose probes stay within one voxel
// of theirs; CC_EXACT the rest (very unequal spacings), every probe by itself. One kernel of the
// second and the last spilled the call's registers in the loop: 0.9 mm at 193 x 229 x 193 393 us (r 3), masked
// 500 (r 4); apart 326 and 388.
enum CcMode { CC_EXACT, CC_AXES, CC_AXES64, CC_ROTATED };

struct CcArgs {
    DevGrid g;
    long long ps;       // plane stride of the derivative fields
    int zchunk;         // slices per CTA
    double isp[3];      // 1 / spacing (the central difference's denominator)
    float ispf[3];      // the same in float32
    int mode;           // the kernel's MODE
    // the probe at -half (p = 2d) and +half (2d + 1) a spacing along physical axis d, relative to
    // its voxel: index offset of its lower corner (-1 or 0; 1 only where the weight is 0, a probe on
    // the neighbour itself: axes permuted and one spacing twice another) and weights of the upper one
    signed char base[6][3];
    float weight[6][3];
    // at a face of index axis r: the physical axes (bit d) whose probes reach more than half a voxel
    // along r and so leave the buffer there, and the one (or 3, none) whose probes end on the half
    // voxel, where the reference's rounding decides
    unsigned char out[3], edge[3];
};

// Shared-memory layout (dynamic): the z-window sums of every halo column, [5][HY][HX] double
// (+ [HY][HX] int counts with a mask); y sums [5][HX][TY+1] double, column-major with an odd
// column stride (+ [TY][HX] int counts); the x sums of the tile's voxels [5][TX][TY+1] double; the
// raw voxels of the tile with a one-voxel halo for four slices, [4][TY+2][TX+2] float2 (f, m), for
// the central differences; block-reduction space. The odd strides keep every pass free of bank
// conflicts: the y pass stores consecutive columns, the x pass reads consecutive rows, and each
// voxel's thread reads its own row of a column.
template <int R, int TY, bool MK>
struct Layout {
    static constexpr int HX = TX + 2 * R;
    static constexpr int HY = TY + 2 * R;
    static constexpr int HC = HX * HY;           // halo columns of the tile
    static constexpr int NT = CC_NT;
    static constexpr int CPT = (HC + NT - 1) / NT;  // halo columns per thread
    static constexpr int NP = MK ? 4 : 3;  // block partials: cc, |dF|^2, |dM|^2 (+ valid voxels)
    static constexpr int RX = TX + 2, RY = TY + 2, RXY = RX * RY;
    static constexpr int RING = RXY - TX * TY;   // raw voxels around the tile, one a thread
    static constexpr int D = 4;                  // raw slices: z - 1, z, z + 1 and the next one
    static constexpr int YS = TY + 1;            // odd: TY is even
    static constexpr int GX = 8;                 // outputs of an item of the x pass
    static constexpr int YI = 5 * HX, XI = 5 * TY * (TX / GX);  // items of the y and x passes
    static_assert(TX % GX == 0 && RING <= NT && YI <= NT && XI <= NT && TX * TY == NT,
                  "one item a thread");
    static constexpr size_t zs1 = sizeof(double) * 5 * HC + (MK ? sizeof(int) * HC : 0);
    static constexpr size_t xs_bytes = sizeof(double) * 5 * HX * YS;  // y sums [5][HX][YS]
    static constexpr size_t xc_bytes = MK ? sizeof(int) * TY * HX : 0;
    static constexpr size_t raw_bytes = sizeof(float2) * D * RXY;
    static constexpr size_t sx_bytes = sizeof(double) * 5 * TX * YS;  // x sums [5][TX][YS]
    static constexpr size_t sx_off = zs1 + xs_bytes + xc_bytes + raw_bytes;
    static constexpr size_t red_off = sx_off + sx_bytes;
    static constexpr size_t bytes = red_off + 64 * sizeof(double);
};

// MK: masked (cpu/mod.rs:134-163 -> evaluate_masked with Some(valid)): a voxel counts only where
// `vimg` is not zero; invalid voxels add nothing to any window sum, the count is the number of
// valid voxels in the window, their outputs are zero and the value is the mean over the valid
// voxels (result[3] receives their number; zero means no voxel in the masks).
//
// Pass order z, y, x. Each thread owns up to CPT halo columns and moves their z-window sums (in
// shared memory, where the y pass reads them) one slice per step: the entering slice is added
// and the leaving slice (read again, from L2) subtracted -- before the step's first barrier, which
// the previous step's y pass has passed. Products of float32 voxels are exact in float64, so the
// running sums carry no drift beyond float64 rounding. The y and x passes make eight outputs an
// item, and each thread then reads its own voxel's window sums.
constexpr int CC_MIN_BLOCKS = 3;

// The window sums' arithmetic. SumF64 (the default): float64, in which the products of float32
// voxels are exact. SumC32: compensated float32, a (hi, lo) float pair per sum -- products split
// exactly by an fma (TwoProduct), additions by Knuth's TwoSum with the rounding errors gathered
// in lo and a Fast2Sum renormalisation; every operation is an explicitly rounded intrinsic, so
// the compiler cannot fuse a product into a neighbouring addition. Both take 8 bytes a sum in
// shared memory.
struct SumF64 {
    using T = double;
    __device__ static __forceinline__ T zero() { return 0.0; }
    __device__ static __forceinline__ T diff(float a, float b) { return (double)a - (double)b; }
    __device__ static __forceinline__ T prod_diff(float a, float b, float c, float d) {
        const double x = a, y = b, z = c, w = d;
        return x * y - z * w;
    }
    __device__ static __forceinline__ T add(T a, T b) { return a + b; }
    __device__ static __forceinline__ double value(T a) { return a; }
};

struct SumC32 {
    using T = float2;  // x: hi, y: lo
    __device__ static __forceinline__ void two_sum(float a, float b, float& s, float& e) {
        s = __fadd_rn(a, b);
        const float bb = __fsub_rn(s, a);
        e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    }
    __device__ static __forceinline__ T zero() { return make_float2(0.0f, 0.0f); }
    __device__ static __forceinline__ T diff(float a, float b) {
        float s, e;
        two_sum(a, -b, s, e);
        return make_float2(s, e);
    }
    __device__ static __forceinline__ T prod_diff(float a, float b, float c, float d) {
        const float p = __fmul_rn(a, b), pe = __fmaf_rn(a, b, -p);
        const float q = __fmul_rn(c, d), qe = __fmaf_rn(c, d, -q);
        float s, e;
        two_sum(p, -q, s, e);
        return make_float2(s, __fadd_rn(e, __fsub_rn(pe, qe)));
    }
    __device__ static __forceinline__ T add(T a, T b) {
        float s, e;
        two_sum(a.x, b.x, s, e);
        const float lo = __fadd_rn(e, __fadd_rn(a.y, b.y));
        const float hi = __fadd_rn(s, lo);
        return make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s)));
    }
    __device__ static __forceinline__ double value(T a) { return (double)a.x + (double)a.y; }
};

// The G sums of 2R + 1 consecutive values out of G + 2R (load(t), t = 0 ..), store(j, sum of
// load(j) .. load(j + 2R)), without a subtraction: the windows of GS neighbouring outputs all
// contain the values GS-1 .. 2R, so each is a suffix sum that ends at 2R plus a prefix sum that
// starts at 2R + 1 (van Herk's and Gil and Werman's running extremum, for sums): about 2.7 additions
// an output at R = 4 in place of 8. A window of zeros sums to exactly zero.
template <class Acc, int R, int G, class Load, class Store>
__device__ __forceinline__ void window_sums(Load load, Store store) {
    using T = typename Acc::T;
    constexpr int GS = R == 1 ? 2 : (R <= 3 ? 4 : 8);  // GS <= 2R + 1
    static_assert(G % GS == 0, "whole groups");
#pragma unroll
    for (int h = 0; h < G; h += GS) {
        T s[GS];
        T c = load(h + GS - 1);
#pragma unroll
        for (int t = GS; t <= 2 * R; ++t) c = Acc::add(c, load(h + t));
        s[GS - 1] = c;
#pragma unroll
        for (int j = GS - 2; j >= 0; --j) s[j] = Acc::add(s[j + 1], load(h + j));
        store(h, s[0]);
        T p = load(h + 2 * R + 1);
        store(h + 1, Acc::add(s[1], p));
#pragma unroll
        for (int j = 2; j < GS; ++j) {
            p = Acc::add(p, load(h + 2 * R + j));
            store(h + j, Acc::add(s[j], p));
        }
    }
}

// The exact central differences of both images (interp.rs:96-120 at voxel (x, y, z)), the probes'
// float64 indices formed once for the two. Inlined into the loop of the one kind of grid that needs it:
// as a call, its operands and the loop's go through local memory (193 x 229 x 193, spacings 0.5 / 8 /
// 0.7 mm turned, r 4: 1749 us with a call an image, 1292 with one for both, 895 inlined).
__device__ __forceinline__ void cc_exact_gradients(const float* __restrict__ fimg,
                                                const float* __restrict__ mimg, const DevGrid& g,
                                                int x, int y, int z, float gf[3], float gm[3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double a[3], b[3];
        probe_index(g, x, y, z, d, -1.0, a);
        probe_index(g, x, y, z, d, +1.0, b);
        gf[d] = gm[d] = 0.0f;
        if (!inside_index(a[0], a[1], a[2], g.nx, g.ny, g.nz) ||
            !inside_index(b[0], b[1], b[2], g.nx, g.ny, g.nz))
            continue;
        const int n[3] = {g.nx, g.ny, g.nz};
        int ia[3], ib[3];
        float wa[3], wb[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            lin_axis(a[r], n[r], ia[r], wa[r]);
            lin_axis(b[r], n[r], ib[r], wb[r]);
        }
        auto diff = [&](const float* img) {
            const float v1 = lin_at_axes(img, g.nx, g.ny, ia[0], wa[0], ia[1], wa[1], ia[2], wa[2]);
            const float v2 = lin_at_axes(img, g.nx, g.ny, ib[0], wb[0], ib[1], wb[1], ib[2], wb[2]);
            return (float)((double)(v2 - v1) / g.sp[d]);
        };
        gf[d] = diff(fimg);
        gm[d] = diff(mimg);
    }
}

// Whether a probe of voxel (x, y, z) along physical axis d is outside the buffer along index axis r,
// by the reference's own arithmetic.
__device__ __noinline__ bool cc_probe_outside(const DevGrid& g, int x, int y, int z, int d, int r,
                                              int n) {
    double a[3], b[3];
    probe_index(g, x, y, z, d, -1.0, a);
    probe_index(g, x, y, z, d, +1.0, b);
    return !(a[r] >= -0.5 && a[r] < (double)n - 0.5 && b[r] >= -0.5 && b[r] < (double)n - 0.5);
}

// One tile (bx, by, bz) of the CC pair: writes the tile's derivative voxels and leaves the
// thread's sums [cc, |dF|^2, |dM|^2, valid voxels] in acc_out. MODE: how the central differences
// are formed, one kind of grid alone (registers that other kinds need would be spilled for in the
// loop).
template <int R, int TY, bool MK, int MODE, class Acc = SumF64>
__device__ __forceinline__ void cc_tile(const CcArgs& a, int bx, int by, int bz,
                                        unsigned char* smem, const float* __restrict__ fimg,
                                        const float* __restrict__ mimg,
                                        const float* __restrict__ vimg,
                                        float* __restrict__ d_fixed, float* __restrict__ d_moving,
                                        int want_norms, double acc_out[4]) {
    using L = Layout<R, TY, MK>;
    using T = typename Acc::T;
    static_assert(sizeof(T) == sizeof(double), "a window sum takes 8 bytes");
    T* zs = reinterpret_cast<T*>(smem);
    int* zc = reinterpret_cast<int*>(zs + 5 * L::HC);
    T* xs = reinterpret_cast<T*>(smem + L::zs1);
    int* xc = reinterpret_cast<int*>(smem + L::zs1 + L::xs_bytes);
    float2* raw = reinterpret_cast<float2*>(smem + L::zs1 + L::xs_bytes + L::xc_bytes);
    T* sx = reinterpret_cast<T*>(smem + L::sx_off);

    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int x0 = bx * TX, y0 = by * TY;
    const int z0 = bz * a.zchunk;
    const int z1 = min(z0 + a.zchunk, nz);
    const int x = x0 + tx, y = y0 + ty;
    const bool own = x < nx && y < ny;
    const long long sxy = (long long)nx * ny;

    double acc_cc = 0.0, acc_nf = 0.0, acc_nm = 0.0, acc_nv = 0.0;

    // the thread's halo columns: offset inside a slice, OUT outside the image (sums stay zero)
    constexpr unsigned int OUT = 0xffffffffu;
    unsigned int coff[L::CPT];
#pragma unroll
    for (int j = 0; j < L::CPT; ++j) {
        const int s = tid + j * L::NT;
        coff[j] = OUT;
        if (s < L::HC) {
            const int hy = s / L::HX, hx = s - hy * L::HX;
            const int gx = x0 - R + hx, gy = y0 - R + hy;
            if (gx >= 0 && gx < nx && gy >= 0 && gy < ny) coff[j] = gy * nx + gx;
        }
    }
    // The last slice where each halo column of an image was not zero. The reference forms every
    // window sum directly from the window's voxels (metric/cc.rs:137-157), so a window where an
    // image is zero sums to exactly zero and its CC takes the degenerate value; a running sum keeps
    // a float64 rounding residue of what entered and left, so an image's sums are reset to zero
    // whenever its last non-zero slice is out of the window.
    int lastf[L::CPT], lastm[L::CPT];
    const int kb = max(z0 - R, 0);
    // the first window's slices but the last: additions only, their loads in flight together
    {
        T zsum[L::CPT][5];
        int cnt[L::CPT];
#pragma unroll
        for (int j = 0; j < L::CPT; ++j) {
            lastf[j] = lastm[j] = kb - 2 * R - 2;
            cnt[j] = 0;
#pragma unroll
            for (int q = 0; q < 5; ++q) zsum[j][q] = Acc::zero();
        }
        const int ke = min(z0 + R, nz);
#pragma unroll 4
        for (int k = kb; k < ke; ++k) {
            const long long zi = (long long)k * sxy;
#pragma unroll
            for (int j = 0; j < L::CPT; ++j) {
                float f = 0.0f, m = 0.0f;
                if (coff[j] != OUT) {
                    f = __ldg((fimg + zi) + coff[j]);
                    m = __ldg((mimg + zi) + coff[j]);
                    if constexpr (MK) {
                        const bool v = __ldg((vimg + zi) + coff[j]) != 0.0f;
                        if (!v) f = m = 0.0f;  // a masked-out voxel adds nothing
                        cnt[j] += (int)v;
                    }
                }
                if (f != 0.0f) lastf[j] = k;
                if (m != 0.0f) lastm[j] = k;
                zsum[j][0] = Acc::add(zsum[j][0], Acc::diff(f, 0.0f));
                zsum[j][1] = Acc::add(zsum[j][1], Acc::diff(m, 0.0f));
                zsum[j][2] = Acc::add(zsum[j][2], Acc::prod_diff(f, f, 0.0f, 0.0f));
                zsum[j][3] = Acc::add(zsum[j][3], Acc::prod_diff(m, m, 0.0f, 0.0f));
                zsum[j][4] = Acc::add(zsum[j][4], Acc::prod_diff(f, m, 0.0f, 0.0f));
            }
        }
#pragma unroll
        for (int j = 0; j < L::CPT; ++j) {
            const int s = tid + j * L::NT;
            if (s < L::HC) {
#pragma unroll
                for (int q = 0; q < 5; ++q) zs[q * L::HC + s] = zsum[j][q];
                if constexpr (MK) zc[s] = cnt[j];
            }
        }
    }
    // entering slice k and leaving slice k - 2R - 1 of the next step, in flight during a step
    float2 pin[L::CPT], pout[L::CPT];
    bool vin[L::CPT], vout[L::CPT];
    auto fetch = [&](int k) {
        const bool add = k < nz, sub = k - 2 * R - 1 >= kb;
        const long long zi = (long long)k * sxy, zo = (long long)(k - 2 * R - 1) * sxy;
        const float *fi = fimg + zi, *mi = mimg + zi, *fo = fimg + zo, *mo = mimg + zo;
#pragma unroll
        for (int j = 0; j < L::CPT; ++j) {
            const bool c = coff[j] != OUT;
            pin[j] = c && add ? make_float2(__ldg(fi + coff[j]), __ldg(mi + coff[j]))
                              : make_float2(0.0f, 0.0f);
            pout[j] = c && sub ? make_float2(__ldg(fo + coff[j]), __ldg(mo + coff[j]))
                               : make_float2(0.0f, 0.0f);
            if constexpr (MK) {
                vin[j] = c && add && __ldg((vimg + zi) + coff[j]) != 0.0f;
                vout[j] = c && sub && __ldg((vimg + zo) + coff[j]) != 0.0f;
                if (!vin[j]) pin[j] = make_float2(0.0f, 0.0f);
                if (!vout[j]) pout[j] = make_float2(0.0f, 0.0f);
            }
        }
    };
    // the raw voxels of the tile and its one-voxel ring, clamped at the image's faces: the thread's
    // own voxel's column (also kept in registers) and, for the first RING threads, one of the ring
    const unsigned int ocol = (unsigned int)(min(y, ny - 1) * nx + min(x, nx - 1));
    unsigned int rcol = 0;
    int rslot = 0;
    if (tid < L::RING) {
        int rx, ry;
        if (tid < 2 * L::RX) {
            ry = tid < L::RX ? 0 : L::RY - 1;
            rx = tid < L::RX ? tid : tid - L::RX;
        } else {
            const int t = tid - 2 * L::RX;
            ry = 1 + (t >> 1);
            rx = (t & 1) ? L::RX - 1 : 0;
        }
        rslot = ry * L::RX + rx;
        rcol = (unsigned int)(min(max(y0 - 1 + ry, 0), ny - 1) * nx + min(max(x0 - 1 + rx, 0), nx - 1));
    }
    const int oslot = (ty + 1) * L::RX + tx + 1;
    auto voxel = [&](int z, unsigned int col) {
        const long long o = (long long)min(max(z, 0), nz - 1) * sxy;
        return make_float2(__ldg((fimg + o) + col), __ldg((mimg + o) + col));
    };
    float2 lo, cur = voxel(z0 - 1, ocol), hi = voxel(z0, ocol);  // shifted by the first step
    float2 nown = voxel(z0 + 1, ocol), nring = make_float2(0.0f, 0.0f);
    raw[((z0 - 1) & 3) * L::RXY + oslot] = cur;
    raw[(z0 & 3) * L::RXY + oslot] = hi;
    if (tid < L::RING) {
        raw[((z0 - 1) & 3) * L::RXY + rslot] = voxel(z0 - 1, rcol);
        raw[(z0 & 3) * L::RXY + rslot] = voxel(z0, rcol);
        nring = voxel(z0 + 1, rcol);
    }
    const T* own_sums = sx + tx * L::YS + ty;
    // identity grids: whether the probes of the faces are inside (a coordinate's probes do not
    // depend on the others): bit 0 x, bits 1 and 2 the first and last slice, bit 3 y
    unsigned int ok = ~0u;
    if ((MODE == CC_AXES || MODE == CC_AXES64) && own) {
        auto inside = [&](int i, int j, int k, int d, int n) {
            return axis_probe_inside(a.g, i, j, k, d, -1.0, n) && axis_probe_inside(a.g, i, j, k, d, +1.0, n);
        };
        if (!inside(x, y0, z0, 0, nx)) ok &= ~1u;
        if (!inside(x, y0, 0, 2, nz)) ok &= ~2u;
        if (!inside(x, y0, nz - 1, 2, nz)) ok &= ~4u;
        if (!inside(x, y, z0, 1, ny)) ok &= ~8u;
    }
    // rotated grids: the physical axes (bits 0-2) whose difference is zero at the voxel's x and y
    // faces, then (bits 4-6, 8-10) at the first and the last slice; a probe that ends on the half
    // voxel depends on the coordinate along that axis alone (cc_args)
    unsigned int gone = 0;
    if (MODE == CC_ROTATED && own) {
        auto face = [&](int r, int n, int i, int j, int k) {
            unsigned int m = a.out[r];
            if (a.edge[r] < 3 && cc_probe_outside(a.g, i, j, k, a.edge[r], r, n)) m |= 1u << a.edge[r];
            return m;
        };
        if (x == 0 || x == nx - 1) gone |= face(0, nx, x, y0, z0);
        if (y == 0 || y == ny - 1) gone |= face(1, ny, x0, y, z0);
        gone |= face(2, nz, x0, y0, 0) << 4 | face(2, nz, x0, y0, nz - 1) << 8;
    }
    // analytic voxel count of the clamped window along x and y
    const int cxy = own ? (min(x + R, nx - 1) - max(x - R, 0) + 1) *
                              (min(y + R, ny - 1) - max(y - R, 0) + 1) : 1;
    int pcnt = 0;
    double icnt = 0.0;
    fetch(z0 + R);
    for (int z = z0; z < z1; ++z) {
        // the raw slice z + 1, then the z step: add slice k = z + R (if it exists), drop slice
        // k - 2R - 1 (if it was added)
        lo = cur;
        cur = hi;
        hi = nown;
        {
            float2* slot = raw + ((z + 1) & 3) * L::RXY;
            slot[oslot] = nown;
            if (tid < L::RING) slot[rslot] = nring;
        }
#pragma unroll
        for (int j = 0; j < L::CPT; ++j) {
            const float f = pin[j].x, m = pin[j].y, g = pout[j].x, n = pout[j].y;
            const int s = tid + j * L::NT;
            if (s < L::HC) {
                // four zeros change nothing (the sums of a zero background are left alone)
                if (((__float_as_uint(f) | __float_as_uint(m) | __float_as_uint(g) |
                      __float_as_uint(n)) << 1) != 0u) {
                    T* zq = zs + s;
                    if (f != 0.0f) lastf[j] = z + R;
                    if (m != 0.0f) lastm[j] = z + R;
                    T v0 = Acc::add(zq[0], Acc::diff(f, g));
                    T v1 = Acc::add(zq[L::HC], Acc::diff(m, n));
                    T v2 = Acc::add(zq[2 * L::HC], Acc::prod_diff(f, f, g, g));
                    T v3 = Acc::add(zq[3 * L::HC], Acc::prod_diff(m, m, n, n));
                    T v4 = Acc::add(zq[4 * L::HC], Acc::prod_diff(f, m, g, n));
                    if (min(lastf[j], lastm[j]) < z - R) {
                        if (lastf[j] < z - R) v0 = v2 = Acc::zero();
                        if (lastm[j] < z - R) v1 = v3 = Acc::zero();
                        v4 = Acc::zero();
                    }
                    zq[0] = v0;
                    zq[L::HC] = v1;
                    zq[2 * L::HC] = v2;
                    zq[3 * L::HC] = v3;
                    zq[4 * L::HC] = v4;
                }
                if constexpr (MK) zc[s] += (int)vin[j] - (int)vout[j];
            }
        }
        if (z + 1 < z1) {
            fetch(z + 1 + R);
            nown = voxel(z + 2, ocol);
            if (tid < L::RING) nring = voxel(z + 2, rcol);
        }
        __syncthreads();  // z sums visible; the previous x pass is done with the y sums
        // y pass: each item makes eight output rows of one halo column for one of the five window
        // sums; a warp's items are consecutive columns, so its loads and stores fall on distinct
        // banks
        if (tid < L::YI) {
            const int q = tid / L::HX, hx = tid - q * L::HX;
            const T* col = zs + q * L::HC + hx;
            T* o = xs + tid * L::YS;
            window_sums<Acc, R, TY>([&](int t) { return col[t * L::HX]; },
                                    [&](int j, T v) { o[j] = v; });
        }
        if constexpr (MK) {
            for (int s = tid; s < L::HX * TY; s += L::NT) {
                const int row = s / L::HX, hx = s - row * L::HX;
                int cn = 0;
#pragma unroll
                for (int t = 0; t <= 2 * R; ++t) cn += zc[(row + t) * L::HX + hx];
                xc[s] = cn;
            }
        }
        __syncthreads();
        // x pass: each item makes eight consecutive outputs of one row; a warp's items are the
        // rows of one column group, then of the next
        if (tid < L::XI) {
            const int q = tid / (TY * (TX / L::GX)), rr = tid - q * (TY * (TX / L::GX));
            const int row = rr % TY, g = rr / TY;
            const T* in = xs + (q * L::HX + g * L::GX) * L::YS + row;
            T* out = sx + (q * TX + g * L::GX) * L::YS + row;
            window_sums<Acc, R, L::GX>([&](int t) { return in[t * L::YS]; },
                                       [&](int j, T v) { out[j * L::YS] = v; });
        }
        __syncthreads();
        if (!own) continue;
        double S[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) S[q] = Acc::value(own_sums[q * TX * L::YS]);

        // ---- output voxel (x, y, z) ----
        const long long slice = (long long)z * sxy;
        float *pf = d_fixed + slice, *pm = d_moving + slice;
        double cnt;
        if constexpr (MK) {
            if (__ldg((vimg + slice) + ocol) == 0.0f) {
                pf[ocol] = (pf + a.ps)[ocol] = (pf + 2 * a.ps)[ocol] = 0.0f;
                pm[ocol] = (pm + a.ps)[ocol] = (pm + 2 * a.ps)[ocol] = 0.0f;
                continue;
            }
            int Sc = 0;
#pragma unroll
            for (int t = 0; t <= 2 * R; ++t) Sc += xc[ty * L::HX + tx + t];
            cnt = (double)Sc;  // >= 1: the centre is valid
            icnt = 1.0 / cnt;
            acc_nv += 1.0;
        } else {
            const int c = cxy * (min(z + R, nz - 1) - max(z - R, 0) + 1);
            cnt = (double)c;
            if (c != pcnt) {  // changes near the z faces only
                icnt = 1.0 / cnt;
                pcnt = c;
            }
        }
        const float2* cs = raw + (z & 3) * L::RXY + oslot;
        const float2 centre = MODE == CC_ROTATED ? cs[0] : cur;
        const float fv = centre.x, mv = centre.y;
        // metric/cc.rs:267-302 (same expression order)
        const double sum_f = S[0], sum_m = S[1], sum_f2 = S[2], sum_m2 = S[3], sum_fm = S[4];
        const double fmean = sum_f * icnt, mmean = sum_m * icnt;
        const double s_ff = sum_f2 - fmean * sum_f - fmean * sum_f + cnt * fmean * fmean;
        const double s_mm = sum_m2 - mmean * sum_m - mmean * sum_m + cnt * mmean * mmean;
        const double s_fm = sum_fm - mmean * sum_f - fmean * sum_m + cnt * mmean * fmean;
        const double fi = (double)fv - fmean, mi = (double)mv - mmean;
        const double product = s_ff * s_mm;
        double cc = 1.0, cf = 0.0, cm = 0.0;
        const bool prod_ok = fabs(product) > DBL_EPSILON;
        const bool coef_ok = s_ff > DBL_EPSILON && s_mm > DBL_EPSILON;  // implies product > 0
        // one reciprocal: 1 / sMM = sFF / product and 1 / sFF = sMM / product
        const double ip = (prod_ok || coef_ok) ? 1.0 / product : 0.0;
        if (prod_ok) cc = s_fm * s_fm * ip;
        if (coef_ok) {
            const double k2 = 2.0 * s_fm * ip;
            cf = k2 * (fi - s_fm * s_ff * ip * mi);  // (fixed, moving)
            cm = k2 * (mi - s_fm * s_mm * ip * fi);  // (moving, fixed)
        }
        acc_cc += cc;
        // gradients of moving (for the first direction) and of fixed (for the second)
        float gm[3], gf[3];
        if (MODE == CC_AXES || MODE == CC_AXES64) {
            // interp.rs:96-120 on an identity-direction grid: the probes at +-half a spacing lerp
            // halfway toward the neighbours along the axis. Upper probe at p + 0.5: lerp to p + 1
            // unless p is the last voxel; lower probe at p - 0.5: base p - 1 with weight 0.5, or
            // the first voxel itself (a face's missing neighbour is the voxel itself here)
            auto diff = [&](int d, bool in, float2 p, float2 q) {
                const float m2 = fmaf(q.y - mv, 0.5f, mv), m1 = fmaf(mv - p.y, 0.5f, p.y);
                const float f2 = fmaf(q.x - fv, 0.5f, fv), f1 = fmaf(fv - p.x, 0.5f, p.x);
                if (MODE == CC_AXES) {  // the float64 product of two floats is exact: one rounding either way
                    gm[d] = (m2 - m1) * a.ispf[d];
                    gf[d] = (f2 - f1) * a.ispf[d];
                } else {
                    gm[d] = (float)((double)(m2 - m1) * a.isp[d]);
                    gf[d] = (float)((double)(f2 - f1) * a.isp[d]);
                }
                if (!in) gm[d] = gf[d] = 0.0f;
            };
            diff(0, ok & 1u, cs[-1], cs[1]);
            diff(1, ok & 8u, cs[-L::RX], cs[L::RX]);
            diff(2, (z > 0 || (ok & 2u)) && (z < nz - 1 || (ok & 4u)), lo, hi);
        } else if (MODE == CC_ROTATED) {
            // a rotated grid: every probe's corners and weights are the same, and a corner outside the
            // buffer is the clamped ring's face voxel, which lin_axis reads there
            const unsigned int no = gone | (z == 0 ? gone >> 4 : 0u) | (z == nz - 1 ? gone >> 8 : 0u);
            const float2* below = raw + ((z - 1) & 3) * L::RXY + oslot;
            const float2* above = raw + ((z + 1) & 3) * L::RXY + oslot;
            float2 v[2];
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const float wx = a.weight[p][0], wy = a.weight[p][1], wz = a.weight[p][2];
                const int at = a.base[p][0] + L::RX * a.base[p][1];
                const int ox = wx > 0.0f ? 1 : 0, oy = wy > 0.0f ? L::RX : 0;
                const int slice = a.base[p][2];
                auto plane = [&](const float2* s) {
                    const float2 v00 = s[at], v10 = s[at + ox], v01 = s[at + oy], v11 = s[at + oy + ox];
                    const float fx0 = fmaf(v10.x - v00.x, wx, v00.x);
                    const float fx1 = fmaf(v11.x - v01.x, wx, v01.x);
                    const float mx0 = fmaf(v10.y - v00.y, wx, v00.y);
                    const float mx1 = fmaf(v11.y - v01.y, wx, v01.y);
                    return make_float2(fmaf(fx1 - fx0, wy, fx0), fmaf(mx1 - mx0, wy, mx0));
                };
                const float2 a0 = plane(slice < 0 ? below : (slice == 0 ? cs : above));
                v[p & 1] = a0;
                if (wz > 0.0f) {
                    const float2 a1 = plane(slice < 0 ? cs : above);
                    v[p & 1] = make_float2(fmaf(a1.x - a0.x, wz, a0.x), fmaf(a1.y - a0.y, wz, a0.y));
                }
                if (p & 1) {
                    gf[p >> 1] = (float)((double)(v[1].x - v[0].x) * a.isp[p >> 1]);
                    gm[p >> 1] = (float)((double)(v[1].y - v[0].y) * a.isp[p >> 1]);
                    if (no >> (p >> 1) & 1u) gf[p >> 1] = gm[p >> 1] = 0.0f;
                }
            }
        } else {
            cc_exact_gradients(fimg, mimg, a.g, x, y, z, gf, gm);
        }
        const float fcf = (float)cf, fcm = (float)cm;
        float dfx = fcf * gm[0], dfy = fcf * gm[1], dfz = fcf * gm[2];
        float dmx = fcm * gf[0], dmy = fcm * gf[1], dmz = fcm * gf[2];
        pf[ocol] = dfx;
        (pf + a.ps)[ocol] = dfy;
        (pf + 2 * a.ps)[ocol] = dfz;
        pm[ocol] = dmx;
        (pm + a.ps)[ocol] = dmy;
        (pm + 2 * a.ps)[ocol] = dmz;
        if (want_norms) {
            acc_nf += (double)dfx * dfx + (double)dfy * dfy + (double)dfz * dfz;
            acc_nm += (double)dmx * dmx + (double)dmy * dmy + (double)dmz * dmz;
        }
    }

    acc_out[0] = acc_cc;
    acc_out[1] = acc_nf;
    acc_out[2] = acc_nm;
    acc_out[3] = acc_nv;
}

// The block's sums of acc (NP of them) into dst[0 .. NP) (warp sums, then warps in order).
template <int NP, int NT>
__device__ __forceinline__ void cc_block_partials(double acc[4], double* red, double* dst) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int q = 0; q < NP; ++q) acc[q] = warp_sum_d(acc[q]);
    __syncthreads();
    if ((tid & 31) == 0) {
#pragma unroll
        for (int q = 0; q < NP; ++q) red[(tid >> 5) * NP + q] = acc[q];
    }
    __syncthreads();
    if (tid < NP) {
        double s = 0.0;
        for (int w = 0; w < NT / 32; ++w) s += red[w * NP + tid];
        dst[tid] = s;
    }
}

// Whether this block is the last of `total` to add its partials (fixed-order reduction).
__device__ __forceinline__ bool cc_last(unsigned int* counter, unsigned int total) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == total - 1;
    __syncthreads();
    return last;
}

// The last block's reduction of `nblocks` partials in a fixed order (every thread of the block,
// block_sum_fixed): [value, |dF|^2, |dM|^2 (, valid voxels)] into result; the counter is reset.
// `red` is the block's shared reduction space (NT / 32 doubles at least).
template <int NP, bool MK>
__device__ __forceinline__ void cc_finish(const double* partials, unsigned int nblocks,
                                          long long n, double* result, unsigned int* counter,
                                          double* red) {
    double tot[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < NP; ++q) tot[q] = block_sum_fixed(partials + q, nblocks, NP, red);
    if (threadIdx.x == 0) {
        // the mean over the valid voxels (all voxels without a mask); no valid voxel: NaN
        result[0] = -tot[0] / (MK ? tot[3] : (double)n);
        result[1] = tot[1];
        result[2] = tot[2];
        if constexpr (MK) result[3] = tot[3];
        *counter = 0;
    }
}

template <int R, int TY, bool MK, int MODE, class Acc = SumF64>
__global__ void __launch_bounds__(CC_NT, CC_MIN_BLOCKS) k_cc_pair(const __grid_constant__ CcArgs a, const float* __restrict__ fimg,
                                                     const float* __restrict__ mimg,
                                                     const float* __restrict__ vimg,
                                                     float* __restrict__ d_fixed,
                                                     float* __restrict__ d_moving,
                                                     double* __restrict__ partials,
                                                     unsigned int* __restrict__ counter,
                                                     double* __restrict__ result, int want_norms) {
    pdl_wait();
    using L = Layout<R, TY, MK>;
    extern __shared__ __align__(16) unsigned char smem[];
    double* red = reinterpret_cast<double*>(smem + L::red_off);
    double acc[4];
    cc_tile<R, TY, MK, MODE, Acc>(a, blockIdx.x, blockIdx.y, blockIdx.z, smem, fimg, mimg, vimg,
                            d_fixed, d_moving, want_norms, acc);
    // block partials, then the fixed-order last-block reduction
    const unsigned int nblocks = gridDim.x * gridDim.y * gridDim.z;
    const unsigned int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    cc_block_partials<L::NP, L::NT>(acc, red, partials + (size_t)bid * L::NP);
    if (!cc_last(counter, nblocks)) return;
    cc_finish<L::NP, MK>(partials, nblocks, a.g.n, result, counter, red);
}

// The CC pair of every active subject of a batch (unmasked): subject b's images at
// fimg / mimg + b * img_stride, its derivative fields at d_fixed / d_moving + b * field_stride,
// its tile partials at partials + b * part_stride, its last-tile counter at counter[b] and its
// [value, |dF|^2, |dM|^2] at result + b * result_stride. Tiles are summed in the single
// kernel's block order, so a subject's value does not depend on the batch.
template <int R, int TY, int MODE>
__global__ void __launch_bounds__(CC_NT, CC_MIN_BLOCKS) k_cc_pair_batch(
    const __grid_constant__ CcArgs a, BatchList Lb, const float* __restrict__ fimg, const float* __restrict__ mimg,
    long long img_stride, float* __restrict__ d_fixed, float* __restrict__ d_moving,
    long long field_stride, double* __restrict__ partials, long long part_stride,
    unsigned int* __restrict__ counter, double* __restrict__ result, int result_stride,
    int want_norms) {
    using L = Layout<R, TY, false>;
    extern __shared__ __align__(16) unsigned char smem[];
    double* red = reinterpret_cast<double*>(smem + L::red_off);
    const int work = *Lb.count * Lb.tiles;
    const int gx = (a.g.nx + TX - 1) / TX, gy = (a.g.ny + TY - 1) / TY;
    for (int w = blockIdx.x; w < work; w += gridDim.x) {
        const int b = Lb.active[w / Lb.tiles], t = w % Lb.tiles;
        int bx, by, bz;
        tile_coords(t, gx, gy, bx, by, bz);
        double acc[4];
        cc_tile<R, TY, false, MODE>(a, bx, by, bz, smem, fimg + b * img_stride, mimg + b * img_stride,
                              nullptr, d_fixed + b * field_stride, d_moving + b * field_stride,
                              want_norms, acc);
        double* pb = partials + b * part_stride;
        cc_block_partials<L::NP, L::NT>(acc, red, pb + (size_t)t * L::NP);
        if (cc_last(counter + b, (unsigned int)Lb.tiles))
            cc_finish<L::NP, false>(pb, (unsigned int)Lb.tiles, a.g.n,
                                    result + (size_t)b * result_stride, counter + b, red);
        __syncthreads();  // the next tile rewrites the shared sums
    }
}

// Grid of a launch: TX x TY column tiles times z chunks. About three and a half waves of resident
// CTAs (measured at the 193 x 229 x 193 finest level, r = 4: 8 chunks 0.287 ms, 5 chunks 0.303, 12
// chunks 0.301, 1 chunk 0.426), with chunks no thinner than 2R slices, the filling steps every chunk
// pays before its first output -- except where that leaves resident slots empty (the coarse levels),
// where chunks go down to 4 slices: at 48 x 57 x 48 the kernel takes 26 us with 5 chunks, 19 with 12, 17
// with 16 or 24, and an iteration 116 us with chunks of 8 slices, 110 with 4 or 3, 112 with 2.
template <int R, int TY, bool MK, int MODE, class Acc = SumF64>
int plan_launch(CcArgs& a, int num_sms, dim3* grid) {
    using L = Layout<R, TY, MK>;
    FW_CUDA(cudaFuncSetAttribute(k_cc_pair<R, TY, MK, MODE, Acc>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::bytes));
    static const int occ = [] {
        int o = 1;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_cc_pair<R, TY, MK, MODE, Acc>, L::NT,
                                                          L::bytes) != cudaSuccess || o < 1)
            o = 1;
        return o;
    }();
    dim3 g((a.g.nx + TX - 1) / TX, (a.g.ny + TY - 1) / TY, 1);
    const long long tiles = (long long)g.x * g.y;
    const long long slots = (long long)occ * num_sms;
    long long best = (7 * slots + tiles) / (2 * tiles);  // round(3.5 slots / tiles)
    best = std::min<long long>(best, a.g.nz / (2 * R));
    if (best * tiles < slots)
        best = std::max<long long>(best, std::min<long long>(slots / tiles, a.g.nz / 4));
    best = std::max<long long>(best, 1);
    a.zchunk = (int)((a.g.nz + best - 1) / best);
    g.z = (a.g.nz + a.zchunk - 1) / a.zchunk;
    *grid = g;
    return 0;
}

template <int R, int TY, bool MK, int MODE, class Acc = SumF64>
int launch_r(fw_ctx* ctx, const CcArgs& a0, const float* f, const float* m, const float* v,
             float* df, float* dm, double* d_result, int want_norms) {
    using L = Layout<R, TY, MK>;
    CcArgs a = a0;
    dim3 grid;
    FW_TRY((plan_launch<R, TY, MK, MODE, Acc>(a, ctx->num_sms, &grid)));
    unsigned int nblocks = grid.x * grid.y * grid.z;
    FW_TRY(ensure_scratch(ctx, SLOT_PARTIALS + (size_t)L::NP * nblocks + 16));
    return launch_pdl(ctx, "k_cc_pair", k_cc_pair<R, TY, MK, MODE, Acc>, grid, dim3(L::NT), L::bytes,
                      a, f, m, v, df, dm, ctx->d_scratch + SLOT_PARTIALS, ctx->d_counter + 1,
                      d_result, want_norms);
}

// The window-sum arithmetic of the unmasked single-image CC pair (FW_CC_SUMS_*), process-wide.
std::atomic<int> g_cc_sums{FW_CC_SUMS_F64};

template <bool MK>
int launch_radius(fw_ctx* ctx, const CcArgs& a, int radius, const float* f, const float* m,
                  const float* v, float* df, float* dm, double* d_result, int want_norms) {
    const bool c32 = !MK && g_cc_sums.load() == FW_CC_SUMS_C32;
#define FW_CC_RADIUS(RR)                                                                         \
    case RR:                                                                                    \
        if constexpr (!MK)                                                                      \
            if (c32)                                                                            \
                return (a.mode == CC_EXACT     ? launch_r<RR, CC_TY, false, CC_EXACT, SumC32>   \
                        : a.mode == CC_ROTATED ? launch_r<RR, CC_TY, false, CC_ROTATED, SumC32> \
                                               : launch_r<RR, CC_TY, false, CC_AXES64, SumC32>)(\
                    ctx, a, f, m, v, df, dm, d_result, want_norms);                             \
        return (a.mode == CC_AXES      ? launch_r<RR, CC_TY, MK, CC_AXES>                       \
                : a.mode == CC_AXES64  ? launch_r<RR, CC_TY, MK, CC_AXES64>                     \
                : a.mode == CC_ROTATED ? launch_r<RR, CC_TY, MK, CC_ROTATED>                    \
                                       : launch_r<RR, CC_TY, MK, CC_EXACT>)(                    \
            ctx, a, f, m, v, df, dm, d_result, want_norms);
    switch (radius) {
        FW_CC_RADIUS(1)
        FW_CC_RADIUS(2)
        FW_CC_RADIUS(3)
        FW_CC_RADIUS(4)
        FW_CC_RADIUS(5)
        FW_CC_RADIUS(6)
        FW_CC_RADIUS(7)
        FW_CC_RADIUS(8)
        default:
            return fail(FW_ERR_INVALID, "cc metric: radius must be in 1..=8 (BOX_RADIUS_MAX)");
    }
#undef FW_CC_RADIUS
}

template <int R, int MODE>
int launch_cc_batch_r(fw_ctx* ctx, const CcArgs& a, const BatchList& L, int blocks,
                      const float* f, const float* m, long long img_stride, float* df, float* dm,
                      long long field_stride, double* partials, long long part_stride,
                      unsigned int* counter, double* result, int result_stride, int want_norms) {
    using Lay = Layout<R, CC_TY, false>;
    FW_CUDA(cudaFuncSetAttribute(k_cc_pair_batch<R, CC_TY, MODE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes));
    k_cc_pair_batch<R, CC_TY, MODE><<<blocks, Lay::NT, Lay::bytes, ctx->stream>>>(
        a, L, f, m, img_stride, df, dm, field_stride, partials, part_stride, counter, result,
        result_stride, want_norms);
    return check_launch(ctx, "k_cc_pair_batch");
}

template <int R>
int cc_batch_occupancy() {
    using Lay = Layout<R, CC_TY, false>;
    int o = 1;
    if (cudaFuncSetAttribute(k_cc_pair_batch<R, CC_TY, CC_AXES>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)Lay::bytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_cc_pair_batch<R, CC_TY, CC_AXES>, Lay::NT,
                                                      Lay::bytes) != cudaSuccess || o < 1) {
        cudaGetLastError();
        o = 1;
    }
    return o;
}

CcArgs cc_args(const HostGrid& g, long long ps) {
    CcArgs a;
    std::memset(&a, 0, sizeof(a));
    a.g = dev_grid(g);
    a.ps = ps;
    for (int d = 0; d < 3; ++d) {
        a.isp[d] = 1.0 / g.sp[d];
        a.ispf[d] = (float)a.isp[d];
    }
    bool identity = true;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c)
            if (g.dir[r * 3 + c] != (r == c ? 1.0 : 0.0)) identity = false;
    const bool exact = (double)a.ispf[0] == a.isp[0] && (double)a.ispf[1] == a.isp[1] &&
                       (double)a.ispf[2] == a.isp[2];
    bool stencil = !identity;
    // How far rounding can move a probe's index: a few float64 units of the largest coordinate in
    // voxels (and no less than 1e-9).
    double reach = 0.0, least = g.sp[0];
    for (int d = 0; d < 3; ++d) {
        reach = std::max(reach, std::fabs(g.org[d]));
        least = std::min(least, g.sp[d]);
    }
    for (int d = 0; d < 3; ++d) reach += (double)g.n[d] * g.sp[d];
    const double slack = std::max(1e-9, 256.0 * DBL_EPSILON * reach / least);
    for (int r = 0; r < 3; ++r) {
        a.edge[r] = 3;
        for (int d = 0; d < 3; ++d) {
            const double h = 0.5 * g.sp[d] * std::fabs(g.inv[r * 3 + d]);
            if (h > 0.5 + slack) {
                a.out[r] |= (unsigned char)(1u << d);
            } else if (h >= 0.5 - slack) {
                // on the half voxel: decided once a column, if index r follows physical axis d alone
                // and d index r alone (the other terms of the probe's index are exact zeros)
                bool alone = a.edge[r] == 3;
                for (int q = 0; q < 3; ++q) {
                    if (q != d && g.inv[r * 3 + q] != 0.0) alone = false;
                    if (q != r && g.dir[d * 3 + q] != 0.0) alone = false;
                }
                if (alone) a.edge[r] = (unsigned char)d;
                else stencil = false;
            }
        }
    }
    for (int p = 0; p < 6; ++p)
        for (int r = 0; r < 3; ++r) {
            // index offset along axis r of the probe along physical axis p / 2
            const double h = (p & 1 ? 0.5 : -0.5) * g.sp[p / 2] * g.inv[r * 3 + p / 2];
            double base = std::floor(h), w = h - base;
            // within rounding of a voxel: that voxel (a probe's own rounding is this large)
            if (w > 1.0 - 1e-12) {
                base += 1.0;
                w = 0.0;
            } else if (w < 1e-12) {
                w = 0.0;
            }
            if (!(base >= -1.0 && base + (w > 0.0 ? 1.0 : 0.0) <= 1.0)) stencil = false;
            else {
                a.base[p][r] = (signed char)base;
                a.weight[p][r] = (float)w;
            }
        }
    a.mode = identity ? (exact ? CC_AXES : CC_AXES64) : (stencil ? CC_ROTATED : CC_EXACT);
    return a;
}

}  // namespace

int cc_batch_tiles(const HostGrid& g, int zchunk) {
    const long long gx = (g.n[0] + TX - 1) / TX, gy = (g.n[1] + CC_TY - 1) / CC_TY;
    const long long gz = (g.n[2] + zchunk - 1) / zchunk;
    return (int)(gx * gy * gz);
}

int cc_batch_blocks_per_sm(int radius) {
    switch (radius) {
        case 1: return cc_batch_occupancy<1>();
        case 2: return cc_batch_occupancy<2>();
        case 3: return cc_batch_occupancy<3>();
        case 4: return cc_batch_occupancy<4>();
        case 5: return cc_batch_occupancy<5>();
        case 6: return cc_batch_occupancy<6>();
        case 7: return cc_batch_occupancy<7>();
        case 8: return cc_batch_occupancy<8>();
        default: return 1;
    }
}

int launch_cc_pair_batch(fw_ctx* ctx, const HostGrid& g, long long ps, int radius, int zchunk,
                         const BatchList& L, int blocks, const float* fimg, const float* mimg,
                         long long img_stride, float* d_fixed, float* d_moving,
                         long long field_stride, double* partials, long long part_stride,
                         unsigned int* counter, double* result, int result_stride,
                         int want_norms) {
    CcArgs a = cc_args(g, ps);
    a.zchunk = zchunk;
#define FW_CC_BATCH(RR)                                                                          \
    case RR:                                                                                    \
        return (a.mode == CC_AXES      ? launch_cc_batch_r<RR, CC_AXES>                         \
                : a.mode == CC_AXES64  ? launch_cc_batch_r<RR, CC_AXES64>                       \
                : a.mode == CC_ROTATED ? launch_cc_batch_r<RR, CC_ROTATED>                      \
                                       : launch_cc_batch_r<RR, CC_EXACT>)(                      \
            ctx, a, L, blocks, fimg, mimg, img_stride, d_fixed, d_moving, field_stride,         \
            partials, part_stride, counter, result, result_stride, want_norms);
    switch (radius) {
        FW_CC_BATCH(1)
        FW_CC_BATCH(2)
        FW_CC_BATCH(3)
        FW_CC_BATCH(4)
        FW_CC_BATCH(5)
        FW_CC_BATCH(6)
        FW_CC_BATCH(7)
        FW_CC_BATCH(8)
        default:
            return fail(FW_ERR_INVALID, "cc metric: radius must be in 1..=8 (BOX_RADIUS_MAX)");
    }
#undef FW_CC_BATCH
}

// d_result receives [value, sum |d_fixed|^2, sum |d_moving|^2] and, with `valid`, the number of
// valid voxels in d_result[3].
int launch_cc_pair_impl(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving, int radius,
                        fw_field* d_fixed, fw_field* d_moving, double* d_result, int want_norms,
                        const fw_image* valid) {
    CcArgs a = cc_args(fixed->grid, d_fixed->ps);
    if (valid)
        return launch_radius<true>(ctx, a, radius, fixed->d, moving->d, valid->d, d_fixed->d,
                                   d_moving->d, d_result, want_norms);
    return launch_radius<false>(ctx, a, radius, fixed->d, moving->d, nullptr, d_fixed->d,
                                d_moving->d, d_result, want_norms);
}

int launch_cc_pair(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving, int radius,
                   fw_field* d_fixed, fw_field* d_moving, double* d_value, double* d_norms) {
    (void)d_norms;
    return launch_cc_pair_impl(ctx, fixed, moving, radius, d_fixed, d_moving, d_value,
                               d_norms != nullptr);
}

}  // namespace fw

using namespace fw;

extern "C" {

static int cc_pair_common(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                          const fw_image* valid, int32_t radius, double values[2],
                          fw_field** d_fixed, fw_field** d_moving, double norms[2]) {
    FW_CHECK(ctx && fixed && moving && values && d_fixed && d_moving, "null argument");
    if (!fixed->grid.same(moving->grid))
        return fail(FW_ERR_INVALID, "cc metric: the images are not on one grid");
    if (valid && !valid->grid.same(fixed->grid))
        return fail(FW_ERR_INVALID, "cc metric: the mask is not on the virtual grid");
    // the scratch grows before the result's place in it is taken (at most one block a column tile,
    // or four waves of them: plan_launch)
    const long long tiles = ((fixed->grid.n[0] + TX - 1) / TX) * ((fixed->grid.n[1] + CC_TY - 1) / CC_TY);
    FW_TRY(ensure_scratch(ctx, SLOT_PARTIALS + 4 * (size_t)(tiles + 32LL * ctx->num_sms) + 16));
    fw_field *a = nullptr, *b = nullptr;
    FW_TRY(new_field(ctx, fixed->grid, &a));
    int rc = new_field(ctx, fixed->grid, &b);
    if (rc) {
        fw_field_free(a);
        return rc;
    }
    // [value, nf, nm, valid voxels] at SLOT_CC_VALUE .. SLOT_CC_VALID
    double* slot = ctx->d_scratch + SLOT_CC_VALUE;
    rc = launch_cc_pair_impl(ctx, fixed, moving, radius, a, b, slot, 1, valid);
    double r[4] = {0, 0, 0, 0};
    if (!rc) rc = read_back(ctx, slot, valid ? 4 : 3, r);
    if (!rc && valid && r[3] == 0.0) rc = fail(FW_ERR_INVALID, std::string("cc metric: ") + FW_NO_VOXEL_IN_MASKS);
    if (rc) {
        fw_field_free(a);
        fw_field_free(b);
        return rc;
    }
    values[0] = r[0];
    values[1] = r[0];
    if (norms) {
        norms[0] = std::sqrt(r[1]);
        norms[1] = std::sqrt(r[2]);
    }
    *d_fixed = a;
    *d_moving = b;
    return 0;
}

int fw_cc_value_derivative_pair(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                                int32_t radius, double values[2], fw_field** d_fixed,
                                fw_field** d_moving) {
    return cc_pair_common(ctx, fixed, moving, nullptr, radius, values, d_fixed, d_moving, nullptr);
}

int fw_cc_value_derivative_pair_with_norms(fw_ctx* ctx, const fw_image* fixed,
                                           const fw_image* moving, int32_t radius,
                                           double values[2], fw_field** d_fixed,
                                           fw_field** d_moving, double norms[2]) {
    FW_CHECK(norms, "null norms");
    return cc_pair_common(ctx, fixed, moving, nullptr, radius, values, d_fixed, d_moving, norms);
}

int fw_cc_value_derivative_pair_masked(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                                       const fw_image* valid, int32_t radius, double values[2],
                                       fw_field** d_fixed, fw_field** d_moving) {
    FW_CHECK(valid, "null mask");
    return cc_pair_common(ctx, fixed, moving, valid, radius, values, d_fixed, d_moving, nullptr);
}

int fw_cc_value_derivative_pair_masked_with_norms(fw_ctx* ctx, const fw_image* fixed,
                                                  const fw_image* moving, const fw_image* valid,
                                                  int32_t radius, double values[2],
                                                  fw_field** d_fixed, fw_field** d_moving,
                                                  double norms[2]) {
    FW_CHECK(valid && norms, "null argument");
    return cc_pair_common(ctx, fixed, moving, valid, radius, values, d_fixed, d_moving, norms);
}

int fw_set_cc_window_sums(int32_t kind) {
    FW_CHECK(kind == FW_CC_SUMS_F64 || kind == FW_CC_SUMS_C32,
             "cc metric: unknown window-sum arithmetic");
    g_cc_sums.store(kind);
    return 0;
}

int fw_cc_value_derivative(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving,
                           int32_t radius, double* value, fw_field** derivative) {
    FW_CHECK(value && derivative, "null argument");
    double v[2];
    fw_field *a = nullptr, *b = nullptr;
    FW_TRY(cc_pair_common(ctx, fixed, moving, nullptr, radius, v, &a, &b, nullptr));
    fw_field_free(b);
    *value = v[0];
    *derivative = a;
    return 0;
}

}  // extern "C"

// ---- allocation-free variant of the CC pair ---------------------------------------------------
//
// For callers that cannot allocate device memory: hosts that hand every byte of the GPU to
// their own pool allocator (a deep-learning framework's caching allocator, a serving process
// with a fixed HBM budget), plug-ins that get only the buffers such a host gives them, and
// real-time pipelines that plan all memory before they start. The
// caller passes the images, the two derivative fields and a 3-double result on the device; the
// kernel's only scratch -- the block partials and the last-block counter -- lives in the
// file-scope array below, which every GPU that loads this library holds until the process exits.

namespace fw {
namespace {

struct NoAllocScratch {
    double partials[3 * FW_NOALLOC_MAX_BLOCKS];
    unsigned int counter[64];
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

std::mutex g_noalloc_mu;
NoAllocScratch* g_noalloc_ptr[128] = {};

// The array's device address on `device` (current), looked up once per device: in host code the
// symbol is only a host-side stand-in, not an address a kernel may use.
int noalloc_scratch(int device, NoAllocScratch** out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (device < 0 || device >= 128) return fail(FW_ERR_INVALID, "cc pair (no alloc): device index out of range");
    if (!g_noalloc_ptr[device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[device] = static_cast<NoAllocScratch*>(p);
    }
    *out = g_noalloc_ptr[device];
    return 0;
}

template <int R, int TY, int MODE>
int noalloc_launch(const CcArgs& a0, int num_sms, const float* f, const float* m, float* df,
                   float* dm, double* result, NoAllocScratch* s, cudaStream_t stream) {
    using L = Layout<R, TY, false>;
    CcArgs a = a0;
    dim3 grid;
    FW_TRY((plan_launch<R, TY, false, MODE>(a, num_sms, &grid)));
    long long nblocks = (long long)grid.x * grid.y * grid.z;
    if (nblocks > FW_NOALLOC_MAX_BLOCKS)
        return fail(FW_ERR_INVALID,
                    "cc pair (no alloc): the grid needs " + std::to_string(nblocks) +
                        " thread blocks, more than the " + std::to_string(FW_NOALLOC_MAX_BLOCKS) +
                        " the static scratch holds (use fw_cc_value_derivative_pair)");
    // the last-block counter must start at zero whatever the previous call left
    FW_CUDA(cudaMemsetAsync(s->counter, 0, sizeof(unsigned int), stream));
    k_cc_pair<R, TY, false, MODE><<<grid, L::NT, L::bytes, stream>>>(a, f, m, nullptr, df, dm,
                                                                s->partials, s->counter, result, 1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "k_cc_pair (no alloc)");
    return 0;
}

}  // namespace
}  // namespace fw

extern "C" int fw_cc_value_derivative_pair_noalloc(const fw_grid* grid, const float* fixed,
                                                   const float* moving, int32_t radius,
                                                   float* d_fixed, float* d_moving,
                                                   int64_t plane_stride, double* result,
                                                   void* stream) {
    FW_CHECK(grid && fixed && moving && d_fixed && d_moving && result, "null argument");
    HostGrid g;
    FW_TRY(make_grid(grid, g));
    FW_CHECK(plane_stride >= g.count(), "cc pair (no alloc): plane stride below the voxel count");
    int device = 0;
    FW_CUDA(cudaGetDevice(&device));
    int num_sms = 0;
    FW_CUDA(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device));
    NoAllocScratch* s = nullptr;
    FW_TRY(noalloc_scratch(device, &s));
    const CcArgs a = cc_args(g, plane_stride);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define FW_CC_NOALLOC(RR)                                                                        \
    case RR:                                                                                    \
        return (a.mode == CC_AXES      ? noalloc_launch<RR, CC_TY, CC_AXES>                     \
                : a.mode == CC_AXES64  ? noalloc_launch<RR, CC_TY, CC_AXES64>                   \
                : a.mode == CC_ROTATED ? noalloc_launch<RR, CC_TY, CC_ROTATED>                  \
                                       : noalloc_launch<RR, CC_TY, CC_EXACT>)(                  \
            a, num_sms, fixed, moving, d_fixed, d_moving, result, s, st);
    switch (radius) {
        FW_CC_NOALLOC(1)
        FW_CC_NOALLOC(2)
        FW_CC_NOALLOC(3)
        FW_CC_NOALLOC(4)
        FW_CC_NOALLOC(5)
        FW_CC_NOALLOC(6)
        FW_CC_NOALLOC(7)
        FW_CC_NOALLOC(8)
        default:
            return fail(FW_ERR_INVALID, "cc metric: radius must be in 1..=8 (BOX_RADIUS_MAX)");
    }
#undef FW_CC_NOALLOC
}
