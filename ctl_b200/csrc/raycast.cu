// Cone-beam ray casting kernels (sm_100a).
//
// One thread per detector pixel; a block covers one detector tile of a few
// neighbouring views of one module, each warp a small pixel patch of one view
// (LaunchShape, chosen per call).  Per ray, in FP64: direction
// A*[x,y,1] normalised and scaled to one step in voxel units, entry/exit
// parameters against the (half-voxel padded) volume box with the 0.01-voxel
// face tolerance, first/last sample index.  The sample loop then runs in FP32
// on positions rebased at the first sample, so their magnitude is bounded by
// the volume extent rather than the source distance.
//
// Reference: modules/src/ocl/cl_src/projectors/raycasterprojector_interp.cl:18-148
// (trilinear, image3d_t + CLK_FILTER_LINEAR + CLK_ADDRESS_CLAMP) and
// raycasterprojector_no_interp.cl:16-154 (nearest voxel), launched per view
// over (channels, rows, modules) by raycasterprojector.cpp:339-343.  Here all
// views of a call go in one launch.
//
// Sampling scheme (identical to the reference): sample i sits at
// source + i*step for i = floor(tmin) .. floor(tmax)+1, tmin/tmax clamped at
// 0; a ray that hits no face takes no samples; the result is
// increment * sum / raysPerPixel.  Samples outside the padded box read zeros.
#include "internal.cuh"

#include <algorithm>
#include <cfloat>

namespace ctlcu {

namespace {

template <typename T>
__device__ __forceinline__ float load_voxel(const T* p);

template <>
__device__ __forceinline__ float load_voxel<float>(const float* p)
{
    return __ldg(p);
}
template <>
__device__ __forceinline__ float load_voxel<__nv_bfloat16>(const __nv_bfloat16* p)
{
    const unsigned short u = __ldg(reinterpret_cast<const unsigned short*>(p));
    return __uint_as_float(static_cast<unsigned int>(u) << 16);
}
template <>
__device__ __forceinline__ float load_voxel<__half>(const __half* p)
{
    const unsigned short u = __ldg(reinterpret_cast<const unsigned short*>(p));
    return __half2float(__ushort_as_half(u));
}

template <Accum A>
struct Accumulator;

// add: one FP32 value.  add_product: m samples of v; FP64 takes the product exactly, the
// others collect it in `part`, an FP32 sum of a few products, which flush hands on.
template <>
struct Accumulator<Accum::F64> {
    double s = 0.0;
    __device__ __forceinline__ void add(float v) { s += static_cast<double>(v); }
    __device__ __forceinline__ void add_product(float m, float v)
    {
        s = fma(static_cast<double>(m), static_cast<double>(v), s);
    }
    __device__ __forceinline__ void add_product(float m, float v, float&) { add_product(m, v); }
    __device__ __forceinline__ void flush(float) {}
    __device__ __forceinline__ double value() const { return s; }
};

template <>
struct Accumulator<Accum::Kahan> {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float v)
    {
        const float y = v - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ void add_product(float m, float v, float& part) { part = fmaf(m, v, part); }
    __device__ __forceinline__ void flush(float part) { add(part); }
    // the compensation still holds what the last additions rounded off s
    __device__ __forceinline__ double value() const { return static_cast<double>(s) - static_cast<double>(c); }
};

template <>
struct Accumulator<Accum::F32> {
    float s = 0.0f;
    __device__ __forceinline__ void add(float v) { s += v; }
    __device__ __forceinline__ void add_product(float m, float v, float& part) { part = fmaf(m, v, part); }
    __device__ __forceinline__ void flush(float part) { add(part); }
    __device__ __forceinline__ double value() const { return static_cast<double>(s); }
};

// One ray ready for the sample loop.  The cell, segment, pair and trilinear loops run in
// FP32 relative to the ray's integer origin (CellFrame); the texture loop runs
// from the rounded absolute base, its 8-bit filter weights being far coarser; the
// nearest-voxel loop takes every sample's voxel from FP64 positions, or from FP32
// ones that cannot differ (march_nearest).
struct Ray {
    double base[3];  // coordinate of the first sample in the loop's index space
    double step[3];  // one step in voxel units
    int n;           // number of samples (0: the ray misses)
    int first;       // index of the first sample
};

// Face test of raycasterprojector_interp.cl:136-148.
__device__ __forceinline__ void check_face(double h0, double h1, double lo0, double lo1, double hi0,
                                           double hi1, double lambda, double& tmin, double& tmax)
{
    const bool inside = (h0 >= lo0) && (h1 >= lo1) && (h0 <= hi0) && (h1 <= hi1);
    if (inside && lambda < tmin)
        tmin = lambda;
    if (inside && lambda > tmax)
        tmax = lambda;
}

// FP64 ray setup for detector coordinate (px, py).  `shift` is added to the
// rebased first-sample position to map it into the loop's index space.
template <Mode M>
__device__ __forceinline__ Ray setup_ray(const ProjectArgs& a, const ViewGeom& g, double px, double py,
                                         int* flags)
{
    Ray r;
    double d0 = g.A[0] * px + g.A[1] * py + g.A[2];
    double d1 = g.A[3] * px + g.A[4] * py + g.A[5];
    double d2 = g.A[6] * px + g.A[7] * py + g.A[8];
    const double nrm = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    d0 = d0 / nrm * (a.increment / a.voxel[0]);
    d1 = d1 / nrm * (a.increment / a.voxel[1]);
    d2 = d2 / nrm * (a.increment / a.voxel[2]);
    const double s0 = g.src[0] / a.voxel[0], s1 = g.src[1] / a.voxel[1], s2 = g.src[2] / a.voxel[2];
    const double k0 = a.corner[0] / a.voxel[0], k1 = a.corner[1] / a.voxel[1],
                 k2 = a.corner[2] / a.voxel[2];
    const double pad = (M == Mode::Nearest || M == Mode::NearestSamples) ? 0.0 : 0.5;
    const double c10 = k0 - pad, c11 = k1 - pad, c12 = k2 - pad;
    const double c20 = k0 + a.grid[0] + pad, c21 = k1 + a.grid[1] + pad, c22 = k2 + a.grid[2] + pad;
    const double l10 = (c10 - s0) / d0, l11 = (c11 - s1) / d1, l12 = (c12 - s2) / d2;
    const double l20 = (c20 - s0) / d0, l21 = (c21 - s1) / d1, l22 = (c22 - s2) / d2;
    const double e = 0.01;
    double tmin = DBL_MAX, tmax = 0.0;
    check_face(s1 + l10 * d1, s2 + l10 * d2, c11 - e, c12 - e, c21 + e, c22 + e, l10, tmin, tmax);
    check_face(s0 + l11 * d0, s2 + l11 * d2, c10 - e, c12 - e, c20 + e, c22 + e, l11, tmin, tmax);
    check_face(s0 + l12 * d0, s1 + l12 * d1, c10 - e, c11 - e, c20 + e, c21 + e, l12, tmin, tmax);
    check_face(s1 + l20 * d1, s2 + l20 * d2, c11 - e, c12 - e, c21 + e, c22 + e, l20, tmin, tmax);
    check_face(s0 + l21 * d0, s2 + l21 * d2, c10 - e, c12 - e, c20 + e, c22 + e, l21, tmin, tmax);
    check_face(s0 + l22 * d0, s1 + l22 * d1, c10 - e, c11 - e, c20 + e, c21 + e, l22, tmin, tmax);
    r.n = 0;
    r.first = 0;
    if (tmin == DBL_MAX) {
        r.base[0] = r.base[1] = r.base[2] = 0.0;
        r.step[0] = r.step[1] = r.step[2] = 0.0;
        return r;
    }
    const double t0 = fmax(tmin, 0.0), t1 = fmax(tmax, 0.0);
    // the box diagonal bounds any honest ray; beyond it the inputs are broken
    if (!(t1 - t0 < 1.0e7) || !isfinite(t0)) {
        if (flags)
            atomicOr(flags, kFlagNonFinite);
        r.n = 0;
        r.base[0] = r.base[1] = r.base[2] = 0.0;
        r.step[0] = r.step[1] = r.step[2] = 0.0;
        return r;
    }
    const double i0 = floor(t0), i1 = floor(t1) + 1.0;
    r.n = static_cast<int>(i1 - i0) + 1;
    r.first = static_cast<int>(fmin(i0, 1.0e9));
    // position relative to the corner: (source - corner) + i * step
    double shift;
    if (M == Mode::Trilinear)
        shift = (a.up == 1) ? (kPad - 0.5) : -0.5;  // taps at floor(p - 0.5) (+ pad)
    else if (M == Mode::Nearest || M == Mode::NearestSamples)
        shift = kPad;                                // voxel floor(p) (+ pad)
    else
        shift = 0.0;                                 // texture: hardware subtracts 0.5
    r.base[0] = (s0 - k0) + i0 * d0 + shift;
    r.base[1] = (s1 - k1) + i0 * d1 + shift;
    r.base[2] = (s2 - k2) + i0 * d2 + shift;
    r.step[0] = d0;
    r.step[1] = d1;
    r.step[2] = d2;
    return r;
}

// The same for the loops over derived arrays (Cells, Segments, their up-sampled forms, Pairs).
// Outside the box, padded by half a voxel, samples read zeros, so these loops run
// over ceil(t0) .. floor(t1) of the slab intersection, which holds every sample that
// the face tests above let in and that is not zero.  Lengths are in grid voxels from
// the box's low corner; the host's scale, inv_voxel and corner_v leave one reciprocal
// square root and three reciprocals of the 18 divisions above (64^3 -> 90 x 128^2:
// 311 -> 299 us; 201x173x155 -> 23 x 479 x 361: 2.03 -> 1.95 ms).  Coordinates are
// v = p - 1 + pad: the cell index is rint(v), the offset from the cell centre v - rint(v).
template <Mode M>
__device__ __forceinline__ Ray setup_ray_cells(const ProjectArgs& a, const ViewGeom& g, double px, double py,
                                               int* flags)
{
    Ray r;
    r.n = 0;
    r.first = 0;
    double d[3], s[3];
    for (int i = 0; i < 3; ++i)
        d[i] = fma(g.A[3 * i], px, fma(g.A[3 * i + 1], py, g.A[3 * i + 2]));
    const double rn = rsqrt(fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2])));
    double near = -DBL_MAX, far = DBL_MAX;
    for (int i = 0; i < 3; ++i) {
        d[i] *= rn * a.scale[i];
        s[i] = fma(g.src[i], a.inv_voxel[i], -a.corner_v[i]);
        // an axis along which the ray stands still gives +-inf, or NaN on a face, which fmin and fmax pass over
        const double inv = 1.0 / d[i];
        const double l1 = (-0.5 - s[i]) * inv, l2 = (a.grid[i] + 0.5 - s[i]) * inv;
        near = fmax(near, fmin(l1, l2));
        far = fmin(far, fmax(l1, l2));
    }
    const double t0 = fmax(near, 0.0);
    double first = t0, last = far;  // of the samples that are not zero
    if (M != Mode::Pairs) {
        // clipped to the slabs of the cells that are not zero, a thousandth of a voxel
        // wider for the FP32 positions; cell i covers i - 1/2 .. i + 1/2 in v
        const double f = M == Mode::CellsUp || M == Mode::SegmentsUp ? (double)a.up : 1.0;
        const double dir[5] = { d[0], d[1], d[2], d[0] + d[1], d[0] - d[1] };
        const double pos[5] = { s[0], s[1], s[2], s[0] + s[1], s[0] - s[1] };
        const double wide[5] = { 0.501, 0.501, 0.501, 1.002, 1.002 };
        const double shift[5] = { 1.0 - kPad, 1.0 - kPad, 1.0 - kPad, 2.0 - 2 * kPad, 0.0 };
        for (int i = 0; i < 5; ++i) {
            const double lo = f * (shift[i] - wide[i] - __ldg(a.support + 2 * i));
            const double hi = f * (shift[i] + wide[i] + __ldg(a.support + 2 * i + 1));
            // a diagonal's reciprocal from FP32 and one Newton step (4e-15), well within
            // the margin; where FP32 cannot hold it, it is NaN and the slab is passed over
            const double r0 = __frcp_rn((float)dir[i]);
            const double inv = i < 3 ? 1.0 / dir[i] : r0 * fma(-dir[i], r0, 2.0);
            const double l1 = (lo - pos[i]) * inv, l2 = (hi - pos[i]) * inv;
            first = fmax(first, fmin(l1, l2));
            last = fmin(last, fmax(l1, l2));
        }
    }
    // a ray that misses, or whose direction is not a number
    const bool hit = near <= far && far >= 0.0 && rn * 0.0 == 0.0;
    // the box diagonal bounds any honest ray; beyond it the inputs are broken
    if (hit && !(far - t0 < 1.0e7)) {
        if (flags)
            atomicOr(flags, kFlagNonFinite);
    } else if (hit) {
        const double i0 = ceil(first), i1 = floor(last);
        r.n = i1 >= i0 ? static_cast<int>(i1 - i0) + 1 : 0;
        r.first = static_cast<int>(fmin(i0, 1.0e9));
        for (int i = 0; i < 3; ++i) {
            r.base[i] = fma(i0, d[i], s[i]);
            r.step[i] = d[i];
            if (M == Mode::CellsUp || M == Mode::SegmentsUp) {
                // the same in stored voxels, a.up of the grid's to one
                const double f = 1.0 / a.up;
                r.base[i] *= f;
                r.step[i] *= f;
            }
            r.base[i] += kPad - 1.0;
        }
    }
    if (r.n <= 0)
        for (int i = 0; i < 3; ++i)
            r.base[i] = r.step[i] = 0.0;
    return r;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

__device__ __forceinline__ int floor_div(int i, int f) { return i >= 0 ? i / f : -((f - 1 - i) / f); }

// Sample loop, trilinear with zero border, volume stored as T (padded).
// Positions are formed relative to the integer part (ox, oy, oz) of the first
// sample, for the reason given at CellFrame; the offset is folded into the
// ray's base pointer and its clamp bounds, so a sample costs what it did with
// absolute coordinates.
template <typename T, Accum ACC, bool UP>
__device__ __forceinline__ void march_trilinear(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const T* __restrict__ vol = static_cast<const T*>(a.vol);
    const int sy = a.sy, sz = a.sz;
    const int mx = a.ext[0] - 2, my = a.ext[1] - 2, mz = a.ext[2] - 2;
    const int ox = (int)rint(r.base[0]), oy = (int)rint(r.base[1]), oz = (int)rint(r.base[2]);
    const float bx = (float)(r.base[0] - ox), by = (float)(r.base[1] - oy), bz = (float)(r.base[2] - oz);
    const float dx = (float)r.step[0], dy = (float)r.step[1], dz = (float)r.step[2];
    // the ray's origin tap; indexes relative to it are clamped so that the
    // absolute tap stays in [0, m] on each axis
    const T* __restrict__ vray = vol + ((ptrdiff_t)ox + (ptrdiff_t)oy * sy + (ptrdiff_t)oz * sz);
    for (int k = 0; k < r.n; ++k) {
        const float kf = static_cast<float>(k);
        const float ux = fmaf(kf, dx, bx);
        const float uy = fmaf(kf, dy, by);
        const float uz = fmaf(kf, dz, bz);
        const float fx = floorf(ux), fy = floorf(uy), fz = floorf(uz);
        const float wx = ux - fx, wy = uy - fy, wz = uz - fz;
        float v000, v100, v010, v110, v001, v101, v011, v111;
        if (!UP) {
            const int ix = clampi(__float2int_rz(fx), -ox, mx - ox);
            const int iy = clampi(__float2int_rz(fy), -oy, my - oy);
            const int iz = clampi(__float2int_rz(fz), -oz, mz - oz);
            const T* p = vray + (ix + iy * sy + iz * sz);
            v000 = load_voxel(p);
            v100 = load_voxel(p + 1);
            v010 = load_voxel(p + sy);
            v110 = load_voxel(p + sy + 1);
            v001 = load_voxel(p + sz);
            v101 = load_voxel(p + sz + 1);
            v011 = load_voxel(p + sz + sy);
            v111 = load_voxel(p + sz + sy + 1);
        } else {
            // virtual replication: grid index g maps to stored voxel floor(g / f)
            const int f = a.up;
            const int gx = __float2int_rz(fmaxf(fminf(fx, 1.0e8f), -1.0e8f)) + ox;
            const int gy = __float2int_rz(fmaxf(fminf(fy, 1.0e8f), -1.0e8f)) + oy;
            const int gz = __float2int_rz(fmaxf(fminf(fz, 1.0e8f), -1.0e8f)) + oz;
            const int x0 = clampi(floor_div(gx, f) + kPad, 0, mx + 1);
            const int x1 = clampi(floor_div(gx + 1, f) + kPad, 0, mx + 1);
            const int y0 = clampi(floor_div(gy, f) + kPad, 0, my + 1) * sy;
            const int y1 = clampi(floor_div(gy + 1, f) + kPad, 0, my + 1) * sy;
            const int z0 = clampi(floor_div(gz, f) + kPad, 0, mz + 1) * sz;
            const int z1 = clampi(floor_div(gz + 1, f) + kPad, 0, mz + 1) * sz;
            v000 = load_voxel(vol + (x0 + y0 + z0));
            v100 = load_voxel(vol + (x1 + y0 + z0));
            v010 = load_voxel(vol + (x0 + y1 + z0));
            v110 = load_voxel(vol + (x1 + y1 + z0));
            v001 = load_voxel(vol + (x0 + y0 + z1));
            v101 = load_voxel(vol + (x1 + y0 + z1));
            v011 = load_voxel(vol + (x0 + y1 + z1));
            v111 = load_voxel(vol + (x1 + y1 + z1));
        }
        const float c00 = fmaf(wx, v100 - v000, v000);
        const float c10 = fmaf(wx, v110 - v010, v010);
        const float c01 = fmaf(wx, v101 - v001, v001);
        const float c11 = fmaf(wx, v111 - v011, v011);
        const float c0 = fmaf(wy, c10 - c00, c00);
        const float c1 = fmaf(wy, c11 - c01, c01);
        acc.add(fmaf(wz, c1 - c0, c0));
    }
}

// Per-ray frame of the cell and pair loops.  Each axis of the first-sample
// position is split into an integer I = rint(base) and an FP32 remainder, and
// positions are formed as v' = (base - I) + k step.  Along an axis on which the
// ray moves little (a ray grazing a face of the volume) v' stays near zero,
// where FP32 is fine-grained; an absolute coordinate of a few hundred voxels
// would carry a rounding offset of up to 3e-5 voxel into every sample, and on
// a grazing ray that offset changes the line integral by up to 1e-3.  I is
// folded into the rounding constant m = kMagic + I (exact in FP32, |I| < 2^22),
// so t = v' + m has the bits kMagicBits + I + rint(v') of the absolute cell.
struct CellFrame {
    float2 bxy;  // base - I, x and y
    float bz;
    float2 mxy;  // kMagic + I, x and y
    float mz;
};

__device__ __forceinline__ CellFrame cell_frame(const Ray& r)
{
    CellFrame f;
    const double ix = rint(r.base[0]), iy = rint(r.base[1]), iz = rint(r.base[2]);
    f.bxy = make_float2((float)(r.base[0] - ix), (float)(r.base[1] - iy));
    f.bz = (float)(r.base[2] - iz);
    f.mxy = make_float2(__fadd_rn(kMagic, (float)ix), __fadd_rn(kMagic, (float)iy));
    f.mz = __fadd_rn(kMagic, (float)iz);
    return f;
}

// One axis of a frame moved on by K steps: K d + (K dl) is formed with its FP32
// rounding error, d + dl being the step to twice FP32's precision, and the integer
// part of the new position goes into m, the remainder (about [-1/2, 1/2]) into b.
__device__ __forceinline__ void advance_axis(float& b, float& m, float d, float dl, float K)
{
    const float p = __fmul_rn(K, d);
    const float low = fmaf(K, dl, fmaf(K, d, -p));
    const float t = __fadd_rn(p, m);
    const float u = __fadd_rn(__fsub_rn(p, __fsub_rn(t, m)), __fadd_rn(b, low));
    m = __fadd_rn(u, t);
    b = __fsub_rn(u, __fsub_rn(m, t));
}

// The coefficients of the cell a ray is in, reloaded only when its cell
// changes (consecutive samples of a ray often share a cell).
struct CellCache {
    uint32_t idx = 0xffffffffu;  // cell whose coefficients c0..c7 hold
    float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f, c4 = 0.f, c5 = 0.f, c6 = 0.f, c7 = 0.f;
};

// The interpolant of the cached cell at offsets (hx, hy, hz) from its centre,
// loading the cell first if `idx` differs from the cached one: a predicated
// 32-byte load, so the registers keep the cached cell when it does not.
__device__ __forceinline__ float cell_eval(const char* __restrict__ cells, uint32_t idx, float hx, float hy,
                                           float hz, CellCache& cc)
{
    {
        const char* p = cells + (size_t)idx * kCellBytes;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %8, %9;\n\t"
                     "@p ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%10];\n\t}"
                     : "+f"(cc.c0), "+f"(cc.c1), "+f"(cc.c2), "+f"(cc.c3), "+f"(cc.c4), "+f"(cc.c5),
                       "+f"(cc.c6), "+f"(cc.c7)
                     : "r"(idx), "r"(cc.idx), "l"(p));
        cc.idx = idx;
    }
    const float2 hx2 = make_float2(hx, hx);
    const float2 ea = __ffma2_rn(hx2, make_float2(cc.c2, cc.c3), make_float2(cc.c0, cc.c1));
    const float2 eb = __ffma2_rn(hx2, make_float2(cc.c6, cc.c7), make_float2(cc.c4, cc.c5));
    const float2 g = __ffma2_rn(make_float2(hy, hy), eb, ea);
    return fmaf(hz, g.y, g.x);
}

// up * h held to [-1/2, 1/2]
__device__ __forceinline__ float2 hold_half(float2 h, float up)
{
    return make_float2(__saturatef(fmaf(up, h.x, 0.5f)) - 0.5f, __saturatef(fmaf(up, h.y, 0.5f)) - 0.5f);
}

// Two consecutive samples of a ray (steps k and k + 1, the lanes of kk) from
// the coefficient cells.  Per axis: v' = (base - I) + k step; t = v' + m rounds
// to the cell index (its bits minus kMagicBits, see CellFrame); h = v' - (t - m)
// is the offset from the cell centre in [-1/2, 1/2].  Each packed f32x2
// operation holds one axis of both samples.  A sample that lands exactly
// between two cells may take either of them; both give the same interpolated
// value.  The cell index is clamped to the array as a guard; the loop bounds
// already keep every sample inside it.
//
// UP (virtual f^3 replication, f = up): between the centres of two stored
// voxels the replicated grid is flat but for one grid voxel about the face between
// them, where it rises linearly.  Along each axis that is the cell's own
// interpolant at f h instead of h, held at -1/2 and 1/2.
template <bool UP>
__device__ __forceinline__ float2 cell_sample_pair(const char* __restrict__ cells, float2 kk, const CellFrame& fr,
                                                   float2 dx2, float2 dy2, float2 dz2, uint32_t sy, uint32_t sz,
                                                   uint32_t cmax, uint32_t offset, float up, CellCache& cc)
{
    const float2 none2 = make_float2(-1.0f, -1.0f);
    const float2 mx2 = make_float2(fr.mxy.x, fr.mxy.x), my2 = make_float2(fr.mxy.y, fr.mxy.y);
    const float2 mz2 = make_float2(fr.mz, fr.mz);
    const float2 vx = __ffma2_rn(kk, dx2, make_float2(fr.bxy.x, fr.bxy.x));
    const float2 vy = __ffma2_rn(kk, dy2, make_float2(fr.bxy.y, fr.bxy.y));
    const float2 vz = __ffma2_rn(kk, dz2, make_float2(fr.bz, fr.bz));
    const float2 tx = __fadd2_rn(vx, mx2), ty = __fadd2_rn(vy, my2), tz = __fadd2_rn(vz, mz2);
    float2 hx = __ffma2_rn(__ffma2_rn(mx2, none2, tx), none2, vx);  // v - (t - m)
    float2 hy = __ffma2_rn(__ffma2_rn(my2, none2, ty), none2, vy);
    float2 hz = __ffma2_rn(__ffma2_rn(mz2, none2, tz), none2, vz);
    if (UP) {
        hx = hold_half(hx, up);
        hy = hold_half(hy, up);
        hz = hold_half(hz, up);
    }
    const uint32_t i0 = min(cell_linear(__float_as_uint(tx.x), __float_as_uint(ty.x), __float_as_uint(tz.x), sy, sz,
                                        offset), cmax);
    const uint32_t i1 = min(cell_linear(__float_as_uint(tx.y), __float_as_uint(ty.y), __float_as_uint(tz.y), sy, sz,
                                        offset), cmax);
    const float f0 = cell_eval(cells, i0, hx.x, hy.x, hz.x, cc);
    const float f1 = cell_eval(cells, i1, hx.y, hy.y, hz.y, cc);
    return make_float2(f0, f1);
}

// Samples after which the up-sampled sample loop forms its positions anew
// (advance_axis).  Counted from the ray's start, FP32 positions of a replicated grid
// are off by f times what the stored volume's are: 180x170x160, f = 3, ray_sampling 1,
// 2-norm error 1.13e-7 against 1.04e-7 of the gather loop; in windows of 192 samples
// 4.8e-8, of 64 3.2e-8 (101x97x89, f = 3, 60 x 512 x 384, ray_sampling 0.75: 4.38, 4.46
// and 4.50 ms).  A multiple of every U.
constexpr int kUpWindow = 192;

// Sample loop over the coefficient cells, U samples per partial sum (FP32)
// handed to the accumulator; up-sampled, an FP64 accumulator takes every sample, as
// in the gather loop that serves the same calls.
template <Accum ACC, int U, bool UP>
__device__ __forceinline__ void march_cells(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const char* __restrict__ cells = static_cast<const char*>(a.cells);
    CellFrame fr = cell_frame(r);
    const float2 dx2 = make_float2((float)r.step[0], (float)r.step[0]);
    const float2 dy2 = make_float2((float)r.step[1], (float)r.step[1]);
    const float2 dz2 = make_float2((float)r.step[2], (float)r.step[2]);
    const uint32_t sy = a.csy, sz = a.csz, cmax = a.cmax, offset = a.coffset;
    const float up = (float)a.up;
    const float2 two2 = make_float2(2.0f, 2.0f);
    CellCache cc;
    for (int from = 0; from < r.n; from += UP ? kUpWindow : r.n) {
        const int n = UP ? min(r.n - from, kUpWindow) : r.n;
        float2 kk = make_float2(0.0f, 1.0f);  // steps k and k + 1
        int k = 0;
        for (; k + U <= n; k += U) {
            float part = 0.0f;
#pragma unroll
            for (int j = 0; j < U; j += 2) {
                const float2 f = cell_sample_pair<UP>(cells, kk, fr, dx2, dy2, dz2, sy, sz, cmax, offset, up, cc);
                if constexpr (UP) {
                    acc.add_product(1.0f, f.x, part);
                    acc.add_product(1.0f, f.y, part);
                } else {
                    part += f.x;
                    part += f.y;
                }
                kk = __fadd2_rn(kk, two2);
            }
            if constexpr (UP)
                acc.flush(part);
            else
                acc.add(part);
        }
        // the last n - k < U samples, pairwise; a lone last sample takes the
        // first value of a pair whose second step lies beyond the ray (its cell
        // index is clamped like any other, its value unused)
        for (; k + 1 < n; k += 2) {
            const float2 f = cell_sample_pair<UP>(cells, kk, fr, dx2, dy2, dz2, sy, sz, cmax, offset, up, cc);
            acc.add(f.x);
            acc.add(f.y);
            kk = __fadd2_rn(kk, two2);
        }
        if (k < n)
            acc.add(cell_sample_pair<UP>(cells, kk, fr, dx2, dy2, dz2, sy, sz, cmax, offset, up, cc).x);
        if (UP) {
            const float K = (float)kUpWindow;
            advance_axis(fr.bxy.x, fr.mxy.x, dx2.x, (float)(r.step[0] - dx2.x), K);
            advance_axis(fr.bxy.y, fr.mxy.y, dy2.x, (float)(r.step[1] - dy2.x), K);
            advance_axis(fr.bz, fr.mz, dz2.x, (float)(r.step[2] - dz2.x), K);
        }
    }
}

// Per-ray constants of the segment loop, one per axis: where the ray leaves a
// cell (a sample at offset h from the cell's centre exits after e + h * i steps,
// i = -1 / step, e = |i| / 2), and the products of two steps that weigh the
// interpolant's mixed second derivatives, over 12.
struct SegmentRay {
    float2 ixy, exy;
    float iz, ez;
    float pxy, pxz, pyz;
};

__device__ __forceinline__ float exit_slope(float d)
{
    // an axis the ray does not move along (or by less than 1e-5 voxel over the
    // longest ray) never ends a segment: its exit lies 5e11 steps away
    return -1.0f / (fabsf(d) > 1.0e-12f ? d : copysignf(1.0e-12f, d));
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// One segment: the samples k, k + 1, .. last of a ray that lie in the cell of
// sample k, summed in closed form.  On a line the interpolant of a cell is a
// cubic in the step, and over samples placed evenly about their midpoint the odd
// powers cancel, so m samples sum to
//   m (f(mid) + (m^2 - 1) / 12 * q),
//   q = dx dy f_xy(mid) + dx dz f_xz(mid) + dy dz f_yz(mid),
// q being the quadratic coefficient (a trilinear interpolant has no f_xx).  The
// position of sample k is formed as in cell_sample_pair; m follows from the exit
// through the nearest face.  A sample within a rounding error of a face may be
// counted to either side, where both interpolants agree to that error.  A lane
// past its last sample (k = last + 1) gets m = 0 and adds nothing: its load stays
// in the array and its values are not used.
template <Accum ACC>
__device__ __forceinline__ void cell_segment(const char* __restrict__ cells, float& k, float last,
                                             const CellFrame& fr, float2 dxy, float dz, const SegmentRay& sr,
                                             uint32_t sy, uint32_t sz, uint32_t cmax, uint32_t offset,
                                             Accumulator<ACC>& acc, float& part)
{
    const float2 none2 = make_float2(-1.0f, -1.0f);
    const float2 vxy = __ffma2_rn(make_float2(k, k), dxy, fr.bxy);
    const float vz = fmaf(k, dz, fr.bz);
    const float2 txy = __fadd2_rn(vxy, fr.mxy);
    const float tz = __fadd_rn(vz, fr.mz);
    const uint32_t idx = min(cell_linear(__float_as_uint(txy.x), __float_as_uint(txy.y), __float_as_uint(tz), sy, sz,
                                         offset), cmax);
    float c0, c1, c2, c3, c4, c5, c6, c7;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(c0), "=f"(c1), "=f"(c2), "=f"(c3), "=f"(c4), "=f"(c5), "=f"(c6), "=f"(c7)
        : "l"(cells + (size_t)idx * kCellBytes));
    const float2 hxy = __ffma2_rn(__ffma2_rn(fr.mxy, none2, txy), none2, vxy);  // v - (t - m)
    const float hz = __fsub_rn(vz, __fsub_rn(tz, fr.mz));
    // whole steps to the exit, none below 0 and at most to the last sample (-1 past it)
    const float2 exy = __ffma2_rn(hxy, sr.ixy, sr.exy);
    const float e = fminf(fmaxf(min3(exy.x, exy.y, fmaf(hz, sr.iz, sr.ez)), 0.0f), last - k);
    const float m = __fadd_rd(e, 8388608.0f) - 8388607.0f;  // floor(e) + 1, e < kWindow
    const float half = fmaf(m, 0.5f, -0.5f);
    const float2 gxy = __ffma2_rn(make_float2(half, half), dxy, hxy);  // offsets of the midpoint
    const float gz = fmaf(half, dz, hz);
    const float2 hx2 = make_float2(gxy.x, gxy.x);
    const float2 ea = __ffma2_rn(hx2, make_float2(c2, c3), make_float2(c0, c1));
    const float2 eb = __ffma2_rn(hx2, make_float2(c6, c7), make_float2(c4, c5));
    const float2 g = __ffma2_rn(make_float2(gxy.y, gxy.y), eb, ea);
    const float f = fmaf(gz, g.y, g.x);
    const float q = fmaf(sr.pyz, eb.y, fmaf(sr.pxz, fmaf(gxy.y, c7, c3), sr.pxy * fmaf(gz, c7, c6)));
    if (k <= last)
        acc.add_product(m, fmaf(fmaf(m, m, -1.0f), q, f), part);
    k += m;
}

// Samples per window of the segment loop: the lanes of a warp, which step from
// cell to cell each at its own pace, meet again at every sample index that is a
// multiple of this, where positions are also formed anew (advance_axis).  Without that
// they drift apart by several cells along a long
// ray, share fewer cells per load and conflict more in L1 (256^3 -> 60 x 512^2
// with windows of 128, 192 and 256 samples: 11.48, 11.26 and 11.39 ms; 512^3
// helical, 180 views: 2.18, 2.17 and 2.19 ms.  Before positions were formed anew at
// the windows: 32, 64, 128 samples and no windows 12.6, 11.6, 11.3 and 11.7 ms).
constexpr int kWindow = 192;

// Sample sum by segments: one cell load and one evaluation per cell in which a
// ray has samples, instead of per sample; U segments per FP32 partial sum.  At
// the default step (0.3 voxel) a segment holds 2.4 samples on average.  Called by
// all 32 lanes of a warp (r.n = 0 for a lane without a ray).  The windows lie at
// fixed sample indexes, so a ray's segments and partial sums do not depend on the
// warp that runs it.  Steps count from the start of the window, whose position is
// carried in more than FP32, so positions and step lengths stay exact to 1e-6 voxel
// along the whole ray (2-norm error against 64 bits at 201x173x155: 2.8e-8, of
// which 2.5e-8 is the rounding of the result; 5.2e-8 with steps counted from the
// ray's start).  An FP64 accumulator takes every segment's m f exactly, in place of
// the FP32 sum of two (201x173x155, 23 views: 1.366 -> 1.383 ms).
template <Accum ACC, int U>
__device__ __forceinline__ void march_segments(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const char* __restrict__ cells = static_cast<const char*>(a.cells);
    CellFrame fr = cell_frame(r);
    const float2 dxy = make_float2((float)r.step[0], (float)r.step[1]);
    const float dz = (float)r.step[2];
    const float lx = (float)(r.step[0] - dxy.x), ly = (float)(r.step[1] - dxy.y), lz = (float)(r.step[2] - dz);
    SegmentRay sr;
    sr.ixy = make_float2(exit_slope(dxy.x), exit_slope(dxy.y));
    sr.iz = exit_slope(dz);
    sr.exy = make_float2(0.5f * fabsf(sr.ixy.x), 0.5f * fabsf(sr.ixy.y));
    sr.ez = 0.5f * fabsf(sr.iz);
    sr.pxy = dxy.x * dxy.y * (1.0f / 12.0f);
    sr.pxz = dxy.x * dz * (1.0f / 12.0f);
    sr.pyz = dxy.y * dz * (1.0f / 12.0f);
    const uint32_t sy = a.csy, sz = a.csz, cmax = a.cmax, offset = a.coffset;
    const bool hit = r.n > 0;
    const int w1 = __reduce_max_sync(0xffffffffu, hit ? (r.first + r.n - 1) / kWindow : -1);
    int w = __reduce_min_sync(0xffffffffu, hit ? r.first / kWindow : 0x7fffffff);
    int at = r.first;                   // the lane's next sample
    const int end = r.first + r.n;
    for (; w <= w1; ++w) {
        const int stop = min(end, (w + 1) * kWindow);
        if (at < stop) {
            const float last = (float)(stop - at - 1);
            float k = 0.0f;
            do {
                float part = 0.0f;
#pragma unroll
                for (int j = 0; j < U; ++j)
                    cell_segment(cells, k, last, fr, dxy, dz, sr, sy, sz, cmax, offset, acc, part);
                acc.flush(part);
            } while (k <= last);
            advance_axis(fr.bxy.x, fr.mxy.x, dxy.x, lx, k);
            advance_axis(fr.bxy.y, fr.mxy.y, dxy.y, ly, k);
            advance_axis(fr.bz, fr.mz, dz, lz, k);
            at = stop;
        }
        __syncwarp();
    }
}

// One axis of a segment of the replicated grid.  Between the centres of two stored
// voxels the grid is flat but for the ramp of one grid voxel about the face between
// them, |f h| < 1/2 with h the offset from the cell's centre.  From h a ray along the
// axis leaves its ramp, or its flat stretch (which runs on into the next cell), after
// e steps; on the way the cell's own interpolant is taken at `at`, moving by `step`
// per sample on the ramp and not at all off it.
struct UpAxis {
    float slope;       // -1 / step, as SegmentRay
    float ramp, flat;  // steps from the cell's centre to the ramp's end, and to the next ramp
    float step;        // f * step
};

__device__ __forceinline__ UpAxis up_axis(float d, float f)
{
    UpAxis u;
    u.slope = exit_slope(d);
    u.ramp = fabsf(u.slope) * (0.5f / f);
    u.flat = fabsf(u.slope) * (1.0f - 0.5f / f);
    u.step = f * d;
    return u;
}

__device__ __forceinline__ float up_exit(const UpAxis& u, float h, float f, float& at, float& step)
{
    const float y = f * h;
    const bool on = fabsf(y) < 0.5f;
    // off the ramp: ahead of it where y and the step have opposite signs (slope and y the same)
    const bool before = (__float_as_int(y) ^ __float_as_int(u.slope)) >= 0;
    at = fminf(fmaxf(y, -0.5f), 0.5f);
    step = on ? u.step : 0.0f;
    return fmaf(h, u.slope, on ? u.ramp : (before ? -u.ramp : u.flat));
}

// One segment of the replicated grid, as cell_segment: the samples k .. of a ray up to
// the nearest end of a ramp or a flat stretch, summed in closed form with the offsets
// and steps of up_exit.  The cell is sample k's; where a flat stretch crosses into the
// next cell, both cells hold the same values on it.
template <Accum ACC>
__device__ __forceinline__ void cell_segment_up(const char* __restrict__ cells, float& k, float last,
                                                const CellFrame& fr, float2 dxy, float dz, const UpAxis& ux,
                                                const UpAxis& uy, const UpAxis& uz, float f, uint32_t sy, uint32_t sz,
                                                uint32_t cmax, uint32_t offset, Accumulator<ACC>& acc,
                                                float& part)
{
    const float2 none2 = make_float2(-1.0f, -1.0f);
    const float2 vxy = __ffma2_rn(make_float2(k, k), dxy, fr.bxy);
    const float vz = fmaf(k, dz, fr.bz);
    const float2 txy = __fadd2_rn(vxy, fr.mxy);
    const float tz = __fadd_rn(vz, fr.mz);
    const uint32_t idx = min(cell_linear(__float_as_uint(txy.x), __float_as_uint(txy.y), __float_as_uint(tz), sy, sz,
                                         offset), cmax);
    float c0, c1, c2, c3, c4, c5, c6, c7;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(c0), "=f"(c1), "=f"(c2), "=f"(c3), "=f"(c4), "=f"(c5), "=f"(c6), "=f"(c7)
        : "l"(cells + (size_t)idx * kCellBytes));
    const float2 hxy = __ffma2_rn(__ffma2_rn(fr.mxy, none2, txy), none2, vxy);
    const float hz = __fsub_rn(vz, __fsub_rn(tz, fr.mz));
    float ax, ay, az, sx, sy_, sz_;
    const float ex = up_exit(ux, hxy.x, f, ax, sx), ey = up_exit(uy, hxy.y, f, ay, sy_), ez = up_exit(uz, hz, f, az, sz_);
    const float e = fminf(fmaxf(min3(ex, ey, ez), 0.0f), last - k);
    const float m = __fadd_rd(e, 8388608.0f) - 8388607.0f;
    const float half = fmaf(m, 0.5f, -0.5f);
    const float gx = fmaf(half, sx, ax), gy = fmaf(half, sy_, ay), gz = fmaf(half, sz_, az);
    const float2 gx2 = make_float2(gx, gx);
    const float2 ea = __ffma2_rn(gx2, make_float2(c2, c3), make_float2(c0, c1));
    const float2 eb = __ffma2_rn(gx2, make_float2(c6, c7), make_float2(c4, c5));
    const float2 g = __ffma2_rn(make_float2(gy, gy), eb, ea);
    const float v = fmaf(gz, g.y, g.x);
    // dx dy f_xy + dx dz f_xz + dy dz f_yz
    const float q = fmaf(sx, fmaf(sz_, fmaf(gy, c7, c3), sy_ * fmaf(gz, c7, c6)), sy_ * sz_ * eb.y);
    if (k <= last)
        acc.add_product(m, fmaf(fmaf(m, m, -1.0f) * (1.0f / 12.0f), q, v), part);
    k += m;
}

// march_segments for the replicated grid (positions in stored voxels).  101x97x89, f =
// 3, 60 x 512 x 384 at the default step: 10.3 -> 6.6 ms against the sample loop.
template <Accum ACC, int U>
__device__ __forceinline__ void march_segments_up(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const char* __restrict__ cells = static_cast<const char*>(a.cells);
    CellFrame fr = cell_frame(r);
    const float2 dxy = make_float2((float)r.step[0], (float)r.step[1]);
    const float dz = (float)r.step[2], f = (float)a.up;
    const float lx = (float)(r.step[0] - dxy.x), ly = (float)(r.step[1] - dxy.y), lz = (float)(r.step[2] - dz);
    const UpAxis ux = up_axis(dxy.x, f), uy = up_axis(dxy.y, f), uz = up_axis(dz, f);
    const uint32_t sy = a.csy, sz = a.csz, cmax = a.cmax, offset = a.coffset;
    const bool hit = r.n > 0;
    const int w1 = __reduce_max_sync(0xffffffffu, hit ? (r.first + r.n - 1) / kWindow : -1);
    int w = __reduce_min_sync(0xffffffffu, hit ? r.first / kWindow : 0x7fffffff);
    int at = r.first;
    const int end = r.first + r.n;
    for (; w <= w1; ++w) {
        const int stop = min(end, (w + 1) * kWindow);
        if (at < stop) {
            const float last = (float)(stop - at - 1);
            float k = 0.0f;
            do {
                float part = 0.0f;
#pragma unroll
                for (int j = 0; j < U; ++j)
                    cell_segment_up(cells, k, last, fr, dxy, dz, ux, uy, uz, f, sy, sz, cmax, offset, acc, part);
                acc.flush(part);
            } while (k <= last);
            advance_axis(fr.bxy.x, fr.mxy.x, dxy.x, lx, k);
            advance_axis(fr.bxy.y, fr.mxy.y, dxy.y, ly, k);
            advance_axis(fr.bz, fr.mz, dz, lz, k);
            at = stop;
        }
        __syncwarp();
    }
}

// Padded-array index of the voxel floor(p) of sample k, formed in FP64; beyond the
// volume it is clamped to the array's zero border.
__device__ __forceinline__ uint32_t nearest_index(const ProjectArgs& a, const Ray& r, int k)
{
    const double kd = static_cast<double>(k);
    const double px = fmin(fmax(fma(kd, r.step[0], r.base[0]), -1.0), 1.0e9);
    const double py = fmin(fmax(fma(kd, r.step[1], r.base[1]), -1.0), 1.0e9);
    const double pz = fmin(fmax(fma(kd, r.step[2], r.base[2]), -1.0), 1.0e9);
    const int ix = clampi(__double2int_rd(px), 0, a.ext[0] - 1);
    const int iy = clampi(__double2int_rd(py), 0, a.ext[1] - 1);
    const int iz = clampi(__double2int_rd(pz), 0, a.ext[2] - 1);
    return (uint32_t)(ix + iy * a.sy + iz * a.sz);
}

// The exact voxel of sample k and the number of samples, at most `most`, that
// follow each other in it.
__device__ __noinline__ uint2 nearest_run(const ProjectArgs& a, const Ray& r, int k, int most)
{
    const uint32_t idx = nearest_index(a, r, k);
    int m = 1;
    while (m < most && nearest_index(a, r, k + m) == idx)
        ++m;
    return make_uint2(idx, (uint32_t)m);
}

// Nearest voxel: a voxel load and a multiply-add per voxel in which a ray has
// samples, by the windows of march_segments.  A position error would move a sample
// into the neighbouring voxel, so the samples go where FP64 positions put them: FP32
// decides where its error bound (del, in voxels: the rounding of v and of the step
// over a window, and of the frame over the windows) leaves no doubt about the voxel
// of the first sample and the number of samples to the exit, nearest_run in FP64
// elsewhere (about one segment in 10^4 at the default step).  The first and the last
// sample of the reference's range lie outside the volume, or on its face, and are
// taken on their own.  256^3 -> 45 x 512^2: 22.0 ms with every sample in FP64, 9.5
// ms by segments.  The sum is FP64's: m v is exact in it, and so, unless the voxels'
// magnitudes differ by 2^20 and more, is the sum, whatever its order.  Both forms then give
// the same bits, and the choice between them can go by the size of the job (30 views: 6.20
// ms, 6.04 with Kahan sums of two voxels' FP32 sums).
template <typename T>
__device__ __forceinline__ void march_nearest(const ProjectArgs& a, const Ray& r, Accumulator<Accum::F64>& acc)
{
    const T* __restrict__ vol = static_cast<const T*>(a.vol);
    if (r.n > 0)
        acc.add(load_voxel(vol + nearest_index(a, r, 0)));
    const float2 dxy = make_float2((float)r.step[0], (float)r.step[1]);
    const float dz = (float)r.step[2];
    const float lx = (float)(r.step[0] - dxy.x), ly = (float)(r.step[1] - dxy.y), lz = (float)(r.step[2] - dz);
    Ray q = r;  // from sample 1, about the voxel centres: the index is rint(v)
    for (int i = 0; i < 3; ++i)
        q.base[i] += r.step[i] - 0.5;
    CellFrame fr = cell_frame(q);
    const float ix = exit_slope(dxy.x), iy = exit_slope(dxy.y), iz = exit_slope(dz);
    const int end = r.first + r.n - 1;  // past the last sample taken here
    int at = r.first + 1;
    const float reach = (float)kWindow * fmaxf(fmaxf(fabsf(dxy.x), fabsf(dxy.y)), fabsf(dz)) + 1.0f;
    const float del = 1.5e-7f * reach + 2.5e-7f * ((float)(r.n / kWindow) + 4.0f);
    // A source so far away that FP64 cannot hold a position to a voxel (1e16 voxels; any
    // finite matrix is served) puts samples anywhere.  FP32 decides only where the samples
    // taken here stay within a voxel of the volume, a voxel inside the padded array; for
    // other rays `lo` leaves every sample to nearest_run, which holds its indexes in the array.
    bool inside = true;
    for (int i = 0; i < 3; ++i) {
        const double p0 = r.base[i] + r.step[i], p1 = fma((double)(r.n - 2), r.step[i], r.base[i]);
        inside = inside && fmin(p0, p1) >= kPad - 1.0 && fmax(p0, p1) < a.ext[i] - 1.0;
    }
    const float lo = inside ? 0.5f - del : -1.0f, hi = 0.5f + del;
    const uint32_t sy = (uint32_t)a.sy, sz = (uint32_t)a.sz, offset = 0u - kMagicBits * (1u + sy + sz);
    const float2 none2 = make_float2(-1.0f, -1.0f);
    // the number of samples alone says whether a ray takes part: one that misses has no
    // place along the ray to compare
    const bool hit = r.n > 2;
    const int w1 = __reduce_max_sync(0xffffffffu, hit ? (end - 1) / kWindow : -1);
    int w = __reduce_min_sync(0xffffffffu, hit ? at / kWindow : 0x7fffffff);
    for (; w <= w1; ++w) {
        const int stop = min(end, (w + 1) * kWindow);
        if (hit && at < stop) {
            const float last = (float)(stop - at - 1);
            float k = 0.0f;
            do {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 vxy = __ffma2_rn(make_float2(k, k), dxy, fr.bxy);
                    const float vz = fmaf(k, dz, fr.bz);
                    const float2 txy = __fadd2_rn(vxy, fr.mxy);
                    const float tz = __fadd_rn(vz, fr.mz);
                    const float2 h = __ffma2_rn(__ffma2_rn(fr.mxy, none2, txy), none2, vxy);
                    const float hz = __fsub_rn(vz, __fsub_rn(tz, fr.mz));
                    const float left = last - k;  // -1 past the last sample
                    const float e0 = fminf(min3(fmaf(h.x, ix, lo * fabsf(ix)), fmaf(h.y, iy, lo * fabsf(iy)),
                                                fmaf(hz, iz, lo * fabsf(iz))), left);
                    const float e1 = fminf(min3(fmaf(h.x, ix, hi * fabsf(ix)), fmaf(h.y, iy, hi * fabsf(iy)),
                                                fmaf(hz, iz, hi * fabsf(iz))), left);
                    float m = __fadd_rd(e0, 8388608.0f);
                    const bool sure = m == __fadd_rd(e1, 8388608.0f) &&
                                      fmaxf(fmaxf(fabsf(h.x), fabsf(h.y)), fabsf(hz)) < lo;
                    m -= 8388607.0f;
                    uint32_t idx = offset + __float_as_uint(txy.x) + __float_as_uint(txy.y) * sy +
                                   __float_as_uint(tz) * sz;
                    if (!sure && left >= 0.0f) {
                        const uint2 run = nearest_run(a, r, at - r.first + (int)k, (int)left + 1);
                        idx = run.x;
                        m = (float)run.y;
                    }
                    if (left >= 0.0f) {
                        acc.add_product(m, load_voxel(vol + idx));
                    } else {
                        m = 0.0f;
                    }
                    k += m;
                }
            } while (k <= last);
            advance_axis(fr.bxy.x, fr.mxy.x, dxy.x, lx, k);
            advance_axis(fr.bxy.y, fr.mxy.y, dxy.y, ly, k);
            advance_axis(fr.bz, fr.mz, dz, lz, k);
            at = stop;
        }
        __syncwarp();
    }
    if (r.n > 1)
        acc.add(load_voxel(vol + nearest_index(a, r, r.n - 1)));
}

// The same, every sample on its own: the faster form where a voxel holds hardly more
// than one, or few rays leave each waiting for its segments (nearest_segment_max_sampling).
template <typename T>
__device__ __forceinline__ void march_nearest_samples(const ProjectArgs& a, const Ray& r, Accumulator<Accum::F64>& acc)
{
    const T* __restrict__ vol = static_cast<const T*>(a.vol);
    for (int k = 0; k < r.n; ++k)
        acc.add(load_voxel(vol + nearest_index(a, r, k)));
}

// x-pair entries of the current cell: rows (y, z), (y+1, z), (y, z+1), (y+1, z+1).
struct PairCache {
    uint32_t idx = 0xffffffffu;
    float m00 = 0.f, d00 = 0.f, m10 = 0.f, d10 = 0.f, m01 = 0.f, d01 = 0.f, m11 = 0.f, d11 = 0.f;
};

// One sample from the x-pair array: the same cell index and centre offsets as
// cell_sample_pair, four 8-byte entries loaded only when the cell changes, x by
// mid + hx diff, then y and z linearly.
__device__ __forceinline__ float pair_sample(const char* __restrict__ pairs, float2 kk, const CellFrame& fr,
                                             float2 dxy, float dz, uint32_t sy, uint32_t sz, uint32_t pmax,
                                             PairCache& pc)
{
    const float2 none2 = make_float2(-1.0f, -1.0f);
    const float2 vxy = __ffma2_rn(kk, dxy, fr.bxy);
    const float vz = fmaf(kk.x, dz, fr.bz);
    const float2 txy = __fadd2_rn(vxy, fr.mxy);
    const float tz = __fadd_rn(vz, fr.mz);
    const float2 fxy = __ffma2_rn(fr.mxy, none2, txy);  // t - m, exact
    const float fz = __fsub_rn(tz, fr.mz);
    const float2 hxy = __ffma2_rn(fxy, none2, vxy);
    const float hz = fmaf(fz, -1.0f, vz);
    uint32_t idx = __float_as_uint(txy.x) + __float_as_uint(txy.y) * sy + __float_as_uint(tz) * sz;
    idx = min(idx, pmax);
    {
        const char* p0 = pairs + (size_t)idx * 8;
        const char* p1 = p0 + (size_t)sy * 8;
        const char* p2 = p0 + (size_t)sz * 8;
        const char* p3 = p2 + (size_t)sy * 8;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %8, %9;\n\t"
                     "@p ld.global.nc.v2.f32 {%0, %1}, [%10];\n\t"
                     "@p ld.global.nc.v2.f32 {%2, %3}, [%11];\n\t"
                     "@p ld.global.nc.v2.f32 {%4, %5}, [%12];\n\t"
                     "@p ld.global.nc.v2.f32 {%6, %7}, [%13];\n\t}"
                     : "+f"(pc.m00), "+f"(pc.d00), "+f"(pc.m10), "+f"(pc.d10), "+f"(pc.m01), "+f"(pc.d01),
                       "+f"(pc.m11), "+f"(pc.d11)
                     : "r"(idx), "r"(pc.idx), "l"(p0), "l"(p1), "l"(p2), "l"(p3));
        pc.idx = idx;
    }
    const float hx = hxy.x;
    const float2 lo = make_float2(fmaf(hx, pc.d00, pc.m00), fmaf(hx, pc.d01, pc.m01));  // (y, z), (y, z+1)
    const float2 hi = make_float2(fmaf(hx, pc.d10, pc.m10), fmaf(hx, pc.d11, pc.m11));  // (y+1, z), (y+1, z+1)
    const float wy = hxy.y + 0.5f, wz = hz + 0.5f;
    const float2 e = __ffma2_rn(make_float2(wy, wy), __ffma2_rn(lo, none2, hi), lo);     // z, z+1
    return fmaf(wz, e.y - e.x, e.x);
}

// Sample loop over the x-pair array (same structure as march_cells).
template <Accum ACC, int U>
__device__ __forceinline__ void march_pairs(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const char* __restrict__ pairs = static_cast<const char*>(a.cells);
    const CellFrame fr = cell_frame(r);
    const float2 dxy = make_float2((float)r.step[0], (float)r.step[1]);
    const float dz = (float)r.step[2];
    const uint32_t sy = a.csy, sz = a.csz, pmax = a.cmax;
    const float2 one2 = make_float2(1.0f, 1.0f);
    float2 kk = make_float2(0.0f, 0.0f);
    PairCache pc;
    int k = 0;
    for (; k + U <= r.n; k += U) {
        float part = 0.0f;
#pragma unroll
        for (int j = 0; j < U; ++j) {
            part += pair_sample(pairs, kk, fr, dxy, dz, sy, sz, pmax, pc);
            kk = __fadd2_rn(kk, one2);
        }
        acc.add(part);
    }
    for (; k < r.n; ++k) {
        acc.add(pair_sample(pairs, kk, fr, dxy, dz, sy, sz, pmax, pc));
        kk = __fadd2_rn(kk, one2);
    }
}

// Sample loop, hardware texture filter (border colour 0, unnormalised coords).
template <Accum ACC>
__device__ __forceinline__ void march_texture(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    const float bx = (float)r.base[0], by = (float)r.base[1], bz = (float)r.base[2];
    const float dx = (float)r.step[0], dy = (float)r.step[1], dz = (float)r.step[2];
    for (int k = 0; k < r.n; ++k) {
        const float kf = static_cast<float>(k);
        acc.add(tex3D<float>(a.tex, fmaf(kf, dx, bx), fmaf(kf, dy, by), fmaf(kf, dz, bz)));
    }
}

// Pixel (with sub-rays spread over lanes, sub-ray of the finer grid of channels <<
// sub_x by rows << sub_y) of thread `tid` of work item (block) `b` of a.block threads, for the
// launch shape in `a` (every factor of the mapping is a power of two).
// ROWS: consecutive lanes run down the rows of a channel, else along the channels.
template <bool ROWS>
__device__ __forceinline__ bool pixel_of_item(const ProjectArgs& a, uint32_t b, uint32_t tid, uint32_t& vm,
                                              uint32_t& x, uint32_t& y)
{
    // Block order: chunks of vm_group view groups; within a chunk (module,
    // tile, view group).  Blocks resident at the same time then cover the same
    // tiles of neighbouring views, whose rays cross nearly the same part of
    // the volume.
    const uint32_t G = a.vm_group;
    const uint32_t T = a.tiles_per_vm;
    const uint32_t per_chunk = G * a.n_modules * T;
    const uint32_t c = b / per_chunk;
    const uint32_t first = c * G;
    const uint32_t gsize = min(G, a.view_groups - first);
    const uint32_t r = b - c * per_chunk;
    const uint32_t q = r / gsize;
    const uint32_t vg = first + (r - q * gsize);
    const uint32_t m = q / T;
    const uint32_t t = q - m * T;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t slot = warp >> a.wpv_shift, w = warp & ((1u << a.wpv_shift) - 1u);
    const uint32_t view = (vg << a.vpb_shift) + slot;
    vm = view * a.n_modules + m;
    const uint32_t ty = t / a.tiles_x, tx = t - ty * a.tiles_x;
    // rays down the rows of a channel share x and y and differ in z, which the cell
    // layout serves without conflicts (CellLayout); along the channels they share lines
    // of the voxel array, x fastest
    const uint32_t ly_shift = 5u - a.lx_shift;
    const uint32_t lx = ROWS ? lane >> ly_shift : lane & ((1u << a.lx_shift) - 1u);
    const uint32_t ly = ROWS ? lane & ((1u << ly_shift) - 1u) : lane >> a.lx_shift;
    x = (tx << a.tx_shift) + ((w & ((1u << a.wx_shift) - 1u)) << a.lx_shift) + lx;
    y = (ty << a.ty_shift) + ((w >> a.wx_shift) << ly_shift) + ly;
    return view < a.n_views && x < a.span_x && y < a.span_y;
}

__device__ __forceinline__ bool pixel_of_thread(const ProjectArgs& a, uint32_t tid, uint32_t& vm, uint32_t& x,
                                                uint32_t& y)
{
    return pixel_of_item<false>(a, blockIdx.x, tid, vm, x, y);
}

__device__ __forceinline__ bool pixel_of(const ProjectArgs& a, uint32_t& vm, uint32_t& x, uint32_t& y)
{
    return pixel_of_thread(a, threadIdx.x, vm, x, y);
}

// Writes the warp's pixel values (called by all 32 lanes): each lane holds
// `val` for pixel (vm, x, y), or ok = false for no pixel.  The lanes of four
// consecutive channels of one detector row follow each other, or lie one patch height
// apart (ROWS; a warp patch is 4 or 8 channels wide); where all four pixels exist and their row
// segment starts on a 16-byte boundary, the first of them gathers the other three
// values and writes the segment as one 16-byte store; otherwise each lane stores
// its own value.
template <bool ROWS>
__device__ __forceinline__ void store_patch(const ProjectArgs& a, uint32_t vm, uint32_t x, uint32_t y, float val,
                                            bool ok)
{
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31u;
    const uint32_t ls = ROWS ? 5u - a.lx_shift : 0u;  // log2 of the lanes from a channel to the next
    const uint32_t lead = lane & ~(3u << ls);
    const float v1 = __shfl_down_sync(full, val, 1u << ls);
    const float v2 = __shfl_down_sync(full, val, 2u << ls);
    const float v3 = __shfl_down_sync(full, val, 3u << ls);
    const uint32_t okmask = __ballot_sync(full, ok);
    const uint32_t quad = 1u | (1u << (1u << ls)) | (1u << (2u << ls)) | (1u << (3u << ls));
    float* dst = a.out + ((size_t)vm * a.rows + y) * a.channels + x;
    const bool whole = ((okmask >> lead) & quad) == quad && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0;
    // the choice of the four is their first lane's
    const bool vec = __shfl_sync(full, whole ? 1 : 0, lead) != 0;
    if (vec) {
        if (lane == lead)
            *reinterpret_cast<float4*>(dst) = make_float4(val, v1, v2, v3);
    } else if (ok) {
        *dst = val;
    }
}

// One ray of the gather loop, up-sampled.  A voxel that is infinite or not a number
// reaches a whole cell through the cell's polynomial, where the replicated grid holds
// it to the samples next to that voxel, and masks near the largest FP32 number overflow
// its coefficients: volumes with such voxels (kWild) take this road.
template <Accum ACC>
__device__ __noinline__ void gather_upsampled(const ProjectArgs& a, const ViewGeom& g, double px, double py, bool live,
                                              Accumulator<ACC>& acc)
{
    if (!live)
        return;
    const Ray r = setup_ray<Mode::Trilinear>(a, g, px, py, a.flags);
    if (a.dtype == 0)
        march_trilinear<float, ACC, true>(a, r, acc);
    else if (a.dtype == 1)
        march_trilinear<__nv_bfloat16, ACC, true>(a, r, acc);
    else
        march_trilinear<__half, ACC, true>(a, r, acc);
}

// The sample loop of a derived array's mode.
template <Mode M, Accum ACC, int U>
__device__ __forceinline__ void march_array(const ProjectArgs& a, const Ray& r, Accumulator<ACC>& acc)
{
    if (M == Mode::Pairs)
        march_pairs<ACC, U>(a, r, acc);
    else if (M == Mode::Segments)
        march_segments<ACC, U>(a, r, acc);
    else if (M == Mode::SegmentsUp)
        march_segments_up<ACC, U>(a, r, acc);
    else
        march_cells<ACC, U, M == Mode::CellsUp>(a, r, acc);
}

// The rays of work item `b` for thread `tid`, cell, segment or pair loop (FP32
// entries).  Called by every lane of a warp (the segment loop and the store are
// warp-cooperative): a lane without a pixel or with an unusable matrix marches a
// ray of no samples.
template <Mode M, Accum ACC, int U>
__device__ __forceinline__ void cells_item(const ProjectArgs& a, uint32_t b, uint32_t tid)
{
    uint32_t vm, x, y;
    const bool ok = pixel_of_item<true>(a, b, tid, vm, x, y);
    const ViewGeom& g = a.geom[ok ? vm : 0u];
    const bool live = ok && g.valid;
    Accumulator<ACC> acc;
    // (up-sampled volumes with wild voxels, see gather_upsampled)
    const bool by_voxel = (M == Mode::CellsUp || M == Mode::SegmentsUp) && __ldg(a.support + kSupportWild) > 0;
    auto ray = [&](double px, double py) {
        if (by_voxel) {
            gather_upsampled<ACC>(a, g, px, py, live, acc);
            return;
        }
        Ray r = setup_ray_cells<M>(a, g, px, py, live ? a.flags : nullptr);
        if (!live)
            r.n = 0;
        march_array<M, ACC, U>(a, r, acc);
    };
    if (a.rays_x == 1 && a.rays_y == 1) {
        // one ray through the pixel centre (x - 0.5 + 0.5 is x exactly): the
        // pixel and its geometry are dead once the ray is set up, so the
        // sample loop carries only the ray
        ray((double)x, (double)y);
        const float val = static_cast<float>(a.increment * acc.value());
        // the pixel again for the store, rather than holding it through the loop
        pixel_of_item<true>(a, b, tid, vm, x, y);
        store_patch<true>(a, vm, x, y, val, ok);
        return;
    }
    const bool spread = (a.sub_x | a.sub_y) != 0;  // a lane per sub-ray
    const double ix = 1.0 / a.rays_x, iy = 1.0 / a.rays_y;
    const uint32_t nx = spread ? 1u : a.rays_x, ny = spread ? 1u : a.rays_y;
    const uint32_t x0 = spread ? x & (a.rays_x - 1u) : 0u, y0 = spread ? y & (a.rays_y - 1u) : 0u;
    for (uint32_t rx = 0; rx < nx; ++rx)
        for (uint32_t ry = 0; ry < ny; ++ry)
            ray((double)(x >> a.sub_x) - 0.5 + 0.5 * ix + (x0 + rx) * ix,
                (double)(y >> a.sub_y) - 0.5 + 0.5 * iy + (y0 + ry) * iy);
    double sum = acc.value();
    if (spread) {
        const uint32_t ls = 5u - a.lx_shift;  // log2 of the patch height
        for (uint32_t o = 1; o < a.rays_y; o <<= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        for (uint32_t o = 1; o < a.rays_x; o <<= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o << ls);
    }
    const float val = static_cast<float>(a.increment * sum / (double)(a.rays_x * a.rays_y));
    pixel_of_item<true>(a, b, tid, vm, x, y);
    if (!spread)
        store_patch<true>(a, vm, x, y, val, ok);
    else if (ok && ((x & (a.rays_x - 1u)) | (y & (a.rays_y - 1u))) == 0)
        a.out[((size_t)vm * a.rows + (y >> a.sub_y)) * a.channels + (x >> a.sub_x)] = val;
}

constexpr int cell_maxreg(Mode m)
{
    return m == Mode::Segments || m == Mode::SegmentsUp || m == Mode::CellsUp ? CTLCU_SEGMENT_MAXREG
                                                                              : CTLCU_CELL_MAXREG;
}

// Cell, segment or pair loop over one block of the regular grid.
template <Mode M, Accum ACC, int U>
__global__ void __maxnreg__(cell_maxreg(M)) cells_kernel(const __grid_constant__ ProjectArgs a)
{
    cells_item<M, ACC, U>(a, blockIdx.x, threadIdx.x);
}

// Persistent batch kernel with warp-granular work: every warp takes one warp
// patch (32 rays: patch w of block tile b of a request) at a time from
// `counter` and runs it, with no barrier between the warps of a block.  A warp
// whose rays are short (a tile edge, rays that miss the volume) takes the next
// patch at once instead of waiting for the longest ray of its tile, so the SMs
// stay busy to the end of the batch.  Warp items run in the order of the
// single-request launch's blocks and, within a block tile, its warps: warps that
// run at the same time work on neighbouring patches and views of one volume.
//
// Per warp, the request of its item is found by scanning forward from the
// previous one (a warp's items only grow), and the request's launch arguments
// are copied into the warp's own slot of shared memory only when the request
// changes.

template <Mode M, Accum ACC, int U>
__global__ void __maxnreg__(cell_maxreg(M))
    batch_cells_kernel(const BatchReq* __restrict__ reqs, uint32_t n_reqs, uint32_t total_warp_items,
                       uint32_t wpb_shift, unsigned int* counter)
{
    extern __shared__ __align__(16) unsigned char s_raw[];  // one ProjectArgs per warp
    static_assert(sizeof(ProjectArgs) % 4 == 0, "word copy");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    ProjectArgs& sa = reinterpret_cast<ProjectArgs*>(s_raw)[warp];
    uint32_t req = 0, loaded = 0xffffffffu;  // the same in every lane of the warp
    for (;;) {
        uint32_t it = 0;
        if (lane == 0)
            it = atomicAdd(counter, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= total_warp_items)
            return;
        const uint32_t item = it >> wpb_shift, w = it & ((1u << wpb_shift) - 1u);
        while (req + 1 < n_reqs && reqs[req + 1].first_item <= item)
            ++req;  // the last request with first_item <= item
        if (req != loaded) {
            __syncwarp();  // every lane is done with the previous request's arguments
            const uint32_t* src = reinterpret_cast<const uint32_t*>(&reqs[req].a);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&sa);
            for (uint32_t i = lane; i < sizeof(ProjectArgs) / 4; i += 32)
                dst[i] = src[i];
            __syncwarp();
            loaded = req;
        }
        cells_item<M, ACC, U>(sa, item - reqs[req].first_item, (w << 5) + lane);
    }
}

// Gather, nearest-voxel and texture loops over one block of the regular grid.
template <typename T, Mode M, Accum ACC, bool UP>
__global__ void __maxnreg__(CTLCU_GATHER_MAXREG) project_kernel(const __grid_constant__ ProjectArgs a)
{
    static_assert(M == Mode::Trilinear || M == Mode::Nearest || M == Mode::NearestSamples || M == Mode::Texture, "cells_kernel runs these");
    uint32_t vm, x, y;
    const bool ok = pixel_of(a, vm, x, y);
    const ViewGeom& g = a.geom[ok ? vm : 0u];
    const bool live = ok && g.valid;
    Accumulator<ACC> acc;
    float val = 0.0f;
    // the windows of march_nearest are the whole warp's; a lane without a ray stays out of
    // the other loops
    if (M == Mode::Nearest || live) {
        const double ix = 1.0 / a.rays_x, iy = 1.0 / a.rays_y;
        for (uint32_t rx = 0; rx < a.rays_x; ++rx)
            for (uint32_t ry = 0; ry < a.rays_y; ++ry) {
                const double px = (double)x - 0.5 + 0.5 * ix + rx * ix;
                const double py = (double)y - 0.5 + 0.5 * iy + ry * iy;
                Ray r = setup_ray<M>(a, g, px, py, live ? a.flags : nullptr);
                if (!live)
                    r.n = 0;
                if constexpr (M == Mode::Trilinear)
                    march_trilinear<T, ACC, UP>(a, r, acc);
                else if constexpr (M == Mode::Nearest)
                    march_nearest<T>(a, r, acc);
                else if constexpr (M == Mode::NearestSamples)
                    march_nearest_samples<T>(a, r, acc);
                else
                    march_texture<ACC>(a, r, acc);
            }
        val = static_cast<float>(a.increment * acc.value() / (double)(a.rays_x * a.rays_y));
    }
    store_patch<false>(a, vm, x, y, val, ok);
}

template <Mode M>
__global__ void __launch_bounds__(kMaxBlock) count_kernel(const ProjectArgs a)
{
    uint32_t vm, x, y;
    unsigned long long n = 0;
    if (pixel_of(a, vm, x, y)) {
        const ViewGeom& g = a.geom[vm];
        if (g.valid) {
            const double ix = 1.0 / a.rays_x, iy = 1.0 / a.rays_y;
            for (uint32_t rx = 0; rx < a.rays_x; ++rx)
                for (uint32_t ry = 0; ry < a.rays_y; ++ry) {
                    const double px = (double)x - 0.5 + 0.5 * ix + rx * ix;
                    const double py = (double)y - 0.5 + 0.5 * iy + ry * iy;
                    n += (unsigned long long)setup_ray<M>(a, g, px, py, nullptr).n;
                }
        }
    }
    for (int o = 16; o > 0; o >>= 1)
        n += __shfl_down_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31u) == 0 && n)
        atomicAdd(a.counter, n);
}

// log2 of the warps in a block of 128, 256 or 512 threads.
uint32_t log2_block_warps(uint32_t block) { return block == 128 ? 2u : (block == 256 ? 3u : 4u); }

// The launch's block size must be one the pixel mapping was built for.
bool block_ok(const ProjectArgs& a)
{
    return a.block == 128 || a.block == 256 || a.block == kMaxBlock;
}

template <Mode M, Accum ACC, bool UP>
cudaError_t launch_typed(const ProjectArgs& a, int dtype, dim3 grid, cudaStream_t s)
{
    switch (dtype) {
    case 0: project_kernel<float, M, ACC, UP><<<grid, a.block, 0, s>>>(a); break;
    case 1: project_kernel<__nv_bfloat16, M, ACC, UP><<<grid, a.block, 0, s>>>(a); break;
    case 2: project_kernel<__half, M, ACC, UP><<<grid, a.block, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Samples, or segments of about two samples, per partial sum of a loop.
constexpr int loop_unroll(Mode m, int unroll)
{
    return m == Mode::Segments || m == Mode::SegmentsUp ? unroll / 2 : unroll;
}

template <Mode M, Accum ACC>
cudaError_t launch_cells(const ProjectArgs& a, dim3 grid, cudaStream_t s)
{
    switch (a.unroll) {
    case 2: cells_kernel<M, ACC, loop_unroll(M, 2)><<<grid, a.block, 0, s>>>(a); break;
    case 4: cells_kernel<M, ACC, loop_unroll(M, 4)><<<grid, a.block, 0, s>>>(a); break;
    case 8: cells_kernel<M, ACC, loop_unroll(M, 8)><<<grid, a.block, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <Accum ACC>
cudaError_t launch_acc(const ProjectArgs& a, Mode mode, int dtype, dim3 grid, cudaStream_t s)
{
    switch (mode) {
    case Mode::Trilinear:
        return a.up != 1 ? launch_typed<Mode::Trilinear, ACC, true>(a, dtype, grid, s)
                         : launch_typed<Mode::Trilinear, ACC, false>(a, dtype, grid, s);
    // their sums are FP64's whatever the accumulator (march_nearest)
    case Mode::Nearest: return launch_typed<Mode::Nearest, Accum::F64, false>(a, dtype, grid, s);
    case Mode::NearestSamples: return launch_typed<Mode::NearestSamples, Accum::F64, false>(a, dtype, grid, s);
    case Mode::Texture:
        project_kernel<float, Mode::Texture, ACC, false><<<grid, a.block, 0, s>>>(a);
        return cudaGetLastError();
    case Mode::Cells: return launch_cells<Mode::Cells, ACC>(a, grid, s);
    case Mode::Segments: return launch_cells<Mode::Segments, ACC>(a, grid, s);
    case Mode::CellsUp: return launch_cells<Mode::CellsUp, ACC>(a, grid, s);
    case Mode::SegmentsUp: return launch_cells<Mode::SegmentsUp, ACC>(a, grid, s);
    case Mode::Pairs: return launch_cells<Mode::Pairs, ACC>(a, grid, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_project(const ProjectArgs& a, Mode mode, Accum acc, int dtype, cudaStream_t s)
{
    const uint64_t blocks = (uint64_t)a.view_groups * a.n_modules * a.tiles_per_vm;
    if (blocks == 0)
        return cudaSuccess;
    if (blocks > 0x7fffffffull || !block_ok(a))
        return cudaErrorInvalidConfiguration;
    const dim3 grid((unsigned)blocks);
    switch (acc) {
    case Accum::F64: return launch_acc<Accum::F64>(a, mode, dtype, grid, s);
    case Accum::Kahan: return launch_acc<Accum::Kahan>(a, mode, dtype, grid, s);
    case Accum::F32: return launch_acc<Accum::F32>(a, mode, dtype, grid, s);
    }
    return cudaErrorInvalidValue;
}

namespace {
template <Mode M, Accum ACC, int U>
cudaError_t launch_batch_typed(const BatchReq* reqs, uint32_t n_reqs, uint32_t total, uint32_t block,
                               unsigned int* counter, int* blocks, cudaStream_t s)
{
    // warp items: each block tile of `block` rays is block / 32 warp patches
    const uint32_t wpb = block / 32u, wpb_shift = log2_block_warps(block);
    const uint64_t warp_items = (uint64_t)total * wpb;
    // the counter runs past the end by one per warp of the grid: keep it clear of wrapping
    if (warp_items > 0xffffffffull - (1ull << 20))
        return cudaErrorInvalidValue;
    const size_t smem = sizeof(ProjectArgs) * wpb;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_cells_kernel<M, ACC, U>, (int)block, smem);
    if (e != cudaSuccess)
        return e;
    uint64_t grid = (uint64_t)sms * (uint64_t)(per_sm > 0 ? per_sm : 1);
    if (grid > total)
        grid = total;
    *blocks = (int)grid;
    batch_cells_kernel<M, ACC, U><<<(unsigned)grid, block, smem, s>>>(reqs, n_reqs, (uint32_t)warp_items, wpb_shift,
                                                                      counter);
    return cudaGetLastError();
}

template <Mode M, Accum ACC>
cudaError_t launch_batch_unroll(const BatchReq* reqs, uint32_t n_reqs, uint32_t total, const LaunchShape& sh,
                                unsigned int* counter, int* blocks, cudaStream_t s)
{
    switch (sh.unroll) {
    case 2: return launch_batch_typed<M, ACC, loop_unroll(M, 2)>(reqs, n_reqs, total, sh.block, counter, blocks, s);
    case 4: return launch_batch_typed<M, ACC, loop_unroll(M, 4)>(reqs, n_reqs, total, sh.block, counter, blocks, s);
    case 8: return launch_batch_typed<M, ACC, loop_unroll(M, 8)>(reqs, n_reqs, total, sh.block, counter, blocks, s);
    }
    return cudaErrorInvalidValue;
}

template <Mode M>
cudaError_t launch_batch_mode(const BatchReq* reqs, uint32_t n_reqs, uint32_t total, Accum acc,
                              const LaunchShape& sh, unsigned int* counter, int* blocks, cudaStream_t s)
{
    switch (acc) {
    case Accum::F64: return launch_batch_unroll<M, Accum::F64>(reqs, n_reqs, total, sh, counter, blocks, s);
    case Accum::Kahan: return launch_batch_unroll<M, Accum::Kahan>(reqs, n_reqs, total, sh, counter, blocks, s);
    case Accum::F32: return launch_batch_unroll<M, Accum::F32>(reqs, n_reqs, total, sh, counter, blocks, s);
    }
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t launch_batch(const BatchReq* reqs, uint32_t n_reqs, uint32_t total_items, Mode mode, Accum acc,
                         const LaunchShape& shape, unsigned int* counter, int* blocks, cudaStream_t s)
{
    if (total_items == 0 || n_reqs == 0)
        return cudaSuccess;
    if (shape_error(shape))
        return cudaErrorInvalidConfiguration;
    if (mode == Mode::Pairs)
        return launch_batch_mode<Mode::Pairs>(reqs, n_reqs, total_items, acc, shape, counter, blocks, s);
    if (mode == Mode::Cells)
        return launch_batch_mode<Mode::Cells>(reqs, n_reqs, total_items, acc, shape, counter, blocks, s);
    if (mode == Mode::Segments)
        return launch_batch_mode<Mode::Segments>(reqs, n_reqs, total_items, acc, shape, counter, blocks, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_count(const ProjectArgs& a, Mode mode, cudaStream_t s)
{
    const uint64_t blocks = (uint64_t)a.view_groups * a.n_modules * a.tiles_per_vm;
    if (blocks == 0)
        return cudaSuccess;
    if (blocks > 0x7fffffffull || !block_ok(a))
        return cudaErrorInvalidConfiguration;
    const dim3 grid((unsigned)blocks);
    if (mode == Mode::Nearest || mode == Mode::NearestSamples)
        count_kernel<Mode::Nearest><<<grid, a.block, 0, s>>>(a);
    else
        count_kernel<Mode::Trilinear><<<grid, a.block, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace ctlcu
