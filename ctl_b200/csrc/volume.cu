// Volume staging kernels: zero-padded resident copies in the storage dtype,
// the f = 0 mean voxel, and materialised up-sampling for the texture path.
//
// Reference: VolumeSpecs::upSampleVolume (modules/src/projectors/raycasterprojector.cpp:576-672)
// builds, on the host and per project() call, either one voxel holding the
// mean (f = 0), the volume as is (f = 1), or an f^3 nearest-neighbour
// replication (f >= 2).  Here f >= 2 is virtual for the software path (index
// math in raycast.cu) and materialised only for the hardware-texture path.
#include "internal.cuh"

#include <algorithm>
#include <climits>

namespace ctlcu {

namespace {

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }

// dst (padded) <- convert(src), borders zero: a warp per row of the padded array, so
// that every element is written once and only a row's place takes a division.
// 256^3 FP32: 73 us for a memset and one thread per voxel, 23 us now.
template <typename T>
__global__ void __launch_bounds__(256)
    pad_convert_kernel(const float* __restrict__ src, T* __restrict__ dst, int nx, int ny, int nz)
{
    const int ex = nx + 2 * kPad, ey = ny + 2 * kPad, ez = nz + 2 * kPad;
    const uint32_t rows = (uint32_t)ey * (uint32_t)ez, lane = threadIdx.x & 31u;
    for (uint32_t r = blockIdx.x * 8u + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8u) {
        const int z = (int)(r / (uint32_t)ey) - kPad, y = (int)(r % (uint32_t)ey) - kPad;
        const bool inside = z >= 0 && z < nz && y >= 0 && y < ny;
        const float* from = src + ((size_t)z * ny + y) * nx - kPad;
        T* to = dst + (size_t)r * ex;
#pragma unroll 4
        for (int x = (int)lane; x < ex; x += 32) {
            const bool in = inside && x >= kPad && x < nx + kPad;
            to[x] = from_float<T>(in ? __ldg(from + x) : 0.0f);
        }
    }
}

// FP64 sum of the (dequantised) stored voxels; one atomicAdd per block
template <typename T>
__global__ void sum_kernel(const T* __restrict__ padded, int nx, int ny, int nz, double* sum)
{
    const int ex = nx + 2 * kPad, ey = ny + 2 * kPad;
    const size_t total = (size_t)nx * ny * nz;
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx);
        const size_t r = i / nx;
        const int y = (int)(r % ny);
        const int z = (int)(r / ny);
        s += (double)to_float<T>(
            padded[(size_t)(x + kPad) + (size_t)ex * ((size_t)(y + kPad) + (size_t)ey * (size_t)(z + kPad))]);
    }
    __shared__ double part[32];
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = (threadIdx.x < (blockDim.x >> 5)) ? part[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0)
            atomicAdd(sum, s);
    }
}

// 1x1x1 volume (padded to (1+2P)^3, zero-initialised by the caller) holding the mean
__global__ void mean_volume_kernel(const double* sum, double count, float* dst)
{
    const int e = 1 + 2 * kPad;
    dst[kPad + e * (kPad + e * kPad)] = (float)(*sum / count);
}

// dst (dense, f*n per axis, storage dtype) <- nearest replication of the stored volume
template <typename T>
__global__ void upsample_kernel(const T* __restrict__ padded, int nx, int ny, int nz, int f,
                                T* __restrict__ dst)
{
    const int ex = nx + 2 * kPad, ey = ny + 2 * kPad;
    const size_t X = (size_t)nx * f, Y = (size_t)ny * f, Z = (size_t)nz * f;
    const size_t total = X * Y * Z;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t x = i % X;
        const size_t r = i / X;
        const size_t y = r % Y;
        const size_t z = r / Y;
        dst[i] = padded[(x / f + kPad) + ex * ((y / f + kPad) + (size_t)ey * (z / f + kPad))];
    }
}

// Coefficient cells.  Cell (i, j, k) spans padded voxels i..i+1, j..j+1, k..k+1.
// With h = w - 1/2 the local offsets from the cell centre, its trilinear
// interpolant is
//   f = C0 + Cx hx + Cy hy + Cz hz + Cxy hx hy + Cxz hx hz + Cyz hy hz + Cxyz hx hy hz,
//   C0 = sum v / 8, Cx = sum sx v / 4, Cxy = sum sx sy v / 2, Cxyz = sum sx sy sz v
// (s = -1 for the low corner, +1 for the high one, per axis).  The 8
// coefficients are computed in FP64 and stored as FP32 in the order
//   (C0, Cz), (Cx, Cxz), (Cy, Cyz), (Cxy, Cxyz)
// so the sampler evaluates f with three packed f32x2 FMAs and one FMA.
//
// Bound by writing the cells (32 bytes each) once.  A thread writes the slots of
// one place in the rows of a slice pair (CellLayout: lanes alternate between the two
// slices, so a warp writes 1 KB runs), `per` rows one after the other, and keeps the z and x sums and
// differences of the previous row: four voxel loads, four conversions and 20 FP64
// additions per cell.  Slots beyond the last cell of a row, a pair or an odd last
// slice are written as zeros.  256^3 FP32: 240 us with 64 FP64 operations per cell
// and a memset of the array before, 123 us without the bounds and 152 us with them.
__device__ __forceinline__ void store_cell(float* p, float4 lo, float4 hi)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "f"(lo.x), "f"(lo.y), "f"(lo.z), "f"(lo.w), "f"(hi.x), "f"(hi.y), "f"(hi.z), "f"(hi.w)
                 : "memory");
}

template <typename T>
__global__ void __launch_bounds__(128)
    build_cells_kernel(const T* __restrict__ padded, int ex, int ey, CellLayout L, uint32_t per,
                       float* __restrict__ cells, int* __restrict__ support)
{
    __shared__ int most[kSupport];
    if (threadIdx.x < kSupport)
        most[threadIdx.x] = kSupportNone;
    __syncthreads();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t pairs = slot < L.sy ? (L.cz + 1) / 2 : 0u;
    const uint32_t rows = (L.sz + L.sy - 1) / L.sy;  // the last one may be the pair's tail alone
    const uint32_t x = slot >> 1;
    int z_lo = INT_MAX, z_hi = -1, y_lo = INT_MAX, y_hi = -1;  // this thread's cells that are not zero
    bool wild = false;  // a voxel is not below kWild
    const size_t ys = (size_t)ex, zs = (size_t)ex * ey;
    for (uint32_t p = blockIdx.z; p < pairs; p += gridDim.z) {
        const uint32_t z = 2 * p + (slot & 1u);
        const bool column = x < L.cx && z < L.cz;
        for (uint32_t y0 = blockIdx.y * per; y0 < rows; y0 += gridDim.y * per) {
            const uint32_t y1 = min(y0 + per, rows);
            const T* v = padded + (x + ys * y0 + zs * z);
            // sums and differences over x, z of one row: s, sx (x), sz (z), sxz
            double s = 0.0, sx = 0.0, sz = 0.0, sxz = 0.0;
            bool some = false;  // a voxel of the row is not zero
            auto row = [&]() {
                const double a = to_float<T>(v[0]), b = to_float<T>(v[1]);
                const double c = to_float<T>(v[zs]), d = to_float<T>(v[zs + 1]);
                some = a != 0.0 || b != 0.0 || c != 0.0 || d != 0.0;
                wild = wild || !(fabs(a) < kWild && fabs(b) < kWild && fabs(c) < kWild && fabs(d) < kWild);
                const double l = a + b, lx = b - a, h = c + d, hx = d - c;
                s = l + h;
                sx = lx + hx;
                sz = h - l;
                sxz = hx - lx;
            };
            if (column && y0 < L.cy)
                row();
            for (uint32_t y = y0; y < y1; ++y) {
                const size_t i = (size_t)p * L.sz + (size_t)y * L.sy + slot;
                float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
                if (column && y < L.cy) {
                    const double s0 = s, x0 = sx, z0 = sz, xz0 = sxz;
                    const bool some0 = some;
                    v += ys;
                    row();
                    if (some || some0) {
                        y_lo = min(y_lo, (int)y);
                        y_hi = max(y_hi, (int)y);
                        z_lo = min(z_lo, (int)z);
                        z_hi = max(z_hi, (int)z);
                    }
                    lo = make_float4((float)((s0 + s) * 0.125), (float)((z0 + sz) * 0.25), (float)((x0 + sx) * 0.25),
                                     (float)((xz0 + sxz) * 0.5));
                    hi = make_float4((float)((s - s0) * 0.25), (float)((sz - z0) * 0.5), (float)((sx - x0) * 0.5),
                                     (float)(sxz - xz0));
                }
                if (i < (size_t)(p + 1) * L.sz)
                    store_cell(cells + 8 * i, lo, hi);
            }
        }
    }
    const int xi = (int)x;
    const bool any = y_hi >= 0;
    const int m[kSupport] = { -xi, xi, -y_lo, y_hi, -z_lo, z_hi, -(xi + y_lo), xi + y_hi, -(xi - y_hi), xi - y_lo,
                              wild ? 1 : kSupportNone };
    for (int i = 0; i < kSupport; ++i) {
        const int w = __reduce_max_sync(0xffffffffu, any ? m[i] : kSupportNone);
        if ((threadIdx.x & 31u) == 0)
            atomicMax(&most[i], w);
    }
    __syncthreads();
    // most blocks lie within what is known already and need no global atomic
    if (threadIdx.x < kSupport && most[threadIdx.x] > *(volatile int*)(support + threadIdx.x))
        atomicMax(support + threadIdx.x, most[threadIdx.x]);
}

// x-pair entries (mid, diff) of the padded volume, see PairLayout.
template <typename T>
__global__ void build_pairs_kernel(const T* __restrict__ padded, int ex, int ey, int ez, uint32_t psy,
                                   uint32_t psz, float2* __restrict__ pairs)
{
    const int px = ex - 1;
    const size_t total = (size_t)px * ey * ez;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % px);
        const size_t r = i / px;
        const int y = (int)(r % ey);
        const int z = (int)(r / ey);
        const size_t o = (size_t)x + (size_t)ex * ((size_t)y + (size_t)ey * z);
        const double a = (double)to_float<T>(padded[o]), b = (double)to_float<T>(padded[o + 1]);
        pairs[(size_t)x + (size_t)psy * y + (size_t)psz * z] = make_float2((float)(0.5 * (a + b)), (float)(b - a));
    }
}

unsigned grid_for(size_t n)
{
    size_t b = (n + 255) / 256;
    if (b > 148 * 64)
        b = 148 * 64;
    return (unsigned)(b ? b : 1);
}

}  // namespace

cudaError_t launch_pad_convert(const float* src, void* dst, const int n[3], int dtype, cudaStream_t s)
{
    const uint32_t rows = (uint32_t)(n[1] + 2 * kPad) * (uint32_t)(n[2] + 2 * kPad);
    const unsigned g = std::min<uint32_t>((rows + 7) / 8, 148u * 32u);
    switch (dtype) {
    case 0: pad_convert_kernel<float><<<g, 256, 0, s>>>(src, (float*)dst, n[0], n[1], n[2]); break;
    case 1: pad_convert_kernel<__nv_bfloat16><<<g, 256, 0, s>>>(src, (__nv_bfloat16*)dst, n[0], n[1], n[2]); break;
    case 2: pad_convert_kernel<__half><<<g, 256, 0, s>>>(src, (__half*)dst, n[0], n[1], n[2]); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_mean(const void* padded, const int n[3], int dtype, double* sum_out, cudaStream_t s)
{
    const unsigned g = grid_for((size_t)n[0] * n[1] * n[2]);
    switch (dtype) {
    case 0: sum_kernel<float><<<g, 256, 0, s>>>((const float*)padded, n[0], n[1], n[2], sum_out); break;
    case 1: sum_kernel<__nv_bfloat16><<<g, 256, 0, s>>>((const __nv_bfloat16*)padded, n[0], n[1], n[2], sum_out); break;
    case 2: sum_kernel<__half><<<g, 256, 0, s>>>((const __half*)padded, n[0], n[1], n[2], sum_out); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_mean_volume(const double* sum, double count, float* dst_padded, cudaStream_t s)
{
    mean_volume_kernel<<<1, 1, 0, s>>>(sum, count, dst_padded);
    return cudaGetLastError();
}

cudaError_t launch_build_cells(const void* padded, const int n[3], int dtype, const CellLayout& L,
                               void* cells, cudaStream_t s)
{
    const int ex = n[0] + 2 * kPad, ey = n[1] + 2 * kPad;
    int* support = cell_support(cells, L);
    cudaError_t e = cudaMemsetAsync(support, kSupportNone & 0xff, kSupportBytes, s);
    if (e != cudaSuccess)
        return e;
    // rows per thread: 16 where that leaves enough blocks to fill the GPU, fewer for
    // small volumes (64^3: 17 us with 16 rows, 7.4 with 2)
    const uint32_t rows = (L.sz + L.sy - 1) / L.sy, pairs = (L.cz + 1) / 2, bx = (L.sy + 127) / 128;
    uint32_t per = 16;
    while (per > 1 && (uint64_t)bx * ((rows + per - 1) / per) * pairs < 148u * 12u)
        per /= 2;
    const dim3 g(bx, std::min<uint32_t>((rows + per - 1) / per, 65535u), std::min<uint32_t>(pairs, 65535u));
    switch (dtype) {
    case 0: build_cells_kernel<float><<<g, 128, 0, s>>>((const float*)padded, ex, ey, L, per, (float*)cells, support); break;
    case 1: build_cells_kernel<__nv_bfloat16><<<g, 128, 0, s>>>((const __nv_bfloat16*)padded, ex, ey, L, per, (float*)cells, support); break;
    case 2: build_cells_kernel<__half><<<g, 128, 0, s>>>((const __half*)padded, ex, ey, L, per, (float*)cells, support); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_build_pairs(const void* padded, const int n[3], int dtype, const PairLayout& L,
                               void* pairs, cudaStream_t s)
{
    const int ex = n[0] + 2 * kPad, ey = n[1] + 2 * kPad, ez = n[2] + 2 * kPad;
    const unsigned g = grid_for((size_t)(ex - 1) * ey * ez);
    cudaError_t e = cudaMemsetAsync(pairs, 0, L.count * sizeof(float2), s);
    if (e != cudaSuccess)
        return e;
    switch (dtype) {
    case 0: build_pairs_kernel<float><<<g, 256, 0, s>>>((const float*)padded, ex, ey, ez, L.sy, L.sz, (float2*)pairs); break;
    case 1: build_pairs_kernel<__nv_bfloat16><<<g, 256, 0, s>>>((const __nv_bfloat16*)padded, ex, ey, ez, L.sy, L.sz, (float2*)pairs); break;
    case 2: build_pairs_kernel<__half><<<g, 256, 0, s>>>((const __half*)padded, ex, ey, ez, L.sy, L.sz, (float2*)pairs); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_unpad_upsample(const void* padded, const int n[3], int dtype, int f, void* dst,
                                  cudaStream_t s)
{
    const unsigned g = grid_for((size_t)n[0] * n[1] * n[2] * f * f * f);
    switch (dtype) {
    case 0: upsample_kernel<float><<<g, 256, 0, s>>>((const float*)padded, n[0], n[1], n[2], f, (float*)dst); break;
    case 1: upsample_kernel<__nv_bfloat16><<<g, 256, 0, s>>>((const __nv_bfloat16*)padded, n[0], n[1], n[2], f, (__nv_bfloat16*)dst); break;
    case 2: upsample_kernel<__half><<<g, 256, 0, s>>>((const __half*)padded, n[0], n[1], n[2], f, (__half*)dst); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace ctlcu
