// Homogeneous-cube radius of every voxel, the table behind FAST-mode free
// flight in the voxelized transport kernels.
//
// radius[v] is the largest k (capped) such that the cube of voxels within
// Chebyshev distance k of v lies inside the grid and holds v's material
// only.  A packet anywhere inside voxel v is then at least k * min(voxel
// size) away from every other material and from the grid's surface, so a
// sampled free path shorter than that can be taken in one move: the
// exponential free path is memoryless, and the reference's walk, which stops
// at every voxel wall and draws a new path length when the next voxel holds
// the same material (xopto/mcvox/kernel/mcvox.template.c:760-1038), samples
// the same interaction points in distribution.
//
// radius[v] is the Chebyshev distance from v to the set B of voxels that lie
// on the grid surface or have one of their 26 neighbours in another
// material (a voxel within distance k - 1 of v that is not in B has all its
// neighbours in its own material, so the cube of radius k around v is
// homogeneous).  It starts from 0 on B and the cap elsewhere.
//
// max(|dx|, |dy|, |dz|) separates: the distance is the least max(|dx|, .) of
// the least max(|dy|, .) of the least max(|dz|, .), so three passes of lines
// in shared memory, one per axis and each in place, give the exact capped
// result; a voxel looks along its line only as far as its own value.  What
// bounds a pass is the shared-memory reads of that search.  200^3 voxels,
// cap 31: 0.71 ms, 2.87 ms by the
// relaxation below.  Lines too long for shared memory take the in-place
// relaxation r(v) <- min(r(v), 1 + min over the 26 neighbours of r(u)): every
// read value is an upper bound of the true distance, the values only
// decrease, and each pass carries the exact distances one voxel further, so
// cap passes give the exact capped result.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/xopto_gb300.h"
#include "errors.h"

namespace {

__global__ void radius_init_kernel(const uint8_t *__restrict__ vox, uint8_t *radius, int nx, int ny,
                                   int nz, uint8_t cap) {
    const size_t n = (size_t)nx * ny * nz;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        int x = (int)(i % nx);
        int y = (int)((i / nx) % ny);
        int z = (int)(i / ((size_t)nx * ny));
        uint8_t r = cap;
        if (x == 0 || y == 0 || z == 0 || x == nx - 1 || y == ny - 1 || z == nz - 1) {
            r = 0;
        } else {
            const uint8_t m = vox[i];
            for (int dz = -1; dz <= 1 && r; ++dz)
                for (int dy = -1; dy <= 1 && r; ++dy)
                    for (int dx = -1; dx <= 1; ++dx) {
                        size_t j = ((size_t)(z + dz) * ny + (y + dy)) * nx + (x + dx);
                        if (vox[j] != m) {
                            r = 0;
                            break;
                        }
                    }
        }
        radius[i] = r;
    }
}

constexpr int AXIS_THREADS = 256;
constexpr size_t AXIS_BYTES = 48 * 1024;   /* of one block's lines */

/* Lines of one axis, `wide` adjacent ones to a block.  Along x (step = 1) the
   lines are rows and the block's region is contiguous; along y and z the
   lines start at adjacent x.  Line element i of line w lies at
   base + i * step + w * next. */
__global__ void __launch_bounds__(AXIS_THREADS)
radius_axis_kernel(uint8_t *radius, int nx, int ny, int nz, int axis, int wide) {
    extern __shared__ uint8_t line[];
    const size_t plane = (size_t)nx * ny;
    int length, lines;
    size_t base, step;
    if (axis == 0) {
        const size_t row = (size_t)blockIdx.x * wide, rows = (size_t)ny * nz;
        length = nx;
        lines = (int)(rows - row < (size_t)wide ? rows - row : (size_t)wide);
        base = row * nx;
        step = 1;
    } else {
        const int tiles = (nx + wide - 1) / wide;
        const int x0 = (int)(blockIdx.x % tiles) * wide, other = (int)(blockIdx.x / tiles);
        length = axis == 1 ? ny : nz;
        lines = nx - x0 < wide ? nx - x0 : wide;
        base = (axis == 1 ? other * plane : (size_t)other * nx) + x0;
        step = axis == 1 ? (size_t)nx : plane;
    }
    /* shared: [line][i] along x, [i][line] along y and z, as in memory */
    const int count = length * lines, hop = axis == 0 ? 1 : lines;
    for (int e = threadIdx.x; e < count; e += AXIS_THREADS) {
        const size_t at = axis == 0 ? base + e : base + (size_t)(e / lines) * step + e % lines;
        line[e] = radius[at];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < count; e += AXIS_THREADS) {
        const int i = axis == 0 ? e % length : e / lines;
        int best = line[e];
        for (int d = 1; d < best; ++d) {
            int near = best;
            if (i >= d) near = min(near, (int)line[e - d * hop]);
            if (i + d < length) near = min(near, (int)line[e + d * hop]);
            best = min(best, max(d, near));
        }
        const size_t at = axis == 0 ? base + e : base + (size_t)(e / lines) * step + e % lines;
        radius[at] = (uint8_t)best;
    }
}

/* Lines per block along an axis of the given length, 0 = too long. */
int axis_lines(int length, int most) {
    const size_t fit = AXIS_BYTES / (size_t)length;
    return fit >= (size_t)most ? most : (int)fit;
}

__global__ void radius_relax_kernel(uint8_t *radius, int nx, int ny, int nz) {
    const size_t n = (size_t)nx * ny * nz;
    volatile uint8_t *rv = radius;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        uint8_t r = rv[i];
        /* 0 on B, which includes the grid surface: a voxel with r > 0 has
           all 26 neighbours inside the grid */
        if (r == 0) continue;
        int x = (int)(i % nx);
        int y = (int)((i / nx) % ny);
        int z = (int)(i / ((size_t)nx * ny));
        uint8_t m = r;
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    size_t j = ((size_t)(z + dz) * ny + (y + dy)) * nx + (x + dx);
                    uint8_t u = rv[j];
                    m = u < m ? u : m;
                }
        uint8_t c = (uint8_t)(m + 1u);
        if (c < r) rv[i] = c;
    }
}

}  // namespace

extern "C" int mcgb_voxel_radius(const uint8_t *dev_voxels, const int32_t shape[3], uint8_t *dev_radius,
                                 uint32_t max_radius, void *stream) {
    if (!dev_voxels || !dev_radius || !shape)
        return mcgb_internal::set_error(MCGB_E_INVALID, "mcgb_voxel_radius: NULL argument");
    const int nx = shape[0], ny = shape[1], nz = shape[2];
    if (nx <= 0 || ny <= 0 || nz <= 0)
        return mcgb_internal::set_error(MCGB_E_INVALID, "mcgb_voxel_radius: shape must be positive");
    if (max_radius < 1 || max_radius > MCGB_VOXEL_RADIUS_MAX)
        return mcgb_internal::set_error(MCGB_E_INVALID, "mcgb_voxel_radius: max_radius must be in [1, 64]");
    const size_t n = (size_t)nx * ny * nz;
    unsigned blocks = (unsigned)((n + 255) / 256);
    if (blocks > 152u * 64u) blocks = 152u * 64u;
    cudaStream_t s = (cudaStream_t)stream;
    radius_init_kernel<<<blocks, 256, 0, s>>>(dev_voxels, dev_radius, nx, ny, nz, (uint8_t)max_radius);
    /* 64 lines a block: whole 64-byte segments along y and z */
    const int wx = axis_lines(nx, 64), wy = axis_lines(ny, 64), wz = axis_lines(nz, 64);
    const uint64_t bx = wx ? ((uint64_t)ny * nz + wx - 1) / wx : 0;
    const uint64_t by = wy ? (uint64_t)((nx + wy - 1) / wy) * nz : 0, bz = wz ? (uint64_t)((nx + wz - 1) / wz) * ny : 0;
    if (wx && wy >= 8 && wz >= 8 && bx <= 0x7fffffffu && by <= 0x7fffffffu && bz <= 0x7fffffffu) {
        radius_axis_kernel<<<(unsigned)bx, AXIS_THREADS, (size_t)wx * nx, s>>>(dev_radius, nx, ny, nz, 0, wx);
        radius_axis_kernel<<<(unsigned)by, AXIS_THREADS, (size_t)wy * ny, s>>>(dev_radius, nx, ny, nz, 1, wy);
        radius_axis_kernel<<<(unsigned)bz, AXIS_THREADS, (size_t)wz * nz, s>>>(dev_radius, nx, ny, nz, 2, wz);
    } else {
        for (uint32_t k = 0; k < max_radius; ++k)
            radius_relax_kernel<<<blocks, 256, 0, s>>>(dev_radius, nx, ny, nz);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return mcgb_internal::set_error(MCGB_E_CUDA, cudaGetErrorString(e));
    return MCGB_OK;
}
