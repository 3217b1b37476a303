// The triangles of the forward warp's vertex grid (forward/mesh.rs), one vertex per pixel: T1 = (v[r][c], v[r][c+1],
// v[r+1][c]) and T2 = (v[r+1][c+1], v[r][c+1], v[r+1][c]) of every cell, for the kernels and for host programs.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TW_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TW_HOST_DEVICE inline
#endif

namespace tw {

// A triangle's vertices: the pixel of its cell's first vertex and their distances from it (a frame may have more
// than 2^31 pixels)
struct GridTriangle {
    long first;
    int at[3];
};

// Triangle t of a grid of w x h vertices; false past the last one
TW_HOST_DEVICE bool grid_triangle_at(long t, int w, int h, GridTriangle& g) {
    const int cw = w - 1;
    if (t >= 2l * cw * (h - 1)) return false;
    const long cell = t >> 1;
    // (a 64 bit division takes some 70 instructions)
    const long r = cell >> 32 ? cell / cw : (long)((uint32_t)cell / (uint32_t)cw);
    g.first = cell + r;  // r * w + c for the cell r * (w - 1) + c
    g.at[0] = (t & 1) == 0 ? 0 : w + 1;
    g.at[1] = 1;
    g.at[2] = w;
    return true;
}

}  // namespace tw
