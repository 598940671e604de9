// mdx_pot.cuh -- the potential form's colour-split layout of Phi and r~
// (described in k_sor_mixed.cu), shared by its kernels.
#pragma once

#include "mdx_internal.cuh"

struct pot_geom {
    int nx, ny, nz;
    int hq;   // row length of one half (positions)
    int rz;   // one plane of one half: hq (ny+2)
    int H;    // one half, a multiple of 64 elements
};

__host__ __device__ __forceinline__ int pot_row(const pot_geom& L, int h, int j, int k) {
    return h * L.H + (k * (L.ny + 2) + j) * L.hq;
}
__host__ __device__ __forceinline__ int pot_idx(const pot_geom& L, int i, int j, int k) {
    return pot_row(L, (i + j + k) & 1, j, k) + 3 + (i + 1) / 2;
}

inline pot_geom pot_make(const mdx_dims& d) {
    pot_geom L;
    L.nx = d.nx;
    L.ny = d.ny;
    L.nz = d.nz;
    L.hq = ((d.nx / 2 + 5) + 3) & ~3;
    L.rz = L.hq * (d.ny + 2);
    L.H = (int)((((long long)L.rz * (d.nz + 2)) + 63) & ~63LL);
    return L;
}
