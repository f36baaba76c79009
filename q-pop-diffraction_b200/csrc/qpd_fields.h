// Boundary-input preparation on the GPU (kernel in qpd_fields.cu): Q-POP-FerroDyn fields in their file order become the
// packed kernel inputs in one pass.
//
// The reference does this on the host in float64 (src/python/cli.py:174-217, loaders in
// src/python/io_utils.py:30-92) and, in its native program, partly in the `columns` kernel
// (src/heffte/kernels.cuh:34-50): transpose (nz, ny, nx) -> (x, y, z), scale P and u, one-hot
// phases of the FE materials, region = (cell is FE) x region file, and the u_z reference ramp
// (cumsum_z dc[mat] - dc[mat] / 2) dz summed over the FULL material stack, then cropped.
//
// Layout: a block owns 32 neighbouring columns of the (y, x) plane, in file order, and one chunk of 32
// layers.  Its planes are read with the columns fastest (coalesced in the file order) by warps 1..7 while
// warp 0 runs each column's ramp serially in float64 from layer 0 up to the chunk, in the order of
// numpy.cumsum (a block repeats the sums of the chunks below it, 1 byte per layer and column, so that
// chunks need not wait for one another); the cropped layers are written transposed with z fastest
// (coalesced in the kernel order) through padded shared tiles.  Bound by memory traffic on volumes and
// by the serial sum on films: 1x400x400 takes 24 us on 13 x 13 blocks, where blocks of one y row and 32 x
// that walked the chunks in turn, reading a plane at a time, took 95 us.
#pragma once

#include "qpd_kernels.cuh"

namespace qpd {

constexpr int kMaxMaterials = 64;
constexpr unsigned kFlagBadMaterial = 4u;  // a material index outside the dc / phase_of tables

template <typename T> struct FieldsArgs {
    const float* P[3];        // nStruc planes, (nz, ny, nx)
    const float* u[3];        // null -> 0
    const float* phase;       // nPhase planes of phase fractions, or null: one-hot from the material
    const float* region;      // null -> 1
    const signed char* mat;   // (nz_full, ny, nx)
    long long nx, ny, nz, z0; // crop size and its first layer in the material stack
    int nStruc, nPhase, nMat;
    double dz, p_scale, u_scale;
    double dc[kMaxMaterials];
    signed char phase_of[kMaxMaterials];
    T* Pout;                  // 3 planes of n, (x, y, z)
    T* Uout;
    signed char* phase_idx;   // single mode
    T* weight;
    T* wdense;                // dense mode: nPhase planes
    unsigned int* flags;
};

constexpr int kFT = 32;        // tile edge (x and z)
constexpr int kFRows = 8;      // threadIdx.y extent
constexpr int kFPitch = kFT + 1;

template <typename T> cudaError_t launch_fields(const FieldsArgs<T>& a, cudaStream_t st);

}  // namespace qpd
