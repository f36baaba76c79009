// Boundary-input preparation on the GPU (kernel in qpd_fields.cu): Q-POP-FerroDyn fields in their file order become the
// packed kernel inputs in one pass.
//
// The reference does this on the host in float64 (src/python/cli.py:174-217, loaders in
// src/python/io_utils.py:30-92) and, in its native program, partly in the `columns` kernel
// (src/heffte/kernels.cuh:34-50): transpose (nz, ny, nx) -> (x, y, z), scale P and u, one-hot
// phases of the FE materials, region = (cell is FE) x region file, and the u_z reference ramp
// (cumsum_z dc[mat] - dc[mat] / 2) dz summed over the FULL material stack, then cropped.
//
// Layout: a block owns 32 neighbouring columns of the (y, x) plane, in file order, and one or more chunks of 32 layers
// (qpd_fields_split.h).  A chunk's planes are read with the columns fastest (coalesced in the file order) by warps 1..7
// while warp 0 runs each column's ramp serially in float64, in the order of numpy.cumsum, from layer 0 up to the block's
// first chunk and then through its chunks (1 byte per layer and column); the cropped layers are written transposed with z
// fastest (coalesced in the kernel order) through padded shared tiles.  Bound by memory traffic on volumes and by the
// serial sum on films, so a film's chunks have blocks of their own, which repeat the sums of the layers below, and a wide
// plane's columns sum every layer once.  us per kernel, blocks that walk all chunks of 32 x in one y row, a plane at a
// time -> a block per chunk -> here: 1x400x400 97 -> 24 -> 24, 256x256x64 111 -> 82 -> 82, 512x512x104 637 -> 658 -> 629,
// 1024x1024x68 1810 -> 2373 -> 1809, 256x256x1024 1614 -> 3278 -> 1340, 512x512x104 from layer 500 1338 -> 2018 -> 885.
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
// blocks that fill the device: three rounds of four per SM (with 6 and 8 per SM 128^3 takes 52 us instead of 49)
constexpr int kFieldsBlocks = 12 * 148;
constexpr int kFPitch = kFT + 1;

template <typename T> cudaError_t launch_fields(const FieldsArgs<T>& a, cudaStream_t st);

}  // namespace qpd
