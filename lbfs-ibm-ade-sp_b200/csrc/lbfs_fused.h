// Plan of the fused fluid step of uniform grids (lbfs_fused.cu).
//
// It applies to axis-aligned meshes whose cells form logical grids: each
// instance's cells are i + nx (j + ny k), every interior face joins two cells one
// apart along one axis, owner the lower; every missing side of a cell is one
// boundary face; a cell's gradient stencil is its six neighbours (or ghosts), each
// with a weight along its axis alone and of one magnitude; every face has one area
// and one dt and lies dt from both centres (a boundary face's ghost straight across
// it); a periodic partner is a boundary cell; and gamma is 1.  Cells and faces are in
// the generator's order.  Its uniform meshes and their ensembles meet this; it is
// checked face by face and cell by cell at create, instance by instance, and any
// other instance keeps the separate kernels.
//
// FP64 handles only.  An FP32 form of the pass was bound by instruction issue: alone
// a handle gained by it (32^3 duct 14.2 -> 12.0 us a step, 64^3 34 -> 31.5), but three
// handles of 57x45x33 cells in turn lost (112 -> 122 us for ten steps).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "lbfs_fluid.cuh"

namespace lbfs {

constexpr int kUniformThreads = 128;   // a column each
constexpr int kUniformBlocks = 4;      // blocks an SM, 128 registers a thread
constexpr int kUniformPlaneMax = 230;  // cells of a tile's plane with two more below and one above along x and y

struct GridTile {
    int x0, y0, z0, w, h, d, inst, set;  // columns [x0, x0 + w) x [y0, y0 + h), planes [z0, z0 + d); its GridSet
};
struct GridInst {
    int cell0, nx, ny, nz;
    int side0[6];  // first entry in `side` of the sides -x, +x (j + ny k), -y, +y (i + nx k), -z, +z (i + nx j)
    int active;    // bit d: some face of side d is not zero-gradient in every component
    int pad;
};
// The ghost of one boundary face as its cell's gradients need it: val the
// Dirichlet values (velocity profiles of types 9 and 10 evaluated), flags which
// components take them (the others copy the cell), or the periodic partner's.
struct GridSide {
    Vec4<double> val;
    // bit 0: rho Dirichlet, 1: velocity Dirichlet, 2: rho periodic, 3: velocity periodic, 4: the face takes
    // the velocity val itself (type 1)
    int flags, partner;
};
// One boundary face: its cell, the cell's strides along y and z, info -- its side d,
// up to two more missing sides of the cell << 3 and << 6 (7: none) with their
// boundary faces in more, bit 10: the interior branch (an instance's first ghost), its
// GridSet << 11;
// partner: a boundary face of the periodic partner cell; face: its index among the mesh's boundary faces.
struct alignas(16) GridBnd {
    int cell, sy, sz, info, more[2], partner, face;
};

// Multiples of the slope weight w = dt x gradient weight: 3 w, 3 w^2, w / 2, 3 w / 2, 3 w^2 / 4.
struct GridWeights {
    double w, w3, ww3, h, h3, hh3;
};

// What the faces of grids of one spacing share.
struct GridSet {
    double bnd_k;                  // dt / (owner-ghost distance x w): a Dirichlet ghost's slope in differences
    GridWeights cw;
    double area, dt;               // of every interior face
};

struct GridArgs {
    int n_tiles, n_bnd, bnd_blocks;
    int n_sets;
    int plane_stride;              // cells of the largest tile's plane
    int stage_max;                 // threads that may hold a ghost's record
    const GridTile *tiles;
    const GridInst *inst;
    const GridSide *side;          // the boundary faces of every side of every instance
    const GridBnd *bnd;            // [n_bnd] the boundary faces
    const GridSide *bnd_side;      // [n_bnd] their records in that order
    GridSet set;                   // of all grids (n_sets 1)
    const GridSet *sets;           // else one each
    Vec4<double> *prev;            // [nc + nb] the state the last step started from
    double4 *res;                  // [nc] sums of the interior face fluxes per unit area, those in edge left out
    Vec4<double> *edge;            // [3][nc] low fluxes per unit area of the tiles' first columns, rows and planes
};

size_t grid_smem_bytes(const GridArgs &ga);
cudaError_t grid_prepare();
// boundary face fluxes and the cells' interior sums of one step
void launch_grid_step(const FluidArgs<double> &a, const GridArgs &ga, cudaStream_t s);

}  // namespace lbfs
