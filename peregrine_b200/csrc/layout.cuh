// Device layout of a case's arrays.
//
// Every register (Q, Q1, ... in the reference's naming,
// peregrine/launch/arrays.py:37-39) is one allocation holding every block.
// With cv[b] the cells of the blocks before b and C components per cell,
// block b's component c starts at C * cv[b] + c * vol[b] doubles, and its cell
// (i, j, k), counted from the first halo layer, sits at i + X * (j + Y * k)
// inside that.  i runs fastest, components outermost: the reference's device
// F order (peregrine/backend/device/backend.py:57-58), with the blocks laid
// end to end.  The metric arrays share the layout, 31 components per cell.
// A face array of axis a keeps face f at the index of the cell on its high
// side (the reference indexes a face like the cell to its right,
// peregrine/launch/policy.py:78-86), so faces use the cell layout too.
#pragma once
#include <cstdint>

namespace pgb {

constexpr int NG = 2;  // halo layers: the fused stage's stencil reaches two cells

// metric components inside the metric allocation
enum {
  M_XCC = 0, M_DETJINV = 3, M_JINV = 4, M_S = 13, M_XF = 22, M_NCOMP = 31
};

struct BlockDev {
  int nx, ny, nz;     // interior cells
  int X, Y, Z;        // full extents, nx + 2 NG ...
  long long vol;      // X * Y * Z
  long long cv;       // cells of the blocks before this one
  int uniform;        // 1: the metrics are the per-axis constants below
  // uniform form, every value read off the block's own metric arrays
  double S[3];        // the area vector's normal component of an a-face
  double detJinv;
  double Jd[3];       // inverse Jacobian diagonal
  double ex[3];       // xcc(R) - xcc(L) along a
  double xL[3];       // xf - xcc(L) along a
  double xR[3];       // xf - xcc(R) along a
  // per-axis face geometry alpha damping forms, precomputed from the above
  double damp[3];     // alpha / |e . n| for an a-face (the normal is the axis)
  int bcg;            // bit f: face f is an inflow or outflow, whose halo cells take their images' gradients
};

__host__ __device__ __forceinline__ long long cell_index(const BlockDev &b, int fi, int fj, int fk) {
  return (long long)fi + (long long)b.X * ((long long)fj + (long long)b.Y * fk);
}

// the index in its block of interior cell t, i fastest (a block's cells fit
// 32 bits: its arrays' component strides do)
__host__ __device__ __forceinline__ long long inner_cell(const BlockDev &b, long long t) {
  const unsigned u = (unsigned)t, r = u / (unsigned)b.nx, i = u - r * (unsigned)b.nx;
  const unsigned k = r / (unsigned)b.ny, j = r - k * (unsigned)b.ny;
  return cell_index(b, (int)i + NG, (int)j + NG, (int)k + NG);
}

// The per-cell state of the per-block path, fields of one cell SW apart in
// vol-strided planes: the EosState (p, T, rhoinv, rho, e, cp, gamma, c), the
// real gas's root Z, and the double flux's tangent plane of rho e
// (theta, eps, kappa, zeta[ns - 1]) (peregrine/simulator/mixture/eos/base.py:85-86,
// realgas/model.py:31-34, realgasdf/model.py:8-10)
constexpr int SW = 24;
// The ideal gases leave the plane's fields unused and, on uniform blocks of the
// fused passes, keep the cell's velocity at the record's end (uniface.cuh); the
// double flux's batched stages keep a second pressure there (12 species leave
// the last field free).
enum { ST_Z = 8, ST_THETA = 9, ST_EPS = 10, ST_KAPPA = 11, ST_ZETA = 12, ST_U = 21, ST_P2 = 23 };

// Where a per-block kernel's thread works: its block and its index t in the
// pass's range over that block.  With a tile table (a packed launch over many
// blocks), CTA x does tile ctab[x].y of block row ctab[x].x, so a launch has
// exactly the CTAs its blocks need; without one, the block is b plus the grid
// row and the tile the CTA's x.  The kernel names its block index b, its
// descriptor table blks and its tile table ctab.
#define PGB_WHERE(B, t)                                                                              \
  const int2 where_ = ctab ? ctab[blockIdx.x] : make_int2(b + (int)blockIdx.y, (int)blockIdx.x); \
  const BlockDev &B = blks[where_.x];                                                                \
  const long long t = (long long)where_.y * blockDim.x + threadIdx.x

// Where a thread of a pass over the faces of all three axes works: RF_TH
// faces a CTA, the CTAs axis by axis (n0 of axis 0, n1 of axis 1, the rest
// axis 2), a grid row a block; with tile tables (the three axes' end to end)
// each 256-face tile is two CTAs.  Returns the axis; the block and the face's
// number in it in row and t.
constexpr int RF_TH = 128;
#ifdef __CUDACC__
__device__ __forceinline__ int face_work(const unsigned n0, const unsigned n1, const int2 *__restrict__ ctab, int &row,
                                         unsigned &t) {
  const unsigned x = blockIdx.x;
  const int axis = x < n0 ? 0 : x < n0 + n1 ? 1 : 2;
  if (ctab) {
    const int2 w = ctab[x >> 1];
    row = w.x;
    t = (unsigned)w.y * 256u + (x & 1) * RF_TH + threadIdx.x;
  } else {
    row = (int)blockIdx.y;
    t = (x - (axis == 0 ? 0 : axis == 1 ? n0 : n0 + n1)) * RF_TH + threadIdx.x;
  }
  return axis;
}
// face t of an axis of a block as the index of the cell on its high side
// and its place along the axis in pos
__device__ __forceinline__ bool face_cell(const BlockDev &B, const int axis, const unsigned t, long long &R, int &pos) {
  const unsigned fx = B.nx + (axis == 0), fy = B.ny + (axis == 1), fz = B.nz + (axis == 2);
  const unsigned r = t / fx, i = t - r * fx, k = r / fy, j = r - k * fy;
  if (k >= fz) return false;
  pos = (int)(axis == 0 ? i : axis == 1 ? j : k);
  R = cell_index(B, (int)i + NG, (int)j + NG, (int)k + NG);
  return true;
}
#endif

// one cell of a halo filled from another cell: each side's block start in
// cells (cv), its cell index inside the block and its component stride
// (vol); rot, when not 0, the rotation (rot - 1 in the case's table) a
// rotationally periodic interface turns the cell's vectors by
struct HaloEntry {
  long long dcv, scv;
  int didx, sidx, dvol, svol;
  int rot;
};

// A box of halo cells of one block whose sources all lie in one block, the
// source index an affine map of the destination cell: a face's halo NG deep,
// an edge line one deep.  The box runs i fastest in the destination, so a
// warp's threads write neighbouring cells; t = x0 + n0 (x1 + n1 x2) is the
// thread's cell in it, the indices d0 + x . dst and s0 + x . sst.
struct HaloPatch {
  long long dcv, scv;
  int dvol, svol;
  int d0, s0;
  int dst[3], sst[3];
  int n0, n1, cells;
  int rot;
};

// what k_halo turns with an entry's rotation: nothing, the vector at a
// component (Q's momentum at 1), or the gradients' tensor (each row's three
// directions, and the velocity rows u, v, w down every direction)
enum { HALO_SCALARS = -1, HALO_TENSOR = -2 };

// a fused work item: a column of tw x th cells of one block over k0 .. k1 - 1
struct TileDev {
  int blk;
  short i0, j0, tw, th, k0, k1;
};

}  // namespace pgb
