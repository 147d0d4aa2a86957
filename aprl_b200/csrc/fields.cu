// fields.cu -- grid kernels of the step: Cowan-z Faraday with the CPML
// magnetic correction, the zero-current Ampere preview with the CPML
// electric correction, PEC termination and inlet overwrite, the commit
// E^{n+1} = E* - dt/eps0 J, and the moving-window plane insertion.
//
// E, B and the CPML histories are binary64 in every mode, and every
// expression keeps the reference's operation order; the library is compiled
// without FMA contraction, so these kernels reproduce the reference's
// translation units bit for bit.  The kernels are templated on the type F of
// the current J, which only the filter passes read.
#include "common.cuh"
#include "dd.cuh"
#include "fields.cuh"

namespace aprl_gpu {

// transformedCorrection (src/eb_cpml.cpp:131-138).
__device__ __forceinline__ double cpml_correction(const CpmlAxis& ax, int index,
                                                  double difference, double* history) {
  const double psi = ax.decay[index] * *history + ax.drive[index] * difference;
  *history = psi;
  return ax.inverse_kappa_minus_one[index] * difference + psi;
}

__device__ __forceinline__ double* history_at(const CpmlHistory& h, int slot, int k, int zbase,
                                              int row_index, DeviceStatus* status) {
  (void)status;
  return h.data + APRL_BOUNDED(status,
                               (unsigned)((slot * h.layers + ring(k, zbase, h.layers)) *
                                              (unsigned)h.row +
                                          row_index),
                               (size_t)h.slots * h.layers * h.row, 16);
}

// advanceMagneticCowan (src/eb_field.cpp:488-558) fused with
// EBConvolutionalPML::afterMagneticUpdate (src/eb_cpml.cpp:406-468).
//
// A block owns a TX x TY tile of (i, j) columns and marches a chunk of z
// planes.  The three E components of planes k-1, k, k+1 live in a shared
// memory ring, one (TX+2) x (TY+2) tile each, loaded once per plane through
// the reference electricValue's parity/halo rules (map_tile).  Every smoothed
// difference (the 9-point smoothedElectric of src/eb_field.cpp:419-486: alpha*centre, the
// four beta edge samples, the four delta corners) is then evaluated from
// shared memory in the reference's order, so the FP64 update is
// bit-identical to the reference.  Each B node is updated by the
// curl, then by its CPML terms in the reference's term order (0,2,1),
// (1,2,0), (2,1,0), (2,0,1), reusing the curl's smoothed difference.
constexpr int kTX = kCowanTileX, kTY = kCowanTileY;

struct ETile {
  double v[3][3][kTY + 2][kTX + 2];  // [component][plane slot][y][x]
};

// Ring slots of the tile planes k-1, k, k+1 of the current z-march step,
// rotated by one per step (no modular arithmetic in the stencil).
struct PlaneSlots {
  int s[3];
};

__device__ __forceinline__ double tile_at(const ETile& t, int c, int li, int lj, int dk,
                                          const PlaneSlots& ps) {
  return t.v[c][ps.s[dk + 1]][lj][li];
}

// smoothedElectric from the tile: centre (li, lj) in tile coordinates, dk
// the plane offset (-1..1) from the marching plane; every offset is a
// compile-time constant after inlining, so the plane choice is a register.
template <class F>
__device__ __forceinline__ double tile_smoothed(const ETile& t, const CowanArgs<F>& a, int c,
                                                int d, int li, int lj, int dk,
                                                const PlaneSlots& ps) {
  const int ta = (d + 1) % 3, tb = (d + 2) % 3;
  const double delta = d == 0 ? a.delta_yz : (d == 1 ? a.delta_zx : a.delta_xy);
  const int p[3] = {li, lj, dk};
  double result = a.alpha[d] * tile_at(t, c, li, lj, dk, ps);
#pragma unroll
  for (int dir = -1; dir <= 1; dir += 2) {
    int qa[3] = {p[0], p[1], p[2]}, qb[3] = {p[0], p[1], p[2]};
    qa[ta] += dir;
    qb[tb] += dir;
    result += a.beta[ta] * tile_at(t, c, qa[0], qa[1], qa[2], ps);
    result += a.beta[tb] * tile_at(t, c, qb[0], qb[1], qb[2], ps);
  }
#pragma unroll
  for (int da = -1; da <= 1; da += 2)
#pragma unroll
    for (int db = -1; db <= 1; db += 2) {
      int q[3] = {p[0], p[1], p[2]};
      q[ta] += da;
      q[tb] += db;
      result += delta * tile_at(t, c, q[0], q[1], q[2], ps);
    }
  return result;
}

// A thread's share of a tile plane: which E value each of its entries holds
// under electricValue's x and y rules (parity extension at the PEC walls).
// The rules do not depend on the plane, so they are evaluated once a march;
// evaluated for every value of every plane they were most of the kernel's
// instructions, in the boundary tiles that are over half of a 129-node row's.
// Only coordinates within one cell of a component's index range are ever used
// by the smoothing (the reference's own reach); tile points farther out, which
// exist only where a small grid ends inside a tile, hold zero.
constexpr int kTileW = kTX + 2, kTileN = (kTX + 2) * (kTY + 2), kTileT = kTX * kTY,
              kTileR = (kTileN + kTileT - 1) / kTileT;

struct TileMap {
  int at[3][kTileR];  // offset in the component's plane, -1: none
  unsigned odd;       // bit kTileR * c + r: the entry is a sign-reversed mirror image
};

template <class F>
__device__ __forceinline__ void map_tile(TileMap& m, const CowanArgs<F>& a, int i0, int j0) {
  const int tid = threadIdx.y * kTX + threadIdx.x;
  m.odd = 0u;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int nxc = a.g.nx + (c != 0), nyc = a.g.ny + (c != 1);
#pragma unroll
    for (int r = 0; r < kTileR; ++r) {
      const int n = tid + r * kTileT;
      const int jj = n / kTileW;
      int i = i0 - 1 + (n - jj * kTileW), j = j0 - 1 + jj;
      m.at[c][r] = -1;
      if (n >= kTileN || i > nxc || j > nyc) continue;
      bool odd = false;
      if (i < 0 || i >= nxc) {
        if (c != 0) odd = !odd;
        i = i < 0 ? (c == 0 ? 0 : -i) : (c == 0 ? nxc - 1 : 2 * (nxc - 1) - i);
      }
      if (j < 0 || j >= nyc) {
        if (c != 1) odd = !odd;
        j = j < 0 ? (c == 1 ? 0 : -j) : (c == 1 ? nyc - 1 : 2 * (nyc - 1) - j);
      }
      m.at[c][r] = j * nxc + i;
      if (odd) m.odd |= 1u << (kTileR * c + r);
    }
  }
}

// Fills one plane of the tile: the inlet's halo plane below the grid, zero
// above it.
template <class F>
__device__ __forceinline__ void load_plane(ETile& t, const TileMap& m, const CowanArgs<F>& a,
                                           int k, int slot) {
  const int tid = threadIdx.y * kTX + threadIdx.x;
  // All of a thread's loads are issued before any shared-memory store, so
  // their latencies overlap instead of adding up.
  double v[3][kTileR];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int nxc = a.g.nx + (c != 0), nyc = a.g.ny + (c != 1), nzc = a.g.nz + (c != 2);
    const unsigned plane = nxc * nyc;
    const double* from =
        k < 0 ? a.lower[c] : a.e[c] + (k < nzc ? ring(k, a.g.zb_e[c], nzc) * plane : 0u);
#pragma unroll
    for (int r = 0; r < kTileR; ++r)
      v[c][r] = m.at[c][r] >= 0 && k < nzc
                    ? from[APRL_BOUNDED(a.g.status, m.at[c][r], plane, 10 + c)]
                    : 0.0;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < kTileR; ++r) {
      const int n = tid + r * kTileT;
      if (n < kTileN)
        (&t.v[c][slot][0][0])[n] = (m.odd >> (kTileR * c + r)) & 1u ? -v[c][r] : v[c][r];
    }
}

template <class F>
__global__ void __launch_bounds__(kTX * kTY, APRL_COWAN_MIN_BLOCKS)
    cowan_magnetic_kernel(CowanArgs<F> a) {
  __shared__ ETile t;
  const GridT<F>& g = a.g;
  const int i0 = blockIdx.x * kTX, j0 = blockIdx.y * kTY;
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  const int k0 = blockIdx.z * a.chunk;
  const int k1 = min(k0 + a.chunk, g.nz + 1);
  const double dtdx = a.dtdx, dtdy = a.dtdy, dtdz = a.dtdz;
  const int li = threadIdx.x + 1, lj = threadIdx.y + 1;
  PlaneSlots ps = {{0, 1, 2}};
  TileMap map;
  map_tile(map, a, i0, j0);
  load_plane(t, map, a, k0 - 1, ps.s[0]);
  load_plane(t, map, a, k0, ps.s[1]);
  // The column's CPML slots are the same on every plane of the march.
  const bool column = i <= g.nx && j <= g.ny;
  const int slot_x = column && i < g.nx ? a.mx.ordinal[i] : -1;
  const int slot_y = column && j < g.ny ? a.my.ordinal[j] : -1;
  // The z differences smooth within one plane (x and y neighbours), so the
  // smoothed Ey and Ex of plane k+1 are, bit for bit, the plane-k operands
  // of the next step: carried in registers instead of evaluated again.
  double ey_above = 0.0, ex_above = 0.0;
  for (int k = k0; k < k1; ++k) {
    load_plane(t, map, a, k + 1, ps.s[2]);
    // The node's three B values are read before the first B store (which
    // may alias them as far as the compiler knows).
    const bool has_bx = column && j < g.ny && k < g.nz;
    const bool has_by = column && i < g.nx && k < g.nz;
    const bool has_bz = column && i < g.nx && j < g.ny;
    double* const bx = has_bx ? &g.b[0][b_index(g, 0, i, j, k)] : nullptr;
    double* const by = has_by ? &g.b[1][b_index(g, 1, i, j, k)] : nullptr;
    double* const bz = has_bz ? &g.b[2][b_index(g, 2, i, j, k)] : nullptr;
    const double bx_old = has_bx ? *bx : 0.0;
    const double by_old = has_by ? *by : 0.0;
    const double bz_old = has_bz ? *bz : 0.0;
    __syncthreads();
    if (i <= g.nx && j <= g.ny) {
      if (j < g.ny && k < g.nz) {  // Bx (nx+1, ny, nz)
        const double dEzDy = tile_smoothed(t, a, 2, 1, li, lj + 1, 0, ps) -
                             tile_smoothed(t, a, 2, 1, li, lj, 0, ps);
        const double ey_here = k > k0 ? ey_above : tile_smoothed(t, a, 1, 2, li, lj, 0, ps);
        ey_above = tile_smoothed(t, a, 1, 2, li, lj, 1, ps);
        const double dEyDz = ey_above - ey_here;
        double v = bx_old - (dtdy * dEzDy - dtdz * dEyDz);
        const int s = slot_y;
        if (s >= 0)
          v += -1.0 * dtdy * cpml_correction(a.my, j, dEzDy,
                                             history_at(a.h[0], s, k, g.zb_b[0], i, g.status));
        *bx = v;
      }
      if (i < g.nx && k < g.nz) {  // By (nx, ny+1, nz)
        const double ex_here = k > k0 ? ex_above : tile_smoothed(t, a, 0, 2, li, lj, 0, ps);
        ex_above = tile_smoothed(t, a, 0, 2, li, lj, 1, ps);
        const double dExDz = ex_above - ex_here;
        const double dEzDx = tile_smoothed(t, a, 2, 0, li + 1, lj, 0, ps) -
                             tile_smoothed(t, a, 2, 0, li, lj, 0, ps);
        double v = by_old - (dtdz * dExDz - dtdx * dEzDx);
        const int s = slot_x;
        if (s >= 0)
          v += 1.0 * dtdx * cpml_correction(a.mx, i, dEzDx,
                                            history_at(a.h[1], s, k, g.zb_b[1], j, g.status));
        *by = v;
      }
      if (i < g.nx && j < g.ny) {  // Bz (nx, ny, nz+1)
        const double dEyDx = tile_smoothed(t, a, 1, 0, li + 1, lj, 0, ps) -
                             tile_smoothed(t, a, 1, 0, li, lj, 0, ps);
        const double dExDy = tile_smoothed(t, a, 0, 1, li, lj + 1, 0, ps) -
                             tile_smoothed(t, a, 0, 1, li, lj, 0, ps);
        double v = bz_old - (dtdx * dEyDx - dtdy * dExDy);
        const int sx = slot_x;
        if (sx >= 0)
          v += -1.0 * dtdx * cpml_correction(a.mx, i, dEyDx,
                                             history_at(a.h[2], sx, k, g.zb_b[2], j, g.status));
        const int sy = slot_y;
        if (sy >= 0)
          v += 1.0 * dtdy * cpml_correction(a.my, j, dExDy,
                                            history_at(a.h[3], sy, k, g.zb_b[2], i, g.status));
        *bz = v;
      }
    }
    __syncthreads();
    ps = PlaneSlots{{ps.s[1], ps.s[2], ps.s[0]}};
  }
}

// advanceElectric with J = 0 (src/eb_field.cpp:582-627) followed by the
// moving-window boundary (src/moving_window_fields.cpp:254-293): the CPML
// electric terms (src/eb_cpml.cpp:470-539; the convolution histories are
// advanced here once, exactly as the later commit would advance them from
// the same B), PEC on the x/y faces, and the inlet Ex/Ey overwrite at k=0.
// Reads E^n from e_old, writes E* to e_star.
//
// One thread per (i, j) column, marching `chunk` planes: the column's
// predicates, offsets and CPML slots are formed once, a plane's base pointers
// are the same for the whole block, and Bx and By of the plane below stay in
// registers.  One thread per node spent 740 instructions on a node's twelve
// reads, four divisions and some 60 floating-point operations.  On the
// 128x128x512 grid, with the orbit sum written: 0.234 -> 0.225 ms at 2 planes
// (1 plane 0.235, 4 planes 0.226, 16 planes 0.25-0.26: a plane's latency is
// then serial); the 805 MB it moves take 0.123 ms at the copy rate.
template <class F>
__global__ void __launch_bounds__(256, 4) electric_preview_kernel(PreviewArgs<F> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const GridT<F>& g = a.g;
  if (i > g.nx || j > g.ny) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int k0 = blockIdx.z * a.chunk, k1 = min(k0 + a.chunk, nz + 1);
  const double cx = a.cx, cy = a.cy, cz = a.cz;
  const bool has_x = i < nx, has_y = j < ny;
  const bool x_row = has_x && j >= 1 && j < ny;  // Ex: y difference of Bz
  const bool y_row = has_y && i >= 1 && i < nx;  // Ey: x difference of Bz
  const bool z_col = i >= 1 && i < nx && j >= 1 && j < ny;
  const int slot_x = has_x ? a.ex_prof.ordinal[i] : -1;
  const int slot_y = has_y ? a.ey_prof.ordinal[j] : -1;
  // Offsets in a plane of rows nx and nx + 1 wide, and the planes' sizes.
  const int on = j * nx + i, ow = j * (nx + 1) + i;
  const unsigned pe0 = nx * (ny + 1), pe1 = (nx + 1) * ny, pe2 = (nx + 1) * (ny + 1),
                 pbz = nx * ny;
  auto plane = [&](const double* v, int k, int zb, int n, unsigned size) {
    return v + ring(k, zb, n) * size;
  };
  auto at = [&](const double* v, unsigned offset, unsigned size, unsigned site) {
    (void)size;
    (void)site;
    return v[APRL_BOUNDED(g.status, offset, size, site)];
  };
  // The plane below: By for Ex and Bx for Ey.
  double by_k = 0.0, bx_k = 0.0;
  if (k0 >= 1 && k0 <= nz) {
    if (x_row) by_k = at(plane(g.b[1], k0 - 1, g.zb_b[1], nz, pe0), on, pe0, 5);
    if (y_row) bx_k = at(plane(g.b[0], k0 - 1, g.zb_b[0], nz, pe1), ow, pe1, 4);
  }
  for (int k = k0; k < k1; ++k) {
    // Every E and B read of the node is issued before its first store (the
    // stores may alias them as far as the compiler knows).
    const bool has_z = k < nz, inner_k = k >= 1 && k < nz;
    const unsigned b0 = ring(k, g.zb_e[0], nz + 1) * pe0, b1 = ring(k, g.zb_e[1], nz + 1) * pe1,
                   b2 = has_z ? ring(k, g.zb_e[2], nz) * pe2 : 0u;
    const double* const pz = plane(g.b[2], k, g.zb_b[2], nz + 1, pbz);
    const double old0 = has_x ? at(g.e_old[0] + b0, on, pe0, 1) : 0.0;
    const double old1 = has_y ? at(g.e_old[1] + b1, ow, pe1, 2) : 0.0;
    const double old2 = has_z ? at(g.e_old[2] + b2, ow, pe2, 3) : 0.0;
    const double bz = x_row || y_row ? (has_x && has_y ? at(pz, on, pbz, 6) : 0.0) : 0.0;
    const double bz_j = x_row ? at(pz, on - nx, pbz, 6) : 0.0;
    const double bz_i = y_row ? at(pz, on - 1, pbz, 6) : 0.0;
    double by = 0.0, by_i = 0.0, bx = 0.0, bx_j = 0.0;
    if (has_z) {
      const double* const py = plane(g.b[1], k, g.zb_b[1], nz, pe0);
      const double* const px = plane(g.b[0], k, g.zb_b[0], nz, pe1);
      if (x_row) by = at(py, on, pe0, 5);
      if (y_row) bx = at(px, ow, pe1, 4);
      if (z_col) {
        by_i = at(py, on - 1, pe0, 5);
        bx_j = at(px, ow - (nx + 1), pe1, 4);
      }
    }
    if (has_x) {  // Ex (nx, ny+1, nz+1)
      double v = old0;
      if (x_row && inner_k) v += cy * (bz - bz_j) - cz * (by - by_k);
      if (x_row && slot_y >= 0) {
        const double diff = bz - bz_j;
        v += 1.0 * cy * cpml_correction(a.ey_prof, j, diff,
                                        history_at(a.h[0], slot_y, k, g.zb_e[0], i, g.status));
      }
      if (j == 0 || j == ny) v = 0.0;
      if (k == 0) {
        if (a.pre_inlet[0]) a.pre_inlet[0][APRL_BOUNDED(g.status, on, pe0, 22)] = v;
        v = inlet_value(a.inlet, 0, i, j);
      }
      g.e_star[0][APRL_BOUNDED(g.status, b0 + on, e_count(g, 0), 67)] = v;
      if (a.sum[0])
        a.sum[0][APRL_BOUNDED(g.status, b0 + on, e_count(g, 0), 70)] = v + old0;
    }
    if (has_y) {  // Ey (nx+1, ny, nz+1)
      double v = old1;
      if (y_row && inner_k) v += cz * (bx - bx_k) - cx * (bz - bz_i);
      if (y_row && slot_x >= 0) {
        const double diff = bz - bz_i;
        v += -1.0 * cx * cpml_correction(a.ex_prof, i, diff,
                                         history_at(a.h[1], slot_x, k, g.zb_e[1], j, g.status));
      }
      if (i == 0 || i == nx) v = 0.0;
      if (k == 0) {
        if (a.pre_inlet[1]) a.pre_inlet[1][APRL_BOUNDED(g.status, ow, pe1, 23)] = v;
        v = inlet_value(a.inlet, 1, i, j);
      }
      g.e_star[1][APRL_BOUNDED(g.status, b1 + ow, e_count(g, 1), 68)] = v;
      if (a.sum[0])
        a.sum[1][APRL_BOUNDED(g.status, b1 + ow, e_count(g, 1), 71)] = v + old1;
    }
    if (has_z) {  // Ez (nx+1, ny+1, nz)
      double v = old2;
      if (z_col) {
        const double dby = by - by_i, dbx = bx - bx_j;
        v += cx * dby - cy * dbx;
        if (slot_x >= 0)
          v += 1.0 * cx * cpml_correction(a.ex_prof, i, dby,
                                          history_at(a.h[2], slot_x, k, g.zb_e[2], j, g.status));
        if (slot_y >= 0)
          v += -1.0 * cy * cpml_correction(a.ey_prof, j, dbx,
                                           history_at(a.h[3], slot_y, k, g.zb_e[2], i, g.status));
      }
      if (i == 0 || i == nx || j == 0 || j == ny) v = 0.0;
      g.e_star[2][APRL_BOUNDED(g.status, b2 + ow, e_count(g, 2), 69)] = v;
      if (a.sum[0])
        a.sum[2][APRL_BOUNDED(g.status, b2 + ow, e_count(g, 2), 72)] = v + old2;
    }
    by_k = by;
    bx_k = bx;
  }
}

// Boundary::begin lower halo planes (src/moving_window_fields.cpp:206-210):
// reference(a, i, j, offset-1, step) for Ex, Ey, Ez.
__global__ void inlet_lower_kernel(InletPlaneArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z;
  const int nxc = a.nx + (c != 0), nyc = a.ny + (c != 1);
  if (i >= nxc || j >= nyc) return;
  a.out[c][(size_t)j * nxc + i] = inlet_value(a.inlet, c, i, j);
}

__global__ void inlet_complete_kernel(InletCompleteArgs a) {
  const DGrid& g = a.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i <= a.cx || i >= g.nx - a.cx || j <= a.cy || j >= g.ny - a.cy) return;
  // The reference evaluates this in long double; double-double here.
  const DD dex = two_sum(g.e_old[0][e_index(g, 0, i, j, 1)], -g.e_old[0][e_index(g, 0, i - 1, j, 1)]);
  const DD dey = two_sum(g.e_old[1][e_index(g, 1, i, j, 1)], -g.e_old[1][e_index(g, 1, i, j - 1, 1)]);
  const DD divxy = dd_add(dd_div(dex, g.dx), dd_div(dey, g.dy));
  const DD source = dd_div(DD{a.rho[(size_t)j * (g.nx + 1) + i], 0.}, kEpsilon0);
  const DD change = dd_mul(dd_add(divxy, dd_neg(source)), g.dz);
  const double value = dd_value(dd_add(DD{g.e_old[2][e_index(g, 2, i, j, 1)], 0.}, change));
  if (!isfinite(value)) {
    raise_error(a.status, kErrInletField, (unsigned long long)((size_t)j * (g.nx + 1) + i));
    return;
  }
  g.e_old[2][e_index(g, 2, i, j, 0)] = value;
}

__global__ void inlet_halo_kernel(InletHaloArgs a) {
  const DGrid& g = a.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i <= a.cx || i >= g.nx - a.cx || j <= a.cy || j >= g.ny - a.cy) return;
  a.lower_ez[(size_t)j * (g.nx + 1) + i] -=
      g.e_old[2][e_index(g, 2, i, j, 0)] - inlet_value(a.inlet, 2, i, j);
}

// MovingWindowFields::shift plane insertion (src/moving_window_fields.cpp:
// 470-517) on the ring: after the bases moved down by one, logical plane 0
// (the dropped upper plane's storage) receives reference(a, i, j, offset,
// step) for E and B, and every CPML history gets a zero layer at k = 0.
template <class F>
__global__ void shift_insert_kernel(ShiftArgs<F> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z;  // 0..5 fields, 6..13 histories
  const GridT<F>& g = a.g;
  if (c < 3) {
    const int nxc = e_nx(g, c), nyc = e_ny(g, c);
    if (i >= nxc || j >= nyc) return;
    g.e_old[c][e_index(g, c, i, j, 0)] = inlet_value(a.inlet, c, i, j);
  } else if (c < 6) {
    const int b = c - 3;
    const int nxc = b_nx(g, b), nyc = b_ny(g, b);
    if (i >= nxc || j >= nyc) return;
    g.b[b][b_index(g, b, i, j, 0)] = inlet_value(a.inlet, c, i, j);
  } else {
    const CpmlHistory& h = a.h[c - 6];
    // i runs over the row, j over the slots.
    if (i >= h.row || j >= h.slots) return;
    *history_at(h, j, 0, a.history_base[c - 6], i, g.status) = 0.0;
  }
}

// The particle shape's filter, applied on the grid once per trial instead of
// once per particle and node.  With raw J the narrow deposits,
//   J = filter(raw J)                       (linear-binomial3: x and z;
//                                            quintic-compensated: z)
//   E_new = E* - dt/eps0 J                  (applyCurrentSource's mask)
//   S = E_new + E^n = S0 - dt/eps0 J        (S0 = E* + E^n from the preview)
// and the gathers read filter(S).  A deposit or gather over the wide stencil
// skips the nodes outside a component, so both filters take zero there.
//
// A warp owns 32 x nodes of one row (j) of one component and marches z: the
// x filter takes its neighbours by shuffle (28 of the 32 lanes write, the
// filter reaching two nodes in all), the z filter keeps the last planes in
// registers.  Nothing couples rows in y, and every array is read and written
// once, but for the planes a chunk shares with its neighbours.
__device__ __forceinline__ double lane_filter(double v) {
  const double lo = __shfl_up_sync(0xffffffffu, v, 1), hi = __shfl_down_sync(0xffffffffu, v, 1);
  return fma(0.25, lo + hi, 0.5 * v);
}

// z filter of S = 0: the three planes' values oldest first; S = 1: seven.
template <int S>
struct ZWindow {
  static constexpr int R = S == 0 ? 1 : 3, N = 2 * R + 1;
  double v[N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int t = 0; t < N; ++t) v[t] = 0.;
  }
  __device__ __forceinline__ void push(double x) {
#pragma unroll
    for (int t = 0; t + 1 < N; ++t) v[t] = v[t + 1];
    v[N - 1] = x;
  }
  __device__ __forceinline__ double value() const {  // at the window's middle plane
    if constexpr (S == 0) {
      return fma(0.25, v[0] + v[2], 0.5 * v[1]);
    } else {
      double r = kQuinticC64[3] * v[3];
      r = fma(kQuinticC64[2], v[2] + v[4], r);
      r = fma(kQuinticC64[1], v[1] + v[5], r);
      return fma(kQuinticC64[0], v[0] + v[6], r);
    }
  }
};

// One lane's column of a filter pass.
struct FilterMarch {
  unsigned plane, nplane;  // plane sizes of the padded arrays and of E
  int row, node;           // the lane's offsets in a plane of either
  int nzc, zb, zlo, zhi;   // planes, ring base, the mask's planes
  bool inside, raw_in, writes, column;
  const double *raw, *sum;
  double* star;
  void* out;
};

// Output planes from k0 on, the candidate sum's planes [s0, s1).  A plane costs
// few arithmetic operations, so the loop is kept to them: 32-bit offsets that
// step by a plane, the ring's wrap a uniform test, two planes' reads together
// (with the tests and 64-bit offsets of every plane the guess pass took 85
// instructions a plane, of which 12 were arithmetic and memory).
template <int S, int MODE, class W, bool WHOLE>
__device__ __forceinline__ void filter_march(const GridT<double>& g, const FilterMarch& m, int c,
                                             int k0, int s0, int s1) {
  constexpr int R = ZWindow<S>::R;
  constexpr bool kOrbit = MODE == kFilterGuess || MODE == kFilterOrbit;
  constexpr bool kRaw = MODE != kFilterGuess;
  ZWindow<S> wj, ws;
  wj.clear();
  ws.clear();
  // Offsets of plane k of the raw current (modulo 2^32 below the array, where
  // nothing is read), and of the ring's plane p.
  unsigned raw_off = (unsigned)(s0 - R + g.jpad) * m.plane + m.row;
  auto raw_at = [&](int k) -> double {
    if (!m.raw_in || (!WHOLE && (k < -g.jpad || k >= m.nzc + g.jpad))) return 0.;
    return m.raw[APRL_BOUNDED(g.status, raw_off, j_count(g, c), 33 + c)];
  };
  int p = ring(max(s0, 0) < m.nzc ? max(s0, 0) : 0, m.zb, m.nzc);
  unsigned ring_off = p * m.nplane + m.node;
  auto next_ring = [&](int k) {  // from plane k on to the next
    if (!WHOLE && k < 0) return;
    ring_off += m.nplane;
    if (++p == m.nzc) {
      p = 0;
      ring_off = m.node;
    }
  };
  auto sum_at = [&](int k) -> double {
    if (!m.inside || (!WHOLE && (k < 0 || k >= m.nzc))) return 0.;
    return m.sum[APRL_BOUNDED(g.status, ring_off, e_count(g, c), 36 + c)];
  };
  if constexpr (kRaw) {
#pragma unroll
    for (int t = -R; t < R; ++t) {
      double v = raw_at(s0 + t);
      raw_off += m.plane;
      if constexpr (S == 0) v = lane_filter(v);
      wj.push(v);
    }
  }
  unsigned out_off = kOrbit ? (unsigned)(k0 + g.jpad) * m.plane + m.row
                            : (unsigned)k0 * m.nplane + m.node;
  constexpr int U = MODE == kFilterCommit ? 4 : 2;
  for (int kb = s0; kb < s1; kb += U) {
    double raw_v[U], sum_v[U];
    unsigned star_off[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      raw_v[u] = sum_v[u] = 0.;
      star_off[u] = ring_off;
      if (kb + u >= s1) break;
      if constexpr (kRaw) {
        raw_v[u] = raw_at(kb + u + R);
        raw_off += m.plane;
      }
      if constexpr (kOrbit) sum_v[u] = sum_at(kb + u);
      if constexpr (kOrbit || MODE == kFilterCommit) next_ring(kb + u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = kb + u;
      if (k >= s1) break;
      double current = 0.;
      if constexpr (kRaw) {
        double v = raw_v[u];
        if constexpr (S == 0) v = lane_filter(v);
        wj.push(v);
        current = wj.value();
      }
      const bool masked = m.column && (WHOLE || (k >= m.zlo && k <= m.zhi));
      if constexpr (MODE == kFilterCommit) {
        if (m.writes && masked && current != 0.)
          m.star[APRL_BOUNDED(g.status, star_off[u], e_count(g, c), 39 + c)] += g.jcoef * current;
      } else if constexpr (MODE == kFilterCurrent) {
        if (m.writes)
          static_cast<double*>(m.out)[APRL_BOUNDED(g.status, out_off, e_count(g, c), 60 + c)] =
              current;
        out_off += m.nplane;
      } else {
        double s = sum_v[u];
        if (masked && current != 0.) s += g.jcoef * current;
        if constexpr (S == 0) s = lane_filter(s);
        ws.push(s);
        if (k - R >= k0) {
          if (m.writes)
            static_cast<W*>(m.out)[APRL_BOUNDED(g.status, out_off, j_count(g, c), 42 + c)] =
                W(ws.value());
          out_off += m.plane;
        }
      }
    }
  }
}

template <int S, int MODE, class W>
__global__ void current_filter_kernel(FilterArgs a) {
  const GridT<double>& g = a.g;
  if (trial_skipped(g)) return;
  constexpr int R = ZWindow<S>::R;
  constexpr bool kOrbit = MODE == kFilterGuess || MODE == kFilterOrbit;
  const int lane = threadIdx.x & 31;
  const int tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  // Select by branch: a run-time index into the parameter arrays would copy
  // them to local memory.
  const int c = blockIdx.z / a.chunks;
  const int nxc = e_nx(g, c), nyc = e_ny(g, c), nzc = e_nz(g, c);
  const int zb = c == 0 ? g.zb_e[0] : (c == 1 ? g.zb_e[1] : g.zb_e[2]);
  const double* raw = c == 0 ? g.j[0] : (c == 1 ? g.j[1] : g.j[2]);
  const double* sum = c == 0 ? a.sum[0] : (c == 1 ? a.sum[1] : a.sum[2]);
  double* star = c == 0 ? g.e_star[0] : (c == 1 ? g.e_star[1] : g.e_star[2]);
  void* out = c == 0 ? a.out[0] : (c == 1 ? a.out[1] : a.out[2]);
  if (MODE == kFilterCurrent && !out) return;  // not the component asked for
  // Tiles: kFilterLanes nodes from -1 on for the orbit modes (lanes 2..29
  // write), 30 from 0 on otherwise (lanes 1..30).
  constexpr int kHalo = kOrbit ? 2 : 1, kWritten = 32 - 2 * kHalo;
  const int i = tile * kWritten + lane - kHalo - (kOrbit ? 1 : 0);
  if (tile * kWritten - (kOrbit ? 1 : 0) > nxc || j >= nyc) return;  // whole warps
  const bool inside = i >= 0 && i < nxc;
  const bool raw_in = i >= -1 && i <= nxc;
  const bool writes = lane >= kHalo && lane < 32 - kHalo && (kOrbit ? raw_in : inside);
  const bool column = inside && (c == 0 ? (j > 0 && j < g.ny)
                                        : (c == 1 ? (i > 0 && i < g.nx)
                                                  : (i > 0 && i < g.nx && j > 0 && j < g.ny)));
  const int zlo = (c != 2) ? 1 : 0, zhi = (c != 2) ? nzc - 2 : nzc - 1;  // the mask's planes
  // Where no raw node of the tile holds a deposit there is no current: E* and
  // (after the guess pass or an earlier trial) the filtered sum stand.
  if constexpr (MODE == kFilterOrbit || MODE == kFilterCommit) {
    const bool touched = raw_in && column_marked(g, i, j);
    if (!__any_sync(0xffffffffu, touched) && !a.full) return;
  }
  // Output planes [k0, k1): the padded array's for the orbit modes.
  const int first = kOrbit ? -g.jpad : 0, last = kOrbit ? nzc + g.jpad : nzc;
  const int k0 = first + (int)(blockIdx.z % a.chunks) * a.planes;
  const int k1 = min(k0 + a.planes, last);
  if (k0 >= k1) return;
  const int s0 = kOrbit ? k0 - R : k0;  // first plane of the (candidate) sum
  const int s1 = kOrbit ? k1 + R : k1;
  FilterMarch m;
  m.plane = nyc * (nxc + 2);
  m.nplane = nyc * nxc;
  m.row = j * (nxc + 2) + (i + 1);
  m.node = j * nxc + i;
  m.nzc = nzc;
  m.zb = zb;
  m.zlo = zlo;
  m.zhi = zhi;
  m.inside = inside;
  m.raw_in = raw_in;
  m.writes = writes;
  m.column = column;
  m.raw = raw;
  m.sum = sum;
  m.star = star;
  m.out = out;
  // A march whose planes are all inside every array tests no plane number.
  if (s0 - R >= 0 && s1 + R <= nzc && s0 >= zlo && s1 - 1 <= zhi)
    filter_march<S, MODE, W, true>(g, m, c, k0, s0, s1);
  else
    filter_march<S, MODE, W, false>(g, m, c, k0, s0, s1);
}

// The x-z filtered B of the linear-binomial3 gathers, one pass per step:
// binomialXZMagneticSample clamps its nodes to the component (open faces), so
// the filter does, and the output covers one node beyond in x and z.
template <class W>
__global__ void magnetic_filter_kernel(BFilterArgs a) {
  const GridT<double>& g = a.g;
  const int lane = threadIdx.x & 31;
  const int tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z / a.chunks;
  const int nxc = b_nx(g, c), nyc = b_ny(g, c), nzc = b_nz(g, c);
  const int zb = c == 0 ? g.zb_b[0] : (c == 1 ? g.zb_b[1] : g.zb_b[2]);
  const double* b = c == 0 ? g.b[0] : (c == 1 ? g.b[1] : g.b[2]);
  W* out = static_cast<W*>(c == 0 ? a.out[0] : (c == 1 ? a.out[1] : a.out[2]));
  if (tile * 30 - 1 > nxc || j >= nyc) return;
  const int i = tile * 30 + lane - 2;  // lanes 1..30 write nodes -1..nxc
  const int ic = min(max(i, 0), nxc - 1);
  const bool writes = lane >= 1 && lane < 31 && i <= nxc;
  const int k0 = -1 + (int)(blockIdx.z % a.chunks) * a.planes;
  const int k1 = min(k0 + a.planes, nzc + 1);
  if (k0 >= k1) return;
  const unsigned nplane = nyc * nxc, plane = nyc * (nxc + 2);
  const int node = j * nxc + ic, row = j * (nxc + 2) + (i + 1);
  auto at = [&](int k) -> double {
    const int kc = min(max(k, 0), nzc - 1);
    return b[APRL_BOUNDED(g.status, ring(kc, zb, nzc) * nplane + node, b_count(g, c), 45 + c)];
  };
  ZWindow<0> w;
  w.clear();
  w.push(lane_filter(at(k0 - 1)));
  w.push(lane_filter(at(k0)));
  W* to = out + (unsigned)((k0 + 1) * plane + row);
  // Four planes' reads are issued together (one at a time left too few bytes
  // in flight: 0.117 against 0.100 ms on the 128x128x512 grid).
  constexpr int U = 4;
  for (int kb = k0; kb < k1; kb += U) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = kb + u < k1 ? at(kb + u + 1) : 0.;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (kb + u >= k1) break;
      w.push(lane_filter(v[u]));
      if (writes) out[APRL_BOUNDED(g.status, to - out, bf_count(g, c), 57 + c)] = W(w.value());
      to += plane;
    }
  }
}

// Lab detector field plane (src/lab_detectors.cpp:39-99, 2836-2905).
__device__ __forceinline__ void interp_axis(double lattice, int size, int* lower,
                                            double* fraction) {
  if (lattice <= 0.0) {
    *lower = 0;
    *fraction = 0.0;
  } else if (lattice >= (double)(size - 1)) {
    *lower = size - 2;
    *fraction = 1.0;
  } else {
    *lower = (int)floor(lattice);
    *fraction = lattice - (double)*lower;
  }
}

template <class F>
__device__ double detector_component(const GridT<F>& g, int comp, double lx, double ly, int zl,
                                     double zf) {
  const bool electric = comp < 3;
  const int c = comp % 3;
  const int nxc = electric ? e_nx(g, c) : b_nx(g, c);
  const int nyc = electric ? e_ny(g, c) : b_ny(g, c);
  int xl, yl;
  double xf, yf;
  interp_axis(lx, nxc, &xl, &xf);
  interp_axis(ly, nyc, &yl, &yf);
  double value = 0.0;
  for (int cz = 0; cz < 2; ++cz) {
    const double wz = cz ? zf : 1.0 - zf;
    if (wz == 0.0) continue;
    for (int b = 0; b < 2; ++b)
      for (int a = 0; a < 2; ++a) {
        const double wx = a ? xf : 1.0 - xf;
        const double wy = b ? yf : 1.0 - yf;
        const double v = electric ? g.e_old[c][e_index(g, c, xl + a, yl + b, zl + cz)]
                                  : g.b[c][b_index(g, c, xl + a, yl + b, zl + cz)];
        value += wx * wy * wz * v;
      }
  }
  return value;
}

template <class F>
__global__ void detector_plane_kernel(DetectorArgs<F> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const GridT<F>& g = a.g;
  if (i >= g.nx || j >= g.ny) return;
  const double py = a.origin_xy[1] + ((double)j + 0.5) * g.dy;
  const double y = (py - a.origin_xy[1]) / g.dy;
  const double px = a.origin_xy[0] + ((double)i + 0.5) * g.dx;
  const double x = (px - a.origin_xy[0]) / g.dx;
  double eb[3], bb[3];
  eb[0] = detector_component(g, 0, x - 0.5, y, a.vertex_lower, a.vertex_fraction);
  eb[1] = detector_component(g, 1, x, y - 0.5, a.vertex_lower, a.vertex_fraction);
  eb[2] = detector_component(g, 2, x, y, a.half_lower, a.half_fraction);
  bb[0] = detector_component(g, 3, x, y - 0.5, a.half_lower, a.half_fraction);
  bb[1] = detector_component(g, 4, x - 0.5, y, a.half_lower, a.half_fraction);
  bb[2] = detector_component(g, 5, x - 0.5, y - 0.5, a.vertex_lower, a.vertex_fraction);
  // fieldsBoxToLab (src/boostframe.cpp:275-285)
  const DFrame& f = a.frame;
  double* o = a.out + 6 * ((size_t)j * g.nx + i);
  o[0] = fma(f.gamma_beta * kC, bb[1], f.gamma * eb[0]);
  o[1] = fma(-f.gamma_beta * kC, bb[0], f.gamma * eb[1]);
  o[2] = eb[2];
  o[3] = fma(-f.gamma_beta / kC, eb[1], f.gamma * bb[0]);
  o[4] = fma(f.gamma_beta / kC, eb[0], f.gamma * bb[1]);
  o[5] = bb[2];
}

// Built for binary64 J (both modes of this library).
#define APRL_FIELD_KERNELS(F)                                                  \
  template __global__ void cowan_magnetic_kernel<F>(CowanArgs<F>);            \
  template __global__ void electric_preview_kernel<F>(PreviewArgs<F>);        \
  template __global__ void shift_insert_kernel<F>(ShiftArgs<F>);              \
  template __global__ void detector_plane_kernel<F>(DetectorArgs<F>);
APRL_FIELD_KERNELS(double)
#define APRL_FILTER_KERNELS(S)                                                       \
  template __global__ void current_filter_kernel<S, kFilterGuess, double>(FilterArgs);  \
  template __global__ void current_filter_kernel<S, kFilterGuess, float>(FilterArgs);   \
  template __global__ void current_filter_kernel<S, kFilterOrbit, double>(FilterArgs);  \
  template __global__ void current_filter_kernel<S, kFilterOrbit, float>(FilterArgs);   \
  template __global__ void current_filter_kernel<S, kFilterCommit, double>(FilterArgs); \
  template __global__ void current_filter_kernel<S, kFilterCurrent, double>(FilterArgs);
APRL_FILTER_KERNELS(0)
APRL_FILTER_KERNELS(1)
template __global__ void magnetic_filter_kernel<double>(BFilterArgs);
template __global__ void magnetic_filter_kernel<float>(BFilterArgs);
#undef APRL_FILTER_KERNELS
#undef APRL_FIELD_KERNELS

// TransverseReferenceCurrent::prepare's values (src/transverse_reference_current.cpp:
// 52-58): curl_z of the reference B at every target point and reference plane,
// ((By(i,j,k) - By(i-1,j,k))/dx - (Bx(i,j,k) - Bx(i,j-1,k))/dy)/mu0.
__global__ void surface_prepare_kernel(SurfaceArgs a) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= a.count * a.planes) return;
  const long long k = n / a.count, p = n % a.count;
  const size_t i = a.points[2 * p], j = a.points[2 * p + 1];
  // native reference layouts: Bx (nx+1, ny, planes), By (nx, ny+1, planes)
  const size_t bx0 = ((size_t)k * a.ny + j) * (a.nx + 1) + i;
  const size_t bx1 = ((size_t)k * a.ny + j - 1) * (a.nx + 1) + i;
  const size_t by0 = ((size_t)k * (a.ny + 1) + j) * a.nx + i;
  const double v = ((a.by[by0] - a.by[by0 - 1]) / a.dx - (a.bx[bx0] - a.bx[bx1]) / a.dy) / kMu0;
  if (!isfinite(v)) raise_error(a.status, kErrSurfaceCurrent, (unsigned long long)n);
  a.table[n] = v;
}

// TransverseReferenceCurrent::apply (src/transverse_reference_current.cpp:104-118):
// Jz(i, j, k) += the lerp of the prepared planes at offset + k - beta*step.
// The current is the same in every trial of a step, so it goes into E* (and
// its orbit sum) once, after the first trial's current-free gather; a
// read-out of J adds it to Jz.
__global__ void surface_add_kernel(SurfaceArgs a) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const DGrid& g = a.g;
  if (n >= a.count * g.nz) return;
  const int k = (int)(n / a.count);
  const long long p = n % a.count;
  const double z = static_cast<double>(a.offset + k) - a.beta * static_cast<double>(a.step);
  const long long lo = (long long)floor(z);
  const long long hi = lo + 1 < a.planes ? lo + 1 : a.planes - 1;
  const double fraction = z - (double)lo;
  const double low = a.table[lo * a.count + p], high = a.table[hi * a.count + p];
  const double value = fraction == 0. ? low : (1. - fraction) * low + fraction * high;
  const int i = (int)a.points[2 * p], j = (int)a.points[2 * p + 1];
  if (a.jz) {
    a.jz[((size_t)k * (g.ny + 1) + j) * (g.nx + 1) + i] += value;
    return;
  }
  if (!current_mask(g, 2, i, j, k)) return;
  const size_t at = e_index(g, 2, i, j, k);
  g.e_star[2][at] += g.jcoef * value;
  if (a.sum) a.sum[at] += g.jcoef * value;
}

}  // namespace aprl_gpu
