// prism_kernels.cu -- the matrix-free prism path around the node sums: background
// layers, the ends of the forward and the adjoint, eight-corner rows.
//
// Work is organised around mesh NODES (see prism_math.cuh): for a station s
// every node n carries the corner terms F_c(s, n).  Three uses, the first two
// summed in node_kernels.cu and the third in sens_kernels.cu:
//   forward   U_c(s) = scale_c * sum_n F_c(s, n) * rho~(n)          (summation by parts)
//   adjoint   G(n)   = sum_s sum_c W_c(s) F_c(s, n),  grad(cell) = 2 * D3[G](cell)
//   J rows    T_c(s, cell) = eight-node sum in the reference's order
// where D3 is the signed eight-corner sum of a cell and rho~ its transpose
// applied to the model.  These reproduce ScalarOMPGravityImp::CalcGridded
// (Gravity/ScalarOMPGravityImp.cpp:138-180), TensorOMPGravityImp::CalcGridded
// (Gravity/TensorOMPGravityImp.cpp:125-182), the magnetic CalcGridded
// (Magnetics/OMPMagneticSusceptibilityImp.cpp:113-194) and the matrix-free
// LQDerivative (GravMag/ThreeDGravMagImplementation.h:177-231), with all
// stations in one launch and the reduction with the model on the device.
//
// All reductions have a fixed order, so results repeat bit for bit.
#include "chained.cuh"
#include "prism_kernels.h"

namespace j3g {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// Background layer terms (GravityBackground.cpp:24-137).  A block takes 32
// stations of one layer; warp k evaluates one prism component (g_z, Uxx, Uyy,
// Uzz, Uxy, Uxz, Uyz; the eighth warp idles) for those 32 stations, each an
// eight-corner sum in the reference's order, so the serial chain of
// transcendentals per thread is one component long and no warp diverges.
// Warp 0 then combines them with the sheet terms exactly as the reference's
// per-station loop does.  A layer's top is summed from the
// thicknesses in layer order.  The kind is a template argument so that the
// term arrays stay in registers.
template <int KIND>
__global__ void __launch_bounds__(256) k_background(StationView st, int nbg,
                                                    const double *__restrict__ thick, double xo,
                                                    double yo, double zo, double xw, double yw,
                                                    double zw, MagField mf,
                                                    double *__restrict__ bgsens) {
  constexpr int kind = KIND;
  constexpr int raw = kind_raw(kind);
  const int slot = threadIdx.x >> 5, li = threadIdx.x & 31;  // component, station
  const int s = blockIdx.x * 32 + li;
  const int j = blockIdx.y;
  const bool live = s < st.n;
  if constexpr (kind_special(kind)) {  // no background response (OMPMagneticGradImp.h:32-40)
    if (live && slot < raw) bgsens[((long long)s * raw + slot) * nbg + j] = 0.0;
    return;
  } else {
    __shared__ double terms[32][8];
    double mx = 0.0, my = 0.0, mz = 0.0;
    if (live) {
      mx = st.x[s];
      my = st.y[s];
      mz = st.z[s];
    }
    double top = zo;
    for (int i = 0; i < j; ++i) top = add(top, thick[i]);
    const double th = thick[j];
    const double bottom = add(top, th);
    // the slab inside the gridded depth, whole or cut at its bottom
    const bool have = top < zw;
    const double h = bottom <= zw ? th : sub(zw, top);
    constexpr bool kGz = kind == KIND_SCALAR || kind == KIND_JOINT;
    constexpr bool kTensor = kind != KIND_SCALAR;
    double b = 0.0;
    if (live && have) {
      if (slot == 0 && kGz) b = grav_box(mx, my, mz, xo, yo, top, xw, yw, h);
      if (kTensor) {
        if (slot == 1) b = uxx_box(mx, my, mz, xo, yo, top, xw, yw, h);
        if (slot == 2) b = uxx_box(my, mx, mz, yo, xo, top, yw, xw, h);
        if (slot == 3) b = uxx_box(mz, mx, my, top, xo, yo, h, xw, yw);
        if (slot == 4) b = uxy_box(mx, my, mz, xo, yo, top, xw, yw, h);
        if (slot == 5) b = uxy_box(mx, mz, my, xo, top, yo, xw, h, yw);
        if (slot == 6) b = uxy_box(mz, my, mx, top, yo, xo, h, yw, xw);
      }
    }
    terms[li][slot] = b;
    __syncthreads();
    if (!live || slot != 0) return;
    const double *t = terms[li];
    double v[raw];
    if constexpr (kGz) {
      double g = inf_sheet(mz, top, bottom);
      if (have) g = sub(g, t[0]);
      v[0] = g;
    }
    if constexpr (kTensor) {
      // 3 x 3 tensor from the unique components (BasicGravElements.cpp:216-244)
      const double box[9] = {t[1], t[4], t[5], t[4], t[2], t[6], t[5], t[6], t[3]};
      double u[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      u[8] = uzz_inf_sheet(mz, top, bottom);
      if (have) {
#pragma unroll
        for (int c = 0; c < 9; ++c) u[c] = sub(u[c], box[c]);
      }
      if constexpr (kind == KIND_MAGNETIC) {
        const double f1 = mf.fs, f2 = mf.factor;
        v[0] = mul(mul(add(add(mul(u[0], mf.bx), mul(u[1], mf.by)), mul(u[2], mf.bz)), f1), f2);
        v[1] = mul(mul(add(add(mul(u[3], mf.bx), mul(u[4], mf.by)), mul(u[5], mf.bz)), f1), f2);
        v[2] = mul(mul(add(add(mul(u[6], mf.bx), mul(u[7], mf.by)), mul(u[8], mf.bz)), f1), f2);
      } else {
        constexpr int o = kind == KIND_JOINT ? 1 : 0;
#pragma unroll
        for (int c = 0; c < 9; ++c) v[o + c] = u[c];
      }
    }
#pragma unroll
    for (int r = 0; r < raw; ++r) bgsens[((long long)s * raw + r) * nbg + j] = v[r];
  }
}

// ---------------------------------------------------------------------------
template <int RAW>
__device__ __forceinline__ double apply_transform(int transform, const double *raw, double bx,
                                                  double by, double bz) {
  if constexpr (RAW >= 9) {
    if (transform == TR_FTG_INVARIANT)  // Gravity/GravityTransforms.h:33-37
      return sub(sub(sub(add(add(mul(raw[0], raw[4]), mul(raw[4], raw[8])), mul(raw[0], raw[8])),
                         mul(raw[3], raw[1])),
                     mul(raw[7], raw[5])),
                 mul(raw[2], raw[6]));
  }
  if constexpr (RAW >= 3) {
    if (transform == TR_TOTAL_FIELD)  // Magnetics/MagneticTransforms.h:27-30
      return sqrt(add(add(mul(raw[0], raw[0]), mul(raw[1], raw[1])), mul(raw[2], raw[2])));
    if (transform == TR_TFA)  // Magnetics/MagneticTransforms.h:122-129
      return add(add(mul(bx, raw[0]), mul(by, raw[1])), mul(bz, raw[2]));
  }
  return raw[0];
}

// A station's raw rows plus background, and their transform, out.
template <int RAW>
__device__ __forceinline__ void finish_station(int transform, double tbx, double tby, double tbz,
                                               int s, double *r, const double *__restrict__ bgsens,
                                               int nbg, const double *__restrict__ bgval,
                                               double *__restrict__ raw_out,
                                               double *__restrict__ data_out) {
#pragma unroll
  for (int c = 0; c < RAW; ++c) {
    double bg = 0.0;
    for (int j = 0; j < nbg; ++j)
      bg = add(bg, mul(bgsens[((long long)s * RAW + c) * nbg + j], bgval[j]));
    r[c] = add(r[c], bg);
    if (raw_out) raw_out[(long long)s * RAW + c] = r[c];
  }
  if (transform == TR_NONE) {
#pragma unroll
    for (int c = 0; c < RAW; ++c) data_out[(long long)s * RAW + c] = r[c];
  } else {
    data_out[s] = apply_transform<RAW>(transform, r, tbx, tby, tbz);
  }
}

template <int RAW>
__global__ void k_assemble(int transform, double tbx, double tby, double tbz, int nmeas,
                           const double *__restrict__ rows, const double *__restrict__ bgsens,
                           int nbg, const double *__restrict__ bgval, double *__restrict__ raw_out,
                           double *__restrict__ data_out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nmeas) return;
  double r[RAW];
#pragma unroll
  for (int c = 0; c < RAW; ++c) r[c] = rows[(long long)s * RAW + c];
  finish_station<RAW>(transform, tbx, tby, tbz, s, r, bgsens, nbg, bgval, raw_out, data_out);
}

// The end of a node-path forward: a station's partial sums added up in block
// order (16 lanes to a station, one per component), then its raw rows,
// background and transform as in k_assemble.  One launch instead of two, and
// the sums' loads side by side: magnetisation over 14 blocks 15.3 + 3.6 -> 5 us.
constexpr int kFinishStations = kThreads / 16;
template <int KIND>
__global__ void __launch_bounds__(kThreads)
    k_forward_finish(int transform, double tbx, double tby, double tbz, int nmeas, int nblk,
                     const double *__restrict__ partial, const double *__restrict__ bgsens,
                     int nbg, const double *__restrict__ bgval, MagField mf,
                     double *__restrict__ raw_out, double *__restrict__ data_out) {
  using T = KindTraits<KIND>;
  __shared__ double sum[kFinishStations][T::ncomp];
  chain_begin();
  chain_wait();
  const int li = threadIdx.x / 16, q = threadIdx.x % 16;
  const int s = blockIdx.x * kFinishStations + li;
  if (s < nmeas && q < T::ncomp) {
    const double *p = partial + (long long)s * T::ncomp + q;
    const long long step = (long long)nmeas * T::ncomp;
    double v = 0.0;
#pragma unroll 8
    for (int b = 0; b < nblk; ++b) v += p[b * step];
    sum[li][q] = v * comp_scale(T::comp(q));
  }
  __syncwarp();  // a station's lanes are in one warp
  if (s >= nmeas || q != 0) return;
  double r[T::raw];
  if constexpr (T::special) {
    raw_from_vc(KIND, sum[li], mf, r);
  } else {
    double u[NC_COUNT];
#pragma unroll
    for (int c = 0; c < T::ncomp; ++c) u[T::comp(c)] = sum[li][c];
    raw_from_comps(KIND, u, mf, r);
  }
  finish_station<T::raw>(transform, tbx, tby, tbz, s, r, bgsens, nbg, bgval, raw_out, data_out);
}

// w = misfit * dT/draw (GravityTransforms.h:72-93, MagneticTransforms.h:65-75,136-145);
// without a transform the misfit is the raw weight.
template <int RAW>
__device__ __forceinline__ void backproject(int transform, double tbx, double tby, double tbz,
                                            const double *__restrict__ misfit,
                                            const double *__restrict__ rawd, int s, double *w) {
  if (transform == TR_NONE) {
#pragma unroll
    for (int c = 0; c < RAW; ++c) w[c] = misfit[(long long)s * RAW + c];
    return;
  }
  const double m = misfit[s];
  const double *d = rawd + (long long)s * RAW;
  if constexpr (RAW == 9) {  // the FTG invariant
    w[0] = mul(m, add(d[4], d[8]));
    w[1] = mul(m, -d[3]);
    w[2] = mul(m, -d[6]);
    w[3] = mul(m, -d[1]);
    w[4] = mul(m, add(d[0], d[8]));
    w[5] = mul(m, -d[7]);
    w[6] = mul(m, -d[2]);
    w[7] = mul(m, -d[5]);
    w[8] = mul(m, add(d[0], d[4]));
  }
  if constexpr (RAW == 3) {
    if (transform == TR_TOTAL_FIELD) {
      const double t = sqrt(add(add(mul(d[0], d[0]), mul(d[1], d[1])), mul(d[2], d[2])));
#pragma unroll
      for (int c = 0; c < 3; ++c) w[c] = mul(m, d[c] / t);
    } else {  // TFA
      w[0] = mul(m, tbx);
      w[1] = mul(m, tby);
      w[2] = mul(m, tbz);
    }
  }
}

template <int RAW>
__global__ void k_backproject(int transform, double tbx, double tby, double tbz, int nmeas,
                              const double *__restrict__ misfit, const double *__restrict__ rawd,
                              double *__restrict__ w_raw) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nmeas) return;
  double w[RAW];
  backproject<RAW>(transform, tbx, tby, tbz, misfit, rawd, s, w);
#pragma unroll
  for (int c = 0; c < RAW; ++c) w_raw[(long long)s * RAW + c] = w[c];
}

// The weights of a node-path adjoint: k_backproject's raw weights (kept for the
// background) and from them the weights of the node components, W
// [nmeas][NC_COUNT], or [nmeas][ncomp] for the special kinds.
template <int KIND>
__global__ void __launch_bounds__(128)
    k_node_weights(int transform, double tbx, double tby, double tbz, int nmeas,
                   const double *__restrict__ misfit, const double *__restrict__ rawd, MagField mf,
                   double *__restrict__ w_raw, double *__restrict__ W) {
  using T = KindTraits<KIND>;
  chain_begin();
  chain_wait();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nmeas) return;
  double w[T::raw];
  backproject<T::raw>(transform, tbx, tby, tbz, misfit, rawd, s, w);
#pragma unroll
  for (int c = 0; c < T::raw; ++c) w_raw[(long long)s * T::raw + c] = w[c];
  if constexpr (T::special) {
    double u[T::ncomp];
    vc_from_raw_weights(KIND, w, mf, u);
#pragma unroll
    for (int q = 0; q < T::ncomp; ++q)
      W[(long long)s * T::ncomp + q] = u[q] * comp_scale(T::comp(q));
  } else {
    double u[NC_COUNT];
    comps_from_raw_weights(KIND, w, mf, u);
#pragma unroll
    for (int c = 0; c < NC_COUNT; ++c) W[(long long)s * NC_COUNT + c] = u[c] * comp_scale(c);
  }
}

// Chunks of the station subset blockIdx.z (all of them without a table).
__device__ __forceinline__ int subset_chunks(const int *first_chunk, int sub, int chunk0,
                                             int nchunk, int &first) {
  first = first_chunk ? first_chunk[sub] - chunk0 : 0;
  return first_chunk ? first_chunk[sub + 1] - first_chunk[sub] : nchunk;
}

// Groups of `group` chunks added up in place, each into its first chunk (block
// y one group of every subset z): chunks in order, a few loads in flight.
__global__ void __launch_bounds__(kThreads)
    k_sum_groups(long long len, const int *__restrict__ first_chunk, int sub0, int chunk0,
                 int nchunk, int group, double *__restrict__ Gpart) {
  chain_begin();
  chain_wait();
  const long long n = (long long)blockIdx.x * kThreads + threadIdx.x;
  int first;
  const int nk = subset_chunks(first_chunk, sub0 + blockIdx.z, chunk0, nchunk, first);
  const int c0 = blockIdx.y * group, c1 = min(nk, c0 + group);
  if (n >= len || c1 - c0 < 2) return;
  double *g = Gpart + (first + c0) * len + n;
  double v = 0.0;
#pragma unroll 8
  for (int c = 0; c < c1 - c0; ++c) v += g[c * len];
  *g = v;
}

// grad(cell) = 2 * sum_{a,b,c} (-1)^(a+b+c) G(corner a, b, c of the cell), G
// the sum of the chunks (or of the first of every `group`).  A block sums the
// nodes of a tile of cells into shared memory and combines them from there;
// block y is the model block, z the station subset.  The chunk sums through
// memory and a combine kernel of their own took two launches per model block
// and subset, 4 to 5 us each.
constexpr int kTileX = 2, kTileY = 4, kTileZ = 16;  // cells of a block: 1.99 node sums per cell
template <bool PLANES>
__global__ void __launch_bounds__(kThreads)
    k_adjoint_finish(MeshView m, MeshView nodes, NodePlanes p, const int *__restrict__ first_chunk,
                     int sub0, int chunk0, int nchunk, int group, long long ld,
                     const double *__restrict__ Gpart, double *__restrict__ grad) {
  // the cells of a tile lie on up to twice as many planes
  __shared__ double g[PLANES ? 8 * kTileX * kTileY * kTileZ
                             : (kTileX + 1) * (kTileY + 1) * (kTileZ + 1)];
  constexpr int kTile[3] = {kTileX, kTileY, kTileZ};
  chain_begin();
  const int size[3] = {m.nx, m.ny, m.nz};
  int t = blockIdx.x, c0[3], nc[3], n0[3], nn[3];
#pragma unroll
  for (int a = 2; a >= 0; --a) {
    const int tiles = (size[a] + kTile[a] - 1) / kTile[a];
    c0[a] = t % tiles * kTile[a];
    t /= tiles;
    nc[a] = min(kTile[a], size[a] - c0[a]);
    n0[a] = PLANES ? p.lower[a][c0[a]] : c0[a];
    nn[a] = (PLANES ? p.upper[a][c0[a] + nc[a] - 1] : c0[a] + nc[a]) - n0[a] + 1;
  }
  chain_wait();
  int first;
  const int nk = subset_chunks(first_chunk, sub0 + blockIdx.z, chunk0, nchunk, first);
  const long long all = nodes.nnodes(), len = all * gridDim.y;
  const double *part = Gpart + first * len + blockIdx.y * all;
  const int ny1 = nodes.ny + 1, nz1 = nodes.nz + 1;
  for (int n = threadIdx.x; n < nn[0] * nn[1] * nn[2]; n += kThreads) {
    const int k = n % nn[2], ij = n / nn[2], j = ij % nn[1], i = ij / nn[1];
    const double *q = part + ((long long)(n0[0] + i) * ny1 + n0[1] + j) * nz1 + n0[2] + k;
    double v = 0.0;
#pragma unroll 8
    for (int c = 0; c < nk; c += group) v += q[c * len];
    g[n] = v;
  }
  __syncthreads();
  const int k = threadIdx.x % kTileZ, j = threadIdx.x / kTileZ % kTileY,
            i = threadIdx.x / (kTileZ * kTileY);
  if (i >= nc[0] || j >= nc[1] || k >= nc[2]) return;
  const int cell[3] = {i, j, k};
  int corner[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    corner[a][0] = PLANES ? p.lower[a][c0[a] + cell[a]] - n0[a] : cell[a];
    corner[a][1] = PLANES ? p.upper[a][c0[a] + cell[a]] - n0[a] : cell[a] + 1;
  }
  double v = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int a = (q >> 2) & 1, b = (q >> 1) & 1, c = q & 1;
    const double x = g[(corner[0][a] * nn[1] + corner[1][b]) * nn[2] + corner[2][c]];
    v = ((a + b + c) & 1) ? v - x : v + x;
  }
  grad[(sub0 + blockIdx.z) * ld + blockIdx.y * m.ngrid() +
       ((long long)(c0[0] + i) * m.ny + c0[1] + j) * m.nz + c0[2] + k] = 2.0 * v;
}

__global__ void k_background_grad(int kind, int nmeas, int nbg, const double *__restrict__ w_raw,
                                  const double *__restrict__ bgsens, double *__restrict__ gbg) {
  chain_begin();
  chain_wait();
  const int j = blockIdx.x;
  const int raw = kind_raw(kind);
  double acc = 0.0;
  for (int s = threadIdx.x; s < nmeas; s += blockDim.x)
    for (int r = 0; r < raw; ++r)
      acc = fma(w_raw[(long long)s * raw + r], bgsens[((long long)s * raw + r) * nbg + j], acc);
  __shared__ double red[kWarps];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < kWarps; ++w) v += red[w];
    gbg[j] = 2.0 * v;
  }
}

// ---------------------------------------------------------------------------
// Sensitivity rows of meshes whose corners are given one by one.

// Raw rows of one cell from its virtual-component box values u[q]:
// the ordinary kinds through raw_from_comps, the vertical gradient through
// raw_from_vc (BzSensBot - BzSensTop, OMPMagneticGradImp.cpp:88-99) and
// magnetisation as factor * U_kj in row k, column block j
// (OMPMagnetizationImp.cpp:58-68, 93-104).
template <int KIND>
__device__ __forceinline__ void store_cell_rows(const double *u, const MagField &mf,
                                                long long ngrid, long long cell, double *rows,
                                                long long ld) {
  using T = KindTraits<KIND>;
  if constexpr (KIND == KIND_MAGNETIZATION) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int jb = 0; jb < 3; ++jb)
        rows[(long long)k * ld + jb * ngrid + cell] = mul(mf.factor, u[3 * k + jb]);
  } else if constexpr (KIND == KIND_MAG_GRADIENT) {
    double raw[3];
    raw_from_vc(KIND, u, mf, raw);
    rows[cell] = raw[0];
  } else {
    double c[NC_COUNT];
#pragma unroll
    for (int q = 0; q < T::ncomp; ++q) c[T::comp(q)] = u[q];
    double raw[10];
    raw_from_comps(KIND, c, mf, raw);
#pragma unroll
    for (int r = 0; r < T::raw; ++r) rows[(long long)r * ld + cell] = raw[r];
  }
}

template <int KIND>
__global__ void __launch_bounds__(kThreads)
    k_cell_direct(MeshView m, StationView st, int s0, MagField mf, double *__restrict__ rows,
                  long long ld) {
  using T = KindTraits<KIND>;
  constexpr int MASK = T::mask;
  const long long cell = (long long)blockIdx.x * kThreads + threadIdx.x;
  const int sl = blockIdx.y;
  if (cell >= m.ngrid()) return;
  const int k = cell % m.nz;
  const long long t = cell / m.nz;
  const int j = t % m.ny;
  const int i = t / m.ny;
  const int s = s0 + sl;
  double c[T::twin ? 2 : 1][NC_COUNT];
  prism_components(MASK, st.x[s], st.y[s], st.z[s], m.X[i], m.Y[j], m.Z[k], m.xs[i], m.ys[j],
                   m.zs[k], c[0]);
  if constexpr (T::twin)
    prism_components(MASK, st.x[s], st.y[s], add(st.z[s], 1.0), m.X[i], m.Y[j], m.Z[k], m.xs[i],
                     m.ys[j], m.zs[k], c[T::twin ? 1 : 0]);
  double u[kMaxVc];
#pragma unroll
  for (int q = 0; q < T::ncomp; ++q) u[q] = c[T::at(q)][T::comp(q)];
  store_cell_rows<KIND>(u, mf, m.ngrid(), cell, rows + (long long)sl * T::raw * ld, ld);
}

__global__ void k_rows_dot(int raw, long long ngrid, const double *__restrict__ rows,
                           long long ld, const double *__restrict__ rho, double *__restrict__ out) {
  const int row = blockIdx.x;  // sl * raw + r
  const double *p = rows + (long long)row * ld;
  double acc = 0.0;
  for (long long c = threadIdx.x; c < ngrid; c += blockDim.x) acc = fma(p[c], rho[c], acc);
  __shared__ double red[kWarps];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < kWarps; ++w) v += red[w];
    out[row] = v;
  }
}

// grad[cell] += sum_{sl, r} w[(sl*raw + r)] * rows[(sl*raw + r)*ld + cell]
__global__ void k_rows_tdot(int nrow, long long ngrid, const double *__restrict__ rows, long long ld,
                            const double *__restrict__ w, double *__restrict__ grad) {
  const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= ngrid) return;
  double acc = grad[cell];
  for (int r = 0; r < nrow; ++r) acc = fma(w[r], rows[(long long)r * ld + cell], acc);
  grad[cell] = acc;
}

__global__ void k_scale(long long n, double f, double *__restrict__ v) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) v[t] *= f;
}

__global__ void k_fp64_probe(double *out, int n_iter) {
  double a0 = threadIdx.x * 1e-3, a1 = a0 + 1.0, a2 = a0 + 2.0, a3 = a0 + 3.0;
  const double b = 0.999999, c = 1e-7;
  for (int it = 0; it < n_iter; ++it) {
    a0 = fma(a0, b, c);
    a1 = fma(a1, b, c);
    a2 = fma(a2, b, c);
    a3 = fma(a3, b, c);
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = a0 + a1 + a2 + a3;
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
#define J3G_DISPATCH(kind, CALL)                                                  \
  switch (kind) {                                                                 \
    case KIND_SCALAR: { constexpr int K = KIND_SCALAR; CALL; } break;             \
    case KIND_TENSOR: { constexpr int K = KIND_TENSOR; CALL; } break;             \
    case KIND_MAGNETIC: { constexpr int K = KIND_MAGNETIC; CALL; } break;         \
    case KIND_JOINT: { constexpr int K = KIND_JOINT; CALL; } break;               \
    case KIND_MAG_GRADIENT: { constexpr int K = KIND_MAG_GRADIENT; CALL; } break; \
    case KIND_MAGNETIZATION: { constexpr int K = KIND_MAGNETIZATION; CALL; } break; \
    default: return cudaErrorInvalidValue;                                        \
  }

cudaError_t launch_forward_finish(int kind, int transform, double tbx, double tby, double tbz,
                                  int nmeas, int nblk, const double *partial,
                                  const double *bgsens, int nbg, const double *bgval,
                                  const MagField &mf, double *raw_out, double *data_out,
                                  cudaStream_t st) {
  J3G_DISPATCH(kind, return launch_chained(k_forward_finish<K>, dim3(cdiv(nmeas, kFinishStations)),
                                           kThreads, 0, st, transform, tbx, tby, tbz, nmeas, nblk,
                                           partial, bgsens, nbg, bgval, mf, raw_out, data_out));
  return cudaSuccess;
}

cudaError_t launch_background(int kind, const MeshView &m, const StationView &s, int nbg,
                              const double *bg_thick, double xo, double yo, double zo, double xw,
                              double yw, double zw, const MagField &mf, double *bgsens,
                              cudaStream_t st) {
  (void)m;
  if (nbg == 0 || s.n == 0) return cudaSuccess;
  if (nbg > 65535) return cudaErrorInvalidValue;
  const dim3 grid(cdiv(s.n, 32), nbg);
  J3G_DISPATCH(kind, (k_background<K><<<grid, 256, 0, st>>>(s, nbg, bg_thick, xo, yo, zo, xw, yw,
                                                              zw, mf, bgsens)));
  return cudaGetLastError();
}

cudaError_t launch_assemble(int kind, int transform, double tbx, double tby, double tbz,
                            int nmeas, const double *rows, const double *bgsens, int nbg,
                            const double *bgval, double *raw_out, double *data_out,
                            cudaStream_t st) {
  J3G_DISPATCH(kind, (k_assemble<kind_raw(K)><<<cdiv(nmeas, 128), 128, 0, st>>>(
                         transform, tbx, tby, tbz, nmeas, rows, bgsens, nbg, bgval, raw_out,
                         data_out)));
  return cudaGetLastError();
}

cudaError_t launch_backproject(int kind, int transform, double tbx, double tby, double tbz,
                               int nmeas, const double *misfit, const double *raw,
                               double *w_raw, cudaStream_t st) {
  J3G_DISPATCH(kind, (k_backproject<kind_raw(K)><<<cdiv(nmeas, 128), 128, 0, st>>>(
                         transform, tbx, tby, tbz, nmeas, misfit, raw, w_raw)));
  return cudaGetLastError();
}

cudaError_t launch_node_weights(int kind, int transform, double tbx, double tby, double tbz,
                                int nmeas, const double *misfit, const double *raw,
                                const MagField &mf, double *w_raw, double *W, cudaStream_t st) {
  J3G_DISPATCH(kind, return launch_chained(k_node_weights<K>, dim3(cdiv(nmeas, 128)), 128, 0, st,
                                           transform, tbx, tby, tbz, nmeas, misfit, raw, mf,
                                           w_raw, W));
  return cudaSuccess;
}

cudaError_t launch_adjoint_finish(const MeshView &m, const MeshView &nodes,
                                  const NodePlanes *planes, int nblock, int sub0, int sub1,
                                  const int *first_chunk, int chunk0, int nchunk, long long ld,
                                  double *Gpart, double *grad, cudaStream_t st, int *launches) {
  // a thread of the last kernel adds up to 32 chunks one after the other; more
  // are first added up in groups, which are then spread over the GPU
  constexpr int kGroup = 32;
  const long long len = nodes.nnodes() * nblock;
  int group = 1;
  if (nchunk > kGroup)
    for (group = kGroup; (long long)group * group < nchunk;) group *= 2;
  const int tiles = cdiv(m.nx, kTileX) * cdiv(m.ny, kTileY) * cdiv(m.nz, kTileZ);
  *launches = 0;
  for (int s0 = sub0; s0 < sub1; s0 += 65535) {  // grid z
    const int ns = sub1 - s0 < 65535 ? sub1 - s0 : 65535;
    if (group > 1) {
      const cudaError_t e = launch_chained(
          k_sum_groups, dim3(cdiv(len, kThreads), cdiv(nchunk, group), ns), kThreads, 0, st, len,
          first_chunk, s0, chunk0, nchunk, group, Gpart);
      if (e != cudaSuccess) return e;
      ++*launches;
    }
    const dim3 grid(tiles, nblock, ns);
    const cudaError_t e =
        planes ? launch_chained(k_adjoint_finish<true>, grid, kThreads, 0, st, m, nodes, *planes,
                                first_chunk, s0, chunk0, nchunk, group, ld, Gpart, grad)
               : launch_chained(k_adjoint_finish<false>, grid, kThreads, 0, st, m, nodes,
                                NodePlanes{}, first_chunk, s0, chunk0, nchunk, group, ld, Gpart,
                                grad);
    if (e != cudaSuccess) return e;
    ++*launches;
  }
  return cudaSuccess;
}

cudaError_t launch_background_grad(int kind, int nmeas, int nbg, const double *w_raw,
                                   const double *bgsens, double *grad_bg, cudaStream_t st) {
  if (nbg == 0) return cudaSuccess;
  return launch_chained(k_background_grad, dim3(nbg), kThreads, 0, st, kind, nmeas, nbg, w_raw,
                        bgsens, grad_bg);
}

cudaError_t launch_direct_rows(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                               const MagField &mf, double *rows, long long ld, cudaStream_t st) {
  const dim3 grid(cdiv(m.ngrid(), kThreads), ns);
  J3G_DISPATCH(kind, (k_cell_direct<K><<<grid, kThreads, 0, st>>>(m, s, s0, mf, rows, ld)));
  return cudaGetLastError();
}

cudaError_t launch_rows_dot(int raw, int ns, long long ngrid, const double *rows, long long ld,
                            const double *rho, double *out, cudaStream_t st) {
  k_rows_dot<<<ns * raw, kThreads, 0, st>>>(raw, ngrid, rows, ld, rho, out);
  return cudaGetLastError();
}

cudaError_t launch_rows_tdot(int nrow, long long ngrid, const double *rows, long long ld,
                             const double *w, double *grad, cudaStream_t st) {
  k_rows_tdot<<<cdiv(ngrid, kThreads), kThreads, 0, st>>>(nrow, ngrid, rows, ld, w, grad);
  return cudaGetLastError();
}

cudaError_t launch_scale(long long n, double f, double *v, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_scale<<<cdiv(n, kThreads), kThreads, 0, st>>>(n, f, v);
  return cudaGetLastError();
}

cudaError_t launch_fp64_probe(double *out, int blocks, int threads, int n_iter,
                              cudaStream_t st) {
  k_fp64_probe<<<blocks, threads, 0, st>>>(out, n_iter);
  return cudaGetLastError();
}

}  // namespace j3g
