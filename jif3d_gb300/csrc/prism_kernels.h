// prism_kernels.h -- launchers of the prism kernels (internal interface
// between the C-ABI layer and the kernels; no CUDA types leak past capi.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include "kinds.h"

namespace j3g {

// Device view of the mesh.  Node coordinates X[0..nx], Y[0..ny], Z[0..nz];
// cell i spans [X[i], X[i] + xs[i]].  When node_exact is true every
// X[i] + xs[i] equals X[i+1] bit for bit, so a corner term is a node term.
struct MeshView {
  int nx, ny, nz;
  const double *X, *Y, *Z;     // nodes (n + 1 each)
  const double *xs, *ys, *zs;  // cell sizes (n each)
  __host__ __device__ long long ngrid() const { return (long long)nx * ny * nz; }
  __host__ __device__ long long nnodes() const {
    return (long long)(nx + 1) * (ny + 1) * (nz + 1);
  }
};

struct StationView {
  int n;
  const double *x, *y, *z;
};

// The node planes of a mesh whose corners are not all running sums of the
// cell sizes: along each axis the distinct corner coordinates, lower and upper
// corners of neighbouring cells apart where they differ (2 n planes at most).
// lower_of / upper_of: the cell that a plane is the lower / upper corner of, or
// -1; lower / upper: the planes of a cell.  The node kernels work on the planes
// as on any node grid (a MeshView of them).
struct NodePlanes {
  const int *lower_of[3], *upper_of[3], *lower[3], *upper[3];
};

// Forward, node formulation:  per station and component
//   U_c(s) = scale_c * sum_nodes F_c(s, node) * rho~(node)
// rho~ = third mixed backward difference of the zero-padded model, for each of
// its nblock blocks.
// nodes: the node grid, m itself or that of its planes.
cudaError_t launch_rho_tilde(const MeshView &m, const MeshView &nodes, const NodePlanes *planes,
                             int nblock, const double *rho, double *rho_t, cudaStream_t st);
// Split of the forward's work: blocks of `cols` node columns and `kper` nodes
// of each (nblk = column blocks x nkc pieces of the columns, at most
// max_blocks of them where more columns per block can see to that), spb
// stations per block.
struct NodeForwardPlan {
  int threads, cols, kper, nkc, spb, nblk;
};
NodeForwardPlan node_forward_plan(int nx, int ny, int nz, int nmeas, long long max_blocks);
// partial: [nblk][nmeas][ncomp] virtual-component sums; rho_t holds one
// nnodes block per model block of the kind.
cudaError_t launch_node_forward(int kind, const MeshView &m, const StationView &s,
                                const double *rho_t, double *partial, const NodeForwardPlan &p,
                                cudaStream_t st);
// The stations' raw rows from their partial sums, background and transform as
// by launch_assemble.
cudaError_t launch_forward_finish(int kind, int transform, double t_bx, double t_by, double t_bz,
                                  int nmeas, int nblk, const double *partial,
                                  const double *bgsens, int nbg, const double *bgval,
                                  const MagField &mf, double *raw_out, double *data_out,
                                  cudaStream_t st);

// Background: bgsens[s][raw][j] for each layer j (GravityBackground.cpp:24-137,
// OMPMagneticSusceptibilityImp.cpp:31-101).
cudaError_t launch_background(int kind, const MeshView &m, const StationView &s, int nbg,
                              const double *bg_thick, double xorig, double yorig, double zorig,
                              double xw, double yw, double zw, const MagField &mf,
                              double *bgsens, cudaStream_t st);

// Per station: raw = rows [nmeas][raw] (+ sum_j bgsens * bgval) and the optional
// transform.  raw_out [nmeas][raw] (may be null), data_out [nmeas][dpm].
cudaError_t launch_assemble(int kind, int transform, double t_bx, double t_by, double t_bz,
                            int nmeas, const double *rows, const double *bgsens, int nbg,
                            const double *bgval, double *raw_out, double *data_out,
                            cudaStream_t st);

// Adjoint.  w_raw [nmeas][raw] are the raw-row weights (misfit already
// back-projected through the transform).  W [nmeas][NC_COUNT] receives the
// node-component weights with the component scale folded in ([nmeas][ncomp]
// virtual-component weights for the vertical gradient and magnetisation).
cudaError_t launch_backproject(int kind, int transform, double t_bx, double t_by, double t_bz,
                               int nmeas, const double *misfit, const double *raw,
                               double *w_raw, cudaStream_t st);
// Both at once.
cudaError_t launch_node_weights(int kind, int transform, double t_bx, double t_by, double t_bz,
                                int nmeas, const double *misfit, const double *raw,
                                const MagField &mf, double *w_raw, double *W, cudaStream_t st);
// Gpart [nchunk][nblock][nnodes] = sum over the chunk's stations of
// sum_q W_q * F_q, per model block.
// chunk_start (device, nchunk + 1 values, may be null): explicit station
// ranges of the chunks instead of spc apiece.
struct NodeAdjointPlan {
  int threads, kper, nkc, spc, nchunk;
};
// room: bytes for the sums of all stations' chunks (one chunk at least).
NodeAdjointPlan node_adjoint_plan(int nx, int ny, int nz, int nblock, int nmeas, long long room);
cudaError_t launch_node_adjoint(int kind, const MeshView &m, const StationView &s,
                                const double *W, const NodeAdjointPlan &p, int nchunk,
                                const int *chunk_start, double *Gpart, cudaStream_t st);
// grad[k * ld + b * ngrid + cell] = 2 * sum_corners (-1)^shifts * sum of
// Gpart[chunk - chunk0][b][node] over the chunks of subset k, for each model block
// b and the subsets sub0 to sub1 - 1.  Subset k has the chunks first_chunk[k] to
// first_chunk[k + 1] - 1 (device), nchunk of them at most; null: one subset of nchunk
// chunks.  Gpart is overwritten.  launches: kernels queued.
cudaError_t launch_adjoint_finish(const MeshView &m, const MeshView &nodes,
                                  const NodePlanes *planes, int nblock, int sub0, int sub1,
                                  const int *first_chunk, int chunk0, int nchunk, long long ld,
                                  double *Gpart, double *grad, cudaStream_t st, int *launches);
// grad[ngrid + j] = 2 * sum_s sum_r w_raw[s][r] * bgsens[s][r][j]
cudaError_t launch_background_grad(int kind, int nmeas, int nbg, const double *w_raw,
                                   const double *bgsens, double *grad_bg, cudaStream_t st);

// Raw sensitivity rows by eight corner evaluations per cell (corners that are
// not node terms): rows[(sl*raw + r) * ld + cell] for stations s0 .. s0+ns-1
// (sl = s - s0); magnetisation rows carry the three blocks at columns
// b * ngrid + cell.
cudaError_t launch_direct_rows(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                               const MagField &mf, double *rows, long long ld, cudaStream_t st);
// The same from the node terms, kept in F: ns * node_terms_stored(kind) *
// nnodes doubles.
int node_terms_stored(int kind);
cudaError_t launch_node_rows(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                             const MagField &mf, double *F, double *rows, long long ld,
                             cudaStream_t st);
// Rows of the device-resident sensitivity for the same stations: per station
// the kind's node components (scalar 1, tensor 6 = xx yy zz xy xz yz, joint 7 =
// gz + tensor) or, for the magnetic kinds, the raw rows.  As floats at stride ld:
cudaError_t launch_stored_rows32(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                                 const MagField &mf, double *F, float *rows, long long ld,
                                 cudaStream_t st);
// or as the fp16 pair (stored.h): row = scale * (hi + lo) with a power-of-two
// scale, max|hi| in (2^13, 2^14], hi / lo with ld columns and the transpose thi /
// tlo with ldt columns, both tiled, and the FP64 row sums J 1.  rows: scratch of
// ns * stored rows * K doubles; rowmax: a zeroed word per row of the whole matrix
// (the largest high word).  Columns beyond K are written as zero, the
// rest of the padding by launch_zero_padding.
struct StoredPair {
  void *hi, *lo, *thi, *tlo;
  long long ld, ldt;
  float *rowscale;
  double *rowsum;
};
cudaError_t launch_stored_pair(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                               const MagField &mf, double *F, double *rows, long long K,
                               unsigned *rowmax, const StoredPair &p, cudaStream_t st);
cudaError_t launch_zero_padding(const StoredPair &p, long long R, long long K, cudaStream_t st);

// d[(s0+sl)*raw + r] = sum_cell rows[(sl*raw + r)*ld + cell] * rho[cell]
cudaError_t launch_rows_dot(int raw, int ns, long long ngrid, const double *rows, long long ld,
                            const double *rho, double *out, cudaStream_t st);

// grad[cell] += sum_r w[r] * rows[r*ld + cell] over nrow rows.
cudaError_t launch_rows_tdot(int nrow, long long ngrid, const double *rows, long long ld,
                             const double *w, double *grad, cudaStream_t st);
cudaError_t launch_scale(long long n, double f, double *v, cudaStream_t st);

// FP64 peak probe: n_iter dependent-chain FMAs per thread (measurement only).
cudaError_t launch_fp64_probe(double *out, int blocks, int threads, int n_iter,
                              cudaStream_t st);

}  // namespace j3g
