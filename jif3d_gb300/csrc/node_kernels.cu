// node_kernels.cu -- the node-term forward and adjoint sums of the matrix-free
// path (prism_kernels.h): every mesh node's corner terms, for all stations,
// summed with the model differences or the weights.
//
// Work is split into node columns (fixed x and y): a thread takes one column
// and walks its nodes, so that dx, dy and dx^2 + dy^2 are formed once per
// column and station and the z offsets once per block and station (in shared
// memory), instead of once per node.  The terms come from node_fixed.cuh; its
// tables are copied to shared memory, where random lookups cost a few bank
// conflicts (through L1 up to a cycle per lane).
//
// Measured (forward + adjoint of one model): joint g_z + FTG, 64 x 64 x 32
// cells, 1024 stations 8.6 ms, from 77.1 ms with the terms on the FP64 pipe;
// g_z on 12 x 10 x 6 cells, 16 stations 13.7 us from 41 us.  A joint node takes
// about 810 instructions; the schedulers issue in 67 % of the cycles, with the
// integer, multiply-add and FP64 pipes 60 to 70 % busy each.
#include <algorithm>

#include "chained.cuh"
#include "node_column.cuh"
#include "prism_kernels.h"

namespace j3g {
namespace {

constexpr int kMaxColumn = 64;  // z offsets of a forward block held at a time
constexpr int kAdjNodes = 8;    // nodes of a column per adjoint thread
constexpr int kAdjStage = 16;   // stations staged at a time

// rho~ of a node: the signed sum of the cells that it is a corner of, zero
// outside, (-1)^(number of axes along which it is the upper corner), in the
// column order of the forward: [k][column].  PLANES: the node planes of an axis
// are given by p (cells whose lower and upper corner planes are apart), else
// plane i is the lower corner of cell i and the upper corner of cell i - 1.
template <bool PLANES>
__global__ void __launch_bounds__(kNodeThreads)
    k_rho_tilde(MeshView m, MeshView nodes, NodePlanes p, const double *__restrict__ rho,
                double *__restrict__ rt) {
  chain_begin();
  chain_wait();
  const int ny1 = nodes.ny + 1, ncol = (nodes.nx + 1) * ny1;
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= ncol * (nodes.nz + 1)) return;
  rho += blockIdx.y * m.ngrid();
  rt += blockIdx.y * nodes.nnodes();
  const int k = n / ncol, col = n - k * ncol, i = col / ny1, j = col - i * ny1;
  const int ci[2] = {PLANES ? p.lower_of[0][i] : i, PLANES ? p.upper_of[0][i] : i - 1};
  const int cj[2] = {PLANES ? p.lower_of[1][j] : j, PLANES ? p.upper_of[1][j] : j - 1};
  const int ck[2] = {PLANES ? p.lower_of[2][k] : k, PLANES ? p.upper_of[2][k] : k - 1};
  double v = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int a = (q >> 2) & 1, b = (q >> 1) & 1, c = q & 1;
    if (ci[a] < 0 || cj[b] < 0 || ck[c] < 0 || ci[a] >= m.nx || cj[b] >= m.ny || ck[c] >= m.nz)
      continue;
    const double r = rho[((long long)ci[a] * m.ny + cj[b]) * m.nz + ck[c]];
    v = ((a + b + c) & 1) ? v - r : v + r;
  }
  rt[n] = v;
}

// Forward partial sums: block x covers cols columns and kper nodes of each,
// block y spb stations; partial[x][station][component].
template <int KIND>
__global__ void __launch_bounds__(kNodeThreads, kNodeResident)
    k_node_forward(MeshView m, StationView st, const double *__restrict__ rt,
                   double *__restrict__ partial, int cols, int kper, int nkc, int spb) {
  using T = KindTraits<KIND>;
  constexpr int MASK = T::mask;
  constexpr int NCMP = T::ncomp;
  constexpr int NZ = T::twin ? 2 : 1;
  // component 0 is g_z: dx ln(dy + r) + dy ln(dx + r) + dz atan2(dz r, dx dy)
  constexpr bool kGz = (MASK & (1 << NC_GZ)) != 0;
  __shared__ FxTables tab;
  __shared__ ZOffset zo[NZ][kMaxColumn];
  __shared__ double red[NCMP][kNodeThreads];
  const int ny1 = m.ny + 1, nz1 = m.nz + 1, ncol = (m.nx + 1) * ny1;
  const long long nn = (long long)ncol * nz1;
  const int cb = blockIdx.x / nkc, k0 = (blockIdx.x - cb * nkc) * kper;
  const int k1 = min(nz1, k0 + kper);
  const int c0 = cb * cols, c1 = min(ncol, c0 + cols);
  const int s0 = blockIdx.y * spb, s1 = min(st.n, s0 + spb);
  const int tid = threadIdx.x, nt = blockDim.x;
  chain_begin();
  tab.set(tid, nt);  // constant, so before the wait
  chain_wait();
  for (int s = s0; s < s1; ++s) {
    const double mx = st.x[s], my = st.y[s], mz = st.z[s];
    double acc[NCMP];
#pragma unroll
    for (int q = 0; q < NCMP; ++q) acc[q] = 0.0;
    for (int kb = k0; kb < k1; kb += kMaxColumn) {
      const int nk = min(kMaxColumn, k1 - kb);
      __syncthreads();  // the offsets and sums of the last pass are read
      for (int k = tid; k < nk; k += nt) {
        const double Z = m.Z[kb + k];
        zo[0][k] = z_offset(mz, Z);
        // the second position of the vertical gradient, z_meas + 1 as the
        // reference forms it (OMPMagneticGradImp.cpp:76-79)
        if constexpr (T::twin) zo[NZ - 1][k] = z_offset(add(mz, 1.0), Z);
      }
      __syncthreads();
      for (int col = c0 + tid; col < c1; col += nt) {
        const int i = col / ny1, j = col - i * ny1;
        const double dx = sub(mx, m.X[i]), dy = sub(my, m.Y[j]);
        const FxColumn c = fx_column<MASK>(fx_axis(dx), fx_axis(dy), tab);
        const double *r = rt + (long long)kb * ncol + col;
        double slx = 0.0, sly = 0.0;  // this column's sums of ln(dx + r), ln(dy + r)
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
          double w[T::nblock];
#pragma unroll
          for (int b = 0; b < T::nblock; ++b) w[b] = r[b * nn + (long long)k * ncol];
#pragma unroll
          for (int p = 0; p < NZ; ++p) {
            const ZOffset &z = zo[p][k];
            double F[NC_COUNT];
            if (fx_node<MASK, kGz>(c, z.a, tab, F)) {
              if constexpr (kGz) {
                slx = fma(F[NC_YZ], w[0], slx);
                sly = fma(F[NC_XZ], w[0], sly);
              }
#pragma unroll
              for (int q = 0; q < NCMP; ++q)
                if (T::at(q) == p && !(kGz && (T::comp(q) == NC_XZ || T::comp(q) == NC_YZ)))
                  acc[q] = fma(F[T::comp(q)], w[T::block(q)], acc[q]);
            } else {
              node_terms<MASK>(dx, dy, z.d, F);
#pragma unroll
              for (int q = 0; q < NCMP; ++q)
                if (T::at(q) == p) acc[q] = fma(F[T::comp(q)], w[T::block(q)], acc[q]);
            }
          }
        }
        if constexpr (kGz) {  // dx and dy belong to the column
          acc[0] = fma(dx, sly, fma(dy, slx, acc[0]));
          if constexpr (NCMP > 1) {
            acc[NC_XZ] += sly;
            acc[NC_YZ] += slx;
          }
        }
      }
    }
    // a warp per component sums the threads' values (13 FP64 additions a warp
    // and component instead of a shuffle tree in every warp)
#pragma unroll
    for (int q = 0; q < NCMP; ++q) red[q][tid] = acc[q];
    __syncthreads();
    for (int q = tid >> 5; q < NCMP; q += nt >> 5) {
      double v = 0.0;
      for (int t = tid & 31; t < nt; t += 32) v += red[q][t];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if ((tid & 31) == 0) partial[((long long)blockIdx.x * st.n + s) * NCMP + q] = v;
    }
  }
}

// Adjoint: block x covers blockDim columns and kper nodes of each, block y a
// chunk of stations from chunk0 on, staged kAdjStage at a time; the sums of a thread's nodes
// are in shared memory, so that the node loop need not be unrolled.
template <int KIND>
__global__ void __launch_bounds__(kNodeThreads, kNodeResident)
    k_node_adjoint(MeshView m, StationView st, const double *__restrict__ W, int kper, int nkc,
                   int spc, const int *__restrict__ chunk_start, int chunk0,
                   double *__restrict__ Gpart) {
  using T = KindTraits<KIND>;
  constexpr int MASK = T::mask;
  constexpr int NCMP = T::ncomp;
  constexpr int NZ = T::twin ? 2 : 1;
  // weights: node-component layout [nmeas][NC_COUNT], or [nmeas][ncomp] for
  // the special kinds
  constexpr int WLD = T::special ? NCMP : NC_COUNT;
  __shared__ FxTables tab;
  __shared__ ZOffset zo[NZ][kAdjStage][kAdjNodes];
  __shared__ double sx[kAdjStage], sy[kAdjStage], sw[kAdjStage][NCMP];
  // g_z weight times dz (component 0 is g_z, see the forward)
  constexpr bool kGz = (MASK & (1 << NC_GZ)) != 0;
  __shared__ double swz[kGz ? kAdjStage : 1][kAdjNodes];
  // g_z alone: a station's three products are added up before they meet the
  // running sum, so that it is rounded once per station (the other kinds'
  // rounding is less than that of the terms they had in FP64)
  constexpr bool kSumFirst = KIND == KIND_SCALAR;
  extern __shared__ double acc[];  // [nblock][kper][blockDim]
  const int ny1 = m.ny + 1, nz1 = m.nz + 1, ncol = (m.nx + 1) * ny1;
  const long long nn = (long long)ncol * nz1;
  const int cb = blockIdx.x / nkc, k0 = (blockIdx.x - cb * nkc) * kper;
  const int nk = min(kper, nz1 - k0);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int c0 = cb * nt, col = c0 + tid;
  const bool live = col < ncol;
  const int i = live ? col / ny1 : 0, j = live ? col - i * ny1 : 0;
  chain_begin();
  tab.set(tid, nt);  // constant, so before the wait
  chain_wait();
  const double X = m.X[i], Y = m.Y[j];
  // stations of this chunk: spc apiece, or the ranges of chunk_start (chunks
  // that never straddle a station subset)
  const int chunk = chunk0 + blockIdx.y;
  const int s0 = chunk_start ? chunk_start[chunk] : chunk * spc;
  const int s1 = chunk_start ? chunk_start[chunk + 1] : min(st.n, s0 + spc);
  for (int k = 0; k < nk; ++k)
#pragma unroll
    for (int b = 0; b < T::nblock; ++b) acc[(b * kper + k) * nt + tid] = 0.0;
  for (int base = s0; base < s1; base += kAdjStage) {
    const int cnt = min(kAdjStage, s1 - base);
    __syncthreads();
    for (int t = tid; t < cnt; t += nt) {
      sx[t] = st.x[base + t];
      sy[t] = st.y[base + t];
    }
    for (int t = tid; t < cnt * NCMP; t += nt) {
      const int s = t / NCMP, q = t - s * NCMP;
      sw[s][q] = W[(long long)(base + s) * WLD + (T::special ? q : T::comp(q))];
    }
    for (int t = tid; t < cnt * nk; t += nt) {
      const int s = t / nk, k = t - s * nk;
      const double mz = st.z[base + s], Z = m.Z[k0 + k];
      const ZOffset o = z_offset(mz, Z);
      zo[0][s][k] = o;
      if constexpr (kGz) swz[s][k] = W[(long long)(base + s) * WLD + NC_GZ] * o.d;
      if constexpr (T::twin) zo[NZ - 1][s][k] = z_offset(add(mz, 1.0), Z);
    }
    __syncthreads();
    if (!live) continue;
#pragma unroll 1
    for (int t = 0; t < cnt; ++t) {
      const double dx = sub(sx[t], X), dy = sub(sy[t], Y);
      const FxColumn c = fx_column<MASK>(fx_axis(dx), fx_axis(dy), tab);
      // g_z's logarithms go with those of Uxz and Uyz
      double wlx = 0.0, wly = 0.0;
      if constexpr (kGz) {
        wlx = sw[t][0] * dy;
        wly = sw[t][0] * dx;
        if constexpr (NCMP > 1) {
          wlx += sw[t][NC_YZ];
          wly += sw[t][NC_XZ];
        }
      }
#pragma unroll 1
      for (int k = 0; k < nk; ++k) {
        double v[T::nblock];
#pragma unroll
        for (int b = 0; b < T::nblock; ++b) v[b] = kSumFirst ? 0.0 : acc[(b * kper + k) * nt + tid];
#pragma unroll
        for (int p = 0; p < NZ; ++p) {
          const ZOffset &z = zo[p][t][k];
          double F[NC_COUNT];
          if (fx_node<MASK>(c, z.a, tab, F)) {
            if constexpr (kGz)
              v[0] = fma(swz[t][k], F[NC_GZ], fma(wly, F[NC_XZ], fma(wlx, F[NC_YZ], v[0])));
#pragma unroll
            for (int q = 0; q < NCMP; ++q)
              if (T::at(q) == p && !(kGz && (q == 0 || T::comp(q) == NC_XZ || T::comp(q) == NC_YZ)))
                v[T::block(q)] = fma(sw[t][q], F[T::comp(q)], v[T::block(q)]);
          } else {
            node_terms<MASK>(dx, dy, z.d, F);
#pragma unroll
            for (int q = 0; q < NCMP; ++q)
              if (T::at(q) == p)
                v[T::block(q)] = fma(sw[t][q], F[T::comp(q)], v[T::block(q)]);
          }
        }
#pragma unroll
        for (int b = 0; b < T::nblock; ++b)
          acc[(b * kper + k) * nt + tid] = kSumFirst ? acc[(b * kper + k) * nt + tid] + v[b] : v[b];
      }
    }
  }
  __syncthreads();
  // out in node order: runs of nk nodes of consecutive columns
  const int ncl = min(nt, ncol - c0);
#pragma unroll
  for (int b = 0; b < T::nblock; ++b) {
    double *g = Gpart + ((long long)chunk * T::nblock + b) * nn;
    for (int t = tid; t < ncl * nk; t += nt) {
      const int c = t / nk, k = t - c * nk;
      g[(long long)(c0 + c) * nz1 + k0 + k] = acc[(b * kper + k) * nt + c];
    }
  }
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

int column_threads(int ncol) { return std::min(kNodeThreads, (ncol + 31) / 32 * 32); }

// Blocks that the GPU holds at a time.
constexpr double kNodeSlots = 152.0 * kNodeResident;

}  // namespace

NodeForwardPlan node_forward_plan(int nx, int ny, int nz, int nmeas, long long max_blocks) {
  NodeForwardPlan p;
  const int ncol = (nx + 1) * (ny + 1), nz1 = nz + 1;
  p.threads = column_threads(ncol);
  p.cols = p.threads;
  // The split with the least of (blocks / slots) * busy + 0.45 * alone, in the
  // time of one node: busy what a block of spb stations and kper nodes costs the
  // SMs, alone how long it takes, its tables' latency included, which is what
  // the first and last blocks add.  Fitted to sweeps over eight meshes of 605 to
  // 52,000 nodes with 16 to 1200 stations, where it is within 5 % of the best
  // split (fixed thresholds on the number of blocks lost up to a quarter there).
  double best = 0.0;
  for (int spb = 8; spb > 0; spb >>= 1)
    for (int n = 1; n <= std::min(nz1, 64); ++n) {
      const int kper = cdiv(nz1, n), nkc = cdiv(nz1, kper);
      const double blocks = (double)cdiv(ncol, p.cols) * nkc * cdiv(nmeas, spb);
      const double cost = blocks / kNodeSlots * (1.5 + spb * (1.5 + kper)) +
                          0.45 * (10.0 + spb * (3.0 + kper));
      if (best != 0.0 && cost >= best) continue;
      best = cost;
      p.spb = spb;
      p.kper = kper;
      p.nkc = nkc;
    }
  auto blocks = [&]() {
    return (long long)cdiv(ncol, p.cols) * p.nkc * cdiv(nmeas, p.spb);
  };
  // short columns on many blocks: several columns per thread share a block's
  // station setup and sums
  while (p.cols < 8 * p.threads && (long long)p.kper * p.cols < 16LL * p.threads &&
         blocks() >= 12 * kNodeSlots)
    p.cols += p.threads;
  // within the caller's room for partial sums
  if ((long long)cdiv(ncol, p.cols) * p.nkc > max_blocks) {
    p.nkc = 1;
    p.kper = nz1;
    while ((long long)cdiv(ncol, p.cols) * p.nkc > max_blocks && p.cols < ncol)
      p.cols += p.threads;
  }
  // station blocks run over grid y: at most 65535 of them
  p.spb = std::max(p.spb, cdiv(nmeas, 65535));
  p.nblk = cdiv(ncol, p.cols) * p.nkc;
  return p;
}

template <int KIND>
static cudaError_t adjoint_launch(int blocks, int nchunk, size_t smem, cudaStream_t st,
                                  const MeshView &m, const StationView &s, const double *W,
                                  const NodeAdjointPlan &p, const int *chunk_start,
                                  double *Gpart) {
  if (smem > 16384) {  // three model blocks: beyond 48 KB with the tables, by opt-in
    const cudaError_t e = cudaFuncSetAttribute(
        k_node_adjoint<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  for (int c0 = 0; c0 < nchunk; c0 += 65535) {  // grid y
    const dim3 grid(blocks, std::min(65535, nchunk - c0));
    const cudaError_t e = launch_chained(k_node_adjoint<KIND>, grid, p.threads, smem, st, m, s, W,
                                         p.kper, p.nkc, p.spc, chunk_start, c0, Gpart);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

#define J3G_NODE_DISPATCH(kind, ...)                                             \
  switch (kind) {                                                                 \
    case KIND_SCALAR: { constexpr int K = KIND_SCALAR; __VA_ARGS__; } break;             \
    case KIND_TENSOR: { constexpr int K = KIND_TENSOR; __VA_ARGS__; } break;             \
    case KIND_MAGNETIC: { constexpr int K = KIND_MAGNETIC; __VA_ARGS__; } break;         \
    case KIND_JOINT: { constexpr int K = KIND_JOINT; __VA_ARGS__; } break;               \
    case KIND_MAG_GRADIENT: { constexpr int K = KIND_MAG_GRADIENT; __VA_ARGS__; } break; \
    case KIND_MAGNETIZATION: { constexpr int K = KIND_MAGNETIZATION; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                                        \
  }

cudaError_t launch_rho_tilde(const MeshView &m, const MeshView &nodes, const NodePlanes *planes,
                             int nblock, const double *rho, double *rho_t, cudaStream_t st) {
  const dim3 grid(cdiv(nodes.nnodes(), kNodeThreads), nblock);
  return planes ? launch_chained(k_rho_tilde<true>, grid, kNodeThreads, 0, st, m, nodes, *planes,
                                 rho, rho_t)
                : launch_chained(k_rho_tilde<false>, grid, kNodeThreads, 0, st, m, nodes,
                                 NodePlanes{}, rho, rho_t);
}

cudaError_t launch_node_forward(int kind, const MeshView &m, const StationView &s,
                                const double *rho_t, double *partial, const NodeForwardPlan &p,
                                cudaStream_t st) {
  const dim3 grid(p.nblk, cdiv(s.n, p.spb));
  J3G_NODE_DISPATCH(kind, return launch_chained(k_node_forward<K>, grid, p.threads, 0, st, m, s,
                                                rho_t, partial, p.cols, p.kper, p.nkc, p.spb));
}

NodeAdjointPlan node_adjoint_plan(int nx, int ny, int nz, int nblock, int nmeas, long long room) {
  NodeAdjointPlan p;
  const int ncol = (nx + 1) * (ny + 1), nz1 = nz + 1;
  p.threads = column_threads(ncol);
  const int ncb = cdiv(ncol, p.threads);
  p.nkc = cdiv(nz1, kAdjNodes);
  p.kper = cdiv(nz1, p.nkc);
  // Chunks of 16 stations: a block's setup costs about four of its nodes, a
  // few per cent of its time, and six rounds of blocks or more end together (64
  // stations to a block: the last round's blocks ran on alone, magnetics on
  // 48 x 48 x 24 cells and 1024 stations 2.19 ms to 1.86).  The same for every
  // survey with blocks enough, so that a station subset alone and within a batch
  // is summed in the same order.
  p.spc = 16;
  // fewer blocks than four rounds: the split with the least of
  // (rounds + 0.9) * time of a block, as for the forward
  const int resident = std::min<long long>(
      kNodeResident, (227 << 10) / ((29 << 10) + 8LL * nblock * p.kper * p.threads));
  if ((double)ncb * p.nkc * cdiv(nmeas, p.spc) < 4.0 * 152 * resident) {
    double best = 0.0;
    for (int spc : {16, 8, 6, 4, 3, 2, 1})
      for (int n = cdiv(nz1, kAdjNodes); n <= std::min(nz1, 64); ++n) {
        const int kper = cdiv(nz1, n), nkc = cdiv(nz1, kper);
        if (kper > kAdjNodes) continue;
        const int fit = std::min<long long>(
            kNodeResident, (227 << 10) / ((29 << 10) + 8LL * nblock * kper * p.threads));
        const double rounds = (double)ncb * nkc * cdiv(nmeas, spc) / (152.0 * fit);
        const double cost = (rounds + 0.9) * (6.0 + spc * (1.5 + kper));
        if (best != 0.0 && cost >= best) continue;
        best = cost;
        p.spc = spc;
        p.kper = kper;
        p.nkc = nkc;
      }
  }
  // the chunks' sums within the caller's room
  const long long fit = std::max(1LL, room / (8LL * nblock * ncol * nz1));
  p.spc = std::max<long long>(p.spc, (nmeas + fit - 1) / fit);
  p.nchunk = cdiv(nmeas, p.spc);
  return p;
}

cudaError_t launch_node_adjoint(int kind, const MeshView &m, const StationView &s,
                                const double *W, const NodeAdjointPlan &p, int nchunk,
                                const int *chunk_start, double *Gpart, cudaStream_t st) {
  const int ncb = cdiv((long long)(m.nx + 1) * (m.ny + 1), p.threads);
  const size_t smem = sizeof(double) * (size_t)kind_nblock(kind) * p.kper * p.threads;
  J3G_NODE_DISPATCH(kind, return adjoint_launch<K>(ncb * p.nkc, nchunk, smem, st, m, s, W, p,
                                                   chunk_start, Gpart));
  return cudaGetLastError();
}

}  // namespace j3g
