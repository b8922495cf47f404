// sens_kernels.cu -- sensitivity rows of meshes whose corners are node terms:
// the explicit rows of j3g_forward_sens and the device-resident sensitivity
// (FP32, or fp16 hi + lo with its transpose).
//
// A chunk of stations (about 1 GiB of intermediates) at a time:
//   k_node_values  the FP64 node terms, [term][node]
//   k_cell_rows    eight-node sums in the reference's order -> FP64 rows, and for
//                  the fp16 pair the largest high word of each row
//   k_row_sums     J 1 of each row
//   k_split_tiles  FP64 rows -> hi + lo in the tiled layout and, through shared
//                  memory, its transpose, in one pass
// The terms keep their FP64 bits (node_terms) and the sums the reference's order:
// the pair keeps 22 bits of entries whose own FP64 rounding reaches 1e-8 in the
// far field, so that terms rounded in any other way, better ones too, would move
// its last bits.  What of it integer arithmetic can do with the same bits is done
// there (fp64_int.cuh), beside the FP64 pipe that bounds the two first kernels.
//
// Measured (joint g_z + FTG, 64 x 64 x 32 cells, 1024 stations, fp16 pair):
// node terms 21.5 ms (36 with FP64 instructions alone; FP64 pipe 84 % busy), cell
// rows 10.9 ms (16; FP64 and integer pipes 78 %), the split with its transpose
// 4.1 ms for 15 GB of traffic, from 20.6 ms as a split that read the FP64 rows
// three times and two transposes.
#include <cuda_fp16.h>

#include <algorithm>

#include "fp64_int.cuh"
#include "fpbits.cuh"
#include "prism_math.cuh"
#include "prism_kernels.h"
#include "stored.h"

namespace j3g {
namespace {

// Distinct node terms of a kind: the components of its mask in component
// order, at one or two positions.
template <int KIND> struct Terms {
  static constexpr int mask = KindTraits<KIND>::mask;
  static constexpr int positions = KindTraits<KIND>::twin ? 2 : 1;
  __host__ __device__ static constexpr int rank(int c) {  // components below c
    int n = 0;
    for (int k = 0; k < c; ++k) n += mask >> k & 1;
    return n;
  }
  static constexpr int per = rank(NC_COUNT);
  static constexpr int n = per * positions;
  __host__ __device__ static constexpr int comp(int u) {  // component of term u
    int c = 0;
    for (int left = u % per; left > 0 || !(mask >> c & 1); ++c) left -= mask >> c & 1;
    return c;
  }
  __host__ __device__ static constexpr int index(int at, int c) { return at * per + rank(c); }
};

constexpr int kThreads = 256;

// A thread per node, z fastest: stations on the mesh's planes then make whole
// warps take the zero cases of the angles together.
template <int KIND>
__global__ void __launch_bounds__(kThreads)
    k_node_values(MeshView m, StationView st, int s0, double *__restrict__ F) {
  using U = Terms<KIND>;
  const int ny1 = m.ny + 1, nz1 = m.nz + 1, nn = (m.nx + 1) * ny1 * nz1;
  const int n = blockIdx.x * kThreads + threadIdx.x, sl = blockIdx.y, s = s0 + sl;
  if (n >= nn) return;
  const int t = n / nz1, k = n - t * nz1, i = t / ny1, j = t - i * ny1;
  const double dx = sub(st.x[s], m.X[i]), dy = sub(st.y[s], m.Y[j]);
#pragma unroll
  for (int p = 0; p < U::positions; ++p) {
    // the second position of the vertical gradient is 1 m below the first
    double v[NC_COUNT];
    node_terms<U::mask, true>(dx, dy, sub(p ? add(st.z[s], 1.0) : st.z[s], m.Z[k]), v);
#pragma unroll
    for (int u = 0; u < U::per; ++u)
      F[((long long)sl * U::n + p * U::per + u) * nn + n] = v[U::comp(u)];
  }
}

// The rows of one cell from its prism values u (Terms order): STORED, the node
// components or the magnetic kinds' raw rows; else the raw rows.  Row r of
// model block b is out[b * rows + r] (rows of magnetisation have three blocks).
template <int KIND, bool STORED> struct RowMap {
  using T = KindTraits<KIND>;
  static constexpr int rows = STORED ? stored_rows(KIND) : T::raw;
  static constexpr int blocks = T::nblock;
  __device__ static __forceinline__ void map(const double *u, const MagField &mf, double *out) {
    using U = Terms<KIND>;
    if constexpr (KIND == KIND_MAGNETIZATION) {
#pragma unroll
      for (int q = 0; q < 9; ++q)
        out[(q % 3) * 3 + q / 3] = mul(mf.factor, u[U::index(0, T::comp(q))]);
    } else if constexpr (KIND == KIND_MAG_GRADIENT) {
      double v[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) v[q] = u[U::index(T::at(q), T::comp(q))];
      raw_from_vc(KIND, v, mf, out);
    } else if constexpr (STORED && !stored_is_raw(KIND)) {
#pragma unroll
      for (int q = 0; q < rows; ++q) out[q] = u[q];
    } else {
      double c[NC_COUNT];
#pragma unroll
      for (int q = 0; q < NC_COUNT; ++q) c[q] = T::mask >> q & 1 ? u[U::index(0, q)] : 0.0;
      raw_from_comps(KIND, c, mf, out);
    }
  }
};

// combine8 with kIntSums of its seven sums on the integer pipes, bit for bit.
// Cell rows of 64 stations of the joint 64 x 64 x 32 survey: none 995 us (FP64
// pipe 82 % busy, integer 8 %), three 700 us (77 % each), four 820.
constexpr int kIntSums = 3;
__device__ __forceinline__ double combine8_split(int c, const double *v) {
  const uint32_t ord = comp_order(c);
  double acc = kIntSums ? int_neg(v[ord & 7u]) : -v[ord & 7u];
#pragma unroll
  for (int p = 1; p < 8; ++p) {
    const double x = v[(ord >> 3 * p) & 7u];
    const bool minus = p >= 4 && p < 7;
    if (p <= kIntSums)
      acc = int_add(acc, minus ? int_neg(x) : x);
    else
      acc = minus ? sub(acc, x) : add(acc, x);
  }
  return (c >= NC_XX && c <= NC_ZZ) ? mul(acc, kGravConst) : mul(-acc, kGravConst);
}

// A thread per cell, z fastest, one station per blockIdx.y.
template <int KIND, bool STORED, class OutT>
__global__ void __launch_bounds__(kThreads)
    k_cell_rows(MeshView m, int s0, const double *__restrict__ F, MagField mf,
                OutT *__restrict__ rows, long long ld, unsigned *__restrict__ rowmax) {
  using U = Terms<KIND>;
  using R = RowMap<KIND, STORED>;
  constexpr int NR = R::rows * R::blocks;
  const int ny1 = m.ny + 1, nz1 = m.nz + 1, nn = (m.nx + 1) * ny1 * nz1;
  const int ngrid = m.nx * m.ny * m.nz;
  const int cell = blockIdx.x * kThreads + threadIdx.x, sl = blockIdx.y;
  double out[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) out[r] = 0.0;
  if (cell < ngrid) {
    const int t = cell / m.nz, k = cell - t * m.nz, i = t / m.ny, j = t - i * m.ny;
    const double *f = F + (long long)sl * U::n * nn + ((long long)i * ny1 + j) * nz1 + k;
    double u[U::n];
#pragma unroll
    for (int q = 0; q < U::n; ++q) {
      double v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        v[c] = f[(long long)q * nn + ((c >> 2 & 1) * ny1 + (c >> 1 & 1)) * nz1 + (c & 1)];
      u[q] = combine8_split(U::comp(q), v);
    }
    R::map(u, mf, out);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      rows[((long long)sl * R::rows + r % R::rows) * ld + (long long)(r / R::rows) * ngrid + cell] =
          (OutT)out[r];
  }
  if (sizeof(OutT) == 8 && rowmax) {
    __shared__ unsigned top[R::rows];  // the largest high words
    if (threadIdx.x < R::rows) top[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R::rows; ++r) {
      unsigned mx = 0;
#pragma unroll
      for (int b = 0; b < R::blocks; ++b)
        mx = max(mx, (unsigned)(f64_bits(out[b * R::rows + r]) >> 32) & 0x7fffffffu);
      // a NaN (station on an edge's line) is not the maximum
      mx = __reduce_max_sync(0xffffffffu, mx > 0x7ff00000u ? 0u : mx);
      if ((threadIdx.x & 31) == 0) atomicMax(&top[r], mx);
    }
    __syncthreads();
    if (threadIdx.x < R::rows)
      atomicMax(rowmax + (long long)(s0 + sl) * R::rows + threadIdx.x, top[threadIdx.x]);
  }
}

// J 1 of a stored row, a block per row: 256 interleaved sums in cell order, added
// up by warps.  Its order belongs to the results: the models' means are added back
// with it, and a last bit of the data decides roundings of the residuals' fp16
// pairs (a sum that telescoped to the mesh's corners, 16 us instead of 95 for 64
// stations, moved single gradients by 2e-7 for some surveys).
__global__ void __launch_bounds__(kThreads)
    k_row_sums(const double *__restrict__ rows, long long ncol, double *__restrict__ rowsum) {
  const double *p = rows + (long long)blockIdx.x * ncol;
  double acc = 0.0;
#pragma unroll 8
  for (long long c = threadIdx.x; c < ncol; c += kThreads) acc += p[c];
  __shared__ double red[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x != 0) return;
  double v = 0.0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) v += red[w];
  rowsum[blockIdx.x] = v;
}

// ---------------------------------------------------------------------------
// x rounded to fp16 (to nearest, as the conversion from double): through a
// float whose last bit collects what it cuts off.
__device__ __forceinline__ __half round_half(double x) {
  const unsigned long long b = (unsigned long long)f64_bits(x);
  const uint32_t s = (uint32_t)(b >> 32) & 0x80000000u, e = (uint32_t)(b >> 52) & 0x7ffu;
  if (e >= 1151u)  // infinities, NaNs, beyond the range of floats
    return __ushort_as_half(e == 0x7ffu && (b & 0xfffffffffffffull)
                                ? (unsigned short)0x7fff : (unsigned short)(s >> 16 | 0x7c00u));
  const uint32_t f = e <= 896u ? 0u : (e - 896u) << 23 | (uint32_t)(b >> 29) & 0x7fffffu;
  return __float2half_rn(__uint_as_float(s | f | ((b & 0x1fffffffull) != 0 && f ? 1u : 0u)));
}

constexpr int kSplitCells = 64, kSplitRows = 64;
constexpr int kSplitPad = 2;  // halves: a row of 33 words, two-way conflicts at most

// hi + lo of 64 rows x 64 cells: J by rows as they are read, the transpose from
// shared memory in runs of 16 rows (two 16-byte stores where they are whole
// and aligned).  nrow rows from row0 of the whole matrix.
__global__ void __launch_bounds__(256)
    k_split_tiles(const double *__restrict__ rows, long long ncol, int nrow,
                  const unsigned *__restrict__ rowmax, float *__restrict__ scale, long long row0,
                  __half *__restrict__ hi, __half *__restrict__ lo, long long ld,
                  __half *__restrict__ thi, __half *__restrict__ tlo, long long ldt) {
  __shared__ __half sh[2][kSplitCells][kSplitRows + kSplitPad];
  const long long c0 = (long long)blockIdx.x * kSplitCells;
  const int r0 = blockIdx.y * kSplitRows, nr = min(kSplitRows, nrow - r0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long c = c0 + 2 * lane;
  for (int r = w; r < nr; r += 8) {
    const long long row = row0 + r0 + r;
    const double *p = rows + (long long)(r0 + r) * ncol;
    // power-of-two scale that brings the row's largest value into (2^13, 2^14];
    // 1 for a row of zeros
    const unsigned h = rowmax[row];
    const int e = h >> 20 ? min(127, max(-126, (int)(h >> 20) - 1022 - 14)) : 0;
    if (blockIdx.x == 0 && lane == 0) scale[row] = __uint_as_float((unsigned)(127 + e) << 23);
    __half hv[2], lv[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double v = c + q < ncol ? scale_pow2_ftz(p[c + q], -e) : 0.0;
      hv[q] = round_half(v);
      lv[q] = round_half(v - f32_to_f64(__half2float(hv[q])));
      sh[0][2 * lane + q][r] = hv[q];
      sh[1][2 * lane + q][r] = lv[q];
    }
    const long long o = tiled_index(row, c, ld);
    *reinterpret_cast<__half2 *>(hi + o) = __halves2half2(hv[0], hv[1]);
    *reinterpret_cast<__half2 *>(lo + o) = __halves2half2(lv[0], lv[1]);
  }
  __syncthreads();
  const int cell = threadIdx.x >> 2, part = (threadIdx.x & 3) * 16;
  if (c0 + cell >= ncol || part >= nr) return;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    __half *t = (q ? tlo : thi);
    const __half *s = sh[q][cell] + part;
    const long long row = row0 + r0 + part;
    // a run inside one 64-column tile of the transpose, on a 16-byte boundary
    if (part + 16 <= nr && (row & 7) == 0 && (row & 63) <= 48) {
      __align__(16) __half v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = s[k];
      uint4 *d = reinterpret_cast<uint4 *>(t + tiled_index(c0 + cell, row, ldt));
      d[0] = reinterpret_cast<const uint4 *>(v)[0];
      d[1] = reinterpret_cast<const uint4 *>(v)[1];
    } else {
      for (int k = 0; k < min(16, nr - part); ++k)
        t[tiled_index(c0 + cell, row + k, ldt)] = s[k];
    }
  }
}

// Zero rows r0 .. r1 - 1, columns c0 .. c1 - 1 of a tiled pair.
__global__ void k_zero_tiled(__half *__restrict__ hi, __half *__restrict__ lo, long long ld,
                             long long r0, long long r1, long long c0, long long c1) {
  const long long n = (r1 - r0) * (c1 - c0);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const long long o = tiled_index(r0 + t / (c1 - c0), c0 + t % (c1 - c0), ld);
    hi[o] = __ushort_as_half(0);
    lo[o] = __ushort_as_half(0);
  }
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

template <int KIND>
cudaError_t node_values(const MeshView &m, const StationView &s, int s0, int ns, double *F,
                        cudaStream_t st) {
  k_node_values<KIND><<<dim3(cdiv(m.nnodes(), kThreads), ns), kThreads, 0, st>>>(m, s, s0, F);
  return cudaGetLastError();
}

template <int KIND, bool STORED, class OutT>
cudaError_t cell_rows(const MeshView &m, int s0, int ns, const double *F, const MagField &mf,
                      OutT *rows, long long ld, unsigned *rowmax, cudaStream_t st) {
  const dim3 grid(cdiv(m.ngrid(), kThreads), ns);
  k_cell_rows<KIND, STORED, OutT><<<grid, kThreads, 0, st>>>(m, s0, F, mf, rows, ld, rowmax);
  return cudaGetLastError();
}

}  // namespace

#define J3G_SENS_DISPATCH(kind, ...)                                                     \
  switch (kind) {                                                                        \
    case KIND_SCALAR: { constexpr int K = KIND_SCALAR; __VA_ARGS__; } break;             \
    case KIND_TENSOR: { constexpr int K = KIND_TENSOR; __VA_ARGS__; } break;             \
    case KIND_MAGNETIC: { constexpr int K = KIND_MAGNETIC; __VA_ARGS__; } break;         \
    case KIND_JOINT: { constexpr int K = KIND_JOINT; __VA_ARGS__; } break;               \
    case KIND_MAG_GRADIENT: { constexpr int K = KIND_MAG_GRADIENT; __VA_ARGS__; } break; \
    case KIND_MAGNETIZATION: { constexpr int K = KIND_MAGNETIZATION; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                                               \
  }

int node_terms_stored(int kind) {
  switch (kind) {
    case KIND_SCALAR: return Terms<KIND_SCALAR>::n;
    case KIND_JOINT: return Terms<KIND_JOINT>::n;
    default: return Terms<KIND_TENSOR>::n;  // the tensor's six, twice three for the gradient
  }
}

cudaError_t launch_node_rows(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                             const MagField &mf, double *F, double *rows, long long ld,
                             cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  J3G_SENS_DISPATCH(kind, e = node_values<K>(m, s, s0, ns, F, st);
                    if (e == cudaSuccess) e = cell_rows<K, false, double>(
                        m, s0, ns, F, mf, rows, ld, nullptr, st));
  return e;
}

cudaError_t launch_stored_rows32(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                                 const MagField &mf, double *F, float *rows, long long ld,
                                 cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  J3G_SENS_DISPATCH(kind, e = node_values<K>(m, s, s0, ns, F, st);
                    if (e == cudaSuccess) e = cell_rows<K, true, float>(
                        m, s0, ns, F, mf, rows, ld, nullptr, st));
  return e;
}

cudaError_t launch_stored_pair(int kind, const MeshView &m, const StationView &s, int s0, int ns,
                               const MagField &mf, double *F, double *rows, long long K_,
                               unsigned *rowmax, const StoredPair &p, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  const int nrow = ns * stored_rows(kind);
  J3G_SENS_DISPATCH(kind, e = node_values<K>(m, s, s0, ns, F, st);
                    if (e == cudaSuccess) e = cell_rows<K, true, double>(
                        m, s0, ns, F, mf, rows, K_, rowmax, st);
                    if (e != cudaSuccess) return e);
  k_row_sums<<<nrow, kThreads, 0, st>>>(rows, K_, p.rowsum + (long long)s0 * stored_rows(kind));
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const dim3 grid(cdiv(p.ld, kSplitCells), cdiv(nrow, kSplitRows));
  k_split_tiles<<<grid, 256, 0, st>>>(
      rows, K_, nrow, rowmax, p.rowscale, (long long)s0 * stored_rows(kind),
      static_cast<__half *>(p.hi), static_cast<__half *>(p.lo), p.ld, static_cast<__half *>(p.thi),
      static_cast<__half *>(p.tlo), p.ldt);
  return cudaGetLastError();
}

cudaError_t launch_zero_padding(const StoredPair &p, long long R, long long K, cudaStream_t st) {
  struct Part {
    void *hi, *lo;
    long long ld, r0, r1, c0, c1;
  };
  // rows below the last, and the transpose's columns beyond R (J's columns
  // beyond K are written with its rows)
  const Part parts[] = {{p.hi, p.lo, p.ld, R, tiled_rows(R), 0, p.ld},
                        {p.thi, p.tlo, p.ldt, K, tiled_rows(K), 0, p.ldt},
                        {p.thi, p.tlo, p.ldt, 0, K, R, p.ldt}};
  for (const Part &q : parts) {
    const long long n = (q.r1 - q.r0) * (q.c1 - q.c0);
    if (n == 0) continue;
    k_zero_tiled<<<(int)std::min<long long>(152 * 16, cdiv(n, 256)), 256, 0, st>>>(
        static_cast<__half *>(q.hi), static_cast<__half *>(q.lo), q.ld, q.r0, q.r1, q.c0, q.c1);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace j3g
