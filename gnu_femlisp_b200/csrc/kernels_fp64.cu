// kernels_fp64.cu -- the FP64 kernels of the multigrid solve path (sm_100a).
//
// Layout in HBM: a level matrix is stored by stencil slot (structure of
// arrays): A[s * Np + i] = A(i, i + off_s), Np = node count rounded up to a
// multiple of 64 so that every slot array starts on a 512-byte boundary.
// Column indices are implicit (off_s = ox + M oy + M^2 oz), so the matvec
// streams only matrix values, coalesced across the warp (a row per thread).
// Entries outside the grid, in eliminated Dirichlet columns and structurally
// absent Q2 couplings are stored as zeros, which lets neighbour indices be
// clamped to the vector instead of tested.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include "fmgpu_kernels.cuh"

namespace fmg {

std::atomic<long long> g_launches{0};
thread_local cudaStream_t t_pdl_stream = nullptr;

// The Q1 row kernels: 128 threads, four blocks per SM.  The bound matters for
// its effect on register allocation: without it ptxas keeps the 3D kernels at
// 32-40 registers by moving each load down to its multiply-add, and a row
// waits for memory several times; with it (up to 128 registers) all 54 loads
// of a row are in flight at once.  Two to eight blocks measured alike.
constexpr int kRowT = 128;
constexpr int kRowMinBlocks = 4;

template <int D, int P>
struct St {
  static constexpr int W = 2 * P + 1;
  static constexpr int NS = D == 1 ? W : (D == 2 ? W * W : W * W * W);
  static constexpr int CENTER = (NS - 1) / 2;
};

// copies 8 bytes to shared memory in the background
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int D, int P>
__device__ __forceinline__ long long slot_off(int s, long long M) {
  constexpr int W = 2 * P + 1;
  long long o = (long long)(s % W - P);
  if (D > 1) o += M * (long long)((s / W) % W - P);
  if (D > 2) o += M * M * (long long)((s / (W * W)) % W - P);
  return o;
}

__device__ __forceinline__ void node_coords(long long i, long long M, int dim, long long c[3]) {
  c[0] = i % M;
  c[1] = dim > 1 ? (i / M) % M : 0;
  c[2] = dim > 2 ? i / (M * M) : 0;
}

// node_coords in 32-bit arithmetic (levels of fewer than 2^31 nodes)
__device__ __forceinline__ void node_coords32(long long i, long long M, int dim, long long c[3]) {
  const unsigned u = (unsigned)i, m = (unsigned)M;
  const unsigned q = u / m;
  c[0] = u - q * m;
  c[1] = dim > 1 ? q % m : 0;
  c[2] = dim > 2 ? q / m : 0;
}

__device__ __forceinline__ bool node_dirichlet(const long long c[3], long long M, int dim, int dmask) {
  for (int k = 0; k < dim; ++k) {
    if (c[k] == 0 && ((dmask >> (2 * k)) & 1)) return true;
    if (c[k] == M - 1 && ((dmask >> (2 * k + 1)) & 1)) return true;
  }
  return false;
}

// --------------------------------------------------- Q2 sliced storage
// A Q2 node couples at offset +-2 along direction k only when its coordinate k
// is even (a cell vertex); an odd coordinate (an edge / face / cell midpoint)
// couples within +-1.  Slot s of a Q2 level therefore stores only the nodes
// that admit it: those even along every direction where |offset_k| = 2 (the
// slot's pattern r, bit k).  They sit at the front of the slot's array, in
// lexicographic order of the coordinates halved along the restricted
// directions, so a level holds exactly its structural nonzeros (boundary and
// Dirichlet zeros aside) and a Q2 sweep streams no structural zero.  Q1
// levels and the centre slot (pattern 0) keep one entry per node.
template <int D>
__host__ __device__ __forceinline__ int q2_pattern(int s) {
  int r = 0;
  for (int k = 0; k < D; ++k) {
    const int o = s % 5 - 2;
    if (o == 2 || o == -2) r |= 1 << k;
    s /= 5;
  }
  return r;
}

// a node's index in the slot arrays of every pattern, and which patterns it admits
template <int D>
struct Q2Rows {
  long long idx[1 << D];
  unsigned valid;  // bit r: the node is stored in pattern-r slots
};

template <int D>
__host__ __device__ __forceinline__ void q2_rows(const long long c[3], long long M, Q2Rows<D>& q) {
  const long long H = (M + 1) / 2;
  q.valid = 0;
  for (int r = 0; r < (1 << D); ++r) {
    bool ok = true;
    long long id = 0, mul = 1;
    for (int k = 0; k < D; ++k) {
      const bool rk = (r >> k) & 1;
      if (rk && (c[k] & 1)) ok = false;
      id += (rk ? c[k] / 2 : c[k]) * mul;
      mul *= rk ? H : M;
    }
    q.idx[r] = id;
    if (ok) q.valid |= 1u << r;
  }
}

// Scalar Q2 levels go one step further: rows are grouped by colour class
// (coordinates mod 3 -- the classes of the multicolour <sor>), classes in
// ascending order, and inside a class a slot array holds the rows that admit
// the slot in lexicographic order of their place in the class grid.  Along a
// direction the class's coordinates are d, d+3, d+6, .. (d = coordinate mod 3),
// or, where the slot restricts the direction to even coordinates, x0(d),
// x0(d)+6, .. with x0 = 0, 4, 2 for d = 0, 1, 2.  A colour sweep then streams
// one contiguous block of every slot array.  off[colour][r] is where the
// class's block starts in the arrays of pattern-r slots.
// (Levels have fewer than 2^31 nodes.  A class's eight offsets sit together:
// a kernel reads them from its parameters, and each line of those it touches
// is a miss at the start of every launch.)
struct Q2Layout {
  int off[27][8];
};

__host__ __device__ __forceinline__ int q2c_x0(int d) { return d == 0 ? 0 : (d == 1 ? 4 : 2); }
// rows of class digit d along one direction (M coordinates), restricted or not
__host__ __device__ __forceinline__ long long q2c_ext(long long M, int d, bool r) {
  if (!r) return (M - d + 2) / 3;
  const int x0 = q2c_x0(d);
  return x0 < M ? (M - x0 + 5) / 6 : 0;
}
// place of coordinate c (digit d = c mod 3) in its class grid along one direction
__host__ __device__ __forceinline__ long long q2c_j(long long c, int d, bool r) {
  return r ? (c - q2c_x0(d)) / 6 : (c - d) / 3;
}

Q2Layout q2_layout(int D, long long M) {
  Q2Layout L{};
  int ncol = 1;
  for (int k = 0; k < D; ++k) ncol *= 3;
  for (int r = 0; r < (1 << D); ++r) {
    long long acc = 0;
    for (int col = 0; col < ncol; ++col) {
      L.off[col][r] = (int)acc;
      long long cnt = 1;
      int t = col;
      for (int k = 0; k < D; ++k) {
        cnt *= q2c_ext(M, t % 3, (r >> k) & 1);
        t /= 3;
      }
      acc += cnt;
    }
  }
  return L;
}

// storage position of node c in the arrays of pattern-r slots (the node must
// be even along the restricted directions)
template <int D>
__host__ __device__ __forceinline__ long long q2c_pos(const Q2Layout& L, const long long c[3], long long M, int r) {
  int col = 0, m3 = 1;
  long long p = 0, mul = 1;
  for (int k = 0; k < D; ++k) {
    const int d = (int)(c[k] % 3);
    const bool rk = (r >> k) & 1;
    col += d * m3;
    m3 *= 3;
    p += q2c_j(c[k], d, rk) * mul;
    mul *= q2c_ext(M, d, rk);
  }
  return L.off[col][r] + p;
}

// A node's position in the slot arrays of every pattern (32-bit: levels have
// fewer than 2^31 nodes) and the patterns it admits, in the colour-major
// layout of scalar Q2 levels (colour) or the natural sliced one (vector
// levels).
template <int D>
struct Q2Base {
  int p[1 << D];
  unsigned valid;
};

// CLAMP: keep every position in bounds (callers that load unstored slots too)
template <int D, bool COLOUR, bool CLAMP = false>
__device__ __forceinline__ void q2_base(const Q2Layout& lay, const long long c[3], long long M, Q2Base<D>& b) {
  long long nmax_l = 1;
  for (int k = 0; k < D; ++k) nmax_l *= M;
  const int nmax = (int)nmax_l;
  // per direction, unrestricted (0) and restricted (1): place and extent in
  // 32-bit arithmetic with constant divisors
  const int Mi = (int)M;
  int j[3][2] = {{0, 0}, {0, 0}, {0, 0}}, e[3][2] = {{1, 1}, {1, 1}, {1, 1}};
  int col = 0, m3 = 1;
  unsigned odd = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const int ck = (int)c[k];
    if (ck & 1) odd |= 1u << k;
    if (COLOUR) {
      const int d = ck % 3, x0 = q2c_x0(d);
      col += d * m3;
      m3 *= 3;
      j[k][0] = (ck - d) / 3;
      j[k][1] = (ck - x0) / 6;
      e[k][0] = (Mi - d + 2) / 3;
      e[k][1] = x0 < Mi ? (Mi - x0 + 5) / 6 : 0;
    } else {
      j[k][0] = ck;
      j[k][1] = ck >> 1;
      e[k][0] = Mi;
      e[k][1] = (Mi + 1) >> 1;
    }
  }
  b.valid = 0;
#pragma unroll
  for (int r = 0; r < (1 << D); ++r) {
    if (!(r & odd)) b.valid |= 1u << r;
    const int rx = r & 1, ry = (r >> 1) & 1, rz = (r >> 2) & 1;
    const int p = j[0][rx] + e[0][rx] * (j[1][ry] + e[1][ry] * j[2][rz]);
    const int q = COLOUR ? lay.off[col][r] + p : p;
    b.p[r] = (CLAMP && q >= nmax) ? nmax - 1 : q;
  }
}

// ------------------------------------------------------------ batches
// A batched level holds nb independent problems of the same geometry, each
// at a fixed stride (vectors: the padded length Np; matrices: slots x Np).
// The 1D-grid kernels take the problem from blockIdx.y, the transfer kernels
// (1D/2D levels) from blockIdx.z; with one problem the offsets are zero.  A
// reduction then runs per problem: its partials, counter and scalar slots
// move with the problem.
__device__ __forceinline__ Reduce batch_reduce(Reduce R, unsigned bq) {
  R.part += (long long)bq * gridDim.x;
  R.counter += bq;
  R.scal += (long long)bq * S_COUNT;
  return R;
}

// ----------------------------------------------------------------- matvec
// One Q1 row: sum_s A(i, s) x(i + off_s) over the 3^D slots in slot order; dg
// gets the diagonal.  All 2 x 3^D loads are issued before the first
// multiply-add, so a row waits for memory once.  Neighbours outside the level
// meet stored zeros and are clamped to its first or last node.
// Bound by HBM on large levels (257^3 nodes: 556 us per matvec, 7.0 TB/s; 659
// us with two rows per thread and eight such steps per block, the loads then
// waited for slot by slot) and by one memory round trip on small ones (17^3:
// 5.3 us instead of 39 us, where that form gave work to two blocks only).  A
// fused dot product needs that form's thread-to-row map, so the reduction is
// a pass of its own (257^3: 42 us, less than the fused form lost).
template <int D>
__device__ __forceinline__ double q1_row_sum(const double* __restrict__ A, long long Np, int N, int M,
                                             const double* x, int i, double& dg) {
  constexpr int NS = St<D, 1>::NS, C = St<D, 1>::CENTER;
  double av[NS], xv[NS];
  const double* a = A + i;
#pragma unroll
  for (int s = 0; s < NS; ++s) av[s] = __ldg(a + s * Np);
  pdl_wait();  // the coefficients do not depend on the previous launch, the unknowns do
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const int o = (s % 3 - 1) + (D > 1 ? M * ((s / 3) % 3 - 1) : 0) + (D > 2 ? M * M * (s / 9 - 1) : 0);
    xv[s] = x[min(max(i + o, 0), N - 1)];
  }
  dg = av[C];
  double sum = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) sum = fma(av[s], xv[s], sum);
  return sum;
}

// y = A x (RES = false) or r = b - A x (RES = true, b may alias r) on a Q1
// level, one row per thread
template <int D, bool RES>
__global__ void __launch_bounds__(kRowT, kRowMinBlocks)
k_row_q1(const double* __restrict__ A, int N, long long Np, int M, const double* x, const double* b,
         double* y) {
  if (D == 1) pdl_next_light();
  else pdl_next();
  const int i = blockIdx.x * kRowT + threadIdx.x;
  if (i >= N) return;
  const long long bq = blockIdx.y;  // problem of a batched level
  A += bq * St<D, 1>::NS * Np;
  x += bq * Np;
  y += bq * Np;
  double dg;
  const double s = q1_row_sum<D>(A, Np, N, M, x, i, dg);
  y[i] = RES ? b[bq * Np + i] - s : s;
}

// compute-residual fused with the following <jacobi> step on a Q1 level:
// t = (b - A x)/d, xout = x + w t, r := t
template <int D>
__global__ void __launch_bounds__(kRowT, kRowMinBlocks)
k_row_jacobi_q1(const double* __restrict__ A, int N, long long Np, int M, double damp,
                const double* __restrict__ omega, const double* x, const double* b,
                double* __restrict__ xout, double* r, int write_r) {
  if (D == 1) pdl_next_light();
  else pdl_next();
  const int i = blockIdx.x * kRowT + threadIdx.x;
  if (i >= N) return;
  const long long bq = blockIdx.y;  // problem of a batched level
  A += bq * St<D, 1>::NS * Np;
  x += bq * Np;
  const double w = omega ? __ldg(omega + bq * Np + i) : damp;
  double dg;
  const double s = q1_row_sum<D>(A, Np, N, M, x, i, dg);
  const double t = (b[bq * Np + i] - s) / dg;
  if (write_r) r[bq * Np + i] = t;
  xout[bq * Np + i] = fma(w, t, x[i]);
}

// k_jacobi on a scalar Q2 level (the diagonal sits at the node's colour-major place)
template <int D>
__global__ void __launch_bounds__(kBlock)
k_jacobi_q2(const double* __restrict__ A, long long N, long long Np, long long M, double damp,
            const double* __restrict__ omega, double* x, double* r, int write_r, const __grid_constant__ Q2Layout lay) {
  pdl_next_light();
  pdl_wait();
  constexpr int C = St<D, 2>::CENTER;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  long long c[3];
  node_coords32(i, M, D, c);
  const double t = r[i] / A[(long long)C * Np + q2c_pos<D>(lay, c, M, 0)];
  if (write_r) r[i] = t;
  x[i] = fma(omega ? omega[i] : damp, t, x[i]);
}

// ------------------------------------- Q2 rows by colour class and parity
// The row kernels of scalar Q2 levels give each block rows of one colour
// class and one parity pattern (bit k: coordinate k odd).  All rows of a
// warp then admit the same slots, so a row is a compile-time list of its
// stored slots -- no per-slot test, no divergence -- and a thread issues a
// whole z-plane of the stencil (up to 25 coefficient and 25 neighbour loads)
// before the plane's first multiply-add; the row sum still runs in slot
// order, skipping only structural zeros.  Along direction k the class (digit
// d = c mod 3) holds c = d + 3 j, j = 0 .. n-1; its rows of parity p are
// j = j0, j0 + 2, .. with j0 = (p + d) & 1.  Inside a class the coefficient
// arrays are contiguous, so a warp's loads of one slot stay within a few
// sectors.
constexpr int kQ2T = 128;  // threads per block
// matvec and Jacobi residual in 3D: four blocks per SM (at most 128
// registers: the batched loads of a stencil plane fit without spills, 16
// warps per SM instead of 12; the SOR sweep measured slower so)
template <int D>
constexpr int kQ2MinBlocks = D == 3 ? 4 : 1;

struct Q2Sub {
  int d[3], j0[3], st[3], n[3];  // class digit, first place, step and row count along each direction
  long long cnt;                 // rows of the (class, parity) subgrid
};

// ssc >= 0: only the rows that belong to vertex blocks of that colour of the
// <geometric-ssc> sweep -- every odd coordinate, and the even ones that are
// vertices of the colour (coordinate = 2 bit mod 4)
template <int D>
__host__ __device__ __forceinline__ void q2_sub(int M, int colour, int pat, Q2Sub& s, int ssc = -1) {
  s.cnt = 1;
  int t = colour;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k < D) {
      const int d = t % 3, nk = (M - d + 2) / 3;
      const bool quarter = ssc >= 0 && !((pat >> k) & 1);
      const int j0 = quarter ? ((2 * ((ssc >> k) & 1) - d) * 3) & 3 : (((pat >> k) & 1) + d) & 1;
      const int st = quarter ? 4 : 2;
      t /= 3;
      s.d[k] = d;
      s.j0[k] = j0;
      s.st[k] = st;
      s.n[k] = nk > j0 ? (nk - j0 + st - 1) / st : 0;
    } else {
      s.d[k] = 0;
      s.j0[k] = 0;
      s.st[k] = 2;
      s.n[k] = 1;
    }
    s.cnt *= s.n[k];
  }
}

// blocks a class takes: its parity subgrids one after another
template <int D>
__host__ __device__ __forceinline__ long long q2_class_blocks(int M, int colour, int ssc = -1) {
  long long nb = 0;
  for (int pat = 0; pat < (1 << D); ++pat) {
    Q2Sub s;
    q2_sub<D>(M, colour, pat, s, ssc);
    nb += (s.cnt + kQ2T - 1) / kQ2T;
  }
  return nb;
}

// block blk of a class: its parity pattern, subgrid and this thread's row u
// in it; false when the thread has no row
template <int D>
__device__ __forceinline__ bool q2_block(int M, int colour, long long blk, int& pat, Q2Sub& s, long long& u,
                                         int ssc = -1) {
  for (pat = 0; pat < (1 << D); ++pat) {
    q2_sub<D>(M, colour, pat, s, ssc);
    const long long nb = (s.cnt + kQ2T - 1) / kQ2T;
    if (blk < nb) {
      u = blk * kQ2T + threadIdx.x;
      return u < s.cnt;
    }
    blk -= nb;
  }
  return false;
}

// a row's coordinates, node index and its positions in the arrays of every
// slot pattern (colour-major layout; patterns it does not admit are never read)
template <int D>
__device__ __forceinline__ long long q2_place(const Q2Layout& lay, int M, int colour, const Q2Sub& s, long long u,
                                              int c[3], int (&p)[1 << D]) {
  const unsigned uu = (unsigned)u;
  const unsigned q = D > 1 ? uu / (unsigned)s.n[0] : 0u;
  const int uk[3] = {(int)(D > 1 ? uu - q * (unsigned)s.n[0] : uu), D > 2 ? (int)(q % (unsigned)s.n[1]) : (int)q,
                     D > 2 ? (int)(q / (unsigned)s.n[1]) : 0};
  int j[3][2], e[3][2];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k < D) {
      const int jj = s.j0[k] + s.st[k] * uk[k], d = s.d[k], x0 = q2c_x0(d);
      c[k] = d + 3 * jj;
      j[k][0] = jj;
      e[k][0] = (M - d + 2) / 3;
      j[k][1] = (c[k] - x0) / 6;
      e[k][1] = x0 < M ? (M - x0 + 5) / 6 : 0;
    } else {
      c[k] = 0;
      j[k][0] = j[k][1] = 0;
      e[k][0] = e[k][1] = 1;
    }
  }
#pragma unroll
  for (int r = 0; r < (1 << D); ++r) {
    const int rx = r & 1, ry = (r >> 1) & 1, rz = (r >> 2) & 1;
    p[r] = lay.off[colour][r] + j[0][rx] + e[0][rx] * (j[1][ry] + e[1][ry] * j[2][rz]);
  }
  return (long long)c[0] + (long long)M * (c[1] + (long long)M * c[2]);
}

// sum over the row's stored slots, in slot order, of A(i, s) x(i + off_s).
// PAT: the row's parity pattern.  Neighbour coordinates are clamped into the
// grid per direction (a slot reaching outside holds a zero).
template <int D, int PAT>
__device__ __forceinline__ double q2_row_sum(const double* __restrict__ A, long long Np, const double* x, int M,
                                             const int c[3], const int (&p)[1 << D]) {
  int cl[3][5];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int o = 0; o < 5; ++o) cl[k][o] = k < D ? min(max(c[k] + o - 2, 0), M - 1) : 0;
  constexpr int NZ = D > 2 ? 5 : 1, NY = D > 1 ? 5 : 1;
  double s = 0.0;
#pragma unroll
  for (int sz = 0; sz < NZ; ++sz) {
    const bool rz = D > 2 && (sz == 0 || sz == 4);
    if (rz && (PAT & 4)) continue;
    // the loads of a plane's rows 0-2, their multiply-adds, then rows 3-4
    // (at most 30 doubles in flight: the 3D kernels fit four or five blocks
    // per SM without spills); the sum stays in slot order
    double av[15], xv[15];
    int q = 0;
#pragma unroll
    for (int sy = 0; sy < NY; ++sy) {
      const bool ry = D > 1 && (sy == 0 || sy == 4);
      if (!(ry && (PAT & 2))) {
        const double* xl = x + (long long)M * (cl[1][sy] + (long long)M * cl[2][sz]);
#pragma unroll
        for (int sx = 0; sx < 5; ++sx) {
          const bool rx = sx == 0 || sx == 4;
          if (rx && (PAT & 1)) continue;
          const int slot = sx + 5 * (sy + 5 * sz);
          const int r = (rx ? 1 : 0) | (ry ? 2 : 0) | (rz ? 4 : 0);
          av[q] = __ldg(A + (long long)slot * Np + p[r]);
          xv[q] = xl[cl[0][sx]];
          ++q;
        }
      }
      if (sy == 2 || sy == NY - 1) {
#pragma unroll
        for (int k = 0; k < q; ++k) s = fma(av[k], xv[k], s);
        q = 0;
      }
    }
  }
  return s;
}

// calls f(integral_constant<int, pat>) for the runtime pattern pat
template <int D, typename F>
__device__ __forceinline__ void q2_pat_dispatch(int pat, F&& f) {
  switch (pat) {
    case 0: f(std::integral_constant<int, 0>{}); break;
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: if constexpr (D > 1) f(std::integral_constant<int, 2>{}); break;
    case 3: if constexpr (D > 1) f(std::integral_constant<int, 3>{}); break;
    case 4: if constexpr (D > 2) f(std::integral_constant<int, 4>{}); break;
    case 5: if constexpr (D > 2) f(std::integral_constant<int, 5>{}); break;
    case 6: if constexpr (D > 2) f(std::integral_constant<int, 6>{}); break;
    default: if constexpr (D > 2) f(std::integral_constant<int, 7>{}); break;
  }
}

// whether a node lies on a Dirichlet face
__device__ __forceinline__ bool q2_face(const int c[3], int M, int dmask) {
  bool on = false;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    on = on || (c[k] == 0 && ((dmask >> (2 * k)) & 1)) || (c[k] == M - 1 && ((dmask >> (2 * k + 1)) & 1));
  return on;
}

// One colour of the multicolour <sor> sweep of a 3D scalar Q2 level of few
// rows: a tile of 32 rows of one class and parity per block.  A row's sum is
// one chain of up to 125 fma in slot order (10 cycles each); a thread that
// also loads its row waits for memory ten times, as its registers hold half a
// stencil plane, and its unrolled code takes longer to fetch than to run.
// Here warp w loads the coefficients and unknowns of the (y, z) slot rows
// 3 w .. 3 w + 2 (the last warp four) of all 32 rows, up to 20 of each at
// once, into shared memory -- the row's stored slots one after another -- and
// one warp runs the 32 chains from there.  The colours of a sweep overlap:
// indices, coefficients, diagonal and damping are fetched while the previous
// colour still runs, only the unknowns wait for it.
constexpr int kTileRows = 32, kTileT = 256;
constexpr size_t kTileSmem = 2 * 125 * kTileRows * sizeof(double);
// Rows of a colour up to which an SOR sweep takes this form, and nodes up to
// which an SSC sweep does; beyond, the strided reads of x bound it and a thread
// per row is faster.  A coarse level of at most 1,024 unknowns leaves 2^k and
// 3 2^k cells a side.  SOR sweep by tiles and by rows, us: 49^3 nodes 112 and
// 198, 65^3 (10,648 rows) 130 and 238, 97^3 (35,937 rows) 310 and 314, 129^3
// 688 and 440.  SSC sweep: 25^3 90 and 132, 33^3 128 and 141, 49^3 232 and 189,
// 65^3 490 and 328.
constexpr long long kTileMax = 12000, kSscTileMax = 40000;

// SSC: the residuals r = b - A x of the rows of one <geometric-ssc> colour
// instead (every class, blockIdx.z; b may be r): see k_ssc_solve_q2.
template <bool SSC>
__global__ void __launch_bounds__(kTileT, 3)
k_q2_tile(const double* __restrict__ A, long long Np, int M, int col, int dmask, double damp,
          const double* __restrict__ omega, double* x, const double* b, double* r,
          const __grid_constant__ Q2Layout lay) {
  extern __shared__ double tsm[];
  pdl_next();
  const int pat = (int)blockIdx.y, colour = SSC ? (int)blockIdx.z : col;
  Q2Sub sub;
  q2_sub<3>(M, colour, pat, sub, SSC ? col : -1);
  const int u0 = blockIdx.x * kTileRows;
  if (u0 >= sub.cnt) {
    pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool live = u0 + lane < sub.cnt;
  const unsigned u = live ? u0 + lane : (unsigned)sub.cnt - 1;  // spare lanes repeat the last row and store nothing
  const unsigned q0 = u / (unsigned)sub.n[0];
  const int uk[3] = {(int)(u - q0 * (unsigned)sub.n[0]), (int)(q0 % (unsigned)sub.n[1]),
                     (int)(q0 / (unsigned)sub.n[1])};
  int c[3], j[3][2], e[3][2];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int jj = sub.j0[k] + sub.st[k] * uk[k], d = sub.d[k], x0 = q2c_x0(d);
    c[k] = d + 3 * jj;
    j[k][0] = jj;
    e[k][0] = (M - d + 2) / 3;
    j[k][1] = (c[k] - x0) / 6;
    e[k][1] = x0 < M ? (M - x0 + 5) / 6 : 0;
  }
  // stored slots per direction (5 or 3) and the first of them
  const int ox = pat & 1, oy = (pat >> 1) & 1, oz = pat >> 2;
  const int nx = 5 - 2 * ox, ny = 5 - 2 * oy, nv = nx * ny * (5 - 2 * oz);
  double* sa = tsm + lane;                    // [stored slot][row] coefficients
  double* sx = tsm + 125 * kTileRows + lane;  // [stored slot][row] unknowns
  double v[4][5];
  bool on[4];
  int at[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int yz = 3 * warp + t, sz = yz / 5, sy = yz - 5 * sz;
    const bool ry = sy == 0 || sy == 4, rz = sz == 0 || sz == 4;
    on[t] = (t < 3 || warp == 7) && !(ry && oy) && !(rz && oz);
    at[t] = ((sz - oz) * ny + sy - oy) * nx - ox;  // where the slot row starts, less its skipped slot
    if (!on[t]) continue;
    const int pl = (ry ? j[1][1] : j[1][0]) + (ry ? e[1][1] : e[1][0]) * (rz ? j[2][1] : j[2][0]);
    const int rr = (ry ? 2 : 0) | (rz ? 4 : 0);
    const double* a = A + (long long)(5 * yz) * Np;
    const double* a1 = a + lay.off[colour][rr | 1] + j[0][1] + e[0][1] * pl;
    a += lay.off[colour][rr] + j[0][0] + e[0][0] * pl;
    if (!ox) v[t][0] = __ldcg(a1);
#pragma unroll
    for (int q = 1; q < 4; ++q) v[t][q] = __ldcg(a + (long long)q * Np);
    if (!ox) v[t][4] = __ldcg(a1 + 4 * Np);
  }
  const long long i = (long long)c[0] + (long long)M * (c[1] + (long long)M * c[2]);
  double d = 1.0, bi = 0.0, xi = 0.0, w = damp;
  if (!SSC && warp == 0) {
    d = __ldcg(A + 62LL * Np + lay.off[colour][0] + j[0][0] + e[0][0] * (j[1][0] + e[1][0] * j[2][0]));
    if (omega) w = __ldcg(omega + i);
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (on[t]) {
#pragma unroll
      for (int q = 0; q < 5; ++q)
        if (!(q == 0 || q == 4) || !ox) sa[(at[t] + q) * kTileRows] = v[t][q];
    }
  pdl_wait();
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    if (!on[t]) continue;
    const int yz = 3 * warp + t, sz = yz / 5, sy = yz - 5 * sz;
    const double* xl = x + (long long)M * (min(max(c[1] + sy - 2, 0), M - 1) +
                                           (long long)M * min(max(c[2] + sz - 2, 0), M - 1));
#pragma unroll
    for (int q = 0; q < 5; ++q)  // outside the grid the coefficient is a stored zero
      if (!(q == 0 || q == 4) || !ox) v[t][q] = xl[min(max(c[0] + q - 2, 0), M - 1)];
  }
  if (warp == 0) {
    if (!SSC) xi = x[i];
    bi = b[i];
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (on[t]) {
#pragma unroll
      for (int q = 0; q < 5; ++q)
        if (!(q == 0 || q == 4) || !ox) sx[(at[t] + q) * kTileRows] = v[t][q];
    }
  __syncthreads();
  if (warp) return;
  double s = 0.0;
  // nine terms at a time (27, 45 or 75 + 6, 125 + 1: the last ones guarded)
  int q0v = 0;
#pragma unroll 1
  for (; q0v + 9 <= nv; q0v += 9) {
    double ta[9], tx[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) { ta[q] = sa[(q0v + q) * kTileRows]; tx[q] = sx[(q0v + q) * kTileRows]; }
#pragma unroll
    for (int q = 0; q < 9; ++q) s = fma(ta[q], tx[q], s);
  }
  for (; q0v < nv; ++q0v) s = fma(sa[q0v * kTileRows], sx[q0v * kTileRows], s);
  if (!live) return;
  if (SSC) {
    if (pat == 0 || !q2_face(c, M, dmask)) r[i] = bi - s;
    return;
  }
  const double t = (bi - s) / d;
  r[i] = t;
  x[i] = fma(w, t, xi);
}

// colour `col` by tiles: blockIdx.x the tiles of the largest parity subgrid,
// .y the parity, .z the class (SSC)
template <bool SSC>
static void launch_q2_tile(const LevelView& L, int col, double damp, double* x, const double* b, double* r,
                           const Q2Layout& lay, cudaStream_t st) {
  const int M = (int)L.M;
  long long most = 1;
  for (int cls = SSC ? 0 : col; cls < (SSC ? 27 : col + 1); ++cls)
    for (int pat = 0; pat < 8; ++pat) {
      Q2Sub s;
      q2_sub<3>(M, cls, pat, s, SSC ? col : -1);
      most = std::max(most, s.cnt);
    }
  if (col == 0) cudaFuncSetAttribute(k_q2_tile<SSC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem);
  launch_early(k_q2_tile<SSC>, dim3((unsigned)((most + kTileRows - 1) / kTileRows), 8, SSC ? 27 : 1), kTileT,
             kTileSmem, st, L.A, L.Np, M, col, L.dmask, damp, L.omega, x, b, r, lay);
}

// the rows of block blk of colour class `colour` in the multicolour <sor>
// sweep of a scalar Q2 level (linit.lisp:288-323): r = (b - A x)/d, x += w r
template <int D>
__device__ __forceinline__ void sor_q2_block(const double* __restrict__ A, long long Np, int M, int colour,
                                             long long blk, double omega_s, const double* __restrict__ omega,
                                             double* x, const double* b, double* r, const Q2Layout& lay) {
  int pat;
  Q2Sub sub;
  long long u;
  if (!q2_block<D>(M, colour, blk, pat, sub, u)) return;
  int c[3], p[1 << D];
  const long long i = q2_place<D>(lay, M, colour, sub, u, c, p);
  constexpr int C = St<D, 2>::CENTER;
  // the row's own operands first, so that their loads overlap the stencil's
  const double d = __ldg(A + (long long)C * Np + p[0]);
  const double bi = b[i], xi = x[i], wi = omega ? __ldg(omega + i) : omega_s;
  double s = 0.0;
  q2_pat_dispatch<D>(pat, [&](auto P) { s = q2_row_sum<D, decltype(P)::value>(A, Np, x, M, c, p); });
  const double tt = (bi - s) / d;
  r[i] = tt;
  x[i] = fma(wi, tt, xi);
}

// one colour of the sweep per launch
template <int D>
__global__ void __launch_bounds__(kQ2T)
k_sor_q2(const double* __restrict__ A, long long Np, int M, int colour, double omega_s,
         const double* __restrict__ omega, double* x, const double* b, double* r,
         const __grid_constant__ Q2Layout lay) {
  pdl_next();
  pdl_wait();
  sor_q2_block<D>(A, Np, M, colour, blockIdx.x, omega_s, omega, x, b, r, lay);
}

// y = A x or r = b - A x on a scalar Q2 level, rows by class (blockIdx.y) and parity
template <int D, bool RES>
__global__ void __launch_bounds__(kQ2T, kQ2MinBlocks<D>)
k_spmv_q2c(const double* __restrict__ A, long long Np, int M, const double* x, const double* b,
           double* y, const __grid_constant__ Q2Layout lay) {
  pdl_next();
  pdl_wait();
  int pat;
  Q2Sub sub;
  long long u;
  const int colour = (int)blockIdx.y;
  if (!q2_block<D>(M, colour, blockIdx.x, pat, sub, u)) return;
  int c[3], p[1 << D];
  const long long i = q2_place<D>(lay, M, colour, sub, u, c, p);
  double s = 0.0;
  q2_pat_dispatch<D>(pat, [&](auto P) { s = q2_row_sum<D, decltype(P)::value>(A, Np, x, M, c, p); });
  y[i] = RES ? b[i] - s : s;
}

// k_row_jacobi_q1 on a scalar Q2 level, rows by class and parity
template <int D>
__global__ void __launch_bounds__(kQ2T, kQ2MinBlocks<D>)
k_jacobi_res_q2c(const double* __restrict__ A, long long Np, int M, double damp, const double* __restrict__ omega,
                 const double* x, const double* b, double* __restrict__ xout, double* r, int write_r,
                 const __grid_constant__ Q2Layout lay) {
  pdl_next();
  pdl_wait();
  int pat;
  Q2Sub sub;
  long long u;
  const int colour = (int)blockIdx.y;
  if (!q2_block<D>(M, colour, blockIdx.x, pat, sub, u)) return;
  int c[3], p[1 << D];
  const long long i = q2_place<D>(lay, M, colour, sub, u, c, p);
  constexpr int C = St<D, 2>::CENTER;
  const double d = __ldg(A + (long long)C * Np + p[0]);
  double s = 0.0;
  q2_pat_dispatch<D>(pat, [&](auto P) { s = q2_row_sum<D, decltype(P)::value>(A, Np, x, M, c, p); });
  const double t = (b[i] - s) / d;
  if (write_r) r[i] = t;
  xout[i] = fma(omega ? omega[i] : damp, t, x[i]);
}

// ------------------------------------------------------------- smoothers
// <jacobi> step with an up-to-date residual: t = r/d, x += w t, r := t
__global__ void __launch_bounds__(kBlock)
k_jacobi(const double* __restrict__ Dg, long long N, double damp, const double* __restrict__ omega,
         double* x, double* r, int write_r, long long vs, long long as) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const long long bq = blockIdx.y;  // problem of a batched level: vector stride vs, matrix stride as
  Dg += bq * as;
  x += bq * vs;
  r += bq * vs;
  if (omega) omega += bq * vs;
  const double t = r[i] / Dg[i];
  if (write_r) r[i] = t;
  const double w = omega ? omega[i] : damp;
  x[i] = fma(w, t, x[i]);
}

// one colour of the multicolour <sor> sweep on a Q1 level (P = 1): rows with
// (i_k mod (P+1)) = col_k (scalar Q2 levels: k_sor_q2).
// SSC: the <geometric-ssc> sweep of a Q1 level, whose vertex blocks hold one
// node -- the same update, with r keeping the unscaled residual
// (blockit.lisp:131-138) instead of the <sor> correction (linit.lisp:312-322)
template <int D, int P, bool SSC = false>
__global__ void __launch_bounds__(kRowT, kRowMinBlocks)
k_sor_colour(const double* __restrict__ A, long long N, long long Np, long long M, int colour,
             double omega_s, const double* __restrict__ omega, double* x, const double* b, double* r) {
  if (D == 1) pdl_next_light();
  else pdl_next();
  constexpr int NS = St<D, P>::NS;
  constexpr int C = St<D, P>::CENTER;
  constexpr int Q = P + 1;
  const int cx = colour % Q, cy = (colour / Q) % Q, cz = colour / (Q * Q);
  const long long nx = (M - cx + Q - 1) / Q;
  const long long ny = D > 1 ? (M - cy + Q - 1) / Q : 1;
  const long long nz = D > 2 ? (M - cz + Q - 1) / Q : 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nx * ny * nz) return;
  const unsigned tu = (unsigned)t, nxu = (unsigned)nx, nyu = (unsigned)ny;
  const unsigned tq = tu / nxu;
  const long long jx = tu - tq * nxu, jy = tq % nyu, jz = tq / nyu;
  const long long i = (cx + Q * jx) + M * ((D > 1 ? cy + Q * jy : 0) + M * (D > 2 ? cz + Q * jz : 0));
  // coefficients and damping do not depend on the previous launch
  double av[NS], xv[NS];
#pragma unroll
  for (int k = 0; k < NS; ++k) av[k] = __ldg(A + (long long)k * Np + i);
  const double w = omega ? __ldg(omega + i) : omega_s;
  pdl_wait();
#pragma unroll
  for (int k = 0; k < NS; ++k) xv[k] = x[clampi(i + slot_off<D, P>(k, M), N)];
  double s = 0.0;
  const double d = av[C];
#pragma unroll
  for (int k = 0; k < NS; ++k) s = fma(av[k], xv[k], s);
  const double rr = b[i] - s;
  const double tt = rr / d;
  r[i] = SSC ? rr : tt;
  x[i] = fma(w, tt, !SSC && x == r ? tt : xv[C]);  // one vector for both: x is what r has become
}

// Step K of the warp's LU factorisation of a vertex block (rows in lanes):
// the pivot is the first position holding the largest magnitude, the lane at
// position K and the pivot's lane exchange positions (the rows stay put), the
// rows below keep their multiplier in column K.  The recursion keeps every
// index a compile-time constant, so the row stays in registers.
template <int NB, int K>
__device__ __forceinline__ void ssc_lu_step(double (&a)[NB], int& pos, int lane) {
  if constexpr (K < NB) {
    constexpr unsigned FULL = 0xffffffffu;
    double val = (lane < NB && pos >= K) ? fabs(a[K]) : -1.0;
    int key = pos, ln = lane;
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      const double ov = __shfl_xor_sync(FULL, val, m);
      const int ok = __shfl_xor_sync(FULL, key, m);
      const int ol = __shfl_xor_sync(FULL, ln, m);
      if (ov > val || (ov == val && ok < key)) { val = ov; key = ok; ln = ol; }
    }
    if (pos == K) pos = key;  // row interchange
    if (lane == ln) pos = K;
    const double piv = __shfl_sync(FULL, a[K], ln);
    const double rcp = 1.0 / piv;
    const bool below = lane < NB && pos > K;
    const double mlt = a[K] * rcp;
#pragma unroll
    for (int j = K + 1; j < NB; ++j) {
      const double pj = __shfl_sync(FULL, a[j], ln);
      if (below) a[j] = a[j] - mlt * pj;
    }
    if (below) a[K] = mlt;
    ssc_lu_step<NB, K + 1>(a, pos, lane);
  }
}

// a / u rounded to nearest, given y = 1 / u rounded to nearest: two residual
// corrections of a y (Markstein, IBM J. Res. Dev. 34, 1990: with y correctly
// rounded and q within an ulp, q + (a - q u) y rounds to the quotient).  Holds
// while the residuals are exact, i.e. away from the ends of the exponent
// range (div_by_ok).  50 cycles in the chain of a substitution instead of the
// division's 137.
__device__ __forceinline__ double div_by(double a, double u, double y) {
  double q = a * y;
  q = fma(fma(-u, q, a), y, q);
  return fma(fma(-u, q, a), y, q);
}
__device__ __forceinline__ bool div_by_ok(double a, double u, double q) {
  auto mid = [](double v) { return (((unsigned)__double2hiint(v) >> 20) & 0x7ff) - 300u < 1400u; };
  return mid(u) && (a == 0.0 || (mid(a) && mid(q)));  // 1 / u may be infinite: then not even 0 / u holds
}

// A_BB c = r_B of a vertex block with its stored factors: lane t brings member
// t's residual and gets member t's correction.  f: the factors in shared
// memory, [column][position]; the rows sit in lanes by their final position,
// mem is the member of lane's row, u and y its pivot and the pivot's
// reciprocal.  Forward: the row at position K is final, the rows below
// subtract their multiplier times it (the operations, in order, of carrying
// the right-hand side through the elimination).  Backward: the row at
// position K divides, the rows above subtract; lane K keeps the solution of
// member K.  The columns run in loops: unrolled, with the factors in
// registers, the code took longer to fetch than to run.
template <int NB>
__device__ __forceinline__ double ssc_block_solve(const double* f, int mem, double u, double y, double rr, int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  rr = __shfl_sync(FULL, rr, mem);
  const int t = lane < NB ? lane : NB - 1;
#pragma unroll 3
  for (int K = 0; K < NB; ++K) {
    const double fk = f[K * NB + t], rk = __shfl_sync(FULL, rr, K);
    if (lane > K) rr = rr - fk * rk;
  }
  const double rf = rr;
  double corr = 0.0;
#pragma unroll 3
  for (int K = NB - 1; K >= 0; --K) {
    const double fk = f[K * NB + t], q = div_by(rr, u, y), xk = __shfl_sync(FULL, q, K);
    if (lane == K) corr = q;
    if (lane < K) rr = rr - xk * fk;
  }
  // lane K's rr is the numerator of its quotient
  if (__any_sync(FULL, lane < NB && !div_by_ok(rr, u, corr))) {
    rr = rf;
#pragma unroll 1
    for (int K = NB - 1; K >= 0; --K) {
      const double fk = f[K * NB + t];
      if (lane == K) corr = rr / u;
      const double xk = __shfl_sync(FULL, corr, K);
      if (lane < K) rr = rr - xk * fk;
    }
  }
  return corr;
}

// copies a block's factors to shared memory, every load before the first store
template <int NB>
__device__ __forceinline__ void ssc_stage(const double* __restrict__ F, double* f, int lane) {
  constexpr int PER = (NB * NB + 31) / 32;
  double v[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) v[q] = q * 32 + lane < NB * NB ? __ldcg(F + q * 32 + lane) : 0.0;
#pragma unroll
  for (int q = 0; q < PER; ++q)
    if (q * 32 + lane < NB * NB) f[q * 32 + lane] = v[q];
}

// Member `lane` of the vertex block of vertex v (2 x vertex index): its node
// coordinates and offsets, whether it is in the domain, and whether it is a
// member of the block (the vertex itself, or a non-Dirichlet node).
template <int D>
struct SscMember {
  int dm[3], c[3];
  bool real;
};

template <int D>
__device__ __forceinline__ SscMember<D> ssc_member(const int v[3], int lane, int Mi, int dmask) {
  constexpr int NB = D == 1 ? 3 : (D == 2 ? 9 : 27);
  SscMember<D> m;
  bool in = lane < NB, dir = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) { m.dm[k] = 0; m.c[k] = v[k]; }
#pragma unroll
  for (int k = 0, q = lane; k < D; ++k, q /= 3) {
    m.dm[k] = q % 3 - 1;
    m.c[k] = v[k] + m.dm[k];
    in = in && m.c[k] >= 0 && m.c[k] < Mi;
    dir = dir || (m.c[k] == 0 && ((dmask >> (2 * k)) & 1)) || (m.c[k] == Mi - 1 && ((dmask >> (2 * k + 1)) & 1));
  }
  m.real = in && (lane == NB / 2 || !dir);
  return m;
}

// The LU factors of every vertex block of a scalar Q2 level (all colours in
// one launch), for the <geometric-ssc> sweeps: the local matrix A_BB
// (blockit.lisp:150-153) gathered by the member lanes -- every entry lies in
// a pattern-0 slot: a row that is odd along a direction meets the box only
// within +-1 there -- members outside the domain, and Dirichlet members
// other than the vertex, as identity rows with zero columns (the pivots and
// the arithmetic of the real rows are those of the compact block), then
// factored as by gesv! (right-looking, partial pivoting).  The factors depend
// on the matrix only, so a sweep that reuses them repeats exactly the
// operations of factoring afresh.  Layout: F[block][k][position], the member
// whose row ended there in P[block][position]; block = lexicographic vertex
// index.
template <int D>
__global__ void __launch_bounds__(128)
k_ssc_factor_q2(const double* __restrict__ A, long long Np, long long M, int dmask, double* F, unsigned char* P,
                const __grid_constant__ Q2Layout lay) {
  constexpr int NB = D == 1 ? 3 : (D == 2 ? 9 : 27);
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // uniform per warp
  const int Mi = (int)M;
  const int nv = (Mi + 1) / 2;
  const long long nblk = D == 1 ? nv : (D == 2 ? (long long)nv * nv : (long long)nv * nv * nv);
  if (w >= nblk) return;  // the whole warp leaves together
  const int wi = (int)w;
  const int v[3] = {2 * (wi % nv), D > 1 ? 2 * ((wi / nv) % nv) : 0, D > 2 ? 2 * (wi / (nv * nv)) : 0};
  const SscMember<D> mb = ssc_member<D>(v, lane, Mi, dmask);
  const unsigned realmask = __ballot_sync(FULL, mb.real);
  double a[NB];
  if (mb.real) {
    const long long cl[3] = {mb.c[0], mb.c[1], mb.c[2]};
    Q2Base<D> qb;
    q2_base<D, true, true>(lay, cl, M, qb);
    const long long p0 = qb.p[0];
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      bool near = true;
      int sl = 0;
#pragma unroll
      for (int k = 0, q = u, m5 = 1; k < D; ++k, q /= 3, m5 *= 5) {
        const int o = (q % 3 - 1) - mb.dm[k];
        near = near && o >= -1 && o <= 1;
        sl += (o + 2) * m5;
      }
      a[u] = (near && ((realmask >> u) & 1)) ? A[(long long)sl * Np + p0] : 0.0;
    }
  } else {
#pragma unroll
    for (int u = 0; u < NB; ++u) a[u] = (u == lane) ? 1.0 : 0.0;
  }
  int pos = lane;  // lanes >= NB are never candidates
  ssc_lu_step<NB, 0>(a, pos, lane);
  if (lane < NB) {
    double* f = F + w * NB * NB + pos;
#pragma unroll
    for (int k = 0; k < NB; ++k) f[k * NB] = a[k];
    P[w * NB + pos] = (unsigned char)lane;
  }
}

// One colour of the <geometric-ssc> sweep on a scalar Q2 level
// (blockit.lisp:118-204 with the vertex-centred blocks of geoblock.lisp:72-158)
// runs in two launches: the residuals r = b - A x (b may alias r: the alias
// inside <cg>) of the rows of the colour's blocks, in class order as the
// other row kernels, then a warp per block that solves A_BB c = r_B with the
// stored factors (forward in position order, backward column by column) and
// adds x_B += omega c.  Blocks of one colour (vertex index mod 2 per
// direction) share no node and read no unknown another one writes, so the
// residuals are those each block would form for itself.  Formed by the block's
// own lanes, 27 rows of a warp scattered over the classes' arrays, they took
// most of the colour's time: 65^3 nodes 107 us a colour, 45-54 us so; 17^3
// 28 us, 8 us.
// A Dirichlet node belongs to no block but its own.
template <int D>
__global__ void __launch_bounds__(kQ2T, kQ2MinBlocks<D>)
k_ssc_res_q2(const double* __restrict__ A, long long Np, int M, int ssc, int dmask, const double* x, const double* b,
             double* r, const __grid_constant__ Q2Layout lay) {
  pdl_next();
  int pat;
  Q2Sub sub;
  long long u;
  const int colour = (int)blockIdx.y;
  const bool row = q2_block<D>(M, colour, blockIdx.x, pat, sub, u, ssc);
  pdl_wait();
  if (!row) return;
  int c[3], p[1 << D];
  const long long i = q2_place<D>(lay, M, colour, sub, u, c, p);
  const double bi = b[i];
  double s = 0.0;
  q2_pat_dispatch<D>(pat, [&](auto P) { s = q2_row_sum<D, decltype(P)::value>(A, Np, x, M, c, p); });
  if (pat == 0 || !q2_face(c, M, dmask)) r[i] = bi - s;
}

template <int D>
__global__ void __launch_bounds__(128, 7)
k_ssc_solve_q2(int Mi, int dmask, int colour, double omega, double* x, const double* r, const double* __restrict__ F,
               const unsigned char* __restrict__ P) {
  constexpr int NB = D == 1 ? 3 : (D == 2 ? 9 : 27);
  __shared__ double fs_all[4][NB * NB];
  pdl_next();
  const int lane = threadIdx.x & 31;
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);  // uniform per warp
  const int nv = (Mi + 1) / 2;  // vertices per direction
  const int bx = colour & 1, by = (colour >> 1) & 1, bz = (colour >> 2) & 1;
  const int ex = (nv - bx + 1) / 2, ey = D > 1 ? (nv - by + 1) / 2 : 1, ez = D > 2 ? (nv - bz + 1) / 2 : 1;
  if (w >= ex * ey * ez) {  // the whole warp leaves together
    pdl_wait();
    return;
  }
  const int jx = w % ex, jq = w / ex, jy = jq % ey, jz = jq / ey;
  const int ax = bx + 2 * jx, ay = D > 1 ? by + 2 * jy : 0, az = D > 2 ? bz + 2 * jz : 0;
  const int v[3] = {2 * ax, 2 * ay, 2 * az};
  const long long blk = ax + (long long)nv * (ay + (long long)nv * az);
  // the factors do not depend on the previous launch
  double* fs = fs_all[threadIdx.x >> 5];
  ssc_stage<NB>(F + blk * NB * NB, fs, lane);
  const int mem = lane < NB ? P[blk * NB + lane] : lane;
  const SscMember<D> mb = ssc_member<D>(v, lane, Mi, dmask);
  const long long i = mb.real ? (long long)mb.c[0] + Mi * ((long long)mb.c[1] + Mi * (long long)mb.c[2]) : 0;
  __syncwarp();
  const double u = lane < NB ? fs[lane * NB + lane] : 1.0, y = 1.0 / u;
  pdl_wait();
  const double rr = mb.real ? r[i] : 0.0, xi = mb.real ? x[i] : 0.0;
  const double corr = ssc_block_solve<NB>(fs, mem, u, y, rr, lane);
  if (mb.real) x[i] = fma(omega, corr, xi);
}

// <geometric-psc> on a scalar Q1 level: one-node blocks, x_i += damp r_i /
// a_ii (the 1 x 1 LU divides by the pivot), r unchanged
template <int D>
__global__ void __launch_bounds__(kBlock)
k_psc_q1(const double* __restrict__ A, long long N, long long Np, double damp, double* x, const double* r) {
  pdl_next_light();
  pdl_wait();
  constexpr int C = St<D, 1>::CENTER;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  x[i] = fma(damp, r[i] / A[(long long)C * Np + i], x[i]);
}

// <geometric-psc> on a scalar Q2 level, first pass: every vertex block (warp
// per block, all blocks in one launch) solves A_BB c = r_B with the stored
// factors and the residual as it stands (r is read, not written); member t's
// correction goes to C[block][t] (zero for padded members).
template <int D>
__global__ void __launch_bounds__(128, 6)
k_psc_block_q2(long long M, int dmask, const double* r, const double* __restrict__ F,
               const unsigned char* __restrict__ P, double* __restrict__ C) {
  pdl_next();
  pdl_wait();
  constexpr int NB = D == 1 ? 3 : (D == 2 ? 9 : 27);
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // uniform per warp
  const int Mi = (int)M;
  const int nv = (Mi + 1) / 2;
  const long long nblk = D == 1 ? nv : (D == 2 ? (long long)nv * nv : (long long)nv * nv * nv);
  if (w >= nblk) return;  // the whole warp leaves together
  const int wi = (int)w;
  const int v[3] = {2 * (wi % nv), D > 1 ? 2 * ((wi / nv) % nv) : 0, D > 2 ? 2 * (wi / (nv * nv)) : 0};
  const SscMember<D> mb = ssc_member<D>(v, lane, Mi, dmask);
  __shared__ double fs_all[4][NB * NB];
  double* fs = fs_all[threadIdx.x >> 5];
  ssc_stage<NB>(F + w * NB * NB, fs, lane);
  const int mem = lane < NB ? P[w * NB + lane] : lane;
  __syncwarp();
  const double u = lane < NB ? fs[lane * NB + lane] : 1.0, y = 1.0 / u;
  double rr = mb.real ? r[(long long)mb.c[0] + M * ((long long)mb.c[1] + M * (long long)mb.c[2])] : 0.0;
  const double corr = ssc_block_solve<NB>(fs, mem, u, y, rr, lane);
  if (lane < NB) C[w * NB + lane] = corr;
}

// second pass: node i adds, in increasing vertex order, damp times its
// correction from each block holding it as a member (the vertices within 1
// of it along every direction; a Dirichlet node belongs to its own block only)
template <int D>
__global__ void __launch_bounds__(kBlock)
k_psc_gather_q2(long long N, long long M, int dmask, double damp, const double* C, double* x) {
  pdl_next_light();
  pdl_wait();
  constexpr int NB = D == 1 ? 3 : (D == 2 ? 9 : 27);
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int Mi = (int)M, nv = (Mi + 1) / 2;
  int c[3] = {(int)(i % M), D > 1 ? (int)((i / M) % M) : 0, D > 2 ? (int)(i / (M * M)) : 0};
  bool dir = false;
#pragma unroll
  for (int k = 0; k < D; ++k)
    dir = dir || (c[k] == 0 && ((dmask >> (2 * k)) & 1)) || (c[k] == Mi - 1 && ((dmask >> (2 * k + 1)) & 1));
  // candidate vertex coordinates per direction, ascending
  int vc[3][2], nvc[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    nvc[k] = 1;
    vc[k][0] = vc[k][1] = 0;
    if (k >= D) continue;
    if (c[k] & 1) {
      nvc[k] = 2;
      vc[k][0] = c[k] - 1;
      vc[k][1] = c[k] + 1;
    } else {
      vc[k][0] = c[k];
    }
  }
  double xi = x[i];
  for (int iz = 0; iz < nvc[2]; ++iz)
    for (int iy = 0; iy < nvc[1]; ++iy)
      for (int ix = 0; ix < nvc[0]; ++ix) {
        const int vx = vc[0][ix], vy = vc[1][iy], vz = vc[2][iz];
        const bool own = vx == c[0] && (D < 2 || vy == c[1]) && (D < 3 || vz == c[2]);  // i is the vertex
        if (dir && !own) continue;
        const long long blk = (vx >> 1) + (long long)nv * ((vy >> 1) + (long long)nv * (vz >> 1));
        int t = c[0] - vx + 1;
        if (D > 1) t += 3 * (c[1] - vy + 1);
        if (D > 2) t += 9 * (c[2] - vz + 1);
        xi = fma(damp, C[blk * NB + t], xi);
      }
  x[i] = xi;
}

// ------------------------------------------------------ algebraic levels
// Compressed-row forms of the level operators (matrices handed over by the
// host, e.g. from sparse-matrix->ccs on an unstructured or adaptive mesh).
// Each row sums its entries in stored (column-ascending) order with fma, the
// order in which the stencil forms sum their slots, so a structured level
// given as compressed rows yields the structured results bit for bit.

// K = 8: the row sums fetch eight entries at a time -- indices and values, then
// the unknowns -- so a row of up to eight entries waits for memory twice (entry
// by entry it was twice per few entries), and the first eight are fetched while
// the previous launch still runs.  K = 1: entry by entry, for launches of many
// rows, whose time is instructions and warps and not a row's waits.  1,046,592
// rows of five entries, eight at a time and one: matvec 25 and 17 us, residual +
// Jacobi 29 and 21, prolongation 25 and 14; 250,000 rows 7.0 and 5.9, 7.4 and
// 5.9, 7.2 and 5.1; 125,000 rows of a colour 6.6 both; 65,000 rows 3.9 and 3.8,
// where the early start gives the eight 1-2 us.  Every caller's thread passes
// pdl_wait here.
constexpr long long kCsrWide = 150000;
template <int K>
__device__ __forceinline__ double csr_row_sum(const CsrView& a, long long i, const double* x) {
  const long long e1 = a.start[i + 1];
  if constexpr (K == 1) {
    pdl_wait();
    double s = 0.0;
    for (long long e = a.start[i]; e < e1; ++e) s = fma(a.value[e], x[a.index[e]], s);
    return s;
  }
  long long e = a.start[i];
  int ix[K];
  double v[K];
  auto fetch = [&]() {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (e + q < e1) {
        ix[q] = __ldg(a.index + e + q);
        v[q] = __ldg(a.value + e + q);
      }
  };
  fetch();
  pdl_wait();
  double s = 0.0;
  while (e < e1) {
    double xv[K];
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (e + q < e1) xv[q] = x[ix[q]];
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (e + q < e1) s = fma(v[q], xv[q], s);
    e += K;
    if (e < e1) fetch();
  }
  return s;
}
// threads per block: small levels spread over more SMs
template <int K>
constexpr int kCsrT = K > 1 ? 64 : kBlock;
template <int K>
__device__ __forceinline__ void csr_next() {
  if (K > 1) pdl_next();
  else pdl_next_light();
}

// a row's diagonal and damping: before the wait with K = 8, when they are needed
// with K = 1 (523,000 rows of a colour 16.6 us, 18.1 early)
__device__ __forceinline__ void csr_own(const double* diag, const double* omega, double damp, long long i, double& d,
                                        double& w) {
  d = __ldg(diag + i);
  w = omega ? __ldg(omega + i) : damp;
}

// y = A x, or r = b - A x (b may alias r)
template <int K>
__global__ void __launch_bounds__(kCsrT<K>, K > 1 ? 8 : 0)
k_csr_spmv(long long N, CsrView a, const double* x, const double* b, double* y, int res) {
  csr_next<K>();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double s = csr_row_sum<K>(a, i, x);
  y[i] = res ? b[i] - s : s;
}

// compute-residual fused with the following <jacobi> step (as k_row_jacobi_q1)
template <int K>
__global__ void __launch_bounds__(kCsrT<K>, K > 1 ? 8 : 0)
k_csr_jacobi_res(long long N, CsrView a, const double* __restrict__ diag, double damp,
                 const double* __restrict__ omega, const double* x, const double* b,
                 double* __restrict__ xout, double* r, int write_r) {
  csr_next<K>();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double d, w;
  if (K > 1) csr_own(diag, omega, damp, i, d, w);
  const double s = csr_row_sum<K>(a, i, x);
  if (K == 1) csr_own(diag, omega, damp, i, d, w);
  const double t = (b[i] - s) / d;
  if (write_r) r[i] = t;
  xout[i] = fma(w, t, x[i]);
}

// one colour of the SOR (SSC = false: r := the scaled correction, the
// <sor> of linit.lisp:288-323) or point-block SSC sweep (r := the residual,
// blockit.lisp:131-138) of an algebraic level: rows of the colour in any
// order (they couple to none of each other), the row sum over the stored
// entries, columns ascending
template <int K>
__global__ void __launch_bounds__(kCsrT<K>, K > 1 ? 8 : 0)
k_csr_sor(const int* __restrict__ rows, long long cnt, CsrView a, const double* __restrict__ diag, double omega_s,
          const double* __restrict__ omega, double* x, const double* b, double* r, int ssc) {
  csr_next<K>();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const long long i = __ldg(rows + t);
  double d, w;
  if (K > 1) csr_own(diag, omega, omega_s, i, d, w);
  const double s = csr_row_sum<K>(a, i, x);
  if (K == 1) csr_own(diag, omega, omega_s, i, d, w);
  const double rr = b[i] - s;
  const double tt = rr / d;
  r[i] = ssc ? rr : tt;
  x[i] = fma(w, tt, x[i]);
}

// rc = I^T rf row by row of I^T (fine entries ascending); the coarse rhs
// takes rc, the coarse solution 0 (the :after methods of restrict)
template <int K>
__global__ void __launch_bounds__(kCsrT<K>, K > 1 ? 8 : 0)
k_csr_restrict(long long NC, CsrView pt, const double* rf, double* rc, double* rhsc, double* solc) {
  csr_next<K>();
  const long long J = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (J >= NC) return;
  const double s = csr_row_sum<K>(pt, J, rf);
  rc[J] = s;
  if (rhsc) rhsc[J] = s;
  if (solc) solc[J] = 0.0;
}

// xf += I xc (coarse entries ascending)
template <int K>
__global__ void __launch_bounds__(kCsrT<K>, K > 1 ? 8 : 0)
k_csr_prolong(long long NF, CsrView p, const double* xc, double* xf) {
  csr_next<K>();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NF || p.start[i] == p.start[i + 1]) {  // constrained rows keep their value
    pdl_wait();  // (were all rows empty, the launch would otherwise end before its predecessor)
    return;
  }
  const double s = csr_row_sum<K>(p, i, xc);
  xf[i] = xf[i] + s;
}

// the level matrix as a dense row-major n x n array (zeros written beforehand)
__global__ void __launch_bounds__(kBlock) k_csr_densify(long long N, CsrView a, double* Dm) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (long long e = a.start[i]; e < a.start[i + 1]; ++e) Dm[i * N + a.index[e]] = a.value[e];
}

// -------------------------------------------------------------- transfers
template <int P>
__device__ __forceinline__ int restrict_1d(long long J, long long* off, double* w) {
  if (P == 1) { off[0] = -1; off[1] = 0; off[2] = 1; w[0] = 0.5; w[1] = 1.0; w[2] = 0.5; return 3; }
  if ((J & 1) == 0) {
    off[0] = -3; off[1] = -1; off[2] = 0; off[3] = 1; off[4] = 3;
    w[0] = -0.125; w[1] = 0.375; w[2] = 1.0; w[3] = 0.375; w[4] = -0.125;
    return 5;
  }
  off[0] = -1; off[1] = 0; off[2] = 1; w[0] = 0.75; w[1] = 1.0; w[2] = 0.75;
  return 3;
}

template <int P>
__device__ __forceinline__ int prolong_1d(long long I, long long* J, double* w) {
  if ((I & 1) == 0) { J[0] = I / 2; w[0] = 1.0; return 1; }
  if (P == 1) { J[0] = (I - 1) / 2; J[1] = (I + 1) / 2; w[0] = 0.5; w[1] = 0.5; return 2; }
  const long long c = I / 4;
  const double s = (double)(I - 4 * c) / 4.0;
  J[0] = 2 * c; J[1] = 2 * c + 1; J[2] = 2 * c + 2;
  w[0] = 2.0 * (s - 0.5) * (s - 1.0);
  w[1] = 4.0 * s * (1.0 - s);
  w[2] = 2.0 * s * (s - 0.5);
  return 3;
}

// Launch shape of the transfer kernels: blocks (32, 8) over x and y, one z
// plane per blockIdx.z, 32-bit node coordinates (levels have < 2^31 nodes).
__device__ __forceinline__ bool face_dir(int c, int M, int k, int dmask) {
  return (c == 0 && ((dmask >> (2 * k)) & 1)) || (c == M - 1 && ((dmask >> (2 * k + 1)) & 1));
}

// rc_J = I^T rf at coarse node cJ (constrained).  A z plane's loads (up to 25)
// are issued before its multiply-adds, which run in z, y, x order; positions
// outside the level and Dirichlet nodes are skipped.  (3D Q1, 129^3 coarse
// nodes: 64 us, 138 us with each load waiting for the previous term; one
// memory wait per plane on small levels, 12.4 -> 6 us at 33^3.)
// NC: components per node; rf points at the component summed (global or, in
// k_tail, shared memory).
template <int D, int P, int NC = 1, typename T = double>
__device__ __forceinline__ T restrict_node(const int cJ[3], int MC, int MF, int dmask, const T* rf) {
#pragma unroll
  for (int k = 0; k < D; ++k)
    if (face_dir(cJ[k], MC, k, dmask)) return T(0);
  constexpr int R = P == 1 ? 3 : 5;
  // per direction: fine coordinate and weight of each position, and whether it is met
  int f[3][R];
  double w[3][R];
  bool on[3][R];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k >= D) continue;
    long long off[5] = {0, 0, 0, 0, 0};
    double wk[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    const int cnt = restrict_1d<P>(cJ[k], off, wk);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      f[k][q] = 2 * cJ[k] + (int)off[q];
      w[k][q] = wk[q];
      on[k][q] = q < cnt && f[k][q] >= 0 && f[k][q] < MF && !face_dir(f[k][q], MF, k, dmask);
    }
  }
  T acc = T(0);
#pragma unroll
  for (int z = 0; z < (D > 2 ? R : 1); ++z) {
    T v[R * R];
#pragma unroll
    for (int y = 0; y < (D > 1 ? R : 1); ++y)
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (on[0][q] && (D < 2 || on[1][y]) && (D < 3 || on[2][z]))
          v[y * R + q] = rf[NC * (f[0][q] + (long long)MF * ((D > 1 ? f[1][y] : 0) +
                                                             (long long)MF * (D > 2 ? f[2][z] : 0)))];
#pragma unroll
    for (int y = 0; y < (D > 1 ? R : 1); ++y)
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (on[0][q] && (D < 2 || on[1][y]) && (D < 3 || on[2][z])) {
          double ww = w[0][q];
          if (D > 1) ww = ww * w[1][y];
          if (D > 2) ww = ww * w[2][z];
          acc = fma((T)ww, v[y * R + q], acc);
        }
  }
  return acc;
}

// (I xc) at fine node fi, not a Dirichlet node (constrained); all loads first
// (3D Q1, 257^3 fine nodes: 197 us, 469 us with a load per term)
template <int D, int P, int NC = 1, typename T = double>
__device__ __forceinline__ T prolong_node(const int fi[3], int MF, int MC, int dmask, const T* xc) {
  constexpr int R = P == 1 ? 2 : 3;
  int j[3][R];
  double w[3][R];
  bool on[3][R];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k >= D) continue;
    long long J[3] = {0, 0, 0};
    double wk[3] = {0.0, 0.0, 0.0};
    const int cnt = prolong_1d<P>(fi[k], J, wk);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      j[k][q] = (int)J[q];
      w[k][q] = wk[q];
      on[k][q] = q < cnt && !face_dir(j[k][q], MC, k, dmask);
    }
  }
  constexpr int NY = D > 1 ? R : 1, NZ = D > 2 ? R : 1;
  T v[NZ * NY * R];
#pragma unroll
  for (int z = 0; z < NZ; ++z)
#pragma unroll
    for (int y = 0; y < NY; ++y)
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (on[0][q] && (D < 2 || on[1][y]) && (D < 3 || on[2][z]))
          v[(z * NY + y) * R + q] = xc[NC * (j[0][q] + (long long)MC * ((D > 1 ? j[1][y] : 0) +
                                                                        (long long)MC * (D > 2 ? j[2][z] : 0)))];
  T acc = T(0);
#pragma unroll
  for (int z = 0; z < NZ; ++z)
#pragma unroll
    for (int y = 0; y < NY; ++y)
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (on[0][q] && (D < 2 || on[1][y]) && (D < 3 || on[2][z])) {
          double ww = w[0][q];
          if (D > 1) ww = ww * w[1][y];
          if (D > 2) ww = ww * w[2][z];
          acc = fma((T)ww, v[(z * NY + y) * R + q], acc);
        }
  return acc;
}

// rc := I^T rf (constrained), rhs_c := rc, sol_c := 0 (restrict + its :after
// methods for the correction scheme, multigrid.lisp:202-224)
template <int D, int P>
__global__ void __launch_bounds__(kBlock)
k_restrict(int MC, int MF, int dmask, const double* rf, double* __restrict__ rc,
           double* __restrict__ rhsc, double* __restrict__ solc, long long fs, long long cs) {
  if (D == 1) pdl_next_light();  // 32 of 256 threads have work there
  else pdl_next();
  pdl_wait();
  if (D == 1 && threadIdx.y != 0) return;
  if (D < 3) {  // problem of a batched level: fine stride fs, coarse stride cs
    const long long bq = blockIdx.z;
    rf += bq * fs;
    rc += bq * cs;
    rhsc += bq * cs;
    solc += bq * cs;
  }
  const int cJ[3] = {(int)(blockIdx.x * 32 + threadIdx.x), D > 1 ? (int)(blockIdx.y * 8 + threadIdx.y) : 0,
                     D > 2 ? (int)blockIdx.z : 0};
  if (cJ[0] >= MC || cJ[1] >= MC) return;
  const long long J = cJ[0] + (long long)MC * (cJ[1] + (long long)MC * cJ[2]);
  const double acc = restrict_node<D, P>(cJ, MC, MF, dmask, rf);
  rc[J] = acc;
  rhsc[J] = acc;
  solc[J] = 0.0;
}

// xf := xf + I xc (see k_prolong) on Q1 levels, a thread per pair of fine nodes
// 2 j, 2 j + 1 along x: the pair shares its coarse values, every thread of a warp
// takes the same terms (y and z are the warp's), and the loads and stores are
// coalesced.  Terms and their order are prolong_node's.  Bound by HBM and the issue of its loads
// (257^3 fine nodes: 99 us, 197 us with a thread per fine node).
template <int D>
__global__ void __launch_bounds__(kBlock)
k_prolong_q1f(int MF, int MC, int dmask, const double* xc, double* __restrict__ xf, long long fs,
              long long cs) {
  if (D == 1) pdl_next_light();  // 32 of 256 threads have work there
  else pdl_next();
  pdl_wait();
  if (D == 1 && threadIdx.y != 0) return;
  if (D < 3) {  // problem of a batched level
    const long long bq = blockIdx.z;
    xc += bq * cs;
    xf += bq * fs;
  }
  const int j = blockIdx.x * 32 + threadIdx.x;
  const int fy = D > 1 ? (int)(blockIdx.y * 8 + threadIdx.y) : 0, fz = D > 2 ? (int)blockIdx.z : 0;
  if (j >= MC || fy >= MF) return;
  if (D > 1 && face_dir(fy, MF, 1, dmask)) return;
  if (D > 2 && face_dir(fz, MF, 2, dmask)) return;
  const int ny = D > 1 && (fy & 1) ? 2 : 1, nz = D > 2 && (fz & 1) ? 2 : 1;
  const bool x0 = !face_dir(j, MC, 0, dmask), x1 = j + 1 < MC && !face_dir(j + 1, MC, 0, dmask);
  constexpr int NY = D > 1 ? 2 : 1, NZ = D > 2 ? 2 : 1;
  bool on[NZ][NY];
  double v[NZ][NY][2];
#pragma unroll
  for (int z = 0; z < NZ; ++z)
#pragma unroll
    for (int y = 0; y < NY; ++y) {
      const int cy = (fy >> 1) + y, cz = (fz >> 1) + z;
      on[z][y] = y < ny && z < nz && (D < 2 || !face_dir(cy, MC, 1, dmask)) && (D < 3 || !face_dir(cz, MC, 2, dmask));
      const double* c = xc + j + (long long)MC * (cy + (long long)MC * cz);
      v[z][y][0] = on[z][y] && x0 ? c[0] : 0.0;
      v[z][y][1] = on[z][y] && x1 ? c[1] : 0.0;
    }
  double* f = xf + 2 * j + (long long)MF * (fy + (long long)MF * fz);
  const bool w0 = !face_dir(2 * j, MF, 0, dmask), w1 = j + 1 < MC;  // an odd node lies on no face
  const double f0 = w0 ? f[0] : 0.0, f1 = w1 ? f[1] : 0.0;
  double e = 0.0, o = 0.0;
#pragma unroll
  for (int z = 0; z < NZ; ++z)
#pragma unroll
    for (int y = 0; y < NY; ++y)
      if (on[z][y]) {
        const double w = (ny == 2 ? 0.5 : 1.0) * (nz == 2 ? 0.5 : 1.0);
        if (x0) {
          e = fma(w, v[z][y][0], e);
          o = fma(0.5 * w, v[z][y][0], o);
        }
        if (x1) o = fma(0.5 * w, v[z][y][1], o);
      }
  if (w0) f[0] = f0 + e;
  if (w1) f[1] = f1 + o;
}

// xf := xf + I xc (constrained) (prolongate, multigrid.lisp:237-239)
template <int D, int P>
__global__ void __launch_bounds__(kBlock)
k_prolong(int MF, int MC, int dmask, const double* xc, double* __restrict__ xf, long long fs,
          long long cs) {
  if (D == 1) pdl_next_light();  // 32 of 256 threads have work there
  else pdl_next();
  pdl_wait();
  if (D == 1 && threadIdx.y != 0) return;
  if (D < 3) {  // problem of a batched level
    const long long bq = blockIdx.z;
    xc += bq * cs;
    xf += bq * fs;
  }
  const int fi[3] = {(int)(blockIdx.x * 32 + threadIdx.x), D > 1 ? (int)(blockIdx.y * 8 + threadIdx.y) : 0,
                     D > 2 ? (int)blockIdx.z : 0};
  if (fi[0] >= MF || fi[1] >= MF) return;
#pragma unroll
  for (int k = 0; k < D; ++k)
    if (face_dir(fi[k], MF, k, dmask)) return;
  const long long i = fi[0] + (long long)MF * (fi[1] + (long long)MF * fi[2]);
  const double xi = xf[i];
  xf[i] = xi + prolong_node<D, P>(fi, MF, MC, dmask, xc);
}

// -------------------------------------------------------------- coarse LU
// The dense LU with partial pivoting of the base level and its explicit
// inverse (the <lu> coarse-grid iteration; the oracle's dense LU).  Every
// form below performs, for every element, the operations of the unblocked
// right-looking loop in the same order -- pivot: the first row holding the
// largest magnitude among the rows not yet eliminated; multiplier: column
// entry / pivot; update: a_ij = fma(-l_ik, a_kj, a_ij) for k ascending;
// inverse: the interchanges, then per column the unit-lower forward and the
// upper backward substitution (x_k = b_k / u_kk, then b_i = fma(-u_ik, x_k,
// b_i) for the rows above) -- so factors, pivots and inverse are the same bit
// for bit whichever form runs.
//
// Blocked form for matrices beyond shared memory: panels of kLuB columns,
// rows interchanged through a logical permutation (physical rows stay put).
constexpr int kLuB = 32;

// the panel k0..k1-1: per column the pivot (the first logical row holding the
// largest magnitude), the interchange, and the updates of the panel's later
// columns; the multipliers (column / pivot) are stored one step later, and
// the panel's last column's after the loop
__global__ void __launch_bounds__(1024) k_lu_panel(double* A, int n, int k0, int k1, int* piv, int* perm) {
  __shared__ double bv[32];
  __shared__ int bi[32];
  const int tid = threadIdx.x, nt = blockDim.x;
  double dprev = 1.0;
  for (int k = k0; k < k1; ++k) {
    double best = -1.0;
    int besti = n;
    for (int i = k + tid; i < n; i += nt) {
      const double v = fabs(A[(long long)perm[i] * n + k]);
      if (v > best || (v == best && i < besti)) { best = v; besti = i; }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
      if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
    }
    if ((tid & 31) == 0) { bv[tid >> 5] = best; bi[tid >> 5] = besti; }
    __syncthreads();
    if (tid == 0) {
      double b = bv[0];
      int ib = bi[0];
      for (int w = 1; w < (nt + 31) / 32; ++w)
        if (bv[w] > b || (bv[w] == b && bi[w] < ib)) { b = bv[w]; ib = bi[w]; }
      piv[k] = ib;
      const int t = perm[k];
      perm[k] = perm[ib];
      perm[ib] = t;
    }
    __syncthreads();
    const long long pr = perm[k];
    const double d = A[pr * n + k];
    const int m = n - k - 1, w = k1 - k - 1;
    const long long mw = (long long)m * w, nprev = k > k0 ? n - k : 0;  // previous column: logical rows k ..
    for (long long idx = tid; idx < mw + nprev; idx += nt) {
      if (idx < mw) {
        const int i = k + 1 + (int)(idx / w), j = k + 1 + (int)(idx % w);
        const long long ri = perm[i];
        const double l = A[ri * n + k] / d;
        A[ri * n + j] = fma(-l, A[pr * n + j], A[ri * n + j]);
      } else {
        const long long ri = perm[k + (int)(idx - mw)];
        A[ri * n + k - 1] = A[ri * n + k - 1] / dprev;
      }
    }
    dprev = d;
    __syncthreads();
  }
  for (int i = k1 + tid; i < n; i += nt) {  // the panel's last column, logical rows k1 ..
    const long long ri = perm[i];
    A[ri * n + k1 - 1] = A[ri * n + k1 - 1] / dprev;
  }
}

// the panel's rows right of the panel: column j (one thread) takes the
// panel's elimination steps in order
__global__ void k_lu_urows(double* A, int n, int k0, int k1, const int* __restrict__ perm) {
  const int j = k1 + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  for (int k = k0; k < k1; ++k) {
    const double ukj = A[(long long)perm[k] * n + j];
    for (int i = k + 1; i < k1; ++i) {
      const long long ri = perm[i];
      A[ri * n + j] = fma(-A[ri * n + k], ukj, A[ri * n + j]);
    }
  }
}

// the trailing rows and columns: each element takes the panel's steps in order
__global__ void __launch_bounds__(256) k_lu_trail(double* A, int n, int k0, int k1, const int* __restrict__ perm) {
  const int j = k1 + blockIdx.x * 32 + threadIdx.x;
  const int i = k1 + blockIdx.y * 8 + threadIdx.y;
  if (i >= n || j >= n) return;
  const long long ri = perm[i];
  double a = A[ri * n + j];
  for (int k = k0; k < k1; ++k) a = fma(-A[ri * n + k], A[(long long)perm[k] * n + j], a);
  A[ri * n + j] = a;
}

__global__ void k_lu_permute(const double* __restrict__ A, int n, const int* __restrict__ perm, double* X) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n * n) return;
  const long long i = t / n, j = t % n;
  X[t] = A[(long long)perm[i] * n + j];
}

__global__ void k_iota(int* p, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = i;
}

// The inverse with one CTA per column of X reading the factors transposed
// (LT[k][i] = LU[i][k], coalesced over the rows)
__global__ void __launch_bounds__(256) k_lu_inverse_colT(const double* __restrict__ LT, const int* __restrict__ piv,
                                                         int n, double* X) {
  extern __shared__ double S[];
  double* xv = S;
  double* out = S + n;
  const int tid = threadIdx.x, nt = blockDim.x, j = blockIdx.x;
  for (int i = tid; i < n; i += nt) xv[i] = (i == j) ? 1.0 : 0.0;
  __syncthreads();
  if (tid == 0)
    for (int k = 0; k < n; ++k) {
      const int p = piv[k];
      if (p != k) { const double t = xv[k]; xv[k] = xv[p]; xv[p] = t; }
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const double bk = xv[k];
    const double* col = LT + (long long)k * n;
    for (int i = k + 1 + tid; i < n; i += nt) xv[i] = fma(-col[i], bk, xv[i]);
    __syncthreads();
  }
  for (int k = n - 1; k >= 0; --k) {
    const double* col = LT + (long long)k * n;
    const double bk = xv[k] / col[k];
    if (tid == 0) out[k] = bk;
    for (int i = tid; i < k; i += nt) xv[i] = fma(-col[i], bk, xv[i]);
    __syncthreads();
  }
  for (int i = tid; i < n; i += nt) X[(long long)i * n + j] = out[i];
}



// The factorisation on a shared-memory copy of A (n x n doubles fit in one
// CTA), two block barriers per column: warp 0 finds the pivot and
// interchanges logical rows through a permutation; every thread then updates
// the trailing submatrix, forming the multiplier it needs as the quotient the
// column will hold, and scales the previous column (which no later step reads
// before that).
__global__ void __launch_bounds__(1024) k_lu_factor_smem2(double* A, int n, int* piv) {
  extern __shared__ double S[];
  int* perm = reinterpret_cast<int*>(S + (size_t)n * n);
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  for (int idx = tid; idx < n * n; idx += nt) S[idx] = A[idx];
  for (int i = tid; i < n; i += nt) perm[i] = i;
  __syncthreads();
  double dprev = 1.0;
  for (int k = 0; k < n; ++k) {
    if (tid < 32) {
      double best = -1.0;
      int besti = n;
      for (int i = k + lane; i < n; i += 32) {
        const double v = fabs(S[perm[i] * n + k]);
        if (v > best || (v == best && i < besti)) { best = v; besti = i; }
      }
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
        if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
      }
      if (lane == 0) {
        piv[k] = besti;
        const int t = perm[k];
        perm[k] = perm[besti];
        perm[besti] = t;
      }
    }
    __syncthreads();
    const int pr = perm[k];
    const double d = S[pr * n + k];
    const int m = n - k - 1;
    const int mm = m * m, nprev = k > 0 ? n - k : 0;  // previous column: logical rows k .. n-1
    for (int idx = tid; idx < mm + nprev; idx += nt) {
      if (idx < mm) {
        const int i = k + 1 + idx / m, j = k + 1 + idx % m;
        const int ri = perm[i];
        const double l = S[ri * n + k] / d;
        S[ri * n + j] = fma(-l, S[pr * n + j], S[ri * n + j]);
      } else {
        const int ri = perm[k + (idx - mm)];
        S[ri * n + k - 1] = S[ri * n + k - 1] / dprev;
      }
    }
    dprev = d;
    __syncthreads();
  }
  for (int idx = tid; idx < n * n; idx += nt) A[idx] = S[perm[idx / n] * n + idx % n];
}

// The inverse with the factors in shared memory and one CTA per column of X:
// the threads share the rows, a block barrier per elimination column.
__global__ void __launch_bounds__(256) k_lu_inverse_col(const double* __restrict__ LU, const int* __restrict__ piv,
                                                        int n, double* X) {
  extern __shared__ double S[];
  double* L = S;              // n x n
  double* xv = S + n * n;     // the column, forward
  double* out = xv + n;       // the column, backward
  const int tid = threadIdx.x, nt = blockDim.x, j = blockIdx.x;
  for (int idx = tid; idx < n * n; idx += nt) L[idx] = LU[idx];
  for (int i = tid; i < n; i += nt) xv[i] = (i == j) ? 1.0 : 0.0;
  __syncthreads();
  if (tid == 0)
    for (int k = 0; k < n; ++k) {
      const int p = piv[k];
      if (p != k) { const double t = xv[k]; xv[k] = xv[p]; xv[p] = t; }
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const double bk = xv[k];
    for (int i = k + 1 + tid; i < n; i += nt) xv[i] = fma(-L[i * n + k], bk, xv[i]);
    __syncthreads();
  }
  for (int k = n - 1; k >= 0; --k) {
    const double bk = xv[k] / L[k * n + k];
    if (tid == 0) out[k] = bk;
    for (int i = tid; i < k; i += nt) xv[i] = fma(-L[i * n + k], bk, xv[i]);
    __syncthreads();
  }
  for (int i = tid; i < n; i += nt) X[(long long)i * n + j] = out[i];
}



__global__ void k_transpose(const double* __restrict__ X, int n, double* __restrict__ XT) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n * n) return;
  const long long i = t / n, j = t % n;
  XT[j * n + i] = X[i * n + j];
}

// <lu> coarse-grid iterator: r := A^-1 r, x := x + damp r.  Each row's sum is
// one chain of fma in ascending j, 10 cycles a term, and the rows' chains run
// side by side, so that is the time if the coefficients are at hand: eight
// warps copy them into shared memory (cp.async), 64 terms of a CTA's rows at a
// time and one group ahead, and a warp per 32 rows does nothing but the sums.
// The rows are spread over a cluster, whose CTAs all read r before any of
// them writes it.  With one CTA and a thread per row that loaded its own
// coefficients 343 unknowns took 52 us (8 so), 1,029 took 125 us (21 so, near
// what eight warps can copy).  A cp.async whose lanes repeat an address is many
// times slower, so rows beyond n are left out and not clamped.
constexpr int kCsStep = 64, kCsLoad = 8;  // terms per group, loading warps

template <int R>  // warps of rows per CTA
__global__ void __launch_bounds__(32 * (R + kCsLoad), 1)
k_coarse_solve(const double* __restrict__ AinvT, int n, double damp, double* x, double* r, long long vs, int cs) {
  constexpr int W = 32 * R, PER = kCsStep / kCsLoad;  // rows, terms per loading warp
  extern __shared__ double csm[];
  double* ring = csm;                    // [2][term][row]
  double* rs = csm + 2 * kCsStep * W;    // the residual
  const long long bq = blockIdx.x / cs;  // a cluster per problem of a batched base level
  const int rank = (int)(blockIdx.x - bq * cs), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  x += bq * vs;
  r += bq * vs;
  const int row0 = rank * W, ngroup = (n + kCsStep - 1) / kCsStep;
  const double* src = AinvT + bq * n * n;
  // loading warp w copies terms w * PER .. of a group, every row of the CTA
  // (rows and terms beyond n are not read)
  auto request = [&](int g) {
    const int t0 = (warp - R) * PER, cnt = min(PER, n - (g * kCsStep + t0));
    double* d = ring + ((g & 1) * kCsStep + t0) * W + lane;
    const double* c = src + (long long)(g * kCsStep + t0) * n;
#pragma unroll
    for (int h = 0; h < R; ++h) {
      const double* ch = c + row0 + 32 * h + lane;
      if (row0 + 32 * h + lane < n) {
#pragma unroll
        for (int q = 0; q < PER; ++q, ch += n)
          if (q < cnt) cp_async8(d + q * W + 32 * h, ch);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_next();
  if (warp >= R) request(0);
  pdl_wait();
  for (int j = threadIdx.x; j < n; j += blockDim.x) rs[j] = r[j];
  if (cs > 1) cooperative_groups::this_cluster().sync();
  double acc = 0.0;
  for (int g = 0; g < ngroup; ++g) {
    if (warp >= R) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // group g is there, and the sums of group g - 1 are done
    if (warp >= R) {
      if (g + 1 < ngroup) request(g + 1);
    } else {
      const double* a = ring + (g & 1) * kCsStep * W + threadIdx.x;
      const double* v = rs + g * kCsStep;
      const int cnt = n - g * kCsStep;
      if (cnt >= kCsStep) {
#pragma unroll 1
        for (int q0 = 0; q0 < kCsStep; q0 += 16) {
          double t[16], u[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) { t[q] = a[(q0 + q) * W]; u[q] = v[q0 + q]; }
#pragma unroll
          for (int q = 0; q < 16; ++q) acc = fma(t[q], u[q], acc);
        }
      } else {
        for (int q = 0; q < cnt; ++q) acc = fma(a[q * W], v[q], acc);
      }
    }
  }
  const int i = row0 + (int)threadIdx.x;
  if (warp < R && i < n) {
    r[i] = acc;
    x[i] = fma(damp, acc, x[i]);
  }
}

// ------------------------------------------------------------ vector ops
__global__ void k_fill(double* x, long long n, double v) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = v;
}

__global__ void k_copy(const double* x, double* __restrict__ y, long long n) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = x[i];
}

// axpy!: y := y + alpha x (alpha from a device slot when aslot >= 0)
__global__ void k_axpy(double alpha, const double* sc, int aslot, const double* x,
                       double* y, long long n) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = aslot >= 0 ? sc[aslot] : alpha;
  y[i] = fma(a, x[i], y[i]);
}

// DR4096 dot product (x, y).  Q pairs of elements in flight a thread, MB blocks
// per SM: four and four while the blocks fit one wave so (one chunk 4.5 us, 4.8
// with two pairs and eight blocks), two and eight beyond, where the second wave
// would be nearly empty (669 chunks 7.8 us and 9.0 in the other form, 1,019 9.5
// and 11.0, 1,184 9.3 and 11.0; from 1,500 on alike).
constexpr unsigned kDotWave = 4 * 148;
template <int Q, int MB>
__global__ void __launch_bounds__(kBlock, MB)
k_dot(const double* x, const double* y, long long n, Reduce R, long long vs) {
  pdl_next();
  pdl_wait();
  __shared__ double smem[8];
  const long long bq = blockIdx.y;  // problem of a batched vector (stride vs)
  x += bq * vs;
  y += bq * vs;
  R = batch_reduce(R, (unsigned)bq);
  const long long base = (long long)blockIdx.x * kChunk + 2 * threadIdx.x;
  // pairs by 16-byte loads, Q at a time before their terms.  The library's
  // own vectors start on 16 bytes; those a caller hands to fmg_dot_noalloc
  // need only the 8 of a double, and then come one by one.
  const bool wide = (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
  double acc = 0.0;
#pragma unroll
  for (int m0 = 0; m0 < kPairsPerThread; m0 += Q) {
    double2 u[Q], v[Q];
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      const long long i0 = base + 512LL * (m0 + m);
      if (wide && i0 + 1 < n) {
        u[m] = *reinterpret_cast<const double2*>(x + i0);
        v[m] = *reinterpret_cast<const double2*>(y + i0);
      } else {
        if (i0 < n) {
          u[m].x = x[i0];
          v[m].x = y[i0];
        }
        if (i0 + 1 < n) {
          u[m].y = x[i0 + 1];
          v[m].y = y[i0 + 1];
        }
      }
    }
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      const long long i0 = base + 512LL * (m0 + m);
      if (i0 < n) acc = fma(u[m].x, v[m].x, acc);
      if (i0 + 1 < n) acc = fma(u[m].y, v[m].y, acc);
    }
  }
  dr_finish(acc, R, smem);
}

// CG update (krylow.lisp:117-121): x += lam p; r -= lam a; fused (r,r);
// then w := r and (optionally) w2 := r, q := 0 for the preconditioner call
__global__ void __launch_bounds__(kBlock, 3)
k_cg_update(const double* sc, double* __restrict__ x, const double* p, double* __restrict__ r, const double* a,
            double* __restrict__ w, double* __restrict__ w2, double* __restrict__ q, long long n, Reduce R, long long vs,
            const double* frozen) {
  pdl_next();
  pdl_wait();
  __shared__ double smem[8];
  const long long bq = blockIdx.y;  // problem of a batched vector (stride vs); frozen: it has converged
  sc += bq * S_COUNT;
  x += bq * vs;
  p += bq * vs;
  r += bq * vs;
  a += bq * vs;
  if (w) w += bq * vs;
  if (w2) w2 += bq * vs;
  if (q) q += bq * vs;
  R = batch_reduce(R, (unsigned)bq);
  const bool fz = frozen && frozen[bq] != 0.0;
  const double lam = sc[S_LAM], nlam = sc[S_NEGLAM];
  const long long base = (long long)blockIdx.x * kChunk + 2 * threadIdx.x;
  double acc = 0.0;
  // pairs by 16-byte accesses (every vector starts on 16 bytes), several in flight
#pragma unroll 4
  for (int m = 0; m < kPairsPerThread; ++m) {
    const long long i = base + 512LL * m;
    if (i + 1 < n) {
      const double2 ri = *reinterpret_cast<const double2*>(r + i);
      double2 rn = ri;
      if (!fz) {
        const double2 ai = *reinterpret_cast<const double2*>(a + i), pi = *reinterpret_cast<const double2*>(p + i),
                      xi = *reinterpret_cast<const double2*>(x + i);
        rn = make_double2(fma(nlam, ai.x, ri.x), fma(nlam, ai.y, ri.y));
        *reinterpret_cast<double2*>(x + i) = make_double2(fma(lam, pi.x, xi.x), fma(lam, pi.y, xi.y));
        *reinterpret_cast<double2*>(r + i) = rn;
      }
      acc = fma(rn.x, rn.x, acc);
      acc = fma(rn.y, rn.y, acc);
      if (w) *reinterpret_cast<double2*>(w + i) = rn;
      if (w2) *reinterpret_cast<double2*>(w2 + i) = rn;
      if (q) *reinterpret_cast<double2*>(q + i) = make_double2(0.0, 0.0);
    } else if (i < n) {
      const double rn = fz ? r[i] : fma(nlam, a[i], r[i]);
      if (!fz) {
        x[i] = fma(lam, p[i], x[i]);
        r[i] = rn;
      }
      acc = fma(rn, rn, acc);
      if (w) w[i] = rn;
      if (w2) w2[i] = rn;
      if (q) q[i] = 0.0;
    }
  }
  dr_finish(acc, R, smem);
}

// p := (new_alpha/alpha) p (scal!), then p := p + q (m+!)
__global__ void k_p_update(const double* sc, double* __restrict__ p, const double* q, long long n, long long vs,
                           const double* frozen) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long bq = blockIdx.y;  // problem of a batched vector; frozen problems keep p
  if (frozen && frozen[bq] != 0.0) return;
  sc += bq * S_COUNT;
  p += bq * vs;
  q += bq * vs;
  const double t = sc[S_RATIO] * p[i];
  p[i] = t + q[i];
}

// -------------------------------------------------------------- assembly
// Gauss-point samples of a cell-wise coefficient for a coarse level:
// kq[c * nq + q] = kcell[top cell containing the q-th Gauss point of c]
template <int D>
__global__ void k_sample_kq(long long ncells_l, long long n_l, long long n_top, double ratio, int np,
                            const double* __restrict__ xi, const double* __restrict__ kcell,
                            double* __restrict__ kq) {
  int nq = 1;
  for (int k = 0; k < D; ++k) nq *= np;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncells_l * nq) return;
  const long long c = t / nq;
  const int q = (int)(t % nq);
  const long long cc[3] = {c % n_l, D > 1 ? (c / n_l) % n_l : 0, D > 2 ? c / (n_l * n_l) : 0};
  const int qi[3] = {q % np, (q / np) % np, q / (np * np)};
  long long f[3] = {0, 0, 0};
  for (int k = 0; k < D; ++k) f[k] = (long long)floor(((double)cc[k] + xi[qi[k]]) * ratio);
  kq[t] = kcell[f[0] + n_top * (f[1] + n_top * f[2])];
}

// Stiffness entries by gather: for node i and slot s with neighbour j, the
// sum over the cells containing both nodes, in increasing cell index, of the
// local matrix entry (assemble-interior + global-local-matrix-operation,
// fedisc.lisp:73-206, sparseif.lisp:308-385).  Dirichlet rows become identity
// rows and Dirichlet columns are dropped (S A S + P).  On the top level the
// right-hand side is gathered the same way.
template <int D, int P>
__global__ void __launch_bounds__(kBlock)
k_assemble(AsmArgs g, const __grid_constant__ Q2Layout lay) {
  constexpr int NS = St<D, P>::NS;
  constexpr int C = St<D, P>::CENTER;
  constexpr int W = 2 * P + 1;
  constexpr int P1 = P + 1;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  long long ci[3];
  node_coords(i, g.M, D, ci);
  // the storage position of slot s of this node (-1: not stored, a structural zero)
  auto pos = [&](int s) -> long long {
    if (P != 2) return (long long)s * g.Np + i;
    const int r = q2_pattern<D>(s);
    for (int k = 0; k < D; ++k)
      if (((r >> k) & 1) && (ci[k] & 1)) return -1;
    return (long long)s * g.Np + q2c_pos<D>(lay, ci, g.M, r);
  };
  if (node_dirichlet(ci, g.M, D, g.dmask)) {
    for (int s = 0; s < NS; ++s) {
      const long long p = pos(s);
      if (p >= 0) g.A[p] = (s == C) ? 1.0 : 0.0;
    }
    if (g.rhs) g.rhs[i] = 0.0;
    return;
  }
  const int nl = g.nl, nq = g.nq;
  for (int s = 0; s < NS; ++s) {
    if (pos(s) < 0) continue;
    long long o[3] = {s % W - P, D > 1 ? (s / W) % W - P : 0, D > 2 ? (s / (W * W)) % W - P : 0};
    long long cj[3], lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    bool ok = true;
    for (int k = 0; k < 3; ++k) cj[k] = ci[k] + o[k];
    for (int k = 0; k < D; ++k) {
      if (cj[k] < 0 || cj[k] >= g.M) ok = false;
      const long long mx = ci[k] > cj[k] ? ci[k] : cj[k];
      const long long mn = ci[k] < cj[k] ? ci[k] : cj[k];
      lo[k] = mx >= P ? (mx - 1) / P : 0;
      hi[k] = mn / P;
      if (hi[k] > g.n - 1) hi[k] = g.n - 1;
    }
    double v = 0.0;
    if (ok && !node_dirichlet(cj, g.M, D, g.dmask)) {
      for (long long cz = lo[2]; cz <= hi[2]; ++cz)
        for (long long cy = lo[1]; cy <= hi[1]; ++cy)
          for (long long cx = lo[0]; cx <= hi[0]; ++cx) {
            const long long cc[3] = {cx, cy, cz};
            const long long cidx = cx + g.n * (cy + g.n * cz);
            int a = 0, b = 0, mul = 1;
            for (int k = 0; k < D; ++k) {
              a += (int)(ci[k] - P * cc[k]) * mul;
              b += (int)(cj[k] - P * cc[k]) * mul;
              mul *= P1;
            }
            double e;
            if (g.kq == nullptr) {
              const double kc = g.kcell ? g.kcell[cidx] : g.kconst;
              e = kc * g.Kbar[a * nl + b];
            } else {
              e = 0.0;
              for (int q = 0; q < nq; ++q)
                e = fma(g.kq[cidx * nq + q], g.Ctab[((long long)q * nl + a) * nl + b], e);
            }
            v = v + e;
          }
    }
    g.A[pos(s)] = v;
  }
  if (g.rhs) {
    long long lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    for (int k = 0; k < D; ++k) {
      lo[k] = ci[k] >= P ? (ci[k] - 1) / P : 0;
      hi[k] = ci[k] / P;
      if (hi[k] > g.n - 1) hi[k] = g.n - 1;
    }
    double acc = 0.0;
    for (long long cz = lo[2]; cz <= hi[2]; ++cz)
      for (long long cy = lo[1]; cy <= hi[1]; ++cy)
        for (long long cx = lo[0]; cx <= hi[0]; ++cx) {
          const long long cc[3] = {cx, cy, cz};
          const long long cidx = cx + g.n * (cy + g.n * cz);
          int a = 0, mul = 1;
          for (int k = 0; k < D; ++k) { a += (int)(ci[k] - P * cc[k]) * mul; mul *= P1; }
          double bl = 0.0;
          for (int q = 0; q < nq; ++q) {
            const double f = g.fip ? g.fip[cidx * nq + q] : g.fconst;
            bl = fma(f, g.Phi[q * nl + a], bl);
          }
          acc = acc + bl;
        }
    g.rhs[i] = acc;
  }
}

// k_assemble for 3D Q1 with the cell loops unrolled at compile time.  Node i
// is corner a = (1-bx) + 2 (1-by) + 4 (1-bz) of its adjacent cell ci - 1 + b
// (b = bx + 2 by + 4 bz), and neighbour j = i + o is corner a + ox + 2 oy +
// 4 oz of that cell when every 1 - b_k + o_k is 0 or 1.  The cells are walked
// in increasing b -- increasing cell index, the order k_assemble sums in --
// each adding its contribution to the 8 slots it touches, and every entry is
// formed with the same operations (e = k Kbar[a][b'], or e = sum_q fma(kq,
// Ctab, e); v = v + e), so the two kernels agree bit for bit.  The element
// tables travel as a kernel parameter (constant bank): operands of the FMAs
// without loads.  KQ: a coarse level's coefficient samples at the 8 Gauss
// points of each cell.
struct Q1Tab {
  double K[64];   // Kbar[a][b]
  double C[512];  // Ctab[q][a][b]
};

template <bool KQ>
__global__ void __launch_bounds__(kBlock)
k_assemble_q1_3d(AsmArgs g, const __grid_constant__ Q1Tab tab) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  const int M = (int)g.M, n = (int)g.n;
  const int ix = (int)(i % M), iy = (int)((i / M) % M), iz = (int)(i / ((long long)M * M));
  const long long ci[3] = {ix, iy, iz};
  if (node_dirichlet(ci, g.M, 3, g.dmask)) {
    if (g.A) {
#pragma unroll
      for (int s = 0; s < 27; ++s) g.A[(long long)s * g.Np + i] = (s == 13) ? 1.0 : 0.0;
    }
    if (g.rhs) g.rhs[i] = 0.0;
    return;
  }
  double v[27];
#pragma unroll
  for (int s = 0; s < 27; ++s) v[s] = 0.0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (!g.A) break;  // the right-hand side alone
    const int cx = ix - 1 + (b & 1), cy = iy - 1 + ((b >> 1) & 1), cz = iz - 1 + (b >> 2);
    if (cx < 0 || cx >= n || cy < 0 || cy >= n || cz < 0 || cz >= n) continue;
    const long long cidx = cx + (long long)n * (cy + (long long)n * cz);
    const int ax = 1 - (b & 1), ay = 1 - ((b >> 1) & 1), az = 1 - (b >> 2);
    const int a = ax + 2 * ay + 4 * az;
    double kq[KQ ? 8 : 1];
    if (KQ) {
#pragma unroll
      for (int q = 0; q < 8; ++q) kq[q] = __ldg(g.kq + cidx * 8 + q);
    } else {
      kq[0] = g.kcell ? __ldg(g.kcell + cidx) : g.kconst;
    }
#pragma unroll
    for (int bb = 0; bb < 8; ++bb) {  // neighbour corner: slot o = corner bb - corner a
      const int ox = (bb & 1) - ax, oy = ((bb >> 1) & 1) - ay, oz = (bb >> 2) - az;
      const int s = (ox + 1) + 3 * (oy + 1) + 9 * (oz + 1);
      double e;
      if (KQ) {
        e = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) e = fma(kq[q], tab.C[(q * 8 + a) * 8 + bb], e);
      } else {
        e = kq[0] * tab.K[a * 8 + bb];
      }
      v[s] = v[s] + e;
    }
  }
  if (g.A) {
#pragma unroll
    for (int s = 0; s < 27; ++s) {
      const int ox = s % 3 - 1, oy = (s / 3) % 3 - 1, oz = s / 9 - 1;
      const long long cj[3] = {ix + ox, iy + oy, iz + oz};
      const bool ok = cj[0] >= 0 && cj[0] < g.M && cj[1] >= 0 && cj[1] < g.M && cj[2] >= 0 && cj[2] < g.M &&
                      !node_dirichlet(cj, g.M, 3, g.dmask);
      g.A[(long long)s * g.Np + i] = ok ? v[s] : 0.0;
    }
  }
  if (g.rhs) {
    double acc = 0.0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int cx = ix - 1 + (b & 1), cy = iy - 1 + ((b >> 1) & 1), cz = iz - 1 + (b >> 2);
      if (cx < 0 || cx >= n || cy < 0 || cy >= n || cz < 0 || cz >= n) continue;
      const long long cidx = cx + (long long)n * (cy + (long long)n * cz);
      const int a = (1 - (b & 1)) + 2 * (1 - ((b >> 1) & 1)) + 4 * (1 - (b >> 2));
      double bl = 0.0;
      for (int q = 0; q < g.nq; ++q) {
        const double f = g.fip ? g.fip[cidx * g.nq + q] : g.fconst;
        bl = fma(f, g.Phi[q * g.nl + a], bl);
      }
      acc = acc + bl;
    }
    g.rhs[i] = acc;
  }
}

// ====================================================== vector form (nc = 3)
// Elasticity with 3 x 3 nodal blocks: vectors [node][3], level matrices
// [slot][k][l][Np] (block row component k, column component l).  Every
// kernel follows the scalar one with the component loops innermost, in the
// order the oracle uses.

// t := B^-1 r for one diagonal block: LU with partial pivoting (the first
// largest |entry| of the column, LAPACK dgetrf semantics) and substitution
// -- the gesv! of <jacobi> on a 3 x 3 block (linit.lisp:234)
template <typename T>
__device__ __forceinline__ void block_solve3(const T* B, const T* r, T* t) {
  T M[3][3], b[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b[k] = r[k];
#pragma unroll
    for (int m = 0; m < 3; ++m) M[k][m] = B[k * 3 + m];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    int pr = c;
    T mx = fabs(M[c][c]);
#pragma unroll
    for (int rr = c + 1; rr < 3; ++rr)
      if (fabs(M[rr][c]) > mx) { mx = fabs(M[rr][c]); pr = rr; }
    if (pr != c) {
#pragma unroll
      for (int rr = c + 1; rr < 3; ++rr)
        if (rr == pr) {
#pragma unroll
          for (int m = 0; m < 3; ++m) { const T tt = M[c][m]; M[c][m] = M[rr][m]; M[rr][m] = tt; }
          const T tb = b[c]; b[c] = b[rr]; b[rr] = tb;
        }
    }
#pragma unroll
    for (int rr = c + 1; rr < 3; ++rr) {
      const T f = M[rr][c] / M[c][c];
#pragma unroll
      for (int m = c + 1; m < 3; ++m) M[rr][m] = fma(-f, M[c][m], M[rr][m]);
      b[rr] = fma(-f, b[c], b[rr]);
    }
  }
#pragma unroll
  for (int c = 2; c >= 0; --c) {
    T sacc = b[c];
#pragma unroll
    for (int m = c + 1; m < 3; ++m) sacc = fma(-M[c][m], t[m], sacc);
    t[c] = sacc / M[c][c];
  }
}

// The block rows of 64 consecutive nodes, a thread per scalar row (node i,
// component k): sum over the slots ascending, columns ascending, of
// A(i, s)[k][m] x(i + off_s)[m].  OP: y = A x, r = b - A x (b may alias r), or
// compute-residual fused with the following block <jacobi> step: r_i = b_i -
// (A x)_i, t = B^-1 r_i, y_i = x_i + w t, r_i := t.
// The stencil's (y, z) slot rows run in a loop (unrolled, the code took longer
// to fetch than to run on small levels), a slot row's coefficients loaded one
// turn ahead.  The unknowns come from shared memory: the nodes a slot row
// meets are consecutive, so each of the (2 P + 1)^2 segments of 64 + 2 P nodes
// is read once, coalesced, before the loop (nodes outside the level as 0,
// where the stored coefficients are 0 too).  FP64 Q2 matvec: 49^3 nodes 191 ->
// 138 us, 25^3 58 -> 25 us, 13^3 41 -> 20 us against a thread per node with
// the slots unrolled.
// Nodes from which the FP32 form takes a thread per node.  A sweep by scalar
// rows and by nodes, us (all levels of the hierarchy, the top one by either):
// Q2 17^3 55 and 61 (the levels below by nodes too), 25^3 42 and 39, 33^3 98
// and 87, 49^3 160 and 120; Q1 21^3 16.4 and 16.4, 29^3 20.6 and 16.7, 41^3 39
// and 29.  At 97^3 nodes 814 and 443 us.  In FP64 the scalar rows are as fast
// there (921 us, 0.69 of the copy peak; a thread per node 1,128 us) and faster
// below.
constexpr long long kNode3Min = 12000;
enum Row3Op { ROW3_MUL, ROW3_RES, ROW3_JACOBI };
constexpr int kRow3Nodes = 64, kRow3T = 3 * kRow3Nodes;

template <int P, typename T, int OP>
__global__ void __launch_bounds__(kRow3T, sizeof(T) == 8 ? 3 : 4)
k_row3(const T* __restrict__ A, int N, long long Np, int M, double damp, const double* __restrict__ omega,
       const T* x, const T* b, T* y, T* r, int write_r) {
  pdl_next();
  constexpr int W = 2 * P + 1, Q = W * W, SEG = 3 * (kRow3Nodes + 2 * P);
  extern __shared__ unsigned char row3_sm[];
  T* xs = reinterpret_cast<T*>(row3_sm);  // [slot row][node - i0 + P][component]
  const int node = threadIdx.x % kRow3Nodes, k = threadIdx.x / kRow3Nodes;
  const int i0 = blockIdx.x * kRow3Nodes, i = min(i0 + node, N - 1);
  const bool live = i0 + node < N;
  // the node's place in the slot arrays of every pattern (Q2: sliced storage)
  const int H = (M + 1) / 2;
  const unsigned q0 = (unsigned)i / (unsigned)M;
  const int c0 = i - (int)q0 * M, c1 = (int)(q0 % (unsigned)M), c2 = (int)(q0 / (unsigned)M);
  const bool ex = P == 1 || !(c0 & 1), ey = !(c1 & 1), ez = !(c2 & 1);
  const T* Ak = A + (long long)(3 * k) * Np;
  T cur[W][3], nxt[W][3];
  auto load = [&](int q, T (&v)[W][3]) {  // slot row q's coefficients, 0 where not stored
    const int sy = q % W, sz = q / W;
    const bool ry = P == 2 && (sy == 0 || sy == 4), rz = P == 2 && (sz == 0 || sz == 4);
    const bool on = q < Q && !(ry && !ey) && !(rz && !ez);
    int p0 = i, p1 = i;
    if (P == 2) {
      const int yz = (ry ? c1 >> 1 : c1) + (ry ? H : M) * (rz ? c2 >> 1 : c2);
      p0 = c0 + M * yz;
      p1 = (c0 >> 1) + H * yz;
    }
    const T* a = Ak + (long long)(9 * W * q) * Np;
#pragma unroll
    for (int sx = 0; sx < W; ++sx) {
      const bool rx = P == 2 && (sx == 0 || sx == 4);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        v[sx][m] = T(0);
        if (on && (!rx || ex)) v[sx][m] = __ldg(a + (long long)(9 * sx + m) * Np + (rx ? p1 : p0));
      }
    }
  };
  load(0, cur);
  pdl_wait();
  // the unknowns, nine loads at a time
  constexpr int PER = (Q * SEG + kRow3T - 1) / kRow3T, BATCH = 9;
#pragma unroll 1
  for (int f0 = 0; f0 < PER; f0 += BATCH) {
    T v[BATCH];
#pragma unroll
    for (int t = 0; t < BATCH; ++t) {
      const int f = (f0 + t) * kRow3T + threadIdx.x, q = f / SEG, e = f - q * SEG;
      const long long g = 3LL * (i0 + (q % W - P) * M + (q / W - P) * M * M - P) + e;
      v[t] = f < Q * SEG && g >= 0 && g < 3LL * N ? x[g] : T(0);
    }
#pragma unroll
    for (int t = 0; t < BATCH; ++t) {
      const int f = (f0 + t) * kRow3T + threadIdx.x;
      if (f < Q * SEG) xs[f] = v[t];
    }
  }
  const T bi = OP == ROW3_MUL ? T(0) : b[3LL * i + k];
  __syncthreads();
  T s = T(0), dk[3] = {T(0), T(0), T(0)};
#pragma unroll 1
  for (int q = 0; q < Q; ++q) {
    load(q + 1, nxt);
    const int sy = q % W, sz = q / W;
    const bool on = P == 1 || (!((sy == 0 || sy == 4) && !ey) && !((sz == 0 || sz == 4) && !ez));
    const T* xp = xs + q * SEG + 3 * node;
    if (on) {
#pragma unroll
      for (int sx = 0; sx < W; ++sx) {
        if (P == 2 && (sx == 0 || sx == 4) && !ex) continue;
#pragma unroll
        for (int m = 0; m < 3; ++m) s = fma(cur[sx][m], xp[3 * sx + m], s);
      }
    }
    if (OP == ROW3_JACOBI && q == Q / 2) {
#pragma unroll
      for (int m = 0; m < 3; ++m) dk[m] = cur[P][m];
    }
#pragma unroll
    for (int sx = 0; sx < W; ++sx)
#pragma unroll
      for (int m = 0; m < 3; ++m) cur[sx][m] = nxt[sx][m];
  }
  const T res = bi - s;
  if (OP != ROW3_JACOBI) {
    if (live) y[3LL * i + k] = OP == ROW3_RES ? res : s;
    return;
  }
  // the node's residual and diagonal block meet in shared memory
  T* ds = xs + Q * SEG + node;  // [entry][node]: 3 residuals, 9 block entries
  ds[k * kRow3Nodes] = res;
#pragma unroll
  for (int m = 0; m < 3; ++m) ds[(3 + 3 * k + m) * kRow3Nodes] = dk[m];
  __syncthreads();
  if (k != 0 || !live) return;
  T rr[3], B[9], t[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) rr[e] = ds[e * kRow3Nodes];
#pragma unroll
  for (int e = 0; e < 9; ++e) B[e] = ds[(3 + e) * kRow3Nodes];
  block_solve3<T>(B, rr, t);
  const T w = omega ? (T)omega[i] : (T)damp;
  const T* xi = xs + (Q / 2) * SEG + 3 * (node + P);
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (write_r) r[3LL * i + e] = t[e];
    y[3LL * i + e] = fma(w, t[e], xi[e]);
  }
}

// The same with a thread per node, for large FP32 levels: the loop's loads are
// then uniform bases plus one 32-bit offset (k is known to the compiler), where
// the scalar-row form spends most of its issue slots on addresses.  Bound by
// the memory waits of its 25 slot rows (16 warps an SM, 45 loads each in
// flight: 4.6 TB/s at 97^3 nodes); requesting a slot row ahead halves the
// warps and measured slower.
template <int P, typename T, int OP>
__global__ void __launch_bounds__(kRow3Nodes, 8)
k_node3(const T* __restrict__ A, int N, long long Np, int M, double damp, const double* __restrict__ omega,
        const T* x, const T* b, T* y, T* r, int write_r) {
  pdl_next();
  pdl_wait();
  constexpr int W = 2 * P + 1, Q = W * W, SEG = 3 * (kRow3Nodes + 2 * P);
  extern __shared__ unsigned char row3_sm[];
  T* xs = reinterpret_cast<T*>(row3_sm);  // [slot row][node - i0 + P][component]
  const int i0 = blockIdx.x * kRow3Nodes, i = min(i0 + (int)threadIdx.x, N - 1);
  const bool live = i0 + (int)threadIdx.x < N;
  const int H = (M + 1) / 2;
  const unsigned q0 = (unsigned)i / (unsigned)M;
  const int c0 = i - (int)q0 * M, c1 = (int)(q0 % (unsigned)M), c2 = (int)(q0 / (unsigned)M);
  const bool ex = P == 1 || !(c0 & 1), ey = !(c1 & 1), ez = !(c2 & 1);
  constexpr int PER = (Q * SEG + kRow3Nodes - 1) / kRow3Nodes, BATCH = 16;
#pragma unroll 1
  for (int f0 = 0; f0 < PER; f0 += BATCH) {
    T v[BATCH];
#pragma unroll
    for (int t = 0; t < BATCH; ++t) {
      const int f = (f0 + t) * kRow3Nodes + threadIdx.x, q = f / SEG, e = f - q * SEG;
      const long long g = 3LL * (i0 + (q % W - P) * M + (q / W - P) * M * M - P) + e;
      v[t] = f < Q * SEG && g >= 0 && g < 3LL * N ? x[g] : T(0);
    }
#pragma unroll
    for (int t = 0; t < BATCH; ++t) {
      const int f = (f0 + t) * kRow3Nodes + threadIdx.x;
      if (f < Q * SEG) xs[f] = v[t];
    }
  }
  T bi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) bi[k] = OP == ROW3_MUL ? T(0) : b[3LL * i + k];
  __syncthreads();
  T s[3] = {T(0), T(0), T(0)}, B[9];
#pragma unroll 1
  for (int sz = 0; sz < W; ++sz) {
    const bool rz = P == 2 && (sz == 0 || sz == 4);
    if (rz && !ez) continue;
#pragma unroll 1
    for (int sy = 0; sy < W; ++sy) {
      const bool ry = P == 2 && (sy == 0 || sy == 4);
      if (ry && !ey) continue;
      const int q = sy + W * sz;
      unsigned p0 = (unsigned)i, p1 = (unsigned)i;
      if (P == 2) {
        const int yz = (ry ? c1 >> 1 : c1) + (ry ? H : M) * (rz ? c2 >> 1 : c2);
        p0 = (unsigned)(c0 + M * yz);
        p1 = (unsigned)((c0 >> 1) + H * yz);
      }
      const T* a = A + (long long)(9 * W * q) * Np;
      T v[W][9];
#pragma unroll
      for (int sx = 0; sx < W; ++sx) {
        const bool rx = P == 2 && (sx == 0 || sx == 4);
#pragma unroll
        for (int e = 0; e < 9; ++e)
          if (!rx || ex) v[sx][e] = __ldg(a + (long long)(9 * sx + e) * Np + (rx ? p1 : p0));
      }
      const T* xp = xs + q * SEG + 3 * threadIdx.x;
#pragma unroll
      for (int sx = 0; sx < W; ++sx) {
        if (P == 2 && (sx == 0 || sx == 4) && !ex) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int m = 0; m < 3; ++m) s[k] = fma(v[sx][3 * k + m], xp[3 * sx + m], s[k]);
      }
      if (OP == ROW3_JACOBI && q == Q / 2) {
#pragma unroll
        for (int e = 0; e < 9; ++e) B[e] = v[P][e];
      }
    }
  }
  if (!live) return;
  T rr[3], t[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) rr[k] = OP == ROW3_MUL ? s[k] : bi[k] - s[k];
  if (OP != ROW3_JACOBI) {
#pragma unroll
    for (int k = 0; k < 3; ++k) y[3LL * i + k] = rr[k];
    return;
  }
  block_solve3<T>(B, rr, t);
  const T w = omega ? (T)omega[i] : (T)damp;
  const T* xi = xs + (Q / 2) * SEG + 3 * (threadIdx.x + P);
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (write_r) r[3LL * i + e] = t[e];
    y[3LL * i + e] = fma(w, t[e], xi[e]);
  }
}

template <typename T, int OP>
static void launch_row3(int order, const T* A, long long N, long long Np, long long M, double damp,
                        const double* omega, const T* x, const T* b, T* y, T* r, bool write_r, cudaStream_t st) {
  auto go = [&](auto PT) {
    constexpr int P = decltype(PT)::value, W = 2 * P + 1;
    constexpr size_t smem = (W * W * 3 * (kRow3Nodes + 2 * P) + (OP == ROW3_JACOBI ? 12 * kRow3Nodes : 0)) * sizeof(T);
    const unsigned grid = (unsigned)((N + kRow3Nodes - 1) / kRow3Nodes);
    if constexpr (sizeof(T) == 4) {
      if (N >= kNode3Min) {
        launch_late(k_node3<P, T, OP>, grid, kRow3Nodes, smem, st, A, (int)N, Np, (int)M, damp, omega, x, b, y, r,
                                                          write_r ? 1 : 0);
        return;
      }
    }
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(k_row3<P, T, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_late(k_row3<P, T, OP>, grid, kRow3T, smem, st,
                A, (int)N, Np, (int)M, damp, omega, x, b, y, r, write_r ? 1 : 0);
  };
  if (order == 2) go(std::integral_constant<int, 2>{});
  else go(std::integral_constant<int, 1>{});
}

// <jacobi> on 3 x 3 blocks with an up-to-date residual: t = B^-1 r_i, x_i += w t, r_i := t
__global__ void __launch_bounds__(kBlock)
k_jacobi3(const double* __restrict__ A, long long N, long long Np, int center, double damp,
          const double* __restrict__ omega, double* x, double* r, int write_r) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double B[9], t[3];
#pragma unroll
  for (int e = 0; e < 9; ++e) B[e] = A[((long long)center * 9 + e) * Np + i];
  const double rr[3] = {r[3 * i], r[3 * i + 1], r[3 * i + 2]};
  block_solve3<double>(B, rr, t);
  const double w = omega ? omega[i] : damp;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (write_r) r[3 * i + k] = t[k];
    x[3 * i + k] = fma(w, t[k], x[3 * i + k]);
  }
}

// The transfer sums of a node's three components with the terms in loops, for
// large Q2 levels: a thread per scalar unknown repeats the node's indices and
// weights three times and is bound by them there, while on small levels memory
// waits are the time.  Thread per unknown and loops, us: restriction to 25^3
// nodes 33.2 and 33.7, to 33^3 59 and 55, to 49^3 150 and 77; prolongation to
// 33^3 10.6 and 14.6, to 49^3 18.9 and 18.4, to 65^3 37 and 27, to 97^3 105 and
// 59.  Q1 has a quarter of the terms and stays per unknown: restriction to 33^3
// 8.7 and 15.7, to 57^3 23 and 31; prolongation to 65^3 14.7 and 18.7, to 113^3
// 56 and 61.
constexpr long long kRestrictLoopMin = 30000, kProlongLoopMin = 100000;

template <int P, typename T>
__device__ __forceinline__ void restrict3_loop(const int cJ[3], int MC, int MF, int dmask, const T* rf,
                                              T (&acc)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) acc[c] = T(0);
  for (int k = 0; k < 3; ++k)
    if (face_dir(cJ[k], MC, k, dmask)) return;
  long long off[3][5] = {{0}, {0}, {0}};
  double w[3][5] = {{1.0}, {1.0}, {1.0}};
  int cnt[3] = {1, 1, 1};
  for (int k = 0; k < 3; ++k) cnt[k] = restrict_1d<P>(cJ[k], off[k], w[k]);
  for (int z = 0; z < cnt[2]; ++z)
    for (int y = 0; y < cnt[1]; ++y)
      for (int xx = 0; xx < cnt[0]; ++xx) {
        const int fi[3] = {2 * cJ[0] + (int)off[0][xx], 2 * cJ[1] + (int)off[1][y], 2 * cJ[2] + (int)off[2][z]};
        bool skip = false;
        for (int k = 0; k < 3; ++k) skip = skip || fi[k] < 0 || fi[k] >= MF || face_dir(fi[k], MF, k, dmask);
        if (skip) continue;
        double ww = w[0][xx];
        ww = ww * w[1][y] * w[2][z];
        const long long f = fi[0] + (long long)MF * (fi[1] + (long long)MF * fi[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = fma((T)ww, rf[3 * f + c], acc[c]);
      }
}

template <int P, typename T>
__device__ __forceinline__ void prolong3_loop(const int fi[3], int MC, int dmask, const T* xc,
                                             T (&acc)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) acc[c] = T(0);
  long long J[3][3] = {{0}, {0}, {0}};
  double w[3][3] = {{1.0}, {1.0}, {1.0}};
  int cnt[3] = {1, 1, 1};
  for (int k = 0; k < 3; ++k) cnt[k] = prolong_1d<P>(fi[k], J[k], w[k]);
  for (int z = 0; z < cnt[2]; ++z)
    for (int y = 0; y < cnt[1]; ++y)
      for (int xx = 0; xx < cnt[0]; ++xx) {
        const int cj[3] = {(int)J[0][xx], (int)J[1][y], (int)J[2][z]};
        bool dj = false;
        for (int k = 0; k < 3; ++k) dj = dj || face_dir(cj[k], MC, k, dmask);
        if (dj) continue;
        double ww = w[0][xx];
        ww = ww * w[1][y] * w[2][z];
        const long long j = cj[0] + (long long)MC * (cj[1] + (long long)MC * cj[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = fma((T)ww, xc[3 * j + c], acc[c]);
      }
}

// rc := I^T rf per component (constrained), rhs_c := rc, sol_c := 0.  LOOP: a
// thread per node, its three components in the loop form; otherwise a thread
// per scalar unknown (x: node and component)
template <int P, bool LOOP, typename T = double>
__global__ void __launch_bounds__(kBlock)
k_restrict3(int MC, int MF, int dmask, const T* rf, T* __restrict__ rc,
            T* __restrict__ rhsc, T* __restrict__ solc) {
  pdl_next();
  pdl_wait();
  constexpr int CT = LOOP ? 3 : 1;
  const int xs = blockIdx.x * 32 + threadIdx.x, c0 = LOOP ? 0 : xs % 3;
  const int cJ[3] = {LOOP ? xs : xs / 3, (int)(blockIdx.y * 8 + threadIdx.y), (int)blockIdx.z};
  if (cJ[0] >= MC || cJ[1] >= MC) return;
  const long long J = 3 * (cJ[0] + (long long)MC * (cJ[1] + (long long)MC * cJ[2])) + c0;
  T acc[CT];
  if constexpr (LOOP) restrict3_loop<P, T>(cJ, MC, MF, dmask, rf, acc);
  else acc[0] = restrict_node<3, P, 3, T>(cJ, MC, MF, dmask, rf + c0);
#pragma unroll
  for (int c = 0; c < CT; ++c) {
    rc[J + c] = acc[c];
    rhsc[J + c] = acc[c];
    solc[J + c] = T(0);
  }
}

// xf := xf + I xc per component (constrained)
template <int P, bool LOOP, typename T = double>
__global__ void __launch_bounds__(kBlock)
k_prolong3(int MF, int MC, int dmask, const T* xc, T* __restrict__ xf) {
  pdl_next();
  pdl_wait();
  constexpr int CT = LOOP ? 3 : 1;
  const int xs = blockIdx.x * 32 + threadIdx.x, c0 = LOOP ? 0 : xs % 3;
  const int fi[3] = {LOOP ? xs : xs / 3, (int)(blockIdx.y * 8 + threadIdx.y), (int)blockIdx.z};
  if (fi[0] >= MF || fi[1] >= MF) return;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (face_dir(fi[k], MF, k, dmask)) return;
  const long long i = 3 * (fi[0] + (long long)MF * (fi[1] + (long long)MF * fi[2])) + c0;
  T acc[CT];
  if constexpr (LOOP) prolong3_loop<P, T>(fi, MC, dmask, xc, acc);
  else acc[0] = prolong_node<3, P, 3, T>(fi, MF, MC, dmask, xc + c0);
#pragma unroll
  for (int c = 0; c < CT; ++c) xf[i + c] = xf[i + c] + acc[c];
}

template <typename T>
static void launch_restrict3(int order, long long MC, long long MF, int dmask, const T* rf, T* rc, T* rhsc, T* solc,
                             cudaStream_t st) {
  const bool big = order == 2 && MC * MC * MC >= kRestrictLoopMin;
  const dim3 g((unsigned)(((big ? 1 : 3) * MC + 31) / 32), (unsigned)((MC + 7) / 8), (unsigned)MC), t(32, 8);
  const int mc = (int)MC, mf = (int)MF;
  if (big) launch_pdl(k_restrict3<2, true, T>, g, t, 0, st, mc, mf, dmask, rf, rc, rhsc, solc);
  else if (order == 2) launch_pdl(k_restrict3<2, false, T>, g, t, 0, st, mc, mf, dmask, rf, rc, rhsc, solc);
  else launch_pdl(k_restrict3<1, false, T>, g, t, 0, st, mc, mf, dmask, rf, rc, rhsc, solc);
}

template <typename T>
static void launch_prolong3(int order, long long MF, long long MC, int dmask, const T* xc, T* xf, cudaStream_t st) {
  const bool big = order == 2 && MF * MF * MF >= kProlongLoopMin;
  const dim3 g((unsigned)(((big ? 1 : 3) * MF + 31) / 32), (unsigned)((MF + 7) / 8), (unsigned)MF), t(32, 8);
  const int mc = (int)MC, mf = (int)MF;
  if (big) launch_pdl(k_prolong3<2, true, T>, g, t, 0, st, mf, mc, dmask, xc, xf);
  else if (order == 2) launch_pdl(k_prolong3<2, false, T>, g, t, 0, st, mf, mc, dmask, xc, xf);
  else launch_pdl(k_prolong3<1, false, T>, g, t, 0, st, mf, mc, dmask, xc, xf);
}

// Elasticity stiffness by gather (the vector form of k_assemble): for node i,
// slot s and block entry (k, l), the sum over the cells containing both nodes,
// in increasing cell index, of E_c Ebar[a][b][k][l] (top level, E per cell)
// or sum_q fma(E(x_q), Etab[q][a][b][k][l], .) (coarse levels, E sampled at
// the cell's Gauss points); Dirichlet nodes get identity blocks, Dirichlet
// columns are dropped.  a.Kbar = Ebar, a.Ctab = Etab, a.fvec the force.
template <int P>
__global__ void __launch_bounds__(kBlock)
k_assemble3(AsmArgs g) {
  constexpr int NS = St<3, P>::NS;
  constexpr int C = St<3, P>::CENTER;
  constexpr int W = 2 * P + 1;
  constexpr int P1 = P + 1;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  long long ci[3];
  node_coords(i, g.M, 3, ci);
  const int nl = g.nl, nq = g.nq;
  Q2Rows<3> q2;
  if (P == 2) q2_rows<3>(ci, g.M, q2);
  auto pos = [&](int s) -> long long {  // the node's entry in slot s (-1: a structural zero, not stored)
    if (P != 2) return i;
    const int r = q2_pattern<3>(s);
    return ((q2.valid >> r) & 1) ? q2.idx[r] : -1;
  };
  if (node_dirichlet(ci, g.M, 3, g.dmask)) {
    for (int s = 0; s < NS; ++s) {
      const long long p = pos(s);
      if (p < 0) continue;
      for (int e = 0; e < 9; ++e) g.A[((long long)s * 9 + e) * g.Np + p] = (s == C && e % 4 == 0) ? 1.0 : 0.0;
    }
    if (g.rhs)
      for (int k = 0; k < 3; ++k) g.rhs[3 * i + k] = 0.0;
    return;
  }
  for (int s = 0; s < NS; ++s) {
    const long long ps = pos(s);
    if (ps < 0) continue;
    const long long o[3] = {s % W - P, (s / W) % W - P, s / (W * W) - P};
    long long cj[3], lo[3], hi[3];
    bool ok = true;
    for (int k = 0; k < 3; ++k) {
      cj[k] = ci[k] + o[k];
      if (cj[k] < 0 || cj[k] >= g.M) ok = false;
      const long long mx = ci[k] > cj[k] ? ci[k] : cj[k];
      const long long mn = ci[k] < cj[k] ? ci[k] : cj[k];
      lo[k] = mx >= P ? (mx - 1) / P : 0;
      hi[k] = mn / P;
      if (hi[k] > g.n - 1) hi[k] = g.n - 1;
    }
    double v[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) v[e] = 0.0;
    if (ok && !node_dirichlet(cj, g.M, 3, g.dmask)) {
      for (long long cz = lo[2]; cz <= hi[2]; ++cz)
        for (long long cy = lo[1]; cy <= hi[1]; ++cy)
          for (long long cx = lo[0]; cx <= hi[0]; ++cx) {
            const long long cc[3] = {cx, cy, cz};
            const long long cidx = cx + g.n * (cy + g.n * cz);
            int a = 0, b = 0, mul = 1;
            for (int k = 0; k < 3; ++k) {
              a += (int)(ci[k] - P * cc[k]) * mul;
              b += (int)(cj[k] - P * cc[k]) * mul;
              mul *= P1;
            }
            const long long ab = ((long long)a * nl + b) * 9;
            if (g.kq == nullptr) {
              const double kc = g.kcell ? g.kcell[cidx] : g.kconst;
#pragma unroll
              for (int e = 0; e < 9; ++e) v[e] = v[e] + kc * __ldg(g.Kbar + ab + e);
            } else {
#pragma unroll
              for (int e = 0; e < 9; ++e) {
                double ee = 0.0;
                for (int q = 0; q < nq; ++q)
                  ee = fma(__ldg(g.kq + cidx * nq + q), __ldg(g.Ctab + (long long)q * nl * nl * 9 + ab + e), ee);
                v[e] = v[e] + ee;
              }
            }
          }
    }
#pragma unroll
    for (int e = 0; e < 9; ++e) g.A[((long long)s * 9 + e) * g.Np + ps] = v[e];
  }
  if (g.rhs) {
    long long lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
      lo[k] = ci[k] >= P ? (ci[k] - 1) / P : 0;
      hi[k] = ci[k] / P;
      if (hi[k] > g.n - 1) hi[k] = g.n - 1;
    }
    double acc[3] = {0.0, 0.0, 0.0};
    for (long long cz = lo[2]; cz <= hi[2]; ++cz)
      for (long long cy = lo[1]; cy <= hi[1]; ++cy)
        for (long long cx = lo[0]; cx <= hi[0]; ++cx) {
          const long long cc[3] = {cx, cy, cz};
          int a = 0, mul = 1;
          for (int k = 0; k < 3; ++k) { a += (int)(ci[k] - P * cc[k]) * mul; mul *= P1; }
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            double bl = 0.0;
            const double f = g.fvec_on ? g.fvec[k] : g.fconst;
            for (int q = 0; q < nq; ++q) bl = fma(f, g.Phi[q * nl + a], bl);
            acc[k] = acc[k] + bl;
          }
        }
    for (int k = 0; k < 3; ++k) g.rhs[3 * i + k] = acc[k];
  }
}

// dense (3N x 3N) copy of a small block level matrix, for the coarse LU
template <int P>
__global__ void k_densify3(const double* __restrict__ A, long long N, long long Np, long long M,
                           double* __restrict__ Dm) {
  constexpr int NS = St<3, P>::NS;
  constexpr int W = 2 * P + 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * NS) return;
  const long long i = t / NS;
  const int s = (int)(t % NS);
  long long ci[3];
  node_coords(i, M, 3, ci);
  const long long o[3] = {s % W - P, (s / W) % W - P, s / (W * W) - P};
  long long cj[3];
  for (int k = 0; k < 3; ++k) {
    cj[k] = ci[k] + o[k];
    if (cj[k] < 0 || cj[k] >= M) return;
  }
  const long long j = cj[0] + M * (cj[1] + M * cj[2]);
  const long long n = 3 * N;
  long long p = i;
  if constexpr (P == 2) {  // sliced storage
    Q2Rows<3> q;
    q2_rows<3>(ci, M, q);
    const int r = q2_pattern<3>(s);
    if (!((q.valid >> r) & 1)) return;
    p = q.idx[r];
  }
  for (int k = 0; k < 3; ++k)
    for (int m = 0; m < 3; ++m) Dm[(3 * i + k) * n + 3 * j + m] = A[((long long)s * 9 + k * 3 + m) * Np + p];
}

// The full slot layout of a level (structural zeros included) in FP32 -- the
// layout the stored-level kernels of the mixed cycle read -- from a Q2
// level's sliced storage; one thread per (slot, node)
template <int D>
__global__ void k_expand_q2_f32(const double* __restrict__ A, long long N, long long Np, long long M, int nslots,
                                float* __restrict__ out, const __grid_constant__ Q2Layout lay) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nslots * N) return;
  const int s = (int)(t / N);
  const long long i = t - (long long)s * N;
  long long c[3];
  node_coords(i, M, D, c);
  const int r = q2_pattern<D>(s);
  bool ok = true;
  for (int k = 0; k < D; ++k)
    if (((r >> k) & 1) && (c[k] & 1)) ok = false;
  out[(long long)s * Np + i] = ok ? (float)A[(long long)s * Np + q2c_pos<D>(lay, c, M, r)] : 0.f;
}

// Galerkin coarse operator A_C = I^T A_F I of a structured level -- scalar
// Q1/Q2 and 3 x 3 node blocks -- with the constrained interpolation (fine
// Dirichlet rows and coarse Dirichlet columns removed; identity blocks at
// coarse Dirichlet nodes).  One thread per (coarse slot S, coarse row I): it
// walks the oracle's order -- fine i over the restriction stencil of I
// (z, y, x), fine slots ascending, the coarse J = I + off_S looked up in j's
// interpolation stencil -- and keeps the terms that land on S, so each entry
// sums the oracle's terms in the oracle's order:
// acc[k][m] = fma(w_iI * a_ij[k][m], w_jJ, acc[k][m]).  Fine entries a level
// does not store (Q2: an odd-coordinate node's +-2 slots) are structural
// zeros and are skipped.
template <int D, int P>
__device__ __forceinline__ long long gal_pos(const Q2Layout& lay, const long long c[3], long long M, int s, int nc) {
  if (P == 1) return c[0] + M * (c[1] + M * c[2]);
  const int r = q2_pattern<D>(s);
  for (int k = 0; k < D; ++k)
    if (((r >> k) & 1) && (c[k] & 1)) return -1;
  if (nc == 1) return q2c_pos<D>(lay, c, M, r);  // scalar Q2: colour-major
  const long long H = (M + 1) / 2;              // node blocks: lexicographic, halved where restricted
  long long id = 0, mul = 1;
  for (int k = 0; k < D; ++k) {
    const bool rk = (r >> k) & 1;
    id += (rk ? c[k] / 2 : c[k]) * mul;
    mul *= rk ? H : M;
  }
  return id;
}

template <int D, int P, int NC>
__global__ void __launch_bounds__(kBlock)
k_galerkin(const double* __restrict__ AF, long long NpF, int MF, double* __restrict__ AC, long long NCN,
           long long NpC, int MC, int dmask, Q2Layout layF, Q2Layout layC) {
  constexpr int W = 2 * P + 1;
  constexpr int NS = D == 1 ? W : (D == 2 ? W * W : W * W * W);
  constexpr int CEN = (NS - 1) / 2;
  constexpr int NE = NC * NC;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)NS * NCN) return;
  const int S = (int)(t / NCN);
  const long long I = t - (long long)S * NCN;
  long long cI[3];
  node_coords(I, MC, D, cI);
  const long long pI = gal_pos<D, P>(layC, cI, MC, S, NC);
  if (pI < 0) return;  // an entry the coarse level does not store
  double acc[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) acc[e] = 0.0;
  if (node_dirichlet(cI, MC, D, dmask)) {
#pragma unroll
    for (int e = 0; e < NE; ++e) AC[((long long)S * NE + e) * NpC + pI] = (S == CEN && e % (NC + 1) == 0) ? 1.0 : 0.0;
    return;
  }
  const int oS[3] = {S % W - P, D > 1 ? (S / W) % W - P : 0, D > 2 ? S / (W * W) - P : 0};
  long long cJ[3] = {0, 0, 0};
  bool okJ = true;
  for (int k = 0; k < D; ++k) {
    cJ[k] = cI[k] + oS[k];
    okJ = okJ && cJ[k] >= 0 && cJ[k] < MC;
  }
  if (okJ && !node_dirichlet(cJ, MC, D, dmask)) {
    long long off[3][5] = {{0}, {0}, {0}};
    double w[3][5] = {{1.0}, {1.0}, {1.0}};
    int cnt[3] = {1, 1, 1};
    for (int k = 0; k < D; ++k) cnt[k] = restrict_1d<P>(cI[k], off[k], w[k]);
    for (int z = 0; z < cnt[2]; ++z)
      for (int y = 0; y < cnt[1]; ++y)
        for (int x = 0; x < cnt[0]; ++x) {
          const long long fi[3] = {2 * cI[0] + off[0][x], D > 1 ? 2 * cI[1] + off[1][y] : 0,
                                   D > 2 ? 2 * cI[2] + off[2][z] : 0};
          bool skip = false;
          for (int k = 0; k < D; ++k) skip = skip || fi[k] < 0 || fi[k] >= MF || face_dir((int)fi[k], MF, k, dmask);
          if (skip) continue;
          double wi = w[0][x];
          if (D > 1) wi = wi * w[1][y];
          if (D > 2) wi = wi * w[2][z];
          for (int oz = (D > 2 ? -P : 0); oz <= (D > 2 ? P : 0); ++oz)
            for (int oy = (D > 1 ? -P : 0); oy <= (D > 1 ? P : 0); ++oy)
              for (int ox = -P; ox <= P; ++ox) {
                const int o[3] = {ox, oy, oz};
                long long fj[3] = {0, 0, 0};
                double wj[3] = {1.0, 1.0, 1.0};
                bool hit = true;
                for (int k = 0; k < D && hit; ++k) {
                  fj[k] = fi[k] + o[k];
                  if (fj[k] < 0 || fj[k] >= MF || face_dir((int)fj[k], MF, k, dmask)) { hit = false; break; }
                  long long Jk[3];
                  double wk[3];
                  const int nk = prolong_1d<P>(fj[k], Jk, wk);
                  bool found = false;
                  for (int q = 0; q < nk; ++q)
                    if (Jk[q] == cJ[k]) { wj[k] = wk[q]; found = true; }
                  hit = found;
                }
                if (!hit) continue;
                const int sf = (ox + P) + W * ((D > 1 ? oy : 0) + (D > 1 ? P : 0)) +
                               W * W * ((D > 2 ? oz : 0) + (D > 2 ? P : 0));
                const long long pF = gal_pos<D, P>(layF, fi, MF, sf, NC);
                if (pF < 0) continue;  // a structural zero
                double ww = wj[0];
                if (D > 1) ww = ww * wj[1];
                if (D > 2) ww = ww * wj[2];
#pragma unroll
                for (int e = 0; e < NE; ++e)
                  acc[e] = fma(wi * AF[((long long)sf * NE + e) * NpF + pF], ww, acc[e]);
              }
        }
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) AC[((long long)S * NE + e) * NpC + pI] = acc[e];
}

// ---- diagonal-block operations of the recorded cycle (vector form)
// mode 0: y_i = B_i^-1 x_i; 1: y_i = w_i B_i^-1 x_i; 2: y_i += w_i B_i^-1 x_i
// (B_i the 3 x 3 diagonal block, symmetric, so the same solve serves the adjoint)
__global__ void __launch_bounds__(kBlock)
k_bdiag3(const double* __restrict__ A, long long N, long long Np, int center, int mode,
         const double* w, const double* x, double* __restrict__ y) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double B[9], t[3];
#pragma unroll
  for (int e = 0; e < 9; ++e) B[e] = A[((long long)center * 9 + e) * Np + i];
  const double xx[3] = {x[3 * i], x[3 * i + 1], x[3 * i + 2]};
  block_solve3<double>(B, xx, t);
  const double wi = mode == 0 ? 1.0 : w[i];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double v = mode == 0 ? t[k] : wi * t[k];
    y[3 * i + k] = mode == 2 ? y[3 * i + k] + v : v;
  }
}

// y = x + w .* v with w per node (y may be x)
__global__ void k_xpwv3(const double* x, const double* w, const double* v, double* y,
                        long long N) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) y[3 * i + k] = x[3 * i + k] + w[i] * v[3 * i + k];
}

// acc_i += sum_k a_ik b_ik (per-node dot of two vectors)
__global__ void k_acc_prod3(double* __restrict__ acc, const double* a, const double* b,
                            long long N) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double s = a[3 * i] * b[3 * i];
  s = fma(a[3 * i + 1], b[3 * i + 1], s);
  s = fma(a[3 * i + 2], b[3 * i + 2], s);
  acc[i] += s;
}

// ---- FP32 forms for the mixed cycle of the vector form
// first smoothing step from a zero guess: x = w B^-1 b
template <typename T>
__global__ void __launch_bounds__(kBlock)
k_jacobi0_3(const T* __restrict__ A, long long N, long long Np, int center, float damp,
            const double* __restrict__ omega, const T* b, T* __restrict__ x) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  T B[9], t[3];
#pragma unroll
  for (int e = 0; e < 9; ++e) B[e] = A[((long long)center * 9 + e) * Np + i];
  const T bb[3] = {b[3 * i], b[3 * i + 1], b[3 * i + 2]};
  block_solve3<T>(B, bb, t);
  const T w = omega ? (T)omega[i] : (T)damp;
#pragma unroll
  for (int k = 0; k < 3; ++k) x[3 * i + k] = w * t[k];
}

// y = f x with f from a grid scalar: mode 0: 1, mode 1: 1/sqrt(sc[slot]), mode 2: sqrt(sc[slot])
template <typename TI, typename TO>
__global__ void k_vscale(const TI* x, const double* sc, int slot, int mode,
                         TO* __restrict__ y, long long n) {
  pdl_next_light();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double f = 1.0;
  if (mode) {
    const double v = sc[slot];
    f = v > 0.0 ? (mode == 1 ? 1.0 / sqrt(v) : sqrt(v)) : 1.0;
  }
  y[i] = (TO)((double)x[i] * f);
}

// the FCG(1) coefficient beta = -(z, a) / (p, a) of the previous step (0 on a restart)
__global__ void k_fcg_beta(double* sc, int first) {
  pdl_next();
  pdl_wait();
  sc[S_RATIO] = first ? 0.0 : -sc[S_TMP] / sc[S_BETA];
}

// ------------------------------------------------------------ small levels
// The collected steps of a cycle on small levels (see Tail).  A launch costs a
// small level 2-3 us whatever it does, and a step that goes to L2 for its
// operands 1,400 cycles and more (so measured with the levels' data in global
// memory, one CTA or a cluster of eight: no faster than the launches).  Here
// the structured matrices come into shared memory while the previous launch
// ends, the vectors the steps read first follow, and a step costs its barrier,
// its chain and its division: 600-1,300 cycles on up to 300 nodes.  The 26
// steps of a V(1,1) cycle on 33^2 nodes and below take 25 us in place of some
// 60; 64^2 Poisson solve 1.09 -> 0.81 ms, adaptive 2D solve 2.38 -> 2.16 ms.
constexpr int kTailT = 512;

// the launch's parameters; CAP: room for the steps (the parameters are copied
// at every launch, and most cycles' tails have fewer than 48 steps)
template <int CAP>
struct TailArgs {
  int dmask, nbase, nops, nlev, nvec;
  const double* ainv;
  TailLevel lev[Tail::kLev];
  TailVec vec[Tail::kVec];
  TailOp ops[CAP];
};

// row sum, the unknowns (and a structured matrix) in shared memory
template <int D, bool CSR>
__device__ __forceinline__ double tail_row(const TailLevel& L, const double* sm, const double* x, int i, double& dg) {
  double s = 0.0;
  if constexpr (CSR) {
    dg = __ldg(L.diag + i);
    constexpr int K = 8;
    const int e1 = (int)L.a.start[i + 1];
    for (int e = (int)L.a.start[i]; e < e1; e += K) {
      int ix[K];
      double v[K];
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (e + q < e1) { ix[q] = __ldg(L.a.index + e + q); v[q] = __ldg(L.a.value + e + q); }
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (e + q < e1) s = fma(v[q], x[ix[q]], s);
    }
  } else {
    const int M = L.M, N = L.N;
    const double* a = sm + L.aoff + i;
    dg = a[St<D, 1>::CENTER * N];
#pragma unroll
    for (int oz = (D > 2 ? -1 : 0); oz <= (D > 2 ? 1 : 0); ++oz)
#pragma unroll
      for (int oy = (D > 1 ? -1 : 0); oy <= (D > 1 ? 1 : 0); ++oy)
#pragma unroll
        for (int ox = -1; ox <= 1; ++ox) {
          s = fma(*a, x[min(max(i + ox + M * (oy + M * oz), 0), N - 1)], s);
          a += N;
        }
  }
  return s;
}

// row sum of a transfer matrix, the vector in shared memory
__device__ __forceinline__ double tail_csr_sum(const CsrView& a, const double* x, int i) {
  double s = 0.0;
  for (long long e = a.start[i]; e < a.start[i + 1]; ++e) s = fma(__ldg(a.value + e), x[__ldg(a.index + e)], s);
  return s;
}

template <int D, bool CSR, int CAP>
__global__ void __launch_bounds__(kTailT, 1)
k_tail(const __grid_constant__ TailArgs<CAP> g) {
  extern __shared__ double sm[];
  __shared__ TailOp ops[CAP];
  __shared__ TailLevel lv[Tail::kLev];
  __shared__ TailVec vc[Tail::kVec];
  const int tid = threadIdx.x;
  const long long bq = blockIdx.x;  // problem of a batch
  pdl_next();
  {
    auto copy = [&](void* dst, const void* src, int bytes) {
      for (int k = tid; k < bytes / 4; k += kTailT) static_cast<int*>(dst)[k] = static_cast<const int*>(src)[k];
    };
    copy(ops, g.ops, g.nops * (int)sizeof(TailOp));
    copy(lv, g.lev, g.nlev * (int)sizeof(TailLevel));
    copy(vc, g.vec, g.nvec * (int)sizeof(TailVec));
  }
  __syncthreads();
  // background copies (cp.async): every level's matrix and every vector in flight
  if constexpr (!CSR) {
    constexpr int NS = St<D, 1>::NS;
    for (int l = 0; l < g.nlev; ++l) {
      const int N = lv[l].N;
      const long long Np = lv[l].Np;
      const double* A = lv[l].A + bq * NS * Np;
      double* d = sm + lv[l].aoff;
      for (int i = tid; i < N; i += kTailT)
#pragma unroll
        for (int s = 0; s < NS; ++s) cp_async8(d + s * N + i, A + s * Np + i);
    }
  }
  pdl_wait();
  for (int k = 0; k < g.nvec; ++k)
    if (vc[k].in) {
      const TailLevel& L = lv[vc[k].lev];
      for (int i = tid; i < L.N; i += kTailT) cp_async8(sm + vc[k].off + i, vc[k].g + bq * L.Np + i);
    }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  const int dmask = g.dmask;
#pragma unroll 1
  for (int o = 0; o < g.nops; ++o) {
    __syncthreads();
    const TailOp& op = ops[o];
    // a warp without work goes straight to the next barrier: on the smallest
    // levels the idle warps' decoding would be the step's time
    const int n = op.n;
    if ((tid & ~31) >= n) continue;
    const TailLevel& L = lv[op.lev];
    const int N = L.N;
    double *x = sm + op.x, *y = sm + op.y, *r = sm + op.r, *b = sm + op.b;
    const double* om = L.omega ? L.omega + bq * L.Np : nullptr;
    switch (op.kind) {
      case TAIL_RES:
        for (int i = tid; i < n; i += kTailT) {
          double dg;
          const double s = tail_row<D, CSR>(L, sm, x, i, dg);
          r[i] = b[i] - s;
        }
        break;
      case TAIL_JACOBI:
        for (int i = tid; i < n; i += kTailT) {
          const double w = om ? __ldg(om + i) : op.w;
          const double d = CSR ? __ldg(L.diag + i) : sm[L.aoff + St<D, 1>::CENTER * N + i];
          const double t = r[i] / d;
          if (op.flag) r[i] = t;
          x[i] = fma(w, t, x[i]);
        }
        break;
      case TAIL_JACOBI_RES:
        for (int i = tid; i < n; i += kTailT) {
          const double w = om ? __ldg(om + i) : op.w;
          double dg;
          const double s = tail_row<D, CSR>(L, sm, x, i, dg);
          const double t = (b[i] - s) / dg;
          if (op.flag) r[i] = t;
          y[i] = fma(w, t, x[i]);
        }
        break;
      case TAIL_SOR:
      case TAIL_SSC: {
        int nx = 1, ny = 1;
        const int cx = op.flag & 1, cy = (op.flag >> 1) & 1, cz = (op.flag >> 2) & 1;
        if (!CSR) {
          nx = (L.M - cx + 1) / 2;
          ny = D > 1 ? (L.M - cy + 1) / 2 : 1;
        }
        for (int u = tid; u < n; u += kTailT) {
          int i;
          if (CSR) {
            i = __ldg(op.rows + u);
          } else {
            const int q = u / nx, jx = u - q * nx, jy = D > 1 ? q % ny : 0, jz = D > 2 ? q / ny : 0;
            i = cx + 2 * jx + L.M * ((D > 1 ? cy + 2 * jy : 0) + L.M * (D > 2 ? cz + 2 * jz : 0));
          }
          const double w = op.kind == TAIL_SOR && om ? __ldg(om + i) : op.w;
          double dg;
          const double s = tail_row<D, CSR>(L, sm, x, i, dg);
          const double rr = b[i] - s, tt = rr / dg;
          r[i] = op.kind == TAIL_SSC ? rr : tt;
          x[i] = fma(w, tt, x[i]);
        }
        break;
      }
      case TAIL_RESTRICT: {
        const TailLevel& C = lv[op.clev];
        for (int j = tid; j < n; j += kTailT) {
          double acc;
          if constexpr (CSR) {
            acc = tail_csr_sum(L.pt, x, j);
          } else {
            const int q = j / C.M;
            const int c[3] = {j - q * C.M, D > 1 ? q % C.M : 0, D > 2 ? q / C.M : 0};
            acc = restrict_node<D, 1>(c, C.M, L.M, dmask, x);
          }
          r[j] = acc;
          b[j] = acc;
          y[j] = 0.0;
        }
        break;
      }
      case TAIL_PROLONG: {
        const TailLevel& C = lv[op.clev];
        for (int i = tid; i < n; i += kTailT) {
          if constexpr (CSR) {
            if (L.p.start[i] == L.p.start[i + 1]) continue;  // constrained rows keep their value
            y[i] = y[i] + tail_csr_sum(L.p, x, i);
          } else {
            const int q = i / L.M;
            const int c[3] = {i - q * L.M, D > 1 ? q % L.M : 0, D > 2 ? q / L.M : 0};
            bool dir = false;
#pragma unroll
            for (int k = 0; k < D; ++k) dir = dir || face_dir(c[k], L.M, k, dmask);
            if (dir) continue;
            y[i] = y[i] + prolong_node<D, 1>(c, L.M, C.M, dmask, x);
          }
        }
        break;
      }
      default: {  // TAIL_COARSE: at most 128 unknowns, four warps; r is read before it is written
        const int nb = g.nbase;
        double acc = 0.0;
        if (tid < nb) {
          const double* a = g.ainv + bq * nb * nb + tid;
          int j = 0;
          for (; j + 16 <= nb; j += 16) {
            double c[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) c[q] = __ldg(a + (j + q) * nb);
#pragma unroll
            for (int q = 0; q < 16; ++q) acc = fma(c[q], r[j + q], acc);
          }
          for (; j < nb; ++j) acc = fma(__ldg(a + j * nb), r[j], acc);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (tid < nb) {
          r[tid] = acc;
          x[tid] = fma(op.w, acc, x[tid]);
        }
      }
    }
  }
  __syncthreads();
  for (int k = 0; k < g.nvec; ++k)
    if (vc[k].out) {
      const TailLevel& L = lv[vc[k].lev];
      for (int i = tid; i < L.N; i += kTailT) vc[k].g[bq * L.Np + i] = sm[vc[k].off + i];
    }
}

// ---------------------------------------------------------- dispatchers
#define FMG_DISPATCH(D_, P_, ...)                                             \
  do {                                                                        \
    if ((D_) == 1 && (P_) == 1) { constexpr int D = 1, P = 1; __VA_ARGS__; }  \
    else if ((D_) == 2 && (P_) == 1) { constexpr int D = 2, P = 1; __VA_ARGS__; } \
    else if ((D_) == 3 && (P_) == 1) { constexpr int D = 3, P = 1; __VA_ARGS__; } \
    else if ((D_) == 1 && (P_) == 2) { constexpr int D = 1, P = 2; __VA_ARGS__; } \
    else if ((D_) == 2 && (P_) == 2) { constexpr int D = 2, P = 2; __VA_ARGS__; } \
    else { constexpr int D = 3, P = 2; __VA_ARGS__; }                         \
  } while (0)

#define Q1_DISPATCH(D_, ...)                                              \
  do {                                                                    \
    if ((D_) == 1) { constexpr int D = 1; __VA_ARGS__; }                  \
    else if ((D_) == 2) { constexpr int D = 2; __VA_ARGS__; }             \
    else { constexpr int D = 3; __VA_ARGS__; }                            \
  } while (0)
#define Q2_DISPATCH Q1_DISPATCH

static inline unsigned grid1(long long n, int bs = kBlock) { return (unsigned)((n + bs - 1) / bs); }

// the row kernels of scalar Q2 levels over every class: blockIdx.y the class,
// blockIdx.x the blocks of its parity subgrids (the largest class's count)
template <int D>
static dim3 q2_grid(int M, int ssc = -1) {
  int ncol = 1;
  for (int k = 0; k < D; ++k) ncol *= 3;
  long long nb = 1;
  for (int col = 0; col < ncol; ++col) nb = std::max(nb, q2_class_blocks<D>(M, col, ssc));
  return dim3((unsigned)nb, (unsigned)ncol);
}

// a compressed-row kernel over `rows` rows in the form for that many
#define CSR_LAUNCH(kern, rows, ...)                                                                      \
  do {                                                                                                   \
    if ((rows) > kCsrWide) launch_pdl(kern<1>, grid1(rows, kCsrT<1>), kCsrT<1>, 0, st, __VA_ARGS__);       \
    else launch_early(kern<8>, grid1(rows, kCsrT<8>), kCsrT<8>, 0, st, __VA_ARGS__);                       \
  } while (0)

void launch_spmv(const LevelView& L, const double* x, const double* b, double* y, const double* dv,
                 const Reduce* R, cudaStream_t st) {
  if (L.csr) {  // the reduction as a separate DR4096 pass
    g_launches.fetch_add(1, std::memory_order_relaxed);
    CSR_LAUNCH(k_csr_spmv, L.N, L.N, L.a, x, b, y, b ? 1 : 0);
    if (dv) launch_dot(y, dv, L.N, *R, st);
    return;
  }
  if (L.nc == 3) {  // 3 x 3 blocks: the reduction, if any, as a separate DR4096 pass
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (b) launch_row3<double, ROW3_RES>(L.order, L.A, L.N, L.Np, L.M, 0.0, nullptr, x, b, y, nullptr, false, st);
    else launch_row3<double, ROW3_MUL>(L.order, L.A, L.N, L.Np, L.M, 0.0, nullptr, x, b, y, nullptr, false, st);
    if (dv) launch_dot(y, dv, 3 * L.N, *R, st);
    return;
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (L.order == 2) {  // rows by colour class and parity, the reduction as a separate DR4096 pass
    const Q2Layout lay = q2_layout(L.dim, L.M);
    Q2_DISPATCH(L.dim, {
      const dim3 g = q2_grid<D>((int)L.M);
      if (b) launch_pdl(k_spmv_q2c<D, true>, g, kQ2T, 0, st, L.A, L.Np, (int)L.M, x, b, y, lay);
      else launch_pdl(k_spmv_q2c<D, false>, g, kQ2T, 0, st, L.A, L.Np, (int)L.M, x, b, y, lay);
    });
    if (dv) launch_dot(y, dv, L.N, *R, st);
    return;
  }
  const dim3 g(grid1(L.N, kRowT), (unsigned)L.nb);
  Q1_DISPATCH(L.dim, {
    if (b) launch_early(k_row_q1<D, true>, g, kRowT, 0, st, L.A, (int)L.N, L.Np, (int)L.M, x, b, y);
    else launch_early(k_row_q1<D, false>, g, kRowT, 0, st, L.A, (int)L.N, L.Np, (int)L.M, x, b, y);
  });
  if (dv) launch_dot_b(y, dv, L.N, L.Np, L.nb, *R, st);
}

void launch_jacobi(const LevelView& L, double damp, double* x, double* r, bool write_r, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (L.csr) {
    launch_early(k_jacobi, grid1(L.N), kBlock, 0, st, L.diag, L.N, damp, L.omega, x, r, write_r ? 1 : 0, 0, 0);
    return;
  }
  if (L.nc == 3) {
    launch_early(k_jacobi3, grid1(L.N), kBlock, 0, st, L.A, L.N, L.Np, L.center, damp, L.omega, x, r, write_r ? 1 : 0);
    return;
  }
  if (L.order == 2) {  // colour-major sliced storage
    const Q2Layout lay = q2_layout(L.dim, L.M);
    Q2_DISPATCH(L.dim, {
      launch_early(k_jacobi_q2<D>, grid1(L.N), kBlock, 0, st,
                   L.A, L.N, L.Np, L.M, damp, L.omega, x, r, write_r ? 1 : 0, lay);
    });
    return;
  }
  const double* Dg = L.A + (long long)L.center * L.Np;
  long long ns = 1;
  for (int k = 0; k < L.dim; ++k) ns *= 3;
  launch_early(k_jacobi, dim3(grid1(L.N), (unsigned)L.nb), kBlock, 0, st, Dg, L.N, damp, L.omega, x, r, write_r ? 1 : 0,
                                                                L.Np, ns * L.Np);
}

void launch_jacobi_res(const LevelView& L, double damp, const double* x, const double* b, double* xout,
                       double* r, bool write_r, const double* dv, const Reduce* R, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (L.csr) {
    CSR_LAUNCH(k_csr_jacobi_res, L.N, L.N, L.a, L.diag, damp, L.omega, x, b, xout, r, write_r ? 1 : 0);
    if (dv) launch_dot(xout, dv, L.N, *R, st);
    return;
  }
  if (L.nc == 3) {
    launch_row3<double, ROW3_JACOBI>(L.order, L.A, L.N, L.Np, L.M, damp, L.omega, x, b, xout, r, write_r, st);
    if (dv) launch_dot(xout, dv, 3 * L.N, *R, st);
    return;
  }
  if (L.order == 2) {  // rows by colour class and parity
    const Q2Layout lay = q2_layout(L.dim, L.M);
    Q2_DISPATCH(L.dim, {
      launch_pdl(k_jacobi_res_q2c<D>, q2_grid<D>((int)L.M), kQ2T, 0, st,
                 L.A, L.Np, (int)L.M, damp, L.omega, x, b, xout, r,
                                                                 write_r ? 1 : 0, lay);
    });
    if (dv) launch_dot(xout, dv, L.N, *R, st);
    return;
  }
  const dim3 g(grid1(L.N, kRowT), (unsigned)L.nb);
  Q1_DISPATCH(L.dim, {
    launch_early(k_row_jacobi_q1<D>, g, kRowT, 0, st, L.A, (int)L.N, L.Np, (int)L.M, damp, L.omega, x, b, xout, r,
                                            write_r ? 1 : 0);
  });
  if (dv) launch_dot_b(xout, dv, L.N, L.Np, L.nb, *R, st);
}

static void launch_csr_sor(const LevelView& L, double omega, const double* om, double* x, const double* b, double* r,
                           bool ssc, cudaStream_t st) {
  g_launches.fetch_add(L.ncol, std::memory_order_relaxed);
  for (int c = 0; c < L.ncol; ++c) {
    const long long cnt = L.coff[c + 1] - L.coff[c];
    if (cnt > 0)
      CSR_LAUNCH(k_csr_sor, cnt, L.crow + L.coff[c], cnt, L.a, L.diag, omega, om, x, b, r, ssc ? 1 : 0);
  }
}

void launch_sor(const LevelView& L, double omega, double* x, const double* b, double* r, cudaStream_t st) {
  if (L.csr) {
    launch_csr_sor(L, omega, L.omega, x, b, r, false, st);
    return;
  }
  const Q2Layout lay = q2_layout(L.dim, L.M);
  int Q = L.order + 1, ncol = 1;
  for (int k = 0; k < L.dim; ++k) ncol *= Q;
  g_launches.fetch_add(ncol, std::memory_order_relaxed);
  const long long most = (L.M + Q - 1) / Q;  // rows of the largest colour along a direction
  const bool tile = L.order == 2 && L.dim == 3 && most * most * most <= kTileMax;
  for (int col = 0; col < ncol; ++col) {
    const int cx = col % Q, cy = (col / Q) % Q, cz = col / (Q * Q);
    long long cnt = (L.M - cx + Q - 1) / Q;
    if (L.dim > 1) cnt *= (L.M - cy + Q - 1) / Q;
    if (L.dim > 2) cnt *= (L.M - cz + Q - 1) / Q;
    if (tile) {
      launch_q2_tile<false>(L, col, omega, x, b, r, lay, st);
    } else if (L.order == 2) {
      Q2_DISPATCH(L.dim, {
        const unsigned nb = (unsigned)q2_class_blocks<D>((int)L.M, col);
        if (nb) launch_pdl(k_sor_q2<D>, nb, kQ2T, 0, st, L.A, L.Np, (int)L.M, col, omega, L.omega, x, b, r, lay);
      });
    } else {
      Q1_DISPATCH(L.dim, {
        launch_early(k_sor_colour<D, 1>, grid1(cnt, kRowT), kRowT, 0, st,
                     L.A, L.N, L.Np, L.M, col, omega, L.omega, x, b, r);
      });
    }
  }
}

long long ssc_blocks(const LevelView& L) {
  if (L.order != 2) return 0;
  long long nv = (L.M + 1) / 2, n = 1;
  for (int k = 0; k < L.dim; ++k) n *= nv;
  return n;
}

int ssc_block_size(int dim) { return dim == 1 ? 3 : (dim == 2 ? 9 : 27); }

void launch_ssc_factor(const LevelView& L, double* F, unsigned char* P, cudaStream_t st) {
  if (L.order != 2) return;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const Q2Layout lay = q2_layout(L.dim, L.M);
  const unsigned grid = (unsigned)((ssc_blocks(L) * 32 + 127) / 128);
  Q2_DISPATCH(L.dim, { k_ssc_factor_q2<D><<<grid, 128, 0, st>>>(L.A, L.Np, L.M, L.dmask, F, P, lay); });
}

void launch_ssc(const LevelView& L, double omega, double* x, const double* b, double* r, const double* F,
                const unsigned char* P, cudaStream_t st) {
  if (L.csr) {  // an algebraic level: one-unknown blocks over its colouring
    launch_csr_sor(L, omega, nullptr, x, b, r, true, st);
    return;
  }
  const int ncol = 1 << L.dim;
  g_launches.fetch_add(ncol, std::memory_order_relaxed);
  if (L.order == 1) {  // one-node blocks: the colour sweep of the SOR with the SSC residual
    for (int col = 0; col < ncol; ++col) {
      const int cx = col & 1, cy = (col >> 1) & 1, cz = (col >> 2) & 1;
      long long cnt = (L.M - cx + 1) / 2;
      if (L.dim > 1) cnt *= (L.M - cy + 1) / 2;
      if (L.dim > 2) cnt *= (L.M - cz + 1) / 2;
      Q1_DISPATCH(L.dim, {
        launch_early(k_sor_colour<D, 1, true>, grid1(cnt, kRowT), kRowT, 0, st,
                     L.A, L.N, L.Np, L.M, col, omega, nullptr, x, b, r);
      });
    }
    return;
  }
  g_launches.fetch_add(ncol, std::memory_order_relaxed);  // two launches a colour
  const Q2Layout lay = q2_layout(L.dim, L.M);
  const long long nv = (L.M + 1) / 2;
  const bool tile = L.dim == 3 && L.N <= kSscTileMax;
  for (int col = 0; col < ncol; ++col) {
    long long cnt = (nv - (col & 1) + 1) / 2;
    if (L.dim > 1) cnt *= (nv - ((col >> 1) & 1) + 1) / 2;
    if (L.dim > 2) cnt *= (nv - ((col >> 2) & 1) + 1) / 2;
    if (cnt == 0) continue;
    const unsigned grid = (unsigned)((cnt * 32 + 127) / 128);
    Q2_DISPATCH(L.dim, {
      if (tile)
        launch_q2_tile<true>(L, col, 0.0, x, b, r, lay, st);
      else
        launch_pdl(k_ssc_res_q2<D>, q2_grid<D>((int)L.M, col), kQ2T, 0, st, L.A, L.Np, (int)L.M, col, L.dmask,
                   x, b, r, lay);
      launch_early(k_ssc_solve_q2<D>, dim3(grid), 128, 0, st, (int)L.M, L.dmask, col, omega, x, r, F, P);
    });
  }
}

void launch_psc(const LevelView& L, double damp, double* x, const double* r, const double* F,
                const unsigned char* P, double* C, cudaStream_t st) {
  if (L.order == 1) {  // one-node blocks: x_i += damp r_i / a_ii, r unchanged
    g_launches.fetch_add(1, std::memory_order_relaxed);
    Q1_DISPATCH(L.dim, { launch_pdl(k_psc_q1<D>, grid1(L.N), kBlock, 0, st, L.A, L.N, L.Np, damp, x, r); });
    return;
  }
  g_launches.fetch_add(2, std::memory_order_relaxed);
  const unsigned grid = (unsigned)((ssc_blocks(L) * 32 + 127) / 128);
  Q2_DISPATCH(L.dim, {
    launch_pdl(k_psc_block_q2<D>, grid, 128, 0, st, L.M, L.dmask, r, F, P, C);
    launch_pdl(k_psc_gather_q2<D>, grid1(L.N), kBlock, 0, st, L.N, L.M, L.dmask, damp, C, x);
  });
}

static inline dim3 xfer_grid(long long M, int dim) {
  return dim3((unsigned)((M + 31) / 32), (unsigned)(dim > 1 ? (M + 7) / 8 : 1), (unsigned)(dim > 2 ? M : 1));
}

void launch_restrict(const LevelView& F, const LevelView& Cl, const double* rf, double* rc, double* rhsc,
                     double* solc, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (F.csr) {
    CSR_LAUNCH(k_csr_restrict, Cl.N, Cl.N, F.pt, rf, rc, rhsc, solc);
    return;
  }
  if (F.nc == 3) {
    launch_restrict3<double>(F.order, Cl.M, F.M, F.dmask, rf, rc, rhsc, solc, st);
    return;
  }
  FMG_DISPATCH(F.dim, F.order, {
    dim3 gr = xfer_grid(Cl.M, D);
    if (D < 3) gr.z = (unsigned)F.nb;  // the problems of a batched level
    launch_early(k_restrict<D, P>, gr, dim3(32, 8), 0, st,
                 (int)Cl.M, (int)F.M, F.dmask, rf, rc, rhsc, solc, F.Np, Cl.Np);
  });
}

void launch_prolong(const LevelView& Cl, const LevelView& F, const double* xc, double* xf, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (F.csr) {
    CSR_LAUNCH(k_csr_prolong, F.N, F.N, F.p, xc, xf);
    return;
  }
  if (F.nc == 3) {
    launch_prolong3<double>(F.order, F.M, Cl.M, F.dmask, xc, xf, st);
    return;
  }
  FMG_DISPATCH(F.dim, F.order, {
    dim3 gr = xfer_grid(F.M, D);
    if (D < 3) gr.z = (unsigned)F.nb;
    if constexpr (P == 1) {
      gr.x = (unsigned)((Cl.M + 31) / 32);
      launch_early(k_prolong_q1f<D>, gr, dim3(32, 8), 0, st, (int)F.M, (int)Cl.M, F.dmask, xc, xf, F.Np, Cl.Np);
    } else
    launch_early(k_prolong<D, P>, gr, dim3(32, 8), 0, st, (int)F.M, (int)Cl.M, F.dmask, xc, xf, F.Np, Cl.Np);
  });
}

void launch_coarse_solve(const double* AinvT, int n, double damp, double* x, double* r, cudaStream_t st, int nb,
                         long long vs) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  // one warp of rows per CTA up to 512 unknowns, then two, then four (the
  // largest block bases, 2,048); clusters beyond 8 CTAs are not portable
  auto go = [&](auto RT) {
    constexpr int R = decltype(RT)::value;
    int cs = 1;
    while (cs * 32 * R < n) cs *= 2;
    auto kern = k_coarse_solve<R>;
    const size_t smem = (size_t)(2 * kCsStep * 32 * R + n) * sizeof(double);
    // a refusal shows as the launch's error
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (cs > 8) cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_pdl
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(nb * cs));
    cfg.blockDim = dim3(32 * (R + kCsLoad));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = t_pdl_stream == st ? 2 : 1;
    t_pdl_stream = st;
    cudaLaunchKernelEx(&cfg, kern, AinvT, n, damp, x, r, vs, cs);
  };
  if (n <= 512) go(std::integral_constant<int, 1>{});
  else if (n <= 1024) go(std::integral_constant<int, 2>{});
  else go(std::integral_constant<int, 4>{});
}

void launch_lu(double* A, int n, int* piv, double* X, double* XT, cudaStream_t st) {
  g_launches.fetch_add(3, std::memory_order_relaxed);
  const size_t f_smem = (size_t)n * n * sizeof(double), i_smem = f_smem + (size_t)n * 32 * sizeof(double);
  constexpr size_t kMaxSmem = 200 * 1024;
  if (i_smem <= kMaxSmem) {  // the factors fit in shared memory (n <= 144)
    static bool init = false;
    if (!init) {
      cudaFuncSetAttribute(k_lu_factor_smem2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
      cudaFuncSetAttribute(k_lu_inverse_col, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
      init = true;
    }
    k_lu_factor_smem2<<<1, 1024, f_smem + (size_t)n * sizeof(int), st>>>(A, n, piv);
    k_lu_inverse_col<<<n, 256, f_smem + 2 * (size_t)n * sizeof(double), st>>>(A, piv, n, X);
  } else {  // blocked in global memory (L2-resident); perm lives in XT until the end
    int* perm = reinterpret_cast<int*>(XT);
    k_iota<<<grid1(n), kBlock, 0, st>>>(perm, n);
    for (int k0 = 0; k0 < n; k0 += kLuB) {
      const int k1 = std::min(n, k0 + kLuB);
      k_lu_panel<<<1, 1024, 0, st>>>(A, n, k0, k1, piv, perm);
      if (k1 < n) {
        k_lu_urows<<<grid1(n - k1, 128), 128, 0, st>>>(A, n, k0, k1, perm);
        k_lu_trail<<<dim3((unsigned)((n - k1 + 31) / 32), (unsigned)((n - k1 + 7) / 8)), dim3(32, 8), 0, st>>>(
            A, n, k0, k1, perm);
      }
      g_launches.fetch_add(3, std::memory_order_relaxed);
    }
    k_lu_permute<<<grid1((long long)n * n), kBlock, 0, st>>>(A, n, perm, X);   // X: the factors, rows interchanged
    k_transpose<<<grid1((long long)n * n), kBlock, 0, st>>>(X, n, A);         // A: the factors transposed
    k_lu_inverse_colT<<<n, 256, 2 * (size_t)n * sizeof(double), st>>>(A, piv, n, X);
    g_launches.fetch_add(4, std::memory_order_relaxed);
  }
  k_transpose<<<grid1((long long)n * n), kBlock, 0, st>>>(X, n, XT);
}

void launch_fill(double* x, long long n, double v, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (n > 0) launch_early(k_fill, grid1(n), kBlock, 0, st, x, n, v);
}
void launch_copy(const double* x, double* y, long long n, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (n > 0) launch_early(k_copy, grid1(n), kBlock, 0, st, x, y, n);
}
void launch_axpy(double alpha, const double* sc, int aslot, const double* x, double* y, long long n,
                 cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (n > 0) launch_early(k_axpy, grid1(n), kBlock, 0, st, alpha, sc, aslot, x, y, n);
}
void launch_dot(const double* x, const double* y, long long n, const Reduce& R, cudaStream_t st) {
  launch_dot_b(x, y, n, 0, 1, R, st);
}
void launch_dot_b(const double* x, const double* y, long long n, long long vs, int nb, const Reduce& R,
                  cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const dim3 g(nchunks(n), (unsigned)nb);
  if (g.x * g.y <= kDotWave) launch_early(k_dot<4, 4>, g, kBlock, 0, st, x, y, n, R, vs);
  else launch_early(k_dot<2, 8>, g, kBlock, 0, st, x, y, n, R, vs);
}
void launch_cg_update(const double* sc, double* x, const double* p, double* r, const double* a, double* w,
                      double* w2, double* q, long long n, const Reduce& R, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_cg_update, nchunks(n), kBlock, 0, st, sc, x, p, r, a, w, w2, q, n, R, 0, nullptr);
}
void launch_p_update(const double* sc, double* p, const double* q, long long n, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_p_update, grid1(n), kBlock, 0, st, sc, p, q, n, 0, nullptr);
}
void launch_cg_update_b(const double* sc, double* x, const double* p, double* r, const double* a, double* w,
                        double* w2, double* q, long long n, long long vs, int nb, const double* frozen,
                        const Reduce& R, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_cg_update, dim3(nchunks(n), (unsigned)nb), kBlock, 0, st, sc, x, p, r, a, w, w2, q, n, R, vs, frozen);
}
void launch_p_update_b(const double* sc, double* p, const double* q, long long n, long long vs, int nb,
                       const double* frozen, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_p_update, dim3(grid1(n), (unsigned)nb), kBlock, 0, st, sc, p, q, n, vs, frozen);
}

void launch_sample_kq(int dim, long long ncells_l, long long n_l, long long n_top, double ratio, int np,
                      const double* xi, const double* kcell, double* kq, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  long long nq = 1;
  for (int k = 0; k < dim; ++k) nq *= np;
  const unsigned g = grid1(ncells_l * nq);
  if (dim == 1) k_sample_kq<1><<<g, kBlock, 0, st>>>(ncells_l, n_l, n_top, ratio, np, xi, kcell, kq);
  else if (dim == 2) k_sample_kq<2><<<g, kBlock, 0, st>>>(ncells_l, n_l, n_top, ratio, np, xi, kcell, kq);
  else k_sample_kq<3><<<g, kBlock, 0, st>>>(ncells_l, n_l, n_top, ratio, np, xi, kcell, kq);
}

bool assemble_splits(int dim, int order, int nc, const AsmArgs& a) {
  return nc == 1 && dim == 3 && order == 1 && a.nl == 8 && a.nq == 8 && a.M < (1 << 20);
}

void launch_assemble(int dim, int order, const AsmArgs& a, const double* kbar_h, const double* ctab_h,
                     cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (a.nc == 3) {  // elasticity: a.Kbar / a.Ctab hold the elastic tables
    if (order == 2) k_assemble3<2><<<grid1(a.N), kBlock, 0, st>>>(a);
    else k_assemble3<1><<<grid1(a.N), kBlock, 0, st>>>(a);
    return;
  }
  if (dim == 3 && order == 1 && a.nl == 8 && a.nq == 8 && kbar_h && ctab_h && a.M < (1 << 20)) {
    Q1Tab tab;
    std::memcpy(tab.K, kbar_h, sizeof tab.K);
    std::memcpy(tab.C, ctab_h, sizeof tab.C);
    if (a.kq) k_assemble_q1_3d<true><<<grid1(a.N), kBlock, 0, st>>>(a, tab);
    else k_assemble_q1_3d<false><<<grid1(a.N), kBlock, 0, st>>>(a, tab);
    return;
  }
  const Q2Layout lay = q2_layout(dim, a.M);
  FMG_DISPATCH(dim, order, { k_assemble<D, P><<<grid1(a.N), kBlock, 0, st>>>(a, lay); });
}

}  // namespace fmg

namespace fmg {

// dense row-major copy of a (small) level matrix, for the coarse LU
template <int D, int P>
__global__ void k_densify(const double* __restrict__ A, long long N, long long Np, long long M,
                          double* __restrict__ Dm, const __grid_constant__ Q2Layout lay) {
  constexpr int NS = St<D, P>::NS;
  constexpr int W = 2 * P + 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * NS) return;
  const long long i = t / NS;
  const int s = (int)(t % NS);
  long long ci[3];
  node_coords(i, M, D, ci);
  const long long o[3] = {s % W - P, D > 1 ? (s / W) % W - P : 0, D > 2 ? (s / (W * W)) % W - P : 0};
  long long cj[3];
  for (int k = 0; k < 3; ++k) cj[k] = ci[k] + o[k];
  for (int k = 0; k < D; ++k) if (cj[k] < 0 || cj[k] >= M) return;
  const long long j = cj[0] + M * (cj[1] + M * cj[2]);
  long long p = i;
  if constexpr (P == 2) {  // colour-major sliced storage
    const int r = q2_pattern<D>(s);
    for (int k = 0; k < D; ++k)
      if (((r >> k) & 1) && (ci[k] & 1)) return;
    p = q2c_pos<D>(lay, ci, M, r);
  }
  Dm[i * N + j] = A[(long long)s * Np + p];
}

void launch_level_to_f32(const LevelView& L, int nslots, float* out, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const long long n = (long long)nslots * L.N;
  const Q2Layout lay = q2_layout(L.dim, L.M);
  Q1_DISPATCH(L.dim, { k_expand_q2_f32<D><<<grid1(n), kBlock, 0, st>>>(L.A, L.N, L.Np, L.M, nslots, out, lay); });
}

void launch_galerkin(const LevelView& F, const LevelView& Cl, double* AC, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const Q2Layout lf = q2_layout(F.dim, F.M), lc = q2_layout(Cl.dim, Cl.M);
  const int ns = F.order == 1 ? (F.dim == 1 ? 3 : F.dim == 2 ? 9 : 27) : (F.dim == 1 ? 5 : F.dim == 2 ? 25 : 125);
  const unsigned g = grid1((long long)ns * Cl.N);
  const int mf = (int)F.M, mc = (int)Cl.M;
  if (F.nc == 3) {
    if (F.order == 2) k_galerkin<3, 2, 3><<<g, kBlock, 0, st>>>(F.A, F.Np, mf, AC, Cl.N, Cl.Np, mc, F.dmask, lf, lc);
    else k_galerkin<3, 1, 3><<<g, kBlock, 0, st>>>(F.A, F.Np, mf, AC, Cl.N, Cl.Np, mc, F.dmask, lf, lc);
    return;
  }
  if (F.order == 2) {
    Q1_DISPATCH(F.dim, { k_galerkin<D, 2, 1><<<g, kBlock, 0, st>>>(F.A, F.Np, mf, AC, Cl.N, Cl.Np, mc, F.dmask, lf, lc); });
  } else {
    Q1_DISPATCH(F.dim, { k_galerkin<D, 1, 1><<<g, kBlock, 0, st>>>(F.A, F.Np, mf, AC, Cl.N, Cl.Np, mc, F.dmask, lf, lc); });
  }
}

void launch_bdiag3(const LevelView& L, int mode, const double* w, const double* x, double* y, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_bdiag3, grid1(L.N), kBlock, 0, st, L.A, L.N, L.Np, L.center, mode, w, x, y);
}
void launch_xpwv3(const double* x, const double* w, const double* v, double* y, long long N, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_xpwv3, grid1(N), kBlock, 0, st, x, w, v, y, N);
}
void launch_acc_prod3(double* acc, const double* a, const double* b, long long N, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_acc_prod3, grid1(N), kBlock, 0, st, acc, a, b, N);
}

void vec32_spmv(int order, const float* A, long long N, long long Np, long long M, const float* x, const float* b,
                float* y, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_row3<float, ROW3_RES>(order, A, N, Np, M, 0.0, nullptr, x, b, y, nullptr, false, st);
}
void vec32_jacobi0(const float* A, long long N, long long Np, int center, float damp, const double* omega,
                   const float* b, float* x, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_pdl(k_jacobi0_3<float>, grid1(N), kBlock, 0, st, A, N, Np, center, damp, omega, b, x);
}
void vec32_jacobi_res(int order, const float* A, long long N, long long Np, long long M, double damp,
                      const double* omega, const float* x, const float* b, float* xout, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_row3<float, ROW3_JACOBI>(order, A, N, Np, M, damp, omega, x, b, xout, (float*)nullptr, false, st);
}
void vec32_restrict(int order, long long MC, long long MF, int dmask, const float* rf, float* bc, float* xc,
                    cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_restrict3<float>(order, MC, MF, dmask, rf, bc, bc, xc, st);
}
void vec32_prolong(int order, long long MF, long long MC, int dmask, const float* xc, float* xf, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_prolong3<float>(order, MF, MC, dmask, xc, xf, st);
}
void vec_to32(const double* x, const double* sc, int slot, int mode, float* y, long long n, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_pdl(k_vscale<double, float>, grid1(n), kBlock, 0, st, x, sc, slot, mode, y, n);
}
void vec_to64(const float* x, const double* sc, int slot, int mode, double* y, long long n, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_pdl(k_vscale<float, double>, grid1(n), kBlock, 0, st, x, sc, slot, mode, y, n);
}
void vec_f64_to_f32(const double* x, float* y, long long n, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_pdl(k_vscale<double, float>, grid1(n), kBlock, 0, st, x, nullptr, 0, 0, y, n);
}
void launch_fcg_beta(double* sc, bool first, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  launch_early(k_fcg_beta, 1, 1, 0, st, sc, first ? 1 : 0);
}

long long q2_slot_pos(int dim, long long M, long long i, int s, bool colour_major) {
  const long long c[3] = {i % M, dim > 1 ? (i / M) % M : 0, dim > 2 ? i / (M * M) : 0};
  if (colour_major) {
    const Q2Layout lay = q2_layout(dim, M);
    int r = 0, t = s;
    for (int k = 0; k < dim; ++k) {
      const int o = t % 5 - 2;
      if (o == 2 || o == -2) {
        if (c[k] & 1) return -1;
        r |= 1 << k;
      }
      t /= 5;
    }
    if (dim == 3) return q2c_pos<3>(lay, c, M, r);
    if (dim == 2) return q2c_pos<2>(lay, c, M, r);
    return q2c_pos<1>(lay, c, M, r);
  }
  if (dim == 3) {
    Q2Rows<3> q;
    q2_rows<3>(c, M, q);
    const int r = q2_pattern<3>(s);
    return ((q.valid >> r) & 1) ? q.idx[r] : -1;
  }
  if (dim == 2) {
    Q2Rows<2> q;
    q2_rows<2>(c, M, q);
    const int r = q2_pattern<2>(s);
    return ((q.valid >> r) & 1) ? q.idx[r] : -1;
  }
  Q2Rows<1> q;
  q2_rows<1>(c, M, q);
  const int r = q2_pattern<1>(s);
  return ((q.valid >> r) & 1) ? q.idx[r] : -1;
}

void launch_densify(const LevelView& L, double* Dm, cudaStream_t st) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (L.csr) {
    k_csr_densify<<<grid1(L.N), kBlock, 0, st>>>(L.N, L.a, Dm);
    return;
  }
  if (L.nc == 3) {
    if (L.order == 2) k_densify3<2><<<grid1(L.N * St<3, 2>::NS), kBlock, 0, st>>>(L.A, L.N, L.Np, L.M, Dm);
    else k_densify3<1><<<grid1(L.N * St<3, 1>::NS), kBlock, 0, st>>>(L.A, L.N, L.Np, L.M, Dm);
    return;
  }
  const Q2Layout lay = q2_layout(L.dim, L.M);
  FMG_DISPATCH(L.dim, L.order, {
    constexpr int NS = St<D, P>::NS;
    k_densify<D, P><<<grid1(L.N * NS), kBlock, 0, st>>>(L.A, L.N, L.Np, L.M, Dm, lay);
  });
}

// ------------------------------------------------------------ small levels
long long tail_need(const LevelView& L) {  // the matrix and four vectors
  long long ns = 0;
  if (!L.csr) {
    ns = 1;
    for (int k = 0; k < L.dim; ++k) ns *= 3;
  }
  return (ns + 4) * L.N;
}

// One CTA has 208 KB for the levels, half of it used in 3D: the only levels
// that fit the whole and not the half are 9^3 and 5^3 nodes together (183 KB),
// and a cycle takes few steps there for the matrices it brings in.  A cycle
// with the half and the whole, us: Jacobi V(1,1) of 32^3 cells 57 and 48, 64^3
// 75 and 79, 128^3 292 and 296, 256^3 1,876 and 1,881; SOR V(1,1) 145 and 127,
// 229 and 216, 765 and 749, 4,540 and 4,535; a 128^3-cell CG solve 8.0 and 8.3
// ms.  A CTA has an SM to itself (512 threads of 96 registers), so the problems
// of a batch of more than 148 take turns, and what they bring into the launch
// is done once per turn: the room is divided by the turns, and the levels left
// out run in launches over the whole batch.  Ten CG steps with the room divided
// and whole, us: 32^2 cells x 149 845 and 879, x 297 1,054 and 1,122; 64^2 x 160
// 1,371 and 1,386, x 400 2,546 and 2,572; 128^2 x 297 5,749 and 5,846.
long long tail_room(int dim, int nb) { return (dim == 3 ? 104 : 208) * 1024 / 8 / ((nb + 147) / 148); }

template <int CAP>
static void tail_launch(const Tail& t, cudaStream_t st) {
  TailArgs<CAP> a;
  a.dmask = t.dmask; a.nbase = t.nbase; a.nops = t.nops; a.nlev = t.nlev; a.nvec = t.nvec;
  a.ainv = t.ainv;
  std::memcpy(a.lev, t.lev, t.nlev * sizeof(TailLevel));
  std::memcpy(a.vec, t.vec, t.nvec * sizeof(TailVec));
  std::memcpy(a.ops, t.ops, t.nops * sizeof(TailOp));
  const size_t smem = t.used * sizeof(double);
  auto go = [&](auto kern) {
    if (smem > 32 * 1024)
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(tail_room(2, 1) * sizeof(double)));
    launch_early(kern, (unsigned)t.nb, kTailT, smem, st, a);
  };
  if (t.csr) go(k_tail<1, true, CAP>);
  else if (t.dim == 1) go(k_tail<1, false, CAP>);
  else if (t.dim == 2) go(k_tail<2, false, CAP>);
  else go(k_tail<3, false, CAP>);
}

void tail_flush(Tail& t, cudaStream_t st, bool leaving) {
  if (!t.nops) return;
  if (leaving) {
    int high = 0;
    for (int k = 1; k < t.nlev; ++k)
      if (t.levid[k] > t.levid[high]) high = k;
    for (int q = 0; q < t.nvec; ++q) t.vec[q].out = t.vec[q].out && t.vec[q].lev == high;
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (t.nops <= 48) tail_launch<48>(t, st);
  else tail_launch<Tail::kOps>(t, st);
  t.nops = t.nlev = t.nvec = t.used = 0;
}

// the table entry of grid level l
static int tail_entry(Tail& t, int l, const LevelView& L) {
  for (int k = 0; k < t.nlev; ++k)
    if (t.levid[k] == l) return k;
  const int k = t.nlev++;
  t.levid[k] = l;
  TailLevel& e = t.lev[k];
  e.A = L.A; e.omega = L.omega; e.Np = L.Np; e.N = (int)L.N; e.M = (int)L.M;
  e.a = L.a; e.p = L.p; e.pt = L.pt; e.diag = L.diag;
  e.aoff = t.used;
  if (!L.csr) t.used += (int)(tail_need(L) - 4 * L.N);
  t.dim = L.dim; t.dmask = L.dmask; t.nb = L.nb; t.csr = L.csr;
  return k;
}

// the place of vector v of table level k; read, written: what the step does
// with it (a step that writes a vector without reading it writes all of it)
static int tail_vec(Tail& t, int k, double* v, bool read, bool written) {
  if (!v) return 0;
  int q = 0;
  while (q < t.nvec && t.vec[q].g != v) ++q;
  if (q == t.nvec) {
    t.vec[t.nvec++] = TailVec{v, t.used, k, read, false};
    t.used += t.lev[k].N;
  }
  t.vec[q].out = t.vec[q].out || written;
  return t.vec[q].off;
}

static bool tail_full(const Tail& t) {  // a step adds one operation, two levels and four vectors at most
  return t.nops == Tail::kOps || t.nlev + 2 > Tail::kLev || t.nvec + 4 > Tail::kVec;
}

void tail_add(Tail& t, int l, const LevelView& L, const TailStep& s, cudaStream_t st, const LevelView* C) {
  if (tail_full(t)) tail_flush(t, st, false);
  TailOp op{};
  op.kind = (short)s.kind;
  op.flag = s.write_r ? 1 : 0;
  op.w = s.w;
  const int k = tail_entry(t, l, L), c = C ? tail_entry(t, l - 1, *C) : k;
  op.lev = (short)k;
  op.clev = (short)c;
  // what each step reads (in) and writes (out) of x, y, r, b
  bool xi = true, xo = false, yi = false, yo = false, ri = false, ro = false, bi = false, bo = false;
  int kx = k, ky = k, kr = k, kb = k;
  switch (s.kind) {
    case TAIL_RES: bi = true; ro = true; break;
    case TAIL_JACOBI: xo = true; ri = true; ro = s.write_r; break;
    case TAIL_JACOBI_RES: bi = true; yo = true; ro = s.write_r; break;
    case TAIL_RESTRICT: ky = kr = kb = c; yo = ro = bo = true; break;
    case TAIL_PROLONG: kx = c; yi = yo = true; break;
    default: xo = true; ri = ro = true;  // TAIL_COARSE
  }
  op.b = tail_vec(t, kb, bi || bo ? s.b : nullptr, bi, bo);
  op.x = tail_vec(t, kx, s.x, xi, xo);
  op.y = tail_vec(t, ky, yi || yo ? s.y : nullptr, yi, yo);
  op.r = tail_vec(t, kr, ri || ro ? s.r : nullptr, ri, ro);
  op.n = s.kind == TAIL_COARSE ? 128 : (int)(s.kind == TAIL_RESTRICT ? C->N : L.N);
  t.ops[t.nops++] = op;
}

void tail_sweep(Tail& t, int l, const LevelView& L, bool ssc, double omega, double* x, double* b, double* r,
                cudaStream_t st) {
  const int ncol = L.csr ? L.ncol : 1 << L.dim;
  for (int c = 0; c < ncol; ++c) {
    if (L.csr && L.coff[c + 1] == L.coff[c]) continue;
    if (tail_full(t)) tail_flush(t, st, false);
    TailOp op{};
    op.kind = ssc ? TAIL_SSC : TAIL_SOR;
    op.flag = (short)c;
    op.w = omega;
    op.lev = (short)tail_entry(t, l, L);
    op.b = tail_vec(t, op.lev, b, true, false);
    op.x = tail_vec(t, op.lev, x, true, true);
    op.r = tail_vec(t, op.lev, r, true, true);  // a colour writes its own rows only
    if (L.csr) {
      op.n = (int)(L.coff[c + 1] - L.coff[c]);
      op.rows = L.crow + L.coff[c];
    } else {
      op.n = 1;
      for (int k = 0; k < L.dim; ++k) op.n *= ((int)L.M - ((c >> k) & 1) + 1) / 2;
    }
    t.ops[t.nops++] = op;
  }
}

}  // namespace fmg
