// Cell residual kernels for the 2D / 3D Euler equations (PGLDA / PGN / PGB): a group of G
// lanes of one warp works on one cell.
//
// The reference's per-cell work (src/solver/rdm/cellsplitters/PGLDA.hpp:171-310,
// PGN.hpp:154-289, PGB.hpp:314-498 with the metrics of src/interpolation/*Metric.hpp) is split
// over the group as follows:
//   A  stage the cell's nodal states (ndof x neq, FP64) in shared memory;
//   B  flux nodes f = lane, lane + G, ...: S_f = Vsf u; V, rho (or invJ^T rho V on cells of
//      constant Jacobian), p, H there                                     -> shared memory;
//   C  quadrature points q = lane, lane + G, ...: the flux divergence r_q, in registers, then in
//      the place of the flux nodes' values;
//   then for the points in chunks of G, one point per lane:
//   D1 u_q = V u, the upwind matrices of all nodes, summed, and one solve with the sum (FP64)
//      v = (sum K+)^-1 r_q and u_bar - u_0 = (sum K+)^-1 sum_m K+_m (u_m - u_0); the point's
//      record (V, a, H, v, u_bar, ...)                                    -> shared memory;
//   D2 nodes n = lane, lane + G, ...: for every point of the chunk K+_n again, applied:
//      lda_n += w_q |J_q| K+_n v  and  diss_n += w_q |J_q| K+_n (u_n - u_bar)
//      (= sum_{m != n} K+_n (sum K+)^-1 K+_m (u_n - u_m), the reference's N dissipation; PGN,
//      whose residual is the sum of the two, applies K+_n to v + u_n - u_bar once);
//   E  PGB blending theta = |Phi_0| / (sum_n |lda_n0 + diss_n0| + 1e-6) with a group sum,
//      nodal residuals to the contribution slots, cell wave speed |K| max lambda.
//
// The upwind matrices are used in the symmetrising variables of the point's state,
//   y = (dp / a, rho dV, drho - dp / a^2),   du = M y,  y = M^-1 du,
// in which the flux Jacobian in direction g = |g| n is symmetric and the entropy component is
// decoupled: M^-1 K+ M = oc I + s (e0 e0^T + n n^T) + d (e0 n^T + n e0^T) on (y_0, y_V), oc on
// the entropy, with lambda_c = |g| V.n, lambda_+- = |g| (V.n +- a), p = max(0, lambda_+) / 2,
// m = max(0, lambda_-) / 2, oc = max(0, lambda_c), s = p + m - oc, d = p - m: the product
// R max(0, Lambda) L of Euler2DCons.hpp:316-536 / Euler3DCons.hpp:332-560 for |n| = 1. (In 2D the
// reference leaves n = g below |g| = 1e-9, where the two differ by oc (1 - |n|^2) on the velocity's
// diagonal: at most |g|^2 |V|, 1e-18 of a node's usual K+.) A node's part of sum K+ costs 9 FP64 operations in 2D (14 in 3D) after its eigenvalues instead of the 36
// (55) of two full rank-one terms with their factors, and the sum is solved as a symmetric
// positive definite 3 x 3 (4 x 4) system and a scalar instead of a general 4 x 4 (5 x 5) one.
// What bounds them: the FP64 pipe (B200, ncu: 61 % busy on the P2 tetrahedra, the issue slots 52 %,
// the shared-memory pipe 56 %); the rest is the latency of the FP64 chains at 12-16 warps per SM.
// Measured, cell kernels of a sweep, against the form with general matrices in conservative
// variables and one launch per 32-96 cells a block: 62,500 P3 cells (half triangles, half bilinear
// quadrilaterals, 25 points), PGB, 614 -> 326 us; 98,304 P2 tetrahedra, PGLDA, 579 -> 214 us;
// 18,300 P2 triangles, PGN, 41 -> 21 us.
// T is the arithmetic type of B, C and the eigenvalues; M, the sums, the solves and all
// accumulations are FP64 in both precisions (so sum_n K+_n v = r_q holds to FP64 rounding).

#include "rds_internal.h"
#include "rds_math.cuh"
#include "rds_per_device.h"
#include "rds_physics.cuh"

namespace rds
{

namespace
{

template <int G>
__device__ __forceinline__ double group_sum(double v)
{
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int G>
__device__ __forceinline__ double group_max(double v)
{
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of upwind matrices in the symmetrising variables: the acoustic block (y_0, y_V),
// symmetric, and oc on the entropy.
template <int D>
struct SymSum
{
  double oc, s00, s0[D], sv[D * (D + 1) / 2]; // sv: xx, xy, yy (2D), xx, xy, xz, yy, yz, zz (3D)
};

// x := A^-1 x for one or two right-hand sides, A = the acoustic block of the sum (oc on the
// diagonal included here), symmetric positive definite: block elimination with 2 x 2 leading
// (3D: and trailing) blocks by their closed-form inverses, no pivoting needed.
template <int D, bool TWO>
__device__ __forceinline__ void sym_solve(const SymSum<D> &k, double *x, double *z)
{
  const double p00 = k.oc + k.s00, p01 = k.s0[0], p11 = k.oc + k.sv[0];
  const double ip  = rcp_fast(p00 * p11 - p01 * p01);
  const double i00 = p11 * ip, i01 = -p01 * ip, i11 = p00 * ip;
  if constexpr (D == 2)
  {
    // rows 0, 1 eliminated: one remaining row (y_Vy)
    const double q0 = k.s0[1], q1 = k.sv[1];
    const double z0 = i00 * q0 + i01 * q1, z1 = i01 * q0 + i11 * q1;
    const double is = rcp_fast((k.oc + k.sv[2]) - (q0 * z0 + q1 * z1));
    auto solve      = [&](double *b) {
      const double b2 = (b[2] - (z0 * b[0] + z1 * b[1])) * is;
      const double b0 = i00 * b[0] + i01 * b[1] - z0 * b2;
      const double b1 = i01 * b[0] + i11 * b[1] - z1 * b2;
      b[0]            = b0;
      b[1]            = b1;
      b[2]            = b2;
    };
    solve(x);
    if (TWO)
      solve(z);
  }
  else
  {
    const double q00 = k.s0[1], q01 = k.s0[D - 1], q10 = k.sv[1], q11 = k.sv[2];
    const double z00 = i00 * q00 + i01 * q10, z01 = i00 * q01 + i01 * q11;
    const double z10 = i01 * q00 + i11 * q10, z11 = i01 * q01 + i11 * q11;
    const double t00 = (k.oc + k.sv[3]) - (q00 * z00 + q10 * z10);
    const double t01 = k.sv[4 % (D * (D + 1) / 2)] - (q00 * z01 + q10 * z11);
    const double t11 = (k.oc + k.sv[5 % (D * (D + 1) / 2)]) - (q01 * z01 + q11 * z11);
    const double it  = rcp_fast(t00 * t11 - t01 * t01);
    auto solve       = [&](double *b) {
      const double c0 = b[2] - (z00 * b[0] + z10 * b[1]);
      const double c1 = b[3] - (z01 * b[0] + z11 * b[1]);
      const double b2 = (t11 * c0 - t01 * c1) * it, b3 = (t00 * c1 - t01 * c0) * it;
      const double b0 = i00 * b[0] + i01 * b[1] - (z00 * b2 + z01 * b3);
      const double b1 = i01 * b[0] + i11 * b[1] - (z10 * b2 + z11 * b3);
      b[0]            = b0;
      b[1]            = b1;
      b[2]            = b2;
      b[3]            = b3;
    };
    solve(x);
    if (TWO)
      solve(z);
  }
}

// 1 / sqrt(x), zero for x below the smallest normal number.
__device__ __forceinline__ double rsqrt_pos(double x)
{
  const double y = rsqrt_fast(x);
  return __double2hiint(x) >= 0x00100000 ? y : 0.0;
}
__device__ __forceinline__ float rsqrt_pos(float x) { return x > 0.f ? rsqrtf(x) : 0.f; }

// The three numbers of K+ in direction g and its unit normal; returns max_k |lambda_k|.
template <typename T, int D>
struct UpwindK
{
  T oc, s, d, um, n[D];
};

template <typename T, int D>
__device__ __forceinline__ T upwind_k(const T *V, T a, const T *g, UpwindK<T, D> &k)
{
  T n2 = g[0] * g[0] + g[1] * g[1];
  if (D == 3)
    n2 = n2 + g[D - 1] * g[D - 1];
  // |g| and 1 / |g| from one reciprocal square root
  const T rn   = rsqrt_pos(n2);
  const T norm = n2 * rn;
  // the reference keeps g unnormalised below |g| = 1e-9 (2D) or at |g| = 0 (3D)
  const bool keep = (D == 2) ? less_pos(norm, T(1.e-9)) : !less_pos(T(0), norm);
  const T inv_n   = keep ? T(1) : rn;
#pragma unroll
  for (int x = 0; x < D; ++x)
    k.n[x] = g[x] * inv_n;
  T um = V[0] * k.n[0] + V[1] * k.n[1];
  if (D == 3)
    um = um + V[D - 1] * k.n[D - 1];
  k.um        = um;
  const T lc  = norm * um, an = norm * a;
  const T lp  = lc + an, lm = lc - an;
  const T p   = pos_part(lp);
  const T m   = pos_part(lm);
  k.oc        = pos_part(lc);
  k.s         = T(0.5) * (p + m) - k.oc;
  k.d         = T(0.5) * (p - m);
  return fabs(lc) + an;
}

// Inverse Jacobian and determinant at quadrature point q from the geometry nodes; dvg
// [D][NGEO][NQ] (lane-indexed table).
template <typename T, int D, int NQ, int NGEO>
__device__ __forceinline__ T jacobian_lt(const T *dvg, int q, const T (&X)[NGEO][D],
                                         T (&ij)[D][D])
{
  T J[D][D];
#pragma unroll
  for (int xi = 0; xi < D; ++xi)
  {
    const T c = dvg[(xi * NGEO) * NQ + q];
#pragma unroll
    for (int x = 0; x < D; ++x)
      J[xi][x] = c * X[0][x];
#pragma unroll
    for (int g = 1; g < NGEO; ++g)
    {
      const T cg = dvg[(xi * NGEO + g) * NQ + q];
#pragma unroll
      for (int x = 0; x < D; ++x)
        J[xi][x] = J[xi][x] + cg * X[g][x];
    }
  }
  if constexpr (D == 2)
  {
    const T det     = J[0][0] * J[1][1] - J[0][1] * J[1][0];
    const T inv_det = rcp_fast(det);
    ij[0][0]        = inv_det * J[1][1];
    ij[1][1]        = inv_det * J[0][0];
    ij[0][1]        = -inv_det * J[0][1];
    ij[1][0]        = -inv_det * J[1][0];
    return det;
  }
  else
  {
    const T c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
    const T c01 = J[1][0] * J[2][2] - J[1][2] * J[2][0];
    const T c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    const T det = J[0][0] * c00 - J[0][1] * c01 + J[0][2] * c02;
    const T inv = rcp_fast(det);
    ij[0][0]    = c00 * inv;
    ij[0][1]    = -(J[0][1] * J[2][2] - J[0][2] * J[2][1]) * inv;
    ij[0][2]    = (J[0][1] * J[1][2] - J[1][1] * J[0][2]) * inv;
    ij[1][0]    = -c01 * inv;
    ij[1][1]    = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * inv;
    ij[1][2]    = -(J[0][0] * J[1][2] - J[0][2] * J[1][0]) * inv;
    ij[2][0]    = c02 * inv;
    ij[2][1]    = -(J[0][0] * J[2][1] - J[0][1] * J[2][0]) * inv;
    ij[2][2]    = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * inv;
    return det;
  }
}

// Lane-indexed copy of a cell group's tables, staged in shared memory by every block: the entries
// that the lanes of a warp read at different points (phases C, D1), flux nodes (B) or nodes (D2),
// each laid out with that index fastest, so that a warp reads one row of banks (the constant bank
// serialises reads at different addresses, and beside the cells' regions L1 is too small to keep
// the 12-31 KB: the tetrahedra took 349 us with the tables read from global memory, 273 us so).
// Offsets in elements; euler_lane_tables fills it.
template <int D, int NDOF, int NQ, int NFL, int NGEO>
struct LaneTab
{
  static constexpr int VSF  = 0;                   // Vsf [NDOF][NFL]
  static constexpr int V    = VSF + NDOF * NFL;    // V [NDOF][NQ]
  static constexpr int DVF  = V + NDOF * NQ;       // dVf [D][NFL][NQ]
  static constexpr int DVG  = DVF + D * NFL * NQ;  // dVgeo [D][NGEO][NQ]
  static constexpr int DVQ  = DVG + D * NGEO * NQ; // dV [D][NDOF][NQ] (lanes over points)
  static constexpr int DVN  = DVQ + D * NDOF * NQ; // dV [D][NQ][NDOF] (lanes over nodes)
  static constexpr int W    = DVN + D * NQ * NDOF; // w [NQ]
  static constexpr int SIZE = W + NQ;
};

// What D1 leaves for D2 at a point (FP64): the state's V, a, 1/a and H, (gamma - 1)/a and |V|^2/2
// for the N part, v in both variables (LDA part; PGLDA: times w |J|), u_bar - u_0 (PGN: minus v),
// and the inverse Jacobian and w |J| where they differ from point to point.
template <int D, int SCHEME, bool AFFINE>
struct PointRec
{
  static constexpr bool LDA = SCHEME != RDS_PGN, NPART = SCHEME != RDS_PGLDA;
  static constexpr int VEL = 0, A = D, IA = D + 1, H = D + 2;
  static constexpr int GA = D + 3, KE = D + 4;          // N part
  static constexpr int VY = NPART ? D + 5 : D + 3;      // LDA part: y_0, y_V
  static constexpr int VC = VY + (LDA ? D + 1 : 0);     // and conservative
  static constexpr int UB = VC + (LDA ? D + 2 : 0);     // N part
  static constexpr int IJ = UB + (NPART ? D + 2 : 0);   // !AFFINE
  static constexpr int WJ = IJ + (AFFINE ? 0 : D * D);  // w |J| (N part)
  static constexpr int SIZE = (WJ + (NPART ? 1 : 0)) | 1; // odd: lanes on different banks
};

// Shared-memory footprint per cell: nodal states (FP64), then the flux nodes' values (T, phases
// B-C) in the place where after C the flux divergence of all points (T) and the point records of
// one chunk (FP64) go. The stride is an odd number of doubles, so that the groups of a warp,
// which work on different cells, fall on different banks.
template <typename T, int D, int SCHEME, bool AFFINE, int NDOF, int NQ, int NFL, int G>
struct EulerSmem
{
  static constexpr int doubles(int n) { return (n * (int)sizeof(T) + 7) / 8; }
  static constexpr int NEQ  = D + 2;
  static constexpr int U    = NDOF * NEQ;
  static constexpr int FV   = AFFINE ? 2 * D + 2 : D + 3; // values per flux node
  static constexpr int R    = doubles(NQ * NEQ);
  static constexpr int REC  = G * PointRec<D, SCHEME, AFFINE>::SIZE;
  static constexpr int FL   = doubles(NFL * FV);
  static constexpr int SIZE = (U + (FL > R + REC ? FL : R + REC)) | 1; // doubles
};

template <int PHYS, int SCHEME, typename T, int NDOF, int NQ, int NFL, int NGEO, bool AFFINE,
          int G, int NT>
__global__ void __launch_bounds__(NT, 1) cells_euler(const __grid_constant__ CellArgs a)
{
  constexpr int D   = (PHYS == RDS_EULER3D) ? 3 : 2;
  constexpr int NEQ = D + 2;
  // nodes per lane: FULL rounds of all lanes, and a last round of NDOF % G nodes. Where that is
  // half the lanes (PAIR: 6 or 10 nodes on 4 lanes), the two halves take it at two points at once
  // and add up at the end: 1.5 or 2.5 rounds a point instead of 2 or 3.
  constexpr int NPT  = (NDOF + G - 1) / G;
  constexpr int FULL = NDOF / G;
  constexpr bool PAIR = NDOF % G == G / 2;
  using SM          = EulerSmem<T, D, SCHEME, AFFINE, NDOF, NQ, NFL, G>;
  using LT          = LaneTab<D, NDOF, NQ, NFL, NGEO>;
  using PR          = PointRec<D, SCHEME, AFFINE>;
  constexpr int FV  = SM::FV;
  constexpr int CPB = NT / G; // cells per block
  constexpr int CPW = 32 / G; // cells per warp

  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (*a.stop)
    return;

  const int lane = threadIdx.x % G;
  const int slot = threadIdx.x / G; // cell within the block

  // per-cell shared-memory regions
  double *su   = reinterpret_cast<double *>(smem_raw) + (size_t)slot * SM::SIZE;
  T *sfl       = reinterpret_cast<T *>(su + SM::U);
  T *sr        = sfl;
  double *srec = su + SM::U + SM::R;

  // the tables, once per block
  T *tab = reinterpret_cast<T *>(reinterpret_cast<double *>(smem_raw) + (size_t)CPB * SM::SIZE);
  for (int i = threadIdx.x; i < LT::SIZE; i += NT)
    tab[i] = __ldg(static_cast<const T *>(a.lt) + i);
  __syncthreads();

  // Every warp walks units of CPW cells on its own (no block-wide barrier below), with fixed
  // shares: the last, partial round then falls on all SMs alike. Units from a counter end on the
  // SMs whose warps came first and cost the P3 hybrid mesh 11 us a launch (175 against 164).
  const int nunits = (a.ncells + CPW - 1) / CPW;
#pragma unroll 1
  for (int unit = (threadIdx.x / 32) * gridDim.x + blockIdx.x; unit < nunits;
       unit += gridDim.x * (NT / 32))
  {
  const int c     = unit * CPW + (threadIdx.x % 32) / G;
  const bool live = c < a.ncells;
  const int cc    = live ? c : a.ncells - 1; // dead groups shadow the last cell, write nothing

  // ---- A: nodal states (every index load of the lane is in flight before the first value load)
  T X[NGEO][D];
  {
    int vs[NPT], vg[NGEO];
#pragma unroll
    for (int s = 0; s < NPT; ++s)
    {
      const int n = lane + s * G;
      vs[s]       = NDOF % G == 0 || n < NDOF ? __ldg(a.sol_conn + (size_t)n * a.ncells + cc) : 0;
    }
#pragma unroll
    for (int g = 0; g < NGEO; ++g)
      vg[g] = __ldg(a.geo_conn + (size_t)g * a.ncells + cc);
    double us[NPT][NEQ];
#pragma unroll
    for (int s = 0; s < NPT; ++s)
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        us[s][e] = __ldg(a.u + (size_t)e * a.nnodes + vs[s]);
#pragma unroll
    for (int g = 0; g < NGEO; ++g)
#pragma unroll
      for (int d = 0; d < D; ++d)
        X[g][d] = T(__ldg(a.X + (size_t)d * a.ngeo_nodes + vg[g]));
#pragma unroll
    for (int s = 0; s < NPT; ++s)
    {
      const int n = lane + s * G;
      if (NDOF % G == 0 || n < NDOF)
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
          su[n * NEQ + e] = us[s][e];
    }
  }
  __syncwarp();

  const double gm1 = a.gamma - 1.0;
  bool bad         = false;

  // constant-Jacobian cells (simplices, parallelogram quadrilaterals): one Jacobian for all points
  T ijc[D][D];
  T detc = T(0);
  if (AFFINE)
    detc = jacobian_lt<T, D, NQ, NGEO>(tab + LT::DVG, 0, X, ijc);

  // ---- B: state at the flux nodes: V, p, H and rho, or (constant Jacobian) the contravariant
  // mass flux m_xi = sum_x invJ[x][xi] rho V_x. Table entries are read once each and applied to
  // all equations (every sum keeps its order over the nodes).
#pragma unroll 1
  for (int f = lane; f < NFL; f += G)
  {
    T s[NEQ];
    {
      const T t = tab[LT::VSF + f];
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        s[e] = t * T(su[e]);
    }
#pragma unroll
    for (int n = 1; n < NDOF; ++n)
    {
      const T t = tab[LT::VSF + n * NFL + f];
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        s[e] = s[e] + t * T(su[n * NEQ + e]);
    }
    const T ir = rcp_fast(s[0]);
    T V[D], v2 = T(0);
#pragma unroll
    for (int d = 0; d < D; ++d)
    {
      V[d] = s[1 + d] * ir;
      v2   = v2 + V[d] * V[d];
    }
    const T P = T(gm1) * (s[D + 1] - T(0.5) * s[0] * v2);
    bad |= !(P > T(0));
    T *o = sfl + f * FV;
#pragma unroll
    for (int d = 0; d < D; ++d)
      o[d] = V[d];
    o[D]     = P;
    o[D + 1] = (s[D + 1] + P) * ir;
    if constexpr (AFFINE)
    {
#pragma unroll
      for (int xi = 0; xi < D; ++xi)
      {
        T m = ijc[0][xi] * s[1];
#pragma unroll
        for (int x = 1; x < D; ++x)
          m = m + ijc[x][xi] * s[1 + x];
        o[D + 2 + xi] = m;
      }
    }
    else
      o[D + 2] = s[0];
  }
  __syncwarp();

  // ---- C: flux divergence r_q, CR points per lane at a time (a flux node's values are read
  // once for all of them). With g_f = invJ dVf the physical gradient of the flux basis and
  // mu = rho V . g_f: r = sum_f (mu, V mu + p g_f, H mu); the pressure part is summed in reference
  // directions first.
  constexpr int NR = (NQ + G - 1) / G;          // rounds of the lanes over the points
  constexpr int CR = AFFINE || NR < 2 ? NR : 2; // varying Jacobian: CR of them in registers
  T r[NR][NEQ];
#pragma unroll
  for (int j0 = 0; j0 < NR; j0 += CR)
  {
    T ij[CR][D][D], pr[CR][D];
    int q[CR];
#pragma unroll
    for (int j = 0; j < CR; ++j)
    {
      q[j] = (j0 + j) * G + lane;
      q[j] = q[j] < NQ ? q[j] : NQ - 1; // idle lanes of the last round repeat the last point
      if constexpr (!AFFINE)
        jacobian_lt<T, D, NQ, NGEO>(tab + LT::DVG, q[j], X, ij[j]);
      else
#pragma unroll
        for (int a0 = 0; a0 < D; ++a0)
#pragma unroll
          for (int a1 = 0; a1 < D; ++a1)
            ij[j][a0][a1] = ijc[a0][a1];
#pragma unroll
      for (int d = 0; d < D; ++d)
        pr[j][d] = T(0);
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        if (j0 + j < NR)
          r[j0 + j][e] = T(0);
    }
#pragma unroll 1
    for (int f = 0; f < NFL; ++f)
    {
      T o[FV];
#pragma unroll
      for (int i = 0; i < FV; ++i)
        o[i] = sfl[f * FV + i];
#pragma unroll
      for (int j = 0; j < CR && j0 + j < NR; ++j)
      {
        T(&rj)[NEQ] = r[j0 + j];
        T dv[D];
#pragma unroll
        for (int xi = 0; xi < D; ++xi)
          dv[xi] = tab[LT::DVF + (xi * NFL + f) * NQ + q[j]];
        T mu;
        if constexpr (AFFINE)
        {
          mu = dv[0] * o[D + 2];
#pragma unroll
          for (int xi = 1; xi < D; ++xi)
            mu = mu + dv[xi] * o[D + 2 + xi];
        }
        else
        {
          T vg = T(0);
#pragma unroll
          for (int x = 0; x < D; ++x)
          {
            T g = ij[j][x][0] * dv[0];
#pragma unroll
            for (int xi = 1; xi < D; ++xi)
              g = g + ij[j][x][xi] * dv[xi];
            vg = x == 0 ? g * o[0] : vg + g * o[x];
          }
          mu = o[D + 2] * vg;
        }
        rj[0] = rj[0] + mu;
#pragma unroll
        for (int d = 0; d < D; ++d)
          rj[1 + d] = rj[1 + d] + o[d] * mu;
        rj[D + 1] = rj[D + 1] + o[D + 1] * mu;
#pragma unroll
        for (int xi = 0; xi < D; ++xi)
          pr[j][xi] = pr[j][xi] + dv[xi] * o[D];
      }
    }
#pragma unroll
    for (int j = 0; j < CR && j0 + j < NR; ++j)
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int xi = 0; xi < D; ++xi)
          r[j0 + j][1 + d] = r[j0 + j][1 + d] + ij[j][d][xi] * pr[j][xi];
  }
  __syncwarp(); // the flux nodes' values are read: r and the point records take their place
#pragma unroll
  for (int j = 0; j < NR; ++j)
    if (j * G + lane < NQ)
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        sr[(j * G + lane) * NEQ + e] = r[j][e];

  double lda[NPT][NEQ], diss[NPT][NEQ];
#pragma unroll
  for (int s = 0; s < NPT; ++s)
#pragma unroll
    for (int e = 0; e < NEQ; ++e)
    {
      lda[s][e]  = 0.0;
      diss[s][e] = 0.0;
    }
  double phi0_l = 0.0, vol_l = 0.0; // this lane's points' part of Phi_0 and of |K|
  T wsmax       = T(1.e-6);

#pragma unroll 1
  for (int q0 = 0; q0 < NQ; q0 += G)
  {
    const int q = q0 + lane;
    if (q < NQ)
    {
      T ij[D][D];
      T det;
      if (AFFINE)
      {
        det = detc;
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j)
            ij[i][j] = ijc[i][j];
      }
      else
        det = jacobian_lt<T, D, NQ, NGEO>(tab + LT::DVG, q, X, ij);

      // u_q = V u and the point's state
      T uq[NEQ];
      {
        const T t = tab[LT::V + q];
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
          uq[e] = t * T(su[e]);
      }
#pragma unroll
      for (int n = 1; n < NDOF; ++n)
      {
        const T t = tab[LT::V + n * NQ + q];
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
          uq[e] = uq[e] + t * T(su[n * NEQ + e]);
      }
      // V and a in the arithmetic type; what M is built of in FP64 from their values, so that M
      // and M^-1 belong together in both precisions
      T VT[D], aT;
      double V[D], ke = 0.0, ad, ia;
      {
        const T ir = rcp_fast(uq[0]);
        T v2       = T(0);
#pragma unroll
        for (int d = 0; d < D; ++d)
        {
          VT[d] = uq[1 + d] * ir;
          v2    = v2 + VT[d] * VT[d];
          V[d]  = double(VT[d]);
          ke += V[d] * V[d];
        }
        ke *= 0.5;
        const T P = T(gm1) * (uq[D + 1] - T(0.5) * uq[0] * v2);
        bad |= !(P > T(0));
        const T a2  = T(a.gamma) * (P * ir);
        aT          = sqrt_and_inverse(a2, ia);
        ad          = double(aT);
      }
      const double ga = gm1 * ia;

      // ---- D1: sum K+ and (N part) sum K+ (u - u_0): the solve then acts on the differences of
      // the states (a nearly uniform flow has them 100x smaller than the states), as the
      // reference's K+_m (u_n - u_m)
      SymSum<D> K;
      K.oc = K.s00 = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d)
        K.s0[d] = 0.0;
#pragma unroll
      for (int i = 0; i < D * (D + 1) / 2; ++i)
        K.sv[i] = 0.0;
      double y[D + 1], ys = 0.0; // N part
#pragma unroll
      for (int i = 0; i <= D; ++i)
        y[i] = 0.0;
#pragma unroll 2
      for (int n = 0; n < NDOF; ++n)
      {
        T g[D];
        {
          T dv[D];
#pragma unroll
          for (int xi = 0; xi < D; ++xi)
            dv[xi] = tab[LT::DVQ + (xi * NDOF + n) * NQ + q];
#pragma unroll
          for (int x = 0; x < D; ++x)
          {
            g[x] = ij[x][0] * dv[0];
#pragma unroll
            for (int xi = 1; xi < D; ++xi)
              g[x] = g[x] + ij[x][xi] * dv[xi];
          }
        }
        UpwindK<T, D> k;
        wsmax = fmax(wsmax, upwind_k<T, D>(VT, aT, g, k));
        const double oc = double(k.oc), s = double(k.s), dd = double(k.d);
        double nn[D];
#pragma unroll
        for (int d = 0; d < D; ++d)
          nn[d] = double(k.n[d]);
        K.oc += oc;
        K.s00 += s;
        int i = 0;
#pragma unroll
        for (int d = 0; d < D; ++d)
        {
          K.s0[d] += dd * nn[d];
          const double sn = s * nn[d];
#pragma unroll
          for (int e = d; e < D; ++e)
            K.sv[i++] += sn * nn[e];
        }
        if (SCHEME != RDS_PGLDA)
        {
          const double du0 = su[n * NEQ] - su[0];
          double dp        = (su[n * NEQ + D + 1] - su[D + 1]) + ke * du0;
          double dv[D], beta = 0.0;
#pragma unroll
          for (int d = 0; d < D; ++d)
          {
            const double dm = su[n * NEQ + 1 + d] - su[1 + d];
            dp -= V[d] * dm;
            dv[d] = dm - V[d] * du0;
            beta += nn[d] * dv[d];
          }
          const double y0 = ga * dp;
          const double t  = dd * y0 + s * beta;
          y[0] += (oc + s) * y0 + dd * beta;
#pragma unroll
          for (int d = 0; d < D; ++d)
            y[1 + d] += oc * dv[d] + t * nn[d];
          ys += oc * (du0 - y0 * ia);
        }
      }

      // v: r (this lane's own) in the symmetrising variables, solved; both back in conservative
      // ones
      double r[NEQ];
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        r[e] = double(sr[q * NEQ + e]);
      const double wj = double(tab[LT::W + q] * det);
      vol_l += wj;
      phi0_l += wj * r[0];
      double x[D + 1], dp = r[D + 1] + ke * r[0];
#pragma unroll
      for (int d = 0; d < D; ++d)
      {
        dp -= V[d] * r[1 + d];
        x[1 + d] = r[1 + d] - V[d] * r[0];
      }
      x[0]            = ga * dp;
      const double is = rcp_fast(K.oc);
      double xs       = (r[0] - x[0] * ia) * is;
      ys *= is;
      sym_solve<D, SCHEME != RDS_PGLDA>(K, x, y);
      if (SCHEME == RDS_PGN)
      {
        // PGN: K+_n (v + u_n - u_bar)
#pragma unroll
        for (int i = 0; i <= D; ++i)
          y[i] -= x[i];
        ys -= xs;
      }
      const double aog = ad / gm1; // dE = ke drho + V . y_V + a / (gamma - 1) y_0
      auto to_cons     = [&](const double *z, double zs, double *o) {
        const double rho = z[0] * ia + zs;
        double E         = ke * rho + aog * z[0];
        o[0]             = rho;
#pragma unroll
        for (int d = 0; d < D; ++d)
        {
          o[1 + d] = V[d] * rho + z[1 + d];
          E += V[d] * z[1 + d];
        }
        o[D + 1] = E;
      };
      double *rec = srec + lane * PR::SIZE;
#pragma unroll
      for (int d = 0; d < D; ++d)
        rec[PR::VEL + d] = V[d];
      rec[PR::A]  = ad;
      rec[PR::IA] = ia;
      rec[PR::H]  = ke + ad * aog;
      if constexpr (PR::NPART)
      {
        rec[PR::GA] = ga;
        rec[PR::KE] = ke;
        to_cons(y, ys, rec + PR::UB);
      }
      if constexpr (PR::LDA)
      {
        if (SCHEME == RDS_PGLDA)
        {
#pragma unroll
          for (int i = 0; i <= D; ++i)
            x[i] *= wj;
          xs *= wj;
        }
#pragma unroll
        for (int i = 0; i <= D; ++i)
          rec[PR::VY + i] = x[i];
        to_cons(x, xs, rec + PR::VC);
      }
      if constexpr (!AFFINE)
      {
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j)
            rec[PR::IJ + i * D + j] = double(ij[i][j]);
      }
      if constexpr (PR::NPART)
        rec[PR::WJ] = wj;
    }
    __syncwarp();

    // ---- D2: nodes over the lanes, every point of the chunk: node n at the chunk's point k
    auto apply_node = [&](int k, int n, double *lda_n, double *diss_n) {
      const double *rec = srec + k * PR::SIZE;
      T g[D];
      {
        T dv[D];
#pragma unroll
        for (int xi = 0; xi < D; ++xi)
          dv[xi] = tab[LT::DVN + (xi * NQ + q0 + k) * NDOF + n];
#pragma unroll
        for (int x = 0; x < D; ++x)
        {
          g[x] = (AFFINE ? ijc[x][0] : T(rec[PR::IJ + x * D])) * dv[0];
#pragma unroll
          for (int xi = 1; xi < D; ++xi)
            g[x] = g[x] + (AFFINE ? ijc[x][xi] : T(rec[PR::IJ + x * D + xi])) * dv[xi];
        }
      }
      double V[D];
      T VT[D];
#pragma unroll
      for (int d = 0; d < D; ++d)
      {
        V[d]  = rec[PR::VEL + d];
        VT[d] = T(V[d]);
      }
      UpwindK<T, D> kk;
      upwind_k<T, D>(VT, T(rec[PR::A]), g, kk);
      double oc = double(kk.oc), sk = double(kk.s), dk = double(kk.d);
      if (PR::NPART)
      {
        const double wj = rec[PR::WJ];
        oc *= wj;
        sk *= wj;
        dk *= wj;
      }
      double nn[D], um = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d)
      {
        nn[d] = double(kk.n[d]);
        um += V[d] * nn[d];
      }
      if (sizeof(T) == 8)
        um = double(kk.um); // the same sum
      const double ia = rec[PR::IA], H = rec[PR::H];
      // acc += K z, with z_0 and beta = n . z_V of the symmetrising variables and the
      // conservative z:  oc z + (s z_0 + d beta) / a (1, V, H) + (d z_0 + s beta) (0, n, V.n)
      auto apply = [&](double z0, double beta, const double *z, double *acc) {
        const double t1 = (sk * z0 + dk * beta) * ia;
        const double t2 = dk * z0 + sk * beta;
        acc[0] += oc * z[0] + t1;
#pragma unroll
        for (int d = 0; d < D; ++d)
          acc[1 + d] += oc * z[1 + d] + t1 * V[d] + t2 * nn[d];
        acc[D + 1] += oc * z[D + 1] + t1 * H + t2 * um;
      };
      if constexpr (PR::LDA)
      {
        double beta = nn[0] * rec[PR::VY + 1];
#pragma unroll
        for (int d = 1; d < D; ++d)
          beta += nn[d] * rec[PR::VY + 1 + d];
        apply(rec[PR::VY], beta, rec + PR::VC, lda_n);
      }
      if constexpr (PR::NPART)
      {
        double du[NEQ]; // u_n - u_bar = (u_n - u_0) - (u_bar - u_0)
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
          du[e] = (su[n * NEQ + e] - su[e]) - rec[PR::UB + e];
        double dp = du[D + 1] + rec[PR::KE] * du[0], beta = -um * du[0];
#pragma unroll
        for (int d = 0; d < D; ++d)
        {
          dp -= V[d] * du[1 + d];
          beta += nn[d] * du[1 + d];
        }
        apply(rec[PR::GA] * dp, beta, du, diss_n);
      }
    };
    const int nq = NQ - q0 < G ? NQ - q0 : G;
#pragma unroll 1
    for (int k = 0; k < nq; k += PAIR ? 2 : 1)
    {
#pragma unroll
      for (int s = 0; s < FULL; ++s)
        apply_node(k, lane + s * G, lda[s], diss[s]);
      if constexpr (PAIR)
      {
        if (k + 1 < nq)
#pragma unroll
          for (int s = 0; s < FULL; ++s)
            apply_node(k + 1, lane + s * G, lda[s], diss[s]);
        const int kp = k + lane / (G / 2);
        if (kp < nq)
          apply_node(kp, FULL * G + lane % (G / 2), lda[FULL], diss[FULL]);
      }
      else if constexpr (FULL < NPT)
      {
        if (lane + FULL * G < NDOF)
          apply_node(k, lane + FULL * G, lda[FULL], diss[FULL]);
      }
    }
    __syncwarp();
  }
  if constexpr (PAIR)
  {
#pragma unroll
    for (int e = 0; e < NEQ; ++e)
    {
      lda[FULL][e] += __shfl_xor_sync(0xffffffffu, lda[FULL][e], G / 2);
      diss[FULL][e] += __shfl_xor_sync(0xffffffffu, diss[FULL][e], G / 2);
    }
  }
  const double phi0 = group_sum<G>(phi0_l);
  const double vol  = group_sum<G>(vol_l);

  // ---- E: blending, outputs
  double theta = 1.0;
  if (SCHEME == RDS_PGB)
  {
    double part = 0.0;
#pragma unroll
    for (int s = 0; s < NPT; ++s)
      if (lane + s * G < NDOF)
        part += fabs(lda[s][0] + diss[s][0]);
    const double abs_phiN = group_sum<G>(part);
    theta                 = fabs(phi0) / (abs_phiN + 1.e-6);
  }
  const double wmax = group_max<G>(double(wsmax));
  // external nodal blending coefficient: theta_n of the lane's nodes, the N part dropped when
  // all of the cell's are below 1e-6 (PGRDMExplicitCellWorker.hpp:508-517,
  // PGB.hpp:141-148,467-477); the group max runs in every lane of the warp
  double tn[NPT];
  bool skip = false;
  if (SCHEME == RDS_PGB && a.blend)
  {
    double tmax = 0.0;
#pragma unroll
    for (int s = 0; s < NPT; ++s)
    {
      const int n = lane + s * G;
      tn[s]       = (live && n < NDOF) ? __ldg(a.blend + __ldg(a.sol_conn + (size_t)n * a.ncells + c))
                                       : 0.0;
      tmax        = fmax(tmax, tn[s]);
    }
    skip = group_max<G>(tmax) < 1.e-6;
  }
  if (live)
  {
#pragma unroll
    for (int s = 0; s < NPT; ++s)
    {
      const int n = lane + s * G;
      if (n < NDOF)
      {
        const long long slot0 = a.out.slot_base + (long long)n * a.ncells + c;
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
        {
          double r = (SCHEME == RDS_PGLDA)  ? lda[s][e]
                     : (SCHEME == RDS_PGN) ? diss[s][e]
                                           : lda[s][e] + theta * diss[s][e];
          if (SCHEME == RDS_PGB && a.blend)
            r = skip ? lda[s][e] : lda[s][e] + tn[s] * diss[s][e];
          a.out.val[e * a.out.S + slot0] = r; // write-back: the gather reads it from L2
        }
      }
    }
    if (lane == 0)
    {
      a.out.wsc[c] = vol * wmax;
      if (SCHEME == RDS_PGB && a.theta)
        a.theta[c] = theta;
    }
    if (bad)
      atomicOr(a.status, kFlagNegPressure);
  }
  __syncwarp(); // the unit's shared memory is free again
  }
}

// One block per SM with all of its shared memory. Warps: 16 (128 registers a thread) where the
// cells' regions and the tables fit and a lane has at most 12 accumulators, 12 of 168 otherwise,
// fewer where 12 do not fit. Both sides measured, us a launch on B200, 12 warps against 16. More
// accumulators: P3 hybrid mesh, PGB, 165 against 176. At most 12 (24,000 triangles, 16,000
// quadrilaterals): P2 triangles, PGN, 47 against 45; P1, P2 and P3 quadrilaterals, PGN, 25, 44 and
// 115 against 22, 39 and 111; level are P3 triangles, PGN, and P3 quadrilaterals, PGLDA, 25 points
// (95), and with 20 points these take 78 against 80. That holds although some spill at 128
// registers: 116 bytes stored by PGN on P2 quadrilaterals, 272 by PGLDA on P3 quadrilaterals, whose
// lanes keep the sums of 4 points in phase C. NT stays a multiple of 64: 14 warps get the
// registers of 16.
template <typename T, int D, int SCHEME, bool AFFINE, int NDOF, int NQ, int NFL, int NGEO, int G>
struct EulerBlock
{
  static constexpr int PER   = 8 * EulerSmem<T, D, SCHEME, AFFINE, NDOF, NQ, NFL, G>::SIZE;
  static constexpr int TAB   = LaneTab<D, NDOF, NQ, NFL, NGEO>::SIZE * (int)sizeof(T);
  static constexpr int LIMIT = 227 * 1024;
  static constexpr int FIT   = (LIMIT - TAB) / (32 / G * PER); // warps
  // accumulators of a lane in D2
  static constexpr int ACC = (NDOF + G - 1) / G * (D + 2) * (SCHEME == RDS_PGB ? 2 : 1);
  static constexpr int NT  = 32 * (FIT >= 16 && ACC <= 12 ? 16 : FIT >= 12 ? 12 : FIT >= 10 ? 10 : 8);
  static constexpr int BYTES = NT / G * PER + TAB;
  static_assert(BYTES <= LIMIT, "per-block shared memory above the sm_100 limit");
};

template <int PHYS, int SCHEME, typename T, int NDOF, int NQ, int NFL, int NGEO, bool AFFINE, int G>
cudaError_t launch_euler_one(const CellArgs &a, cudaStream_t s)
{
  constexpr int D = (PHYS == RDS_EULER3D) ? 3 : 2;
  using B         = EulerBlock<T, D, SCHEME, AFFINE, NDOF, NQ, NFL, NGEO, G>;
  auto k          = cells_euler<PHYS, SCHEME, T, NDOF, NQ, NFL, NGEO, AFFINE, G, B::NT>;
  // the shared-memory opt-in, once per instantiation and device (not a stream operation, so it
  // also stays out of captured graphs), and the device's SMs
  static PerDevice sms;
  int nsm             = 0;
  const cudaError_t e = sms.get(&nsm, [&](int dev, int *n) {
    const cudaError_t f =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, B::BYTES);
    return f != cudaSuccess ? f : cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev);
  });
  if (e != cudaSuccess)
    return e;
  const int units = (a.ncells + 32 / G - 1) / (32 / G);
  k<<<units < nsm ? units : nsm, B::NT, B::BYTES, s>>>(a);
  return cudaGetLastError();
}

template <int PHYS, int SCHEME, typename T, int NDOF, int NQ, int NFL, int NGEO, int G>
cudaError_t launch_euler(const HostCellGroup &g, const CellArgs &a, cudaStream_t s)
{
  constexpr int D = (PHYS == RDS_EULER3D) ? 3 : 2;
  CellArgs al     = a;
  if constexpr (sizeof(T) == 8)
    al.lt = g.d_lt64;
  else
    al.lt = g.d_lt32;
  if (!al.lt)
    return cudaErrorInvalidValue;
  // straight-sided simplices always have a constant Jacobian
  if constexpr (NGEO == D + 1)
    return launch_euler_one<PHYS, SCHEME, T, NDOF, NQ, NFL, NGEO, true, G>(al, s);
  else
    return g.const_jac ? launch_euler_one<PHYS, SCHEME, T, NDOF, NQ, NFL, NGEO, true, G>(al, s)
                       : launch_euler_one<PHYS, SCHEME, T, NDOF, NQ, NFL, NGEO, false, G>(al, s);
}

template <int PHYS, int SCHEME, typename T>
cudaError_t dispatch_euler(const HostCellGroup &g, const CellArgs &a, cudaStream_t s, bool *ok)
{
  const rds_cell_group &d = g.desc;
  *ok                     = true;
  if constexpr (PHYS == RDS_EULER2D)
  {
    if (d.shape == RDS_TRIAG && d.ngeo == 3)
    {
      if (d.ndof == 3 && d.nq == 6 && d.nfl == 6)
        return launch_euler<PHYS, SCHEME, T, 3, 6, 6, 3, 4>(g, a, s);
      if (d.ndof == 6 && d.nq == 6 && d.nfl == 10)
        return launch_euler<PHYS, SCHEME, T, 6, 6, 10, 3, 4>(g, a, s);
      if (d.ndof == 6 && d.nq == 7 && d.nfl == 10)
        return launch_euler<PHYS, SCHEME, T, 6, 7, 10, 3, 4>(g, a, s);
      if (d.ndof == 10 && d.nq == 12 && d.nfl == 15)
        return launch_euler<PHYS, SCHEME, T, 10, 12, 15, 3, 4>(g, a, s);
      if (d.ndof == 10 && d.nq == 16 && d.nfl == 15)
        return launch_euler<PHYS, SCHEME, T, 10, 16, 15, 3, 4>(g, a, s);
    }
    if (d.shape == RDS_QUAD && d.ngeo == 4)
    {
      // P1 with the 2x2 Gauss rule (orders 2-3), P1 and P2 with the reference's 8-point rule of
      // orders 4-5 or a 3x3 Gauss rule, P3 with the reference's 20-point rule of order 8 or a 5x5
      // Gauss rule
      if (d.ndof == 4 && d.nq == 4 && d.nfl == 9)
        return launch_euler<PHYS, SCHEME, T, 4, 4, 9, 4, 4>(g, a, s);
      if (d.ndof == 4 && d.nq == 8 && d.nfl == 9)
        return launch_euler<PHYS, SCHEME, T, 4, 8, 9, 4, 4>(g, a, s);
      if (d.ndof == 4 && d.nq == 9 && d.nfl == 9)
        return launch_euler<PHYS, SCHEME, T, 4, 9, 9, 4, 4>(g, a, s);
      if (d.ndof == 9 && d.nq == 8 && d.nfl == 16)
        return launch_euler<PHYS, SCHEME, T, 9, 8, 16, 4, 4>(g, a, s);
      if (d.ndof == 9 && d.nq == 9 && d.nfl == 16)
        return launch_euler<PHYS, SCHEME, T, 9, 9, 16, 4, 4>(g, a, s);
      if (d.ndof == 16 && d.nq == 20 && d.nfl == 25)
        return launch_euler<PHYS, SCHEME, T, 16, 20, 25, 4, 8>(g, a, s);
      if (d.ndof == 16 && d.nq == 25 && d.nfl == 25)
        return launch_euler<PHYS, SCHEME, T, 16, 25, 25, 4, 8>(g, a, s);
    }
  }
  else
  {
    if (d.shape == RDS_TETRA && d.ngeo == 4)
    {
      // P1 with the order-2 rule (4 points), P2 with the order-4 (11) and order-5 (14) rules
      if (d.ndof == 4 && d.nq == 4 && d.nfl == 10)
        return launch_euler<PHYS, SCHEME, T, 4, 4, 10, 4, 4>(g, a, s);
      if (d.ndof == 10 && d.nq == 11 && d.nfl == 20)
        return launch_euler<PHYS, SCHEME, T, 10, 11, 20, 4, 4>(g, a, s);
      if (d.ndof == 10 && d.nq == 14 && d.nfl == 20)
        return launch_euler<PHYS, SCHEME, T, 10, 14, 20, 4, 4>(g, a, s);
    }
  }
  *ok = false;
  return cudaSuccess;
}

const char *euler_name(int physics, int scheme)
{
  static const char *names[2][3] = {{"cells_euler2d_lda", "cells_euler2d_n", "cells_euler2d_b"},
                                    {"cells_euler3d_lda", "cells_euler3d_n", "cells_euler3d_b"}};
  return names[physics == RDS_EULER3D ? 1 : 0][scheme];
}

} // namespace

void euler_lane_tables(const HostCellGroup &g, int dim, std::vector<double> &out)
{
  // the layout of LaneTab, with run-time sizes
  const int D = dim, NDOF = g.desc.ndof, NQ = g.desc.nq, NFL = g.desc.nfl, NGEO = g.desc.ngeo;
  out.assign((size_t)NDOF * NFL + (size_t)NDOF * NQ + (size_t)D * NFL * NQ + (size_t)D * NGEO * NQ +
                 2 * (size_t)D * NDOF * NQ + NQ,
             0.0);
  size_t o = 0;
  for (int n = 0; n < NDOF; ++n)
    for (int f = 0; f < NFL; ++f)
      out[o++] = g.Vsf[(size_t)f * NDOF + n];
  for (int n = 0; n < NDOF; ++n)
    for (int q = 0; q < NQ; ++q)
      out[o++] = g.V[(size_t)q * NDOF + n];
  for (int d = 0; d < D; ++d)
    for (int f = 0; f < NFL; ++f)
      for (int q = 0; q < NQ; ++q)
        out[o++] = g.dVf[((size_t)d * NQ + q) * NFL + f];
  for (int d = 0; d < D; ++d)
    for (int k = 0; k < NGEO; ++k)
      for (int q = 0; q < NQ; ++q)
        out[o++] = g.dVgeo[((size_t)d * NQ + q) * NGEO + k];
  for (int d = 0; d < D; ++d)
    for (int n = 0; n < NDOF; ++n)
      for (int q = 0; q < NQ; ++q)
        out[o++] = g.dV[((size_t)d * NQ + q) * NDOF + n];
  for (int d = 0; d < D; ++d)
    for (int q = 0; q < NQ; ++q)
      for (int n = 0; n < NDOF; ++n)
        out[o++] = g.dV[((size_t)d * NQ + q) * NDOF + n];
  for (int q = 0; q < NQ; ++q)
    out[o++] = g.w[q];
}

cudaError_t launch_cells_euler(const HostCellGroup &g, const CellArgs &a, int physics, int scheme,
                               int precision, cudaStream_t s, const char **name, bool *ok)
{
  *name = euler_name(physics, scheme);
#define RDS_EULER_CASE(PH, SC)                                                                     \
  if (physics == PH && scheme == SC)                                                               \
    return precision == RDS_MIXED ? dispatch_euler<PH, SC, float>(g, a, s, ok)                     \
                                  : dispatch_euler<PH, SC, double>(g, a, s, ok);
  RDS_EULER_CASE(RDS_EULER2D, RDS_PGLDA)
  RDS_EULER_CASE(RDS_EULER2D, RDS_PGN)
  RDS_EULER_CASE(RDS_EULER2D, RDS_PGB)
  RDS_EULER_CASE(RDS_EULER3D, RDS_PGLDA)
  RDS_EULER_CASE(RDS_EULER3D, RDS_PGN)
  RDS_EULER_CASE(RDS_EULER3D, RDS_PGB)
#undef RDS_EULER_CASE
  *ok = false;
  return cudaSuccess;
}

} // namespace rds
