// Weak boundary-condition kernels: one thread per boundary facet (scalar physics), or a group of
// lanes, one per quadrature point (Euler).
//
// Per facet quadrature point a ghost flux is formed and distributed to the facet dofs with the
// facet basis, V(q,n) w_q |J_q| (ghost flux), and summed into the facet total; the dof
// residuals are then rescaled so that they sum to the facet total (src/solver/rdm/bc/
// WeakBC.hpp:786-832). The facet's wave speed is max_q max(1e-9, |lambda|) for every dof and
// enters the nodal wave speed multiplied by the dual volume (WeakBC.hpp:315-352).
//   WeakDirichlet (bc/WeakDirichletBC.hpp:159-265): K-(n) (g - u_q).
//   WeakWall (bc/WeakWall.hpp:93-250): F(u_mirror).n - F(u_q).n, u_mirror with the normal
//     velocity removed, same density and pressure; the dof part is scaled by 1/(3p) for p > 1.
//   WeakSubInlet (bc/WeakSubInlet.hpp:113-215): K-(n) (u_in - u_q), u_in from the total
//     temperature and pressure at the local Mach number (gas constant 287.046 as there).
//   WeakSubOutlet (bc/WeakSubOutlet.hpp:105-190): K-(n) (u_out - u_q), u_out = u_q with the
//     energy of the outlet pressure.
//   WeakFarfield (bc/WeakFarfield.hpp:125-240, the active branch): K-(n) (u_ref - u_q) with the
//     reference state u_ref, lambda floor 1e-8.
//   WeakSuperInlet (bc/WeakSuperInlet.hpp:62-160): no residual; only the facet's wave speed.
//   WeakSymmetry (bc/WeakSymmetry.hpp:100-190): K-(n) (u_mirror - u_q), u_mirror with the same
//     density and energy and the momentum rho (V - 2 (V.n) n).
// StrongDirichletBC::apply (bc/StrongDirichletBC.hpp:202-233) has its own kernel: the listed
// dofs take their values (one thread per distinct dof, the value of the last facet naming it).
// Facet normals are (dy/dxi, -dx/dxi)/|.| in 2D and the normalised cross product of the two
// tangents in 3D, with |J| the length / area factor (src/interpolation/GeometryMetric.hpp:560-660).

#include "rds_bc_facet.cuh"
#include "rds_internal.h"
#include "rds_physics.cuh"

namespace rds
{

namespace
{

// The weak conditions of one launch: up to kMaxBCSet with the same physics and facet type, each
// with its own data, tables and kind; condition k takes the blocks [first[k], first[k + 1]). One
// launch for all of them instead of one each: a sweep of a small mesh waits for every branch of
// its graph to join, and a batch has up to 15 conditions. 24 host-driven steps of 512 P2 cells
// with three conditions took 1.31 ms, 1.16 ms so.
template <int D, int NFDOF, int NFQ, int NFGEO>
struct BCSet
{
  int n;
  int first[kMaxBCSet + 1];
  int kind[kMaxBCSet];
  BCArgs a[kMaxBCSet];
  FacetTables<double, D, NFDOF, NFQ, NFGEO> tb[kMaxBCSet];
};

template <typename Set>
__device__ __forceinline__ int bc_of_block(const Set &set)
{
  int k = 0;
  while (k + 1 < set.n && (int)blockIdx.x >= set.first[k + 1])
    ++k;
  return k;
}

// Scalar physics (weak Dirichlet only): one thread per facet.
template <int PHYS, int NFDOF, int NFQ, int NFGEO>
__global__ void __launch_bounds__(kBlock)
    bc_weak(const __grid_constant__ BCSet<2, NFDOF, NFQ, NFGEO> set)
{
  if (*set.a[0].stop)
    return;
  const int k = bc_of_block(set);
  const int f = (blockIdx.x - set.first[k]) * blockDim.x + threadIdx.x;
  if (f >= set.a[k].nfacets)
    return;
  bc_weak_facet<RDS_BC_WEAK_DIRICHLET, PHYS, 2, 1, NFDOF, NFQ, NFGEO>(set.a[k], set.tb[k], f);
}

// Euler: the points of a facet on the lanes of a group, then one lane per equation sums the dof
// residuals over the points, in the order and with the operations of bc_weak_facet (the same
// bits). The conditions have too few facets to fill the GPU and run beside the cells, so what
// counts is the length of one thread's work: 512 subsonic-inlet facets of P2 tetrahedra (12
// points) took 60 us with one thread per facet, 11 us so, and until they end the SMs they hold are
// missing to the cells, whose blocks take a whole SM each: a sweep of 98,304 tetrahedra 307 us
// before, 267 us now.
template <int KIND, int PHYS, int D, int NEQ, int NFDOF, int NFQ, int NFGEO, int G>
__device__ __forceinline__ void
bc_points(const BCArgs &a, const FacetTables<double, D, NFDOF, NFQ, NFGEO> &tb, const int block,
          double (*s_w)[NFQ], double (*s_g)[NFQ][NEQ])
{
  static_assert(G >= NFQ && 32 % G == 0, "a lane per point");
  const int lane  = threadIdx.x % G, slot = threadIdx.x / G;
  const int f0    = block * (kBlock / G) + slot;
  const bool live = f0 < a.nfacets;
  const int f     = live ? f0 : a.nfacets - 1; // idle groups shadow the last facet, write nothing
  const double relax = (KIND == RDS_BC_WEAK_WALL) ? a.relax : 1.0;
  double coeff       = 0.0;
  if (lane < NFQ)
  {
    double X[NFGEO][D], un[NFDOF][NEQ];
#pragma unroll
    for (int g = 0; g < NFGEO; ++g)
    {
      const int v = a.geo_conn[(size_t)g * a.nfacets + f];
#pragma unroll
      for (int d = 0; d < D; ++d)
        X[g][d] = a.X[(size_t)d * a.ngeo_nodes + v];
    }
#pragma unroll
    for (int n = 0; n < NFDOF; ++n)
    {
      const int v = a.sol_conn[(size_t)n * a.nfacets + f];
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        un[n][e] = a.u[(size_t)e * a.nnodes + v];
    }
    double wq, eig_max, gflux[NEQ];
    bool bad = false;
    bc_weak_point<KIND, PHYS, D, NEQ, NFDOF, NFQ, NFGEO>(a, tb, f, lane, X, un, wq, gflux, eig_max,
                                                         bad);
    coeff            = fmax(0.0, eig_max);
    s_w[slot][lane]  = wq;
#pragma unroll
    for (int e = 0; e < NEQ; ++e)
      s_g[slot][lane][e] = gflux[e];
    if (bad && live)
      atomicOr(a.status, kFlagNegPressure);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
    coeff = fmax(coeff, __shfl_xor_sync(0xffffffffu, coeff, o));
  __syncwarp();
  if (!live)
    return;
  for (int e = lane; e < NEQ; e += G)
  {
    double bres[NFDOF], total = 0.0;
#pragma unroll
    for (int n = 0; n < NFDOF; ++n)
      bres[n] = 0.0;
#pragma unroll
    for (int q = 0; q < NFQ; ++q)
    {
      const double wq = s_w[slot][q], g = s_g[slot][q][e];
      total += wq * g;
#pragma unroll
      for (int n = 0; n < NFDOF; ++n)
        bres[n] += relax * tb.fV[q][n] * wq * g;
    }
    double sum = 0.0;
#pragma unroll
    for (int n = 0; n < NFDOF; ++n)
      sum += bres[n];
    const double scale = fabs(sum) > 1.e-14 ? total / sum : 1.0;
#pragma unroll
    for (int n = 0; n < NFDOF; ++n)
      a.out.val[e * a.out.S + a.out.slot_base + (long long)n * a.nfacets + f] = bres[n] * scale;
  }
  for (int n = lane; n < NFDOF; n += G)
    a.out.wsc[(size_t)n * a.nfacets + f] =
        a.vol[a.sol_conn[(size_t)n * a.nfacets + f]] * coeff;
}

template <int PHYS, int D, int NEQ, int NFDOF, int NFQ, int NFGEO, int G>
__global__ void __launch_bounds__(kBlock)
    bc_weak_points(const __grid_constant__ BCSet<D, NFDOF, NFQ, NFGEO> set)
{
  __shared__ double s_w[kBlock / G][NFQ], s_g[kBlock / G][NFQ][NEQ];
  if (*set.a[0].stop)
    return;
  const int k     = bc_of_block(set);
  const int block = blockIdx.x - set.first[k];
#define RDS_KIND(KIND)                                                                             \
  case KIND:                                                                                       \
    bc_points<KIND, PHYS, D, NEQ, NFDOF, NFQ, NFGEO, G>(set.a[k], set.tb[k], block, s_w, s_g);      \
    break;
  switch (set.kind[k]) // uniform over the block
  {
    RDS_KIND(RDS_BC_WEAK_DIRICHLET)
    RDS_KIND(RDS_BC_WEAK_WALL)
    RDS_KIND(RDS_BC_WEAK_SUB_INLET)
    RDS_KIND(RDS_BC_WEAK_SUB_OUTLET)
    RDS_KIND(RDS_BC_WEAK_FARFIELD)
    RDS_KIND(RDS_BC_WEAK_SUPER_INLET)
    RDS_KIND(RDS_BC_WEAK_SYMMETRY)
  default:
    break;
  }
#undef RDS_KIND
}

template <int PHYS, int D, int NEQ, int NFDOF, int NFQ, int NFGEO>
cudaError_t launch_weak(const HostBC *const *bcs, const BCArgs *args, int n, cudaStream_t s)
{
  BCSet<D, NFDOF, NFQ, NFGEO> set{};
  constexpr int G   = NFQ <= 4 ? 4 : NFQ <= 8 ? 8 : 16;
  constexpr int FPB = NEQ > 1 ? kBlock / G : kBlock; // facets per block
  set.n             = n;
  for (int k = 0; k < n; ++k)
  {
    const HostBC &b = *bcs[k];
    set.kind[k]     = b.desc.kind;
    set.a[k]        = args[k];
    FacetTables<double, D, NFDOF, NFQ, NFGEO> &tb = set.tb[k];
    for (int q = 0; q < NFQ; ++q)
    {
      tb.fw[q] = b.fw[q];
      for (int i = 0; i < NFDOF; ++i)
        tb.fV[q][i] = b.fV[q * NFDOF + i];
      for (int xi = 0; xi < D - 1; ++xi)
        for (int g = 0; g < NFGEO; ++g)
          tb.fdVgeo[xi][q][g] = b.fdVgeo[(xi * NFQ + q) * NFGEO + g];
    }
    set.first[k + 1] = set.first[k] + (args[k].nfacets + FPB - 1) / FPB;
  }
  if constexpr (NEQ > 1)
    bc_weak_points<PHYS, D, NEQ, NFDOF, NFQ, NFGEO, G><<<set.first[n], kBlock, 0, s>>>(set);
  else
    bc_weak<PHYS, NFDOF, NFQ, NFGEO><<<set.first[n], kBlock, 0, s>>>(set);
  return cudaGetLastError();
}

// Facet types: 2D lines P1-P3 with 3-5 point Gauss rules; 3D P1 triangles with 4 points and P2
// triangles with 7 or 12.
template <int PHYS, int D, int NEQ>
cudaError_t dispatch_facets(const HostBC *const *bcs, const BCArgs *args, int n, cudaStream_t s,
                            bool *ok)
{
  const rds_bc_group &d = bcs[0]->desc;
  *ok                   = true;
  if constexpr (D == 2)
  {
    if (d.nfgeo == 2)
    {
#define RDS_WEAK(NFDOF, NFQ)                                                                       \
  if (d.nfdof == NFDOF && d.nfq == NFQ)                                                            \
    return launch_weak<PHYS, D, NEQ, NFDOF, NFQ, 2>(bcs, args, n, s);
      RDS_WEAK(2, 3)
      RDS_WEAK(2, 4)
      RDS_WEAK(3, 3)
      RDS_WEAK(3, 4)
      RDS_WEAK(4, 5)
      RDS_WEAK(4, 4)
#undef RDS_WEAK
    }
  }
  else
  {
    if (d.nfgeo == 3 && d.nfdof == 6 && d.nfq == 12)
      return launch_weak<PHYS, D, NEQ, 6, 12, 3>(bcs, args, n, s);
    if (d.nfgeo == 3 && d.nfdof == 3 && d.nfq == 4)
      return launch_weak<PHYS, D, NEQ, 3, 4, 3>(bcs, args, n, s);
    if (d.nfgeo == 3 && d.nfdof == 6 && d.nfq == 7)
      return launch_weak<PHYS, D, NEQ, 6, 7, 3>(bcs, args, n, s);
  }
  *ok = false;
  return cudaSuccess;
}

const char *bc_name(int kind)
{
  switch (kind)
  {
  case RDS_BC_WEAK_WALL:
    return "bc_weak_wall";
  case RDS_BC_WEAK_SUB_INLET:
    return "bc_weak_sub_inlet";
  case RDS_BC_WEAK_SUB_OUTLET:
    return "bc_weak_sub_outlet";
  case RDS_BC_WEAK_FARFIELD:
    return "bc_weak_farfield";
  case RDS_BC_WEAK_SUPER_INLET:
    return "bc_weak_super_inlet";
  case RDS_BC_WEAK_SYMMETRY:
    return "bc_weak_symmetry";
  case RDS_BC_STRONG_DIRICHLET:
    return "bc_strong_dirichlet";
  default:
    return "bc_weak_dirichlet";
  }
}

// Strong Dirichlet: ndofs distinct dofs, their values SoA [neq][ndofs].
__global__ void __launch_bounds__(kBlock)
    bc_strong(int ndofs, int neq, int nnodes, const int32_t *__restrict__ dofs,
              const double *__restrict__ vals, double *__restrict__ u, const int *stop)
{
  if (*stop)
    return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ndofs)
    return;
  const int v = dofs[i];
  for (int e = 0; e < neq; ++e)
    u[(size_t)e * nnodes + v] = vals[(size_t)e * ndofs + i];
}

} // namespace

cudaError_t launch_strong(const BCArgs &a, int neq, cudaStream_t s, const char **name)
{
  *name = bc_name(RDS_BC_STRONG_DIRICHLET);
  if (a.nfacets > 0)
    bc_strong<<<(a.nfacets + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        a.nfacets, neq, a.nnodes, a.sol_conn, a.gq, a.u_strong, a.stop);
  return cudaGetLastError();
}

bool same_bc_set(const HostBC &a, const HostBC &b)
{
  return a.desc.kind != RDS_BC_STRONG_DIRICHLET && b.desc.kind != RDS_BC_STRONG_DIRICHLET &&
         a.physics == b.physics && a.desc.nfdof == b.desc.nfdof && a.desc.nfq == b.desc.nfq &&
         a.desc.nfgeo == b.desc.nfgeo;
}

cudaError_t launch_bc_set(const HostBC *const *bcs, const BCArgs *args, int n, int dim, int neq,
                          cudaStream_t s, const char **name)
{
  bool ok         = false;
  cudaError_t err = cudaSuccess;
  *name           = bc_name(bcs[0]->desc.kind);
  for (int k = 0; k < n; ++k)
  {
    if (bcs[k]->desc.kind != bcs[0]->desc.kind)
      *name = "bc_weak";
    // scalar physics have weak Dirichlet conditions only
    if (neq == 1 && bcs[k]->desc.kind != RDS_BC_WEAK_DIRICHLET)
    {
      *name = bc_name(bcs[k]->desc.kind);
      return cudaErrorNotSupported;
    }
  }
  const int physics = bcs[0]->physics;
  if (physics == RDS_ADVECTION_CONST && dim == 2 && neq == 1)
    err = dispatch_facets<RDS_ADVECTION_CONST, 2, 1>(bcs, args, n, s, &ok);
  else if (physics == RDS_BURGERS2D && dim == 2 && neq == 1)
    err = dispatch_facets<RDS_BURGERS2D, 2, 1>(bcs, args, n, s, &ok);
  else if (physics == RDS_EULER2D && dim == 2 && neq == 4)
    err = dispatch_facets<RDS_EULER2D, 2, 4>(bcs, args, n, s, &ok);
  else if (physics == RDS_EULER3D && dim == 3 && neq == 5)
    err = dispatch_facets<RDS_EULER3D, 3, 5>(bcs, args, n, s, &ok);
  if (!ok)
    return cudaErrorNotSupported;
  return err;
}

} // namespace rds
