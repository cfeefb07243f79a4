// Batched Hexa8 element kernels (FP64): stiffness K_e = sum_gp w B^T D B and
// consistent mass, the device twins of CalcH8GaussMatrices + CalcH8K
// (FEMElements/FEMElements/rElHexa8.f90:422-464, 489-543) and
// Hexa8.CalculateConsistentMass (ISAAR.MSolve.PreProcessor/Elements/Hexa8.cs:403-435).
//
// One CTA handles 8 elements. Phase 1: 64 threads, one per (element, Gauss
// point), compute the shape-function natural derivatives, the Jacobian, its
// determinant and inverse, the Cartesian derivatives dN/dx (the nonzeros of
// B) and the weight, into shared memory. Phase 2: all threads produce the 300
// packed entries of each element, each entry summed over the 8 Gauss points
// in the reference's order (xi outer, zeta inner). Output writes are
// contiguous across threads.
#include <algorithm>

#include "msg_internal.h"

namespace msg {
namespace {

constexpr int kEPB = 8;      // elements per CTA
constexpr int kThreads = 256;

__constant__ unsigned short c_pair_i[300];
__constant__ unsigned short c_pair_j[300];

struct GaussData {
  double dx[kEPB][8][8][3];  // [elem][gp][node][x,y,z] = dN_node/dx_c
  double w[kEPB][8];
  double S[8][8];            // shape values [gp][node] (same for every element)
};

// rElHexa8.f90:435-445 literal 2-point rule.
__device__ __forceinline__ double gauss_pt(int i) { return i ? .5773502691896 : -.5773502691896; }

__device__ void gauss_point(const double* __restrict__ xyz, int gp, double* dxyz /*[8][3]*/, double* w,
                            double* S8, int* status) {
  const int ix = gp >> 2, iy = (gp >> 1) & 1, iz = gp & 1;
  const double xi = gauss_pt(ix), eta = gauss_pt(iy), zeta = gauss_pt(iz);
  // CalcH8NablaShape (:25-69)
  const double s = 0.35355339059327376220042218105242;
  const double xp = (1.0 + xi) * s, ep = (1.0 + eta) * s, zp = (1.0 + zeta) * s;
  const double xm = (1.0 - xi) * s, em = (1.0 - eta) * s, zm = (1.0 - zeta) * s;
  double ds[24];
  ds[0] = -(em * zm); ds[1] = -ds[0]; ds[2] = ep * zm; ds[3] = -ds[2];
  ds[4] = -(em * zp); ds[5] = -ds[4]; ds[6] = ep * zp; ds[7] = -ds[6];
  ds[8] = -(xm * zm); ds[9] = -(xp * zm); ds[10] = -ds[9]; ds[11] = -ds[8];
  ds[12] = -(xm * zp); ds[13] = -(xp * zp); ds[14] = -ds[13]; ds[15] = -ds[12];
  ds[16] = -(xm * em); ds[17] = -(xp * em); ds[18] = -(xp * ep); ds[19] = -(xm * ep);
  ds[20] = -ds[16]; ds[21] = -ds[17]; ds[22] = -ds[18]; ds[23] = -ds[19];
  // CalcH8JDetJ (:141-208)
  double J[9];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double acc = ds[8 * a] * xyz[i];
#pragma unroll
      for (int n = 1; n < 8; ++n) acc = acc + ds[8 * a + n] * xyz[3 * n + i];
      J[3 * a + i] = acc;
    }
  const double d1 = J[0] * (J[4] * J[8] - J[7] * J[5]);
  const double d2 = -J[1] * (J[3] * J[8] - J[6] * J[5]);
  const double d3 = J[2] * (J[3] * J[7] - J[6] * J[4]);
  const double det = d1 + d2 + d3;
  if (det < 0.00000001) atomicMin(status, MSG_ERR_NEG_DET);
  // CalcH8B inverse (:232-250)
  const double inv = 1.0 / det;
  double Ji[9];
  Ji[0] = (J[4] * J[8] - J[7] * J[5]) * inv;
  Ji[3] = (J[6] * J[5] - J[3] * J[8]) * inv;
  Ji[6] = (J[3] * J[7] - J[6] * J[4]) * inv;
  Ji[1] = (J[7] * J[2] - J[1] * J[8]) * inv;
  Ji[4] = (J[0] * J[8] - J[6] * J[2]) * inv;
  Ji[7] = (J[6] * J[1] - J[7] * J[0]) * inv;
  Ji[2] = (J[1] * J[5] - J[4] * J[2]) * inv;
  Ji[5] = (J[3] * J[2] - J[0] * J[5]) * inv;
  Ji[8] = (J[0] * J[4] - J[3] * J[1]) * inv;
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    dxyz[3 * n + 0] = Ji[0] * ds[n] + Ji[1] * ds[8 + n] + Ji[2] * ds[16 + n];
    dxyz[3 * n + 1] = Ji[3] * ds[n] + Ji[4] * ds[8 + n] + Ji[5] * ds[16 + n];
    dxyz[3 * n + 2] = Ji[6] * ds[n] + Ji[7] * ds[8 + n] + Ji[8] * ds[16 + n];
  }
  *w = 1.0 * 1.0 * 1.0 * det;
  if (S8) {  // CalcH8Shape (:93-117)
    const double c = 0.5;
    const double Xp = (1.0 + xi) * c, Ep = (1.0 + eta) * c, Zp = (1.0 + zeta) * c;
    const double Xm = (1.0 - xi) * c, Em = (1.0 - eta) * c, Zm = (1.0 - zeta) * c;
    S8[0] = Xm * Em * Zm; S8[1] = Xp * Em * Zm; S8[2] = Xp * Ep * Zm; S8[3] = Xm * Ep * Zm;
    S8[4] = Xm * Em * Zp; S8[5] = Xp * Em * Zp; S8[6] = Xp * Ep * Zp; S8[7] = Xm * Ep * Zp;
  }
}

// Column i of B (6 strains) from dN/dx of node a = i/3, component c = i%3
// (rElHexa8.f90:253-396: rows exx, eyy, ezz, gxy, gyz, gzx).
__device__ __forceinline__ void b_column(const double* d /*dN_a/dx[3]*/, int c, double* B6) {
  B6[0] = c == 0 ? d[0] : 0.0;
  B6[1] = c == 1 ? d[1] : 0.0;
  B6[2] = c == 2 ? d[2] : 0.0;
  B6[3] = c == 0 ? d[1] : (c == 1 ? d[0] : 0.0);
  B6[4] = c == 1 ? d[2] : (c == 2 ? d[1] : 0.0);
  B6[5] = c == 0 ? d[2] : (c == 2 ? d[0] : 0.0);
}

__global__ void __launch_bounds__(kThreads) k_h8_ke(int n, const double* __restrict__ xyz,
                                                    const double* __restrict__ Ev, double E_scalar, double nu,
                                                    double* __restrict__ K, int* __restrict__ status) {
  __shared__ GaussData g;
  __shared__ double sD[kEPB][3];  // e3 (diag), e2 (off), e4 (shear) per element
  const int e0 = blockIdx.x * kEPB;
  const int t = threadIdx.x;
  if (t < kEPB * 8) {
    const int le = t >> 3, gp = t & 7, e = e0 + le;
    if (e < n) {
      double x[24];
#pragma unroll
      for (int k = 0; k < 24; ++k) x[k] = xyz[(size_t)e * 24 + k];
      gauss_point(x, gp, &g.dx[le][gp][0][0], &g.w[le][gp], nullptr, status);
    }
  } else if (t < kEPB * 8 + kEPB) {
    const int le = t - kEPB * 8, e = e0 + le;
    if (e < n) {  // ElasticMaterial3D.GetConstitutiveMatrix (:20-44)
      const double E = Ev ? Ev[e] : E_scalar;
      const double e1 = E / (1.0 + nu);
      const double e2 = e1 * nu / (1.0 - 2.0 * nu);
      sD[le][0] = e1 + e2;
      sD[le][1] = e2;
      sD[le][2] = e1 * 0.5;
    }
  }
  __syncthreads();
  for (int q = t; q < kEPB * 300; q += kThreads) {
    const int le = q / 300, idx = q - le * 300, e = e0 + le;
    if (e >= n) break;
    const int i = c_pair_i[idx], j = c_pair_j[idx];
    const int a = i / 3, ci = i - 3 * a, b = j / 3, cj = j - 3 * b;
    const double d3 = sD[le][0], d2 = sD[le][1], d4 = sD[le][2];
    double acc = 0.0;
#pragma unroll 1
    for (int gp = 0; gp < 8; ++gp) {
      double Bi[6], Bj[6];
      b_column(g.dx[le][gp][a], ci, Bi);
      b_column(g.dx[le][gp][b], cj, Bj);
      // eb = D B_i with the isotropic D (rows summed left to right as CalcH8K :514-531)
      double eb[6];
      eb[0] = d3 * Bi[0] + d2 * Bi[1] + d2 * Bi[2];
      eb[1] = d2 * Bi[0] + d3 * Bi[1] + d2 * Bi[2];
      eb[2] = d2 * Bi[0] + d2 * Bi[1] + d3 * Bi[2];
      eb[3] = d4 * Bi[3];
      eb[4] = d4 * Bi[4];
      eb[5] = d4 * Bi[5];
      double st = Bj[0] * eb[0] + Bj[1] * eb[1] + Bj[2] * eb[2] + Bj[3] * eb[3] + Bj[4] * eb[4] + Bj[5] * eb[5];
      acc = acc + st * g.w[le][gp];
    }
    K[(size_t)e * 300 + idx] = acc;
  }
}

__global__ void __launch_bounds__(kThreads) k_h8_me(int n, const double* __restrict__ xyz, double rho,
                                                    double* __restrict__ M, int* __restrict__ status) {
  __shared__ GaussData g;
  const int e0 = blockIdx.x * kEPB;
  const int t = threadIdx.x;
  if (t < kEPB * 8) {
    const int le = t >> 3, gp = t & 7, e = e0 + le;
    if (e < n) {
      double x[24];
#pragma unroll
      for (int k = 0; k < 24; ++k) x[k] = xyz[(size_t)e * 24 + k];
      double S8[8];
      gauss_point(x, gp, &g.dx[le][gp][0][0], &g.w[le][gp], S8, status);
      if (le == 0)
        for (int k = 0; k < 8; ++k) g.S[gp][k] = S8[k];
    }
  }
  __syncthreads();
  for (int q = t; q < kEPB * 300; q += kThreads) {
    const int le = q / 300, idx = q - le * 300, e = e0 + le;
    if (e >= n) break;
    const int i = c_pair_i[idx], j = c_pair_j[idx];
    const int a = i / 3, ci = i - 3 * a, b = j / 3, cj = j - 3 * b;
    double acc = 0.0;
    if (ci == cj) {
      for (int gp = 0; gp < 8; ++gp) acc = acc + g.S[gp][a] * g.S[gp][b] * (g.w[le][gp] * rho);
    }
    M[(size_t)e * 300 + idx] = acc;
  }
}

// Strain / stress recovery and internal forces of a batch of element
// instances (an instance = one element of one realization), the device twin
// of Hexa8.CalculateStresses + CalculateForces (ISAAR.MSolve.PreProcessor/
// Elements/Hexa8.cs:453-510) over CalcH8Strains and CalcH8Forces
// (FEMElements/FEMElements/rElHexa8.f90:636-648, 724-747) with the elastic
// material update (ElasticMaterial3D.cs:20-44, 75-81: the stored strain is the
// increment, stresses = D * increment). Per Gauss point m: strains = B_m u,
// stresses = D(E) B_m du; forces = sum_m w_m B_m^T stresses_m. Sums follow the
// reference's order (24 columns of B; 6 columns of D; 6 rows of B^T; Gauss
// points xi outer, zeta inner). The displacements come from an instance array
// u [n][24] or are gathered from a realization batch X [R][n_dofs] through
// the connectivity and the DOF map (constrained DOFs: 0).
struct StressIn {
  const double* xyz;   // [n_e][24]
  const double* E;     // [n] or nullptr (E_scalar)
  double E_scalar, nu;
  const double* u;     // [n][24] or nullptr (gather from X)
  const double* du;    // [n][24] or nullptr (du = u)
  const double* X;     // [R][n_dofs]
  const int* conn;     // [n_e][8]
  const int* dof;      // [n_nodes][3]
  int n_e, n_dofs;
};

// A warp takes 4 elements, a lane one (element, Gauss point) with the Cartesian
// derivatives in registers, and walks a range of realizations: the geometry is
// formed once for all of them. A lane loads its node's displacements one
// realization ahead and the element's lanes read them from shared memory.
// Strains and stresses go through shared memory to coalesced stores, the Gauss
// points' force contributions are summed there in Gauss order. Terms with a zero
// of B or D are left out, but where a value is not finite (0 * inf is not 0).
// Bound by the shared-memory pipe (81 % busy), then FP64 (43 %); HBM 2.9 TB/s.
// 20^3 elements x 64 realizations: 153 us, 1,029 when every instance formed its
// own geometry on a quarter of the threads and stored 8 bytes at a stride of 48
// (299 with a lane loading all 24 displacements itself, waiting for them).
constexpr int kStWarps = 4, kStElems = 4;  // warps of a CTA, elements of a warp
constexpr int kStPad = 25;                 // doubles a lane in shared memory (24 used; odd: no bank conflicts)
constexpr int kStU = 26;                   // doubles of an element's displacements there (24 used)
constexpr double kMaxDouble = 1.7976931348623157e308;

template <bool kDu>
__global__ void __launch_bounds__(32 * kStWarps, kDu ? 2 : 4)
    k_h8_stress(int R, int r_per, StressIn in, double* __restrict__ strains, double* __restrict__ stresses,
                double* __restrict__ forces, int* __restrict__ status) {
  __shared__ __align__(16) double sh[kStWarps][32 * kStPad + 8];
  __shared__ __align__(16) double su[kStWarps][kDu ? 2 : 1][kStElems * kStU];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e0 = (blockIdx.x * kStWarps + w) * kStElems;  // the warps are independent of each other
  if (e0 >= in.n_e) return;
  const int ne = min(kStElems, in.n_e - e0);  // elements of this warp
  const int le = lane >> 3, gp = lane & 7;
  const bool live = le < ne;
  const int e = live ? e0 + le : e0;  // spare lanes repeat the first element
  double* st = sh[w];
  double d[24], wgt;  // d[3 node + axis] = dN_node/dx_axis
  {
    double x[24];
#pragma unroll
    for (int k = 0; k < 24; ++k) x[k] = in.xyz[(size_t)e * 24 + k];
    gauss_point(x, gp, d, &wgt, nullptr, status);
  }
  // the lane's three displacements: node gp of its element
  int dof[3] = {-1, -1, -1};
  if (!in.u) {
    const int node = in.conn[(size_t)e * 8 + gp];
#pragma unroll
    for (int c = 0; c < 3; ++c) dof[c] = in.dof[(size_t)node * 3 + c];
  }
  const double inv1 = 1.0 / (1.0 + in.nu), lam = in.nu / (1.0 - 2.0 * in.nu);
  const int r0 = blockIdx.y * r_per, r1 = min(R, r0 + r_per);
  // displacements and modulus of the next realization, loaded one ahead
  double un[3], dn[3] = {0, 0, 0}, En;
  auto fetch = [&](int r) {
    const size_t i = (size_t)r * in.n_e + e;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      un[c] = in.u ? in.u[i * 24 + 3 * gp + c] : dof[c] >= 0 ? in.X[(size_t)r * in.n_dofs + dof[c]] : 0.0;
      if constexpr (kDu) dn[c] = in.du[i * 24 + 3 * gp + c];
    }
    En = in.E ? in.E[i] : in.E_scalar;
  };
  if (r0 < r1) fetch(r0);
  for (int r = r0; r < r1; ++r) {
    const size_t i0 = (size_t)r * in.n_e + e0;  // first instance of the warp
    bool bad = false;                           // a displacement that is not finite
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      su[w][0][le * kStU + 3 * gp + c] = un[c];
      bad |= !(fabs(un[c]) <= kMaxDouble);
      if constexpr (kDu) {
        su[w][kDu ? 1 : 0][le * kStU + 3 * gp + c] = dn[c];
        bad |= !(fabs(dn[c]) <= kMaxDouble);
      }
    }
    const double E = En;
    if (r + 1 < r1) fetch(r + 1);
    bad = __any_sync(0xffffffffu, bad);  // (and the shared values are there)
    __syncwarp();
    const double* ul = &su[w][0][le * kStU];
    const double* dl = &su[w][kDu ? 1 : 0][le * kStU];
    double ep[6] = {0, 0, 0, 0, 0, 0}, de[6] = {0, 0, 0, 0, 0, 0};
    // B u: rows exx, eyy, ezz, gxy, gyz, gzx
    auto column = [&](double (&v)[6], const double* dn, double ux, double uy, double uz) {
      v[0] = fma(dn[0], ux, v[0]);
      v[1] = fma(dn[1], uy, v[1]);
      v[2] = fma(dn[2], uz, v[2]);
      v[3] = fma(dn[0], uy, fma(dn[1], ux, v[3]));
      v[4] = fma(dn[1], uz, fma(dn[2], uy, v[4]));
      v[5] = fma(dn[0], uz, fma(dn[2], ux, v[5]));
    };
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      column(ep, d + 3 * n, ul[3 * n], ul[3 * n + 1], ul[3 * n + 2]);
      if constexpr (kDu) column(de, d + 3 * n, dl[3 * n], dl[3 * n + 1], dl[3 * n + 2]);
    }
    if (bad) {  // the zero coefficients' products with the values that are not finite
      double z[3] = {0, 0, 0}, zd[3] = {0, 0, 0};
      for (int n = 0; n < 8; ++n)
        for (int c = 0; c < 3; ++c) {
          z[c] += 0.0 * ul[3 * n + c];
          zd[c] += 0.0 * dl[3 * n + c];
        }
      auto rest = [](double (&v)[6], const double (&q)[3]) {
        v[0] += q[1] + q[2]; v[1] += q[0] + q[2]; v[2] += q[0] + q[1];
        v[3] += q[2]; v[4] += q[0]; v[5] += q[1];
      };
      rest(ep, z);
      if constexpr (kDu) rest(de, zd);
    }
    // ElasticMaterial3D: stresses = D * (strain increment)
    const double e1 = E * inv1, e2 = e1 * lam, e3 = e1 + e2, e4 = e1 * 0.5;
    const double* g = kDu ? de : ep;
    double sg[6];
    sg[0] = fma(e2, g[2], fma(e2, g[1], e3 * g[0]));
    sg[1] = fma(e2, g[2], fma(e3, g[1], e2 * g[0]));
    sg[2] = fma(e3, g[2], fma(e2, g[1], e2 * g[0]));
    sg[3] = e4 * g[3];
    sg[4] = e4 * g[4];
    sg[5] = e4 * g[5];
    const double sum = ((g[0] + g[1]) + (g[2] + g[3])) + (g[4] + g[5]);
    const bool odd = !(fabs(sum) <= kMaxDouble) || !(fabs(e1) <= kMaxDouble);
    if (odd) {  // the zeros of D
      const double n0 = 0.0 * g[0] + 0.0 * g[1] + 0.0 * g[2], s0 = 0.0 * g[3], s1 = 0.0 * g[4], s2 = 0.0 * g[5];
      for (int k = 0; k < 3; ++k) sg[k] += s0 + s1 + s2;
      sg[3] += n0 + s1 + s2;
      sg[4] += n0 + s0 + s2;
      sg[5] += n0 + s0 + s1;
    }
    // the warp's strains and stresses: 48 doubles an element, one after another
    auto put = [&](const double (&v)[6], double* out) {
#pragma unroll
      for (int k = 0; k < 6; ++k) st[lane * 6 + k] = v[k];
      __syncwarp();
      double* o = out + i0 * 48;
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (lane + 32 * k < 48 * ne) o[lane + 32 * k] = st[lane + 32 * k];
      __syncwarp();
    };
    if (strains) put(ep, strains);
    if (stresses) put(sg, stresses);
    if (forces) {
      // CalcH8Forces: w B^T stresses of the lane's Gauss point, summed in Gauss order
      // with the zeros of B, where a stress is not finite (by overflow too)
      double zf[3] = {0, 0, 0};
      const double total = ((sg[0] + sg[1]) + (sg[2] + sg[3])) + (sg[4] + sg[5]);
      if (!(fabs(total) <= kMaxDouble)) {
        zf[0] = 0.0 * sg[1] + 0.0 * sg[2] + 0.0 * sg[4];
        zf[1] = 0.0 * sg[0] + 0.0 * sg[2] + 0.0 * sg[5];
        zf[2] = 0.0 * sg[0] + 0.0 * sg[1] + 0.0 * sg[3];
      }
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const double dx = d[3 * n], dy = d[3 * n + 1], dz = d[3 * n + 2];
        st[lane * kStPad + 3 * n] = wgt * (fma(dz, sg[5], fma(dy, sg[3], dx * sg[0])) + zf[0]);
        st[lane * kStPad + 3 * n + 1] = wgt * (fma(dz, sg[4], fma(dx, sg[3], dy * sg[1])) + zf[1]);
        st[lane * kStPad + 3 * n + 2] = wgt * (fma(dx, sg[5], fma(dy, sg[4], dz * sg[2])) + zf[2]);
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int o = lane + 32 * k, el = o / 24, col = o - 24 * el;
        if (el < ne) {
          double f = 0.0;
#pragma unroll
          for (int m = 0; m < 8; ++m) f = f + st[(el * 8 + m) * kStPad + col];
          forces[i0 * 24 + o] = f;
        }
      }
      __syncwarp();
    }
  }
}

bool g_pairs_ready[64] = {false};
std::mutex g_pairs_mu;

int ensure_pairs(Context* ctx) {
  std::lock_guard<std::mutex> lk(g_pairs_mu);
  if (ctx->device >= 0 && ctx->device < 64 && g_pairs_ready[ctx->device]) return MSG_OK;
  unsigned short pi[300], pj[300];
  int k = 0;
  for (int i = 0; i < 24; ++i)
    for (int j = i; j < 24; ++j) { pi[k] = (unsigned short)i; pj[k] = (unsigned short)j; ++k; }
  MSG_CUDA(ctx, cudaMemcpyToSymbol(c_pair_i, pi, sizeof(pi)));
  MSG_CUDA(ctx, cudaMemcpyToSymbol(c_pair_j, pj, sizeof(pj)));
  if (ctx->device >= 0 && ctx->device < 64) g_pairs_ready[ctx->device] = true;
  return MSG_OK;
}

}  // namespace

int launch_h8_ke(Context* ctx, int n, const double* d_xyz, const double* d_E, double E_scalar, double nu,
                 double* d_K, int* d_status) {
  if (n <= 0) return MSG_OK;
  MSG_TRY(ensure_pairs(ctx));
  k_h8_ke<<<(n + kEPB - 1) / kEPB, kThreads, 0, ctx->stream>>>(n, d_xyz, d_E, E_scalar, nu, d_K, d_status);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_h8_stress(Context* ctx, int n, const double* d_xyz, const double* d_E, double E_scalar, double nu,
                     const double* d_u, const double* d_du, const double* d_X, const int* d_conn, const int* d_dof,
                     int n_e, int n_dofs, double* d_strains, double* d_stresses, double* d_forces, int* d_status) {
  if (n <= 0) return MSG_OK;
  StressIn in{d_xyz, d_E, E_scalar, nu, d_u, d_du, d_X, d_conn, d_dof, n_e, n_dofs};
  // realizations of a warp: enough warps for four rounds of 12 an SM, and no more
  const int R = n / n_e, warps = (n_e + kStElems - 1) / kStElems;
  const int chunks = std::max(1, std::min(R, (ctx->sm_count * 48 + warps - 1) / warps));
  const int r_per = (R + chunks - 1) / chunks;
  const dim3 grid((warps + kStWarps - 1) / kStWarps, (R + r_per - 1) / r_per);
  if (d_du)
    k_h8_stress<true><<<grid, 32 * kStWarps, 0, ctx->stream>>>(R, r_per, in, d_strains, d_stresses, d_forces, d_status);
  else
    k_h8_stress<false><<<grid, 32 * kStWarps, 0, ctx->stream>>>(R, r_per, in, d_strains, d_stresses, d_forces, d_status);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

int launch_h8_me(Context* ctx, int n, const double* d_xyz, double rho, double* d_M, int* d_status) {
  if (n <= 0) return MSG_OK;
  MSG_TRY(ensure_pairs(ctx));
  k_h8_me<<<(n + kEPB - 1) / kEPB, kThreads, 0, ctx->stream>>>(n, d_xyz, rho, d_M, d_status);
  count_launch(ctx);
  MSG_CUDA(ctx, cudaGetLastError());
  return MSG_OK;
}

}  // namespace msg
