// Explicit all-pairs ATTRACT energy (and pose gradient): every ligand bead
// against every receptor bead, no grid -- the rescoring path of the reference,
// test-energy.py:46-58 (delta over all pairs, nonbon of every d^2, summed per
// structure), with ATTRACT's --rcut as an optional distance cutoff.
//
// An item is one ligand bead of one pose.  A lane serves two items at a time in
// packed float operations (or four, in two packed sets), and a warp's lanes meet
// the same receptor bead together: it is one broadcast from shared memory, the
// type test is uniform, and the pair rows of a lane's items stay in registers
// while the receptor type lasts (the host wrapper sorts the receptor by type).
// The receptor is split over `rw` groups of the block's warps and over the `cl`
// blocks of a cluster.  ap_plan() weighs the splits: a library of poses fills the GPU
// with whole receptors, a handful of poses needs every split there is.
//
// A pose's results do not depend on the split, nor on the poses beside it.  The
// receptor is divided into leaves (a power of two, 17 to 64 beads each) that
// follow from its length alone.  A lane sums an item's energy and force over a
// leaf in float, then in double: the leaves of a branch in order (four; two or
// more of 64 branches beyond 4096 beads), the branches in a binary tree, whose lower levels a
// lane forms by itself and whose upper ones the groups and the cluster's blocks.
// A pose's sum takes its beads 64 at a time.
//
// Bound by the FMA pipe (a packed operation takes it twice as long as a plain
// one: 19 of them per two pairs) and by issue: 17.4 instructions per pair at four items per
// lane, the pipe 60 % and the issue slots 55 % busy, against 52.7 for a warp that met 32
// receptor beads at once (a row test and shuffles of its own per bead).  2500 x
// 24 beads: 16 384 poses 1958 -> 880 us (1.1 T pairs/s), 10 poses 48 us on one block each -> 13.4,
// below the host's part of the call.  (Splits chosen without regard to the sums' order took
// 889 and 12.9 us; 300 poses 31 us against 41, 150 x 24 beads, 16 384 poses 135 against 145, 5000 x 24
// beads, 10 poses 16 against 21, 5000 x 301 beads, 300 poses 609 against 511.)
#include <cooperative_groups.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace att {
int report_error(int code, const char* msg);
namespace cg = cooperative_groups;

constexpr int AP_THREADS = 256;
constexpr int AP_WARPS = AP_THREADS / 32;
constexpr int AP_TILE = 1024;    // receptor beads in shared memory (32 B each), over the block's groups
constexpr int AP_LEAF = 64;      // receptor beads summed in float, at most
constexpr int AP_LEVELS = 6;     // of the tree of branches, at most (its upper levels: 8 eights)
constexpr int AP_CHUNK = 64;     // ligand beads of a pose summed at a time
constexpr int AP_POSES = 128;    // poses of a block

struct AllPairsParams {
  const float4* rec;   // [n_rec] x, y, z, receptor type (int bits)
  const float4* lig;   // [n_lig] x, y, z, ligand type (int bits)
  const float* pose;   // [B][6] Euler + translation, or [B][16] row-vector 4x4
  const float4* pair;  // [n_ltypes][n_rtypes][2]: rc, ac, emin, rmin2 / ivor, eplat, -, rcap2
  float* energy;       // [B]
  float* grad;         // [B][6] or [B][16], may be NULL
  float rcut2;         // <= 0: no cutoff
  int n_rec, n_lig, n_poses, pose_format, n_rtypes, n_ltypes;
  int rw, cl;          // receptor groups per block, blocks per cluster
  int pb, nb;          // poses per block, ligand beads per pass (all of them unless pb = 1, then a multiple of 64)
  int leaves_log2, branches_log2;  // of the receptor
};

// two floats in one register pair: every operation rounds as the plain one
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// a double of shared memory in the cluster's block `rank`, by its address there
__device__ __forceinline__ double ld_cluster(unsigned at, int rank) {
  unsigned a;
  double v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned at, int rank, double v) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// a pose's row-vector rotation M (X = x M + t) and, for Euler poses, what its
// gradient takes of the angles
struct PoseM {
  float m[9], t[3], sphi, cphi, spsi, cpsi;
};
__device__ __forceinline__ PoseM load_pose(const AllPairsParams& p, int b) {
  PoseM q;
  q.sphi = q.spsi = 0.f;
  q.cphi = q.cpsi = 1.f;
  if (p.pose_format == 1) {
    const float* P = p.pose + (long long)b * 16;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) q.m[r * 3 + c] = __ldg(P + r * 4 + c);
#pragma unroll
    for (int c = 0; c < 3; ++c) q.t[c] = __ldg(P + 12 + c);
  } else {
    const float* P = p.pose + (long long)b * 6;
    float sth, cth;
    sincosf(__ldg(P + 0), &q.sphi, &q.cphi);
    sincosf(__ldg(P + 1), &q.spsi, &q.cpsi);
    sincosf(__ldg(P + 2), &sth, &cth);
    // column-form Q = Rz(phi) Ry(psi) Rz(-theta); the row-vector M is its transpose
    q.m[0] = q.cphi * q.cpsi * cth + q.sphi * sth;
    q.m[1] = q.sphi * q.cpsi * cth - q.cphi * sth;
    q.m[2] = -q.spsi * cth;
    q.m[3] = q.cphi * q.cpsi * sth - q.sphi * cth;
    q.m[4] = q.sphi * q.cpsi * sth + q.cphi * cth;
    q.m[5] = -q.spsi * sth;
    q.m[6] = q.cphi * q.spsi;
    q.m[7] = q.sphi * q.spsi;
    q.m[8] = q.cpsi;
#pragma unroll
    for (int c = 0; c < 3; ++c) q.t[c] = __ldg(P + 3 + c);
  }
  return q;
}

// The receptor's leaves, the smallest power of two that leaves each 32 beads or fewer, from 64
// leaves on 64 beads, and its branches.  A leaf is the shortest piece that few poses can be split into: with 64
// beads throughout 10 poses of 24 beads took 15.8 us on 150 beads (now 11.5), 14.8 on 700 (11.9), and
// 16 384 poses 137 (now 145) and 310 (332).  (Leaves as branches: 2500 x 24 beads, 16 384 poses 1 %,
// 300 x 8 beads 4 % slower.)
static int ap_leaves_log2(int n_rec) {
  int n = 0;
  while (((long long)(n < 6 ? AP_LEAF / 2 : AP_LEAF) << n) < n_rec) ++n;
  return n;
}
static int ap_branches_log2(int leaves_log2) {
  return leaves_log2 > 6 ? AP_LEVELS : leaves_log2 > 2 ? leaves_log2 - 2 : 0;
}

constexpr int ap_slots(int NP) { return AP_WARPS * 64 * NP; }  // items of a block, over its receptor groups
constexpr size_t ap_smem(int NP) {
  return (size_t)(AP_TILE + 1) * 2 * sizeof(float4) + (size_t)ap_slots(NP) * 4 * sizeof(double) +
         (size_t)AP_POSES * (13 * sizeof(double) + sizeof(PoseM));
}

// NP: packed pairs of items per lane; CUT: rcut; GRAD: the gradient too
template <int NP, bool CUT, bool GRAD>
__global__ void __launch_bounds__(AP_THREADS, NP == 1 ? 3 : 2) allpairs_kernel(const __grid_constant__ AllPairsParams p) {
  extern __shared__ __align__(16) unsigned char ap_smem_raw[];
  float4* s_rec = reinterpret_cast<float4*>(ap_smem_raw);                // [AP_TILE + 1][2]: -x -x -y -y, -z -z type -
  double* s_item = reinterpret_cast<double*>(s_rec + (AP_TILE + 1) * 2);  // [group][E, Gx, Gy, Gz][item]
  double* s_sum = s_item + ap_slots(NP) * 4;                              // [pose][13]
  PoseM* s_m = reinterpret_cast<PoseM*>(s_sum + AP_POSES * 13);           // [pose]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool mat = p.pose_format == 1;
  const int rank = (int)(blockIdx.x % (unsigned)p.cl);
  const int pose0 = (int)(blockIdx.x / (unsigned)p.cl) * p.pb;
  const int np = min(p.pb, p.n_poses - pose0);
  const int iw = AP_WARPS / p.rw, slots = iw * 64 * NP;
  const int group = warp / iw, first = (warp % iw) * 64 * NP + lane;  // this lane's items: first + 32 k
  // a group's leaves: `own` from the (rank rw + group) own-th on; `branch` of them a branch.  A split
  // takes whole branches or single leaves (ap_plan).
  const int parts = p.rw * p.cl, own = (1 << p.leaves_log2) / parts;
  const int branch = 1 << (p.leaves_log2 - p.branches_log2);
  auto leaf_start = [&](int g, int l) {
    return (int)((long long)p.n_rec * ((rank * p.rw + g) * own + l) >> p.leaves_log2);
  };
  const int tile = AP_TILE / p.rw, per_tile = tile / AP_LEAF;  // leaves of a tile
  for (int k = threadIdx.x; k < np; k += AP_THREADS) s_m[k] = load_pose(p, pose0 + k);
  for (int k = threadIdx.x; k < np * 13; k += AP_THREADS) s_sum[k] = 0.0;

  for (int i0 = 0; i0 < p.n_lig; i0 += p.nb) {
    const int nb = min(p.nb, p.n_lig - i0);
    const int items = np * nb;
    __syncthreads();  // the poses are there; the last pass's sums are read
    // this lane's items: moved beads, ligand types (-1: no item, or no pair row)
    f2 X[NP], Y[NP], Z[NP];
    int lt[2 * NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      float c[2][3];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int it = first + 32 * (2 * k + h);
        c[h][0] = c[h][1] = c[h][2] = 0.f;
        lt[2 * k + h] = -1;
        if (it < items) {
          const float4 x = __ldg(p.lig + i0 + it % nb);
          const PoseM& q = s_m[it / nb];
          const int t = __float_as_int(x.w);
          lt[2 * k + h] = (unsigned)t < (unsigned)p.n_ltypes ? t : -1;
#pragma unroll
          for (int d = 0; d < 3; ++d) c[h][d] = fmaf(x.x, q.m[d], fmaf(x.y, q.m[3 + d], fmaf(x.z, q.m[6 + d], q.t[d])));
        }
      }
      X[k] = pk(c[0][0], c[1][0]);
      Y[k] = pk(c[0][1], c[1][1]);
      Z[k] = pk(c[0][2], c[1][2]);
    }
    // its items' sums in double: E, Gx, Gy, Gz, each a row of the group's items
    double* sums = s_item + (size_t)group * slots * 4 + first;
#pragma unroll
    for (int k = 0; k < 2 * NP; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) sums[c * slots + 32 * k] = 0.0;
    const bool idle = __all_sync(0xffffffffu, first >= items);
    // the pair rows of the lane's items with the current receptor type
    f2 rc[NP], ac[NP], rc8[NP], ac6[NP];
    float cap[2 * NP];
    bool simple = true, use = false;
    int cur = -1;
    double pending[AP_LEVELS][(GRAD ? 4 : 1) * 2 * NP];  // subtrees that wait for their right neighbour
#pragma unroll
    for (int k = 0; k < 2 * NP; ++k) cap[k] = 0.f;
#pragma unroll
    for (int k = 0; k < NP; ++k) rc[k] = ac[k] = rc8[k] = ac6[k] = 0ull;

    for (int l0 = 0; l0 < own; l0 += per_tile) {
      __syncthreads();  // the previous tile has been read
      const int l1 = min(own, l0 + per_tile);
      for (int k = threadIdx.x; k < AP_TILE; k += AP_THREADS) {
        const int g = k / tile, j = leaf_start(g, l0) + k % tile;
        if (g < p.rw && j < leaf_start(g, l1)) {
          const float4 r = __ldg(p.rec + j);
          s_rec[2 * k] = make_float4(-r.x, -r.x, -r.y, -r.y);
          s_rec[2 * k + 1] = make_float4(-r.z, -r.z, r.w, 0.f);
        }
      }
      __syncthreads();
      const int first_bead = leaf_start(group, l0);
      const float4* rec = s_rec + 2 * group * tile;
      for (int l = l0; l < (idle ? l0 : l1); ++l) {
        const int c0 = leaf_start(group, l) - first_bead, c1 = leaf_start(group, l + 1) - first_bead;
        f2 e[NP], gx[NP], gy[NP], gz[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) e[k] = gx[k] = gy[k] = gz[k] = 0ull;
        for (int j = c0; j < c1;) {
          float4 A = rec[2 * j], B = rec[2 * j + 1];
          const int rt = __float_as_int(B.z);
          if (rt != cur) {  // a new receptor type: the rows of this lane's items
            cur = rt;
            use = (unsigned)rt < (unsigned)p.n_rtypes;  // (no row: the bead contributes nothing)
            simple = true;
            if (use) {
              float v[2 * NP][2];
#pragma unroll
              for (int k = 0; k < 2 * NP; ++k) {
                const float4* row = p.pair + ((size_t)max(lt[k], 0) * p.n_rtypes + rt) * 2;
                const float4 q0 = __ldg(row), q1 = __ldg(row + 1);
                v[k][0] = q0.x;
                v[k][1] = q0.y;
                cap[k] = q1.w;
                // attractive, no shift: the plain form on both sides of the minimum
                simple &= q1.x == 1.f && q1.y == 0.f && isfinite(q0.z);
              }
#pragma unroll
              for (int k = 0; k < NP; ++k) {
                rc[k] = pk(v[2 * k][0], v[2 * k + 1][0]);
                ac[k] = pk(v[2 * k][1], v[2 * k + 1][1]);
                rc8[k] = pk(8.f * v[2 * k][0], 8.f * v[2 * k + 1][0]);
                ac6[k] = pk(6.f * v[2 * k][1], 6.f * v[2 * k + 1][1]);
              }
              simple = __all_sync(0xffffffffu, simple);
            }
          }
          // the receptor beads of one type
          auto run = [&](auto simple_form) {
            constexpr bool SIMPLE = decltype(simple_form)::value;
            const f2 two = pk(2.f, 2.f);
            // what only the general form takes; it gives rows of the simple form the same bits
            float emin[2 * NP], rmin2[2 * NP], ivor[2 * NP], epl[2 * NP];
            if (!SIMPLE) {
#pragma unroll
              for (int k = 0; k < 2 * NP; ++k) {
                const float4* row = p.pair + ((size_t)max(lt[k], 0) * p.n_rtypes + cur) * 2;
                const float4 q0 = __ldg(row), q1 = __ldg(row + 1);
                emin[k] = q0.z;
                rmin2[k] = q0.w;
                ivor[k] = q1.x;
                epl[k] = q1.y;
              }
            }
            do {
              const float4 A1 = rec[2 * j + 2], B1 = rec[2 * j + 3];  // (the tile has one more)
              const f2 nx = pk(A.x, A.y), ny = pk(A.z, A.w), nz = pk(B.x, B.y);
#pragma unroll
              for (int k = 0; k < NP; ++k) {
                const f2 dx = add2(X[k], nx), dy = add2(Y[k], ny), dz = add2(Z[k], nz);
                const f2 dsq = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                float q0, q1;
                upk(dsq, q0, q1);
                const float d0 = fmaxf(q0, cap[2 * k]), d1 = fmaxf(q1, cap[2 * k + 1]);
                const f2 d2 = pk(d0, d1);
                // n = -1/d2: the approximate reciprocal and one Newton step (within 1 ulp)
                const f2 a = pk(rcp_approx(-d0), rcp_approx(-d1));
                const f2 n = mul2(a, fma2(d2, a, two));
                const f2 n3 = mul2(mul2(n, n), n);
                const f2 u = fma2(rc[k], n, ac[k]);                         // (rc r^-2 - ac) r^-6 = u n3
                f2 gm = mul2(mul2(n3, n), fma2(rc8[k], n, ac6[k]));  // 2 dnonbon/d(d^2)
                float g0_, g1_;
                upk(gm, g0_, g1_);
                const bool b0 = SIMPLE || d0 < rmin2[2 * k], b1 = SIMPLE || d1 < rmin2[2 * k + 1];
                if (SIMPLE && !CUT) {
                  e[k] = fma2(u, n3, e[k]);
                } else if (!CUT) {
                  float u0, u1;
                  upk(u, u0, u1);
                  e[k] = fma2(pk(b0 ? u0 : ivor[2 * k] * u0, b1 ? u1 : ivor[2 * k + 1] * u1), n3, e[k]);
                  e[k] = add2(e[k], pk(b0 ? fmaf(ivor[2 * k] - 1.f, emin[2 * k], -epl[2 * k]) : -epl[2 * k],
                                       b1 ? fmaf(ivor[2 * k + 1] - 1.f, emin[2 * k + 1], -epl[2 * k + 1]) : -epl[2 * k + 1]));
                } else {
                  float e0, e1;
                  upk(mul2(u, n3), e0, e1);
                  if (!SIMPLE) {
                    e0 = (b0 ? fmaf(ivor[2 * k] - 1.f, emin[2 * k], e0) : ivor[2 * k] * e0) - epl[2 * k];
                    e1 = (b1 ? fmaf(ivor[2 * k + 1] - 1.f, emin[2 * k + 1], e1) : ivor[2 * k + 1] * e1) - epl[2 * k + 1];
                  }
                  e0 = q0 < p.rcut2 ? e0 : 0.f;
                  e1 = q1 < p.rcut2 ? e1 : 0.f;
                  e[k] = add2(e[k], pk(e0, e1));
                }
                if (GRAD) {
                  if (!SIMPLE) {
                    g0_ = b0 ? g0_ : ivor[2 * k] * g0_;
                    g1_ = b1 ? g1_ : ivor[2 * k + 1] * g1_;
                  }
                  g0_ = (CUT ? (q0 < cap[2 * k]) | !(q0 < p.rcut2) : q0 < cap[2 * k]) ? 0.f : g0_;
                  g1_ = (CUT ? (q1 < cap[2 * k + 1]) | !(q1 < p.rcut2) : q1 < cap[2 * k + 1]) ? 0.f : g1_;
                  gm = pk(g0_, g1_);
                  gx[k] = fma2(gm, dx, gx[k]);
                  gy[k] = fma2(gm, dy, gy[k]);
                  gz[k] = fma2(gm, dz, gz[k]);
                }
              }
              A = A1;
              B = B1;
              ++j;
            } while (j < c1 && __float_as_int(B.z) == cur);
          };
          if (!use) ++j;
          else if (simple) run(std::true_type{});
          else run(std::false_type{});
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) {
          const f2 v[4] = {e[k], gx[k], gy[k], gz[k]};
#pragma unroll
          for (int c = 0; c < (GRAD ? 4 : 1); ++c) {
            float a, b;
            upk(v[c], a, b);
            sums[c * slots + 64 * k] += a;
            sums[c * slots + 64 * k + 32] += b;
          }
        }
        if (own > branch && ((l + 1) & (branch - 1)) == 0) {  // a branch is done, others follow or went before
          const int b = l / branch;
          double v[(GRAD ? 4 : 1) * 2 * NP];
#pragma unroll
          for (int k = 0; k < (GRAD ? 4 : 1) * 2 * NP; ++k) {
            double* a = sums + k / (2 * NP) * slots + 32 * (k % (2 * NP));
            v[k] = *a;
            *a = 0.0;
          }
          int level = 0;
          for (; b >> level & 1; ++level)
#pragma unroll
            for (int k = 0; k < (GRAD ? 4 : 1) * 2 * NP; ++k) v[k] = pending[level][k] + v[k];
#pragma unroll
          for (int k = 0; k < (GRAD ? 4 : 1) * 2 * NP; ++k) {
            if (l + 1 == own) sums[k / (2 * NP) * slots + 32 * (k % (2 * NP))] = v[k];
            else pending[level][k] = v[k];
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 2 * NP; ++k)
      if (lt[k] < 0) {  // no pair row: the bead contributes nothing
#pragma unroll
        for (int c = 0; c < 4; ++c) sums[c * slots + 32 * k] = 0.0;
      }
    // the upper levels of the tree: the groups' (and the cluster's) sums of an item and value are
    // taken to group 0's place in the block that sums the item's pose, the (pose mod cl)-th; only
    // the lanes that take them read or write that place meanwhile
    cg::cluster_group cluster = cg::this_cluster();
    if (p.cl > 1) cluster.sync();
    else __syncthreads();
    if (parts > 1) {
      const int rw_log2 = __ffs(p.rw) - 1, units = items * (GRAD ? 4 : 1);
      const unsigned item0 = (unsigned)__cvta_generic_to_shared(s_item), group_bytes = (unsigned)slots * 32u;
      const int n_branch = min(parts, 1 << p.branches_log2), each = parts / n_branch;  // (up to 4 leaves of a branch)
      auto place = [&](int u) { return item0 + (unsigned)(u / items * slots + u % items) * 8u; };
      auto part = [&](unsigned at, int n) {
        return ld_cluster(at + (unsigned)(n & (p.rw - 1)) * group_bytes, n >> rw_log2);
      };
      if (parts <= 8) {  // by one thread
        auto take = [&](auto count) {
          constexpr int N = decltype(count)::value;
          for (int u = rank * AP_THREADS + (int)threadIdx.x; u < units; u += p.cl * AP_THREADS) {
            const unsigned at = place(u);
            double t[N];
#pragma unroll 1
            for (int f = 0; f < each; ++f)
#pragma unroll
              for (int c = 0; c < N; ++c) {
                const double a = part(at, c * each + f);
                t[c] = f > 0 ? t[c] + a : a;
              }
#pragma unroll
            for (int w = 1; w < N; w *= 2)
#pragma unroll
              for (int c = 0; c < N; c += 2 * w) t[c] += t[c + w];
            st_cluster(at, u % items / nb % p.cl, t[0]);
          }
        };
        if (n_branch == 1) take(std::integral_constant<int, 1>{});
        else if (n_branch == 2) take(std::integral_constant<int, 2>{});
        else if (n_branch == 4) take(std::integral_constant<int, 4>{});
        else take(std::integral_constant<int, 8>{});
      } else {  // by eight lanes, a branch of eight each
        const int sub = lane & 7;
        for (int u0 = (rank * AP_WARPS + warp) * 4; u0 < units; u0 += p.cl * AP_WARPS * 4) {  // (warp-uniform)
          const int u = min(u0 + (lane >> 3), units - 1);
          const unsigned at = place(u);
          double sum = 0.0, wait[3] = {0.0, 0.0, 0.0};  // one, two and four eights that wait for their neighbour
#pragma unroll 1
          for (int c0 = 0; c0 < n_branch; c0 += 8) {
            double a[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) a[f] = part(at, min(c0 + sub, n_branch - 1) * each + min(f, each - 1));
            sum = a[0];
#pragma unroll
            for (int f = 1; f < 4; ++f) sum = f < each ? sum + a[f] : sum;
            if (c0 + sub >= n_branch) sum = 0.0;
#pragma unroll
            for (int w = 1; w < 8; w *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            bool done = false;
#pragma unroll
            for (int k = 0; k < 3; ++k)
              if (!done) {
                done = (c0 >> (3 + k) & 1) == 0;
                if (done) wait[k] = sum;
                else sum = wait[k] + sum;
              }
          }
          if (sub == 0 && u0 + (lane >> 3) < units) st_cluster(at, u % items / nb % p.cl, sum);
        }
      }
      if (p.cl > 1) cluster.sync();
      else __syncthreads();
    }
    // a pose's sums over its beads, 64 at a time: 8 lanes per pose
    for (int q0 = rank; q0 < np; q0 += AP_THREADS / 8 * p.cl) {
      const int q = q0 + (int)threadIdx.x / 8 * p.cl;
      for (int c0 = 0; c0 < nb; c0 += AP_CHUNK) {
        double acc[13];
#pragma unroll
        for (int k = 0; k < 13; ++k) acc[k] = 0.0;
        if (q < np) {
          const PoseM& pm = s_m[q];
          for (int i = c0 + (threadIdx.x & 7); i < min(nb, c0 + AP_CHUNK); i += 8) {
            double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < (GRAD ? 4 : 1); ++k) v[k] = s_item[k * slots + q * nb + i];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] += v[k];
            if (GRAD) {
              const float4 x = __ldg(p.lig + i0 + i);
              if (mat) {  // dE/dM[r][c] = sum_i x_r g_c
                const double xr[3] = {x.x, x.y, x.z};
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                  for (int c = 0; c < 3; ++c) acc[4 + r * 3 + c] += xr[r] * v[1 + c];
              } else {  // torque about the pose centre: (X - t) x g, X - t = x M
                double a[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) a[d] = fmaf(x.x, pm.m[d], fmaf(x.y, pm.m[3 + d], x.z * pm.m[6 + d]));
                acc[4] += a[1] * v[3] - a[2] * v[2];
                acc[5] += a[2] * v[1] - a[0] * v[3];
                acc[6] += a[0] * v[2] - a[1] * v[1];
              }
            }
          }
        }
        const int nv = !GRAD ? 1 : mat ? 13 : 7;
#pragma unroll
        for (int k = 0; k < 13; ++k)
          if (k < nv) {
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
            if (q < np && (threadIdx.x & 7) == 0) s_sum[q * 13 + k] += acc[k];
          }
      }
    }
  }
  __syncthreads();
  for (int q = rank + (int)threadIdx.x * p.cl; q < np; q += AP_THREADS * p.cl) {
    const double* a = s_sum + q * 13;
    const long long b = pose0 + q;
    p.energy[b] = (float)a[0];
    if (GRAD) {
      if (mat) {
        float* g = p.grad + b * 16;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
          for (int c = 0; c < 3; ++c) g[r * 4 + c] = (float)a[4 + r * 3 + c];
          g[r * 4 + 3] = 0.f;
        }
        g[12] = (float)a[1]; g[13] = (float)a[2]; g[14] = (float)a[3]; g[15] = 0.f;
      } else {
        // dE/d(angle_k) = w_k . torque with w_phi = (0,0,1), w_psi = (-sin phi, cos phi, 0),
        // w_theta = -(cos phi sin psi, sin phi sin psi, cos psi)
        const PoseM& m = s_m[q];
        float* g = p.grad + b * 6;
        const double tx = a[4], ty = a[5], tz = a[6];
        g[0] = (float)tz;
        g[1] = (float)(-m.sphi * tx + m.cphi * ty);
        g[2] = (float)(-(m.cphi * m.spsi * tx + m.sphi * m.spsi * ty + m.cpsi * tz));
        g[3] = (float)a[1]; g[4] = (float)a[2]; g[5] = (float)a[3];
      }
    }
  }
}

typedef void (*ApKernel)(AllPairsParams);
template <int NP>
static ApKernel ap_kernel(bool cut, bool grad) {
  return cut ? (grad ? allpairs_kernel<NP, true, true> : allpairs_kernel<NP, true, false>)
             : (grad ? allpairs_kernel<NP, false, true> : allpairs_kernel<NP, false, false>);
}

// The split of a call: packed pairs per lane, receptor groups per block, blocks
// per cluster.  The time is taken as waves of resident blocks (3 per SM at one
// packed pair per lane, 2 at two, by registers; clusters of 4 and 8 leave 8 and 16 % of the SMs
// without a block).  A block alone on an SM takes its steps (a receptor bead against a lane's
// items; 1.2 at two packed pairs), 20 steps per pass over the ligand, 20 for its start and
// sums and 2.7 per block of its cluster; each further block of busy warps adds 0.2 (0.435)
// of a step to a step.  Fitted to all splits of 75 calls of 60-17 000 receptor beads, 8-301 ligand beads
// and 1-60 000 poses: the split taken is within 3 % of the fastest on average (10 poses of 301 beads: 26 %),
// where the slowest is 3 to 10 times slower.
struct ApPlan {
  int np, rw, cl, pb, nb;
};
static ApPlan ap_plan(long long n_poses, int n_lig, int n_rec, int sms) {
  const int leaves_log2 = ap_leaves_log2(n_rec), branches = 1 << ap_branches_log2(leaves_log2);
  ApPlan best = {1, 1, 1, 1, 1};
  double best_t = 1e300;
  for (int np = 1; np <= 2; ++np)
    for (int rw = 1; rw <= AP_WARPS; rw *= 2)
      for (int cl = 1; cl <= 8; cl *= 2) {
        if (rw * cl > branches && rw * cl != 1 << leaves_log2) continue;  // whole branches, or single leaves
        const int slots = (AP_WARPS / rw) * 64 * np;
        ApPlan q = {np, rw, cl, 1, slots};
        if (n_lig <= slots) {
          q.pb = slots / n_lig < AP_POSES ? slots / n_lig : AP_POSES;
          q.nb = n_lig;
        }
        if (q.pb > n_poses) q.pb = (int)n_poses;
        const double passes = (double)(((long long)n_lig + q.nb - 1) / q.nb);
        const int items = q.pb * (q.nb < n_lig ? q.nb : n_lig);
        const double busy = ((items + 64 * np - 1) / (64 * np)) * rw / (double)AP_WARPS;  // of a block's warps
        const double b = np == 1 ? 0.2 : 0.435;
        auto wave = [&](int k) {  // k blocks per SM
          const double step = 1.0 - b + b * k * busy, slow = step > 1.0 ? step : 1.0;
          return passes * ((np == 1 ? 1.0 : 1.2) * step * n_rec / (rw * cl) + 20.0 * slow) + (20.0 + 2.7 * cl) * slow;
        };
        const int resident = np == 1 ? 3 : 2;
        const double at_once = cl == 8 ? 0.84 * sms : cl == 4 ? 0.916 * sms : sms;  // blocks, one per SM
        const long long blocks = (n_poses + q.pb - 1) / q.pb * cl;
        const double full = floor(blocks / (resident * at_once));
        const int last = (int)ceil((blocks - full * resident * at_once) / at_once - 1e-9);  // on an SM, in the last wave
        const double t = full * wave(resident) + (last > 0 ? wave(last) : 0.0);
        if (t < best_t) {
          best_t = t;
          best = q;
        }
      }
  return best;
}

}  // namespace att

using namespace att;

extern "C" int att_allpairs_energy(const float* rec_dev, int n_rec, const float* lig_dev, int n_lig,
                                   const float* pose_dev, int n_poses, int pose_format, const float* pair_dev,
                                   int n_rtypes, int n_ltypes, float rcut, float* energy_dev, float* grad_dev,
                                   void* stream) {
  auto bad = [](const char* m) { return report_error(ATT_E_INVALID, m); };
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (n_rec < 0 || n_lig < 1 || n_poses < 0) return bad("att_allpairs_energy: n_rec >= 0, n_lig >= 1, n_poses >= 0");
  if (n_rtypes < 1 || n_ltypes < 1) return bad("att_allpairs_energy: empty pair table");
  if (pose_format != 0 && pose_format != 1) return bad("att_allpairs_energy: pose_format must be 0 or 1");
  if ((n_rec && !rec_dev) || !lig_dev || !pair_dev || (n_poses && (!pose_dev || !energy_dev)))
    return bad("att_allpairs_energy: NULL buffer");
  if ((rec_dev && !al16(rec_dev)) || !al16(lig_dev) || (reinterpret_cast<uintptr_t>(pair_dev) & 31u))
    return bad("att_allpairs_energy: receptor and ligand must be 16-byte, the pair table 32-byte aligned");
  if (!(rcut >= 0.f)) return bad("att_allpairs_energy: rcut must be >= 0 (0 = no cutoff)");
  if (n_poses == 0) return ATT_OK;
  AllPairsParams p;
  p.rec = reinterpret_cast<const float4*>(rec_dev);
  p.lig = reinterpret_cast<const float4*>(lig_dev);
  p.pose = pose_dev;
  p.pair = reinterpret_cast<const float4*>(pair_dev);
  p.energy = energy_dev;
  p.grad = grad_dev;
  p.rcut2 = rcut > 0.f ? rcut * rcut : 0.f;
  p.n_rec = n_rec;
  p.n_lig = n_lig;
  p.n_poses = n_poses;
  p.pose_format = pose_format;
  p.n_rtypes = n_rtypes;
  p.n_ltypes = n_ltypes;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const ApPlan plan = ap_plan(n_poses, n_lig, n_rec, sms);
  p.rw = plan.rw;
  p.cl = plan.cl;
  p.pb = plan.pb;
  p.nb = plan.nb;
  p.leaves_log2 = ap_leaves_log2(n_rec);
  p.branches_log2 = ap_branches_log2(p.leaves_log2);
  const bool cut = p.rcut2 > 0.f, grad = grad_dev != nullptr;
  const ApKernel kernel = plan.np == 1 ? ap_kernel<1>(cut, grad) : ap_kernel<2>(cut, grad);
  const size_t smem = plan.np == 1 ? ap_smem(1) : ap_smem(2);
  cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return report_error(ATT_E_CUDA, cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)plan.cl;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(((long long)n_poses + plan.pb - 1) / plan.pb * plan.cl));
  cfg.blockDim = dim3(AP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = &attr;
  cfg.numAttrs = plan.cl > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) return report_error(ATT_E_CUDA, cudaGetErrorString(e));
  return ATT_OK;
}
