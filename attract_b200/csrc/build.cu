// Receptor-side kernels: potential grid builder (K3), neighbour-grid builder
// (K4: count -> scan -> fill) and the dense-grid -> brick repack (K5).
#include <math.h>

#include "common.cuh"

namespace att {

// ---------------------------------------------------------------------------
// Receptor beads near a set of grid points
// ---------------------------------------------------------------------------
// The builders' sums and lists take a point's beads in index order, from those
// within a radius.  A block first keeps the beads that come within the radius
// of its points' bounding box -- in index order, so that sums and lists are
// those of a loop over all beads -- and its threads look at these only.  The
// box test takes the box's nearest coordinate on each axis through the same
// rounded operations as the point test; those are monotone, so no bead that
// passes at some point of the box fails it.

// The ranks of this thread's elements among those that the block's threads take,
// and their number.  Element k of a thread is the (THREADS k + thread)-th: ranks
// follow the index.  (w: 32 words; a barrier has to lie between two uses)
template <int THREADS>
__device__ __forceinline__ void block_ranks(const bool (&take)[1024 / THREADS], unsigned* w, int (&rank)[1024 / THREADS],
                                            int& total) {
  constexpr int W = THREADS / 32, N = 1024 / THREADS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned m[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    m[k] = __ballot_sync(0xffffffffu, take[k]);
    if (lane == 0) w[k * W + warp] = __popc(m[k]);
  }
  __syncthreads();
  const unsigned c = w[lane];
  unsigned inc = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += t;
  }
  total = (int)__shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
  for (int k = 0; k < N; ++k)
    rank[k] = (int)(__shfl_sync(0xffffffffu, inc - c, k * W + warp) + __popc(m[k] & ((1u << lane) - 1u)));
}

__device__ __forceinline__ float nearest_in(float r, float lo, float hi) { return fminf(fmaxf(r, lo), hi); }

// ---------------------------------------------------------------------------
// K3: energy + force voxels (test-calc-grid-energy.py:154-196, with forces)
// ---------------------------------------------------------------------------
// A block serves 4 x 8 x 8 grid points and 8 ligand types.  Bound by the FP64
// pipe: per point, bead within the cutoff and type, 10 double operations (sums
// are held in double), the distance, its reciprocal and the square root once for the 8
// types.  The box keeps about 113 of 2500 beads (0.0093 / A^3, cutoff 10 A) of
// which 39 reach a point; the pair rows are staged as doubles, read by a whole
// warp at once.  2500 beads, 32 types, 1.44 M + 0.74 M points: 132.3 ms with
// every bead tested per point and type, 1.96 ms with this kernel.
constexpr int BP_THREADS = 256;
constexpr int BP_TYPES = 8;    // ligand types per block
constexpr int BP_STAGE = 32;   // beads whose pair rows are staged at a time
constexpr int BP_LIST = 1408;  // beads kept by the box before their sums are formed
constexpr int BP_STEP = 1024;  // beads tested against the box between two barriers

struct PairRowD {  // one (bead, ligand type) in double
  double rc, ac, rc4, ac3;            // 4 rc, 3 ac
  double ep, gp;                      // plateau energy, derivative
  double cap, rmin2, ivor, shift;     // the general form: cap, sign, (ivor - 1) emin
};

__device__ __forceinline__ double dist2_d(double dx, double dy, double dz) { return fma(dz, dz, fma(dy, dy, dx * dx)); }

__global__ void __launch_bounds__(BP_THREADS, 2)
build_potential_kernel(AttGridGeom g, const float4* __restrict__ rec, int n_rec, const float4* __restrict__ pair,
                       int n_rtypes, int n_ltypes, float cutoff2, int outer, int tiles_y, int tiles_z,
                       float4* __restrict__ out) {
  __shared__ float4 s_rec[BP_LIST];
  __shared__ PairRowD s_row[BP_STAGE][BP_TYPES];
  __shared__ double s_xyz[BP_STAGE][3];
  __shared__ unsigned s_w[32];
  const int nx = outer ? g.dim2[0] : g.dim[0];
  const int ny = outer ? g.dim2[1] : g.dim[1];
  const int nz = outer ? g.dim2[2] : g.dim[2];
  const int lt0 = blockIdx.y * BP_TYPES;
  const int nt = min(BP_TYPES, n_ltypes - lt0);
  const int tz = blockIdx.x % tiles_z, txy = blockIdx.x / tiles_z;
  const int x0 = (txy / tiles_y) * 4, y0 = (txy % tiles_y) * 8, z0 = tz * 8;
  // a warp serves 2 x 4 x 4 points: its points meet the same beads
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ix = x0 + ((warp >> 2) & 1) * 2 + (lane >> 4);
  const int iy = y0 + ((warp >> 1) & 1) * 4 + ((lane >> 2) & 3);
  const int iz = z0 + (warp & 1) * 4 + (lane & 3);
  const bool live = ix < nx && iy < ny && iz < nz;
  auto at = [&](int axis, int i) {
    return !outer ? g.origin[axis] + i * g.spacing : g.origin[axis] + (2.f * i - g.extension) * g.spacing;
  };
  const double px = at(0, ix), py = at(1, iy), pz = at(2, iz);
  const float lx = at(0, x0), hx = at(0, min(x0 + 3, nx - 1)), ly = at(1, y0), hy = at(1, min(y0 + 7, ny - 1));
  const float lz = at(2, z0), hz = at(2, min(z0 + 7, nz - 1));
  const double p = g.plateau;
  const double p2 = p * p;
  double e[BP_TYPES], fx[BP_TYPES], fy[BP_TYPES], fz[BP_TYPES];
#pragma unroll
  for (int t = 0; t < BP_TYPES; ++t) e[t] = fx[t] = fy[t] = fz[t] = 0.0;

  int kept = 0;
  for (int base = 0; base < n_rec; base += BP_STEP) {
    constexpr int N = BP_STEP / BP_THREADS;
    float4 r[N];
    bool take[N];
    int rank[N], n = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = base + k * BP_THREADS + (int)threadIdx.x;
      take[k] = i < n_rec;
      if (take[k]) r[k] = rec[i];
    }
#pragma unroll
    for (int k = 0; k < N; ++k)
      take[k] = take[k] && (unsigned)__float_as_int(r[k].w) < (unsigned)n_rtypes &&
                dist2_d((double)nearest_in(r[k].x, lx, hx) - r[k].x, (double)nearest_in(r[k].y, ly, hy) - r[k].y,
                        (double)nearest_in(r[k].z, lz, hz) - r[k].z) < cutoff2;
    block_ranks<BP_THREADS>(take, s_w, rank, n);
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (take[k]) s_rec[kept + rank[k]] = r[k];
    kept += n;
    __syncthreads();  // the list written, the warps' counts read
    if (kept + BP_STEP <= BP_LIST && base + BP_STEP < n_rec) continue;
    for (int k0 = 0; k0 < kept; k0 += BP_STAGE) {
      const int m = min(BP_STAGE, kept - k0);
      bool simple = true;
      for (int q = threadIdx.x; q < m * BP_TYPES; q += BP_THREADS) {
        const int k = q / BP_TYPES, t = q % BP_TYPES;
        const float4 rk = s_rec[k0 + k];
        if (t < 3) s_xyz[k][t] = t == 0 ? rk.x : t == 1 ? rk.y : rk.z;
        if (t >= nt) continue;
        const float4* prow = pair + ((long long)(lt0 + t) * n_rtypes + __float_as_int(rk.w)) * 2;
        const float4 q0 = prow[0], q1 = prow[1];  // rc ac emin rmin2 | ivor eplat gplat rcap2
        PairRowD& w = s_row[k][t];
        w.rc = q0.x; w.ac = q0.y; w.rc4 = 4.0 * q0.x; w.ac3 = 3.0 * q0.y;
        w.ep = q1.y; w.gp = q1.z;
        w.cap = q1.w; w.rmin2 = q0.w; w.ivor = q1.x; w.shift = ((double)q1.x - 1.0) * q0.z;
        simple &= q1.x == 1.f && w.shift == 0.0 && (double)q1.w <= p2;
      }
      // simple: attractive pairs (ivor = 1) with a cap inside the plateau only
      const bool all_simple = __syncthreads_and(simple);
      if (live) {
        for (int k = 0; k < m; ++k) {
          const double dx = px - s_xyz[k][0], dy = py - s_xyz[k][1], dz = pz - s_xyz[k][2];
          const double dsq = dist2_d(dx, dy, dz);
          if (!(dsq < cutoff2)) continue;
          if (dsq < p2) {
            const double pl = dsq > 0.0 ? -2.0 * p / sqrt(dsq) : 0.0;
#pragma unroll
            for (int t = 0; t < BP_TYPES; ++t) {
              if (t < nt) {
                const PairRowD& w = s_row[k][t];
                const double sc = w.gp * pl;
                e[t] += w.ep;
                fx[t] = fma(sc, dx, fx[t]);
                fy[t] = fma(sc, dy, fy[t]);
                fz[t] = fma(sc, dz, fz[t]);
              }
            }
          } else {
            const double rr2 = 1.0 / dsq;
            const double rr6 = rr2 * rr2 * rr2;
            const double m8 = -2.0 * (rr6 * rr2);
            if (all_simple) {
#pragma unroll
              for (int t = 0; t < BP_TYPES; ++t) {
                if (t < nt) {
                  const PairRowD& w = s_row[k][t];
                  e[t] = fma(fma(w.rc, rr2, -w.ac), rr6, e[t]);
                  const double sc = m8 * fma(-w.rc4, rr2, w.ac3);
                  fx[t] = fma(sc, dx, fx[t]);
                  fy[t] = fma(sc, dy, fy[t]);
                  fz[t] = fma(sc, dz, fz[t]);
                }
              }
            } else {
#pragma unroll
              for (int t = 0; t < BP_TYPES; ++t) {
                if (t < nt) {
                  const PairRowD& w = s_row[k][t];
                  double r2 = rr2, r6 = rr6, d2 = dsq, sc = m8;
                  if (dsq < w.cap) {  // constant below the cap: its energy, no force
                    d2 = w.cap;
                    r2 = 1.0 / d2;
                    r6 = r2 * r2 * r2;
                    sc = 0.0;
                  }
                  const double vlj = fma(w.rc, r2, -w.ac) * r6;
                  const bool near = d2 < w.rmin2;
                  e[t] += near ? vlj + w.shift : w.ivor * vlj;
                  if (sc != 0.0) sc *= (near ? 1.0 : w.ivor) * fma(-w.rc4, r2, w.ac3);
                  fx[t] = fma(sc, dx, fx[t]);
                  fy[t] = fma(sc, dy, fy[t]);
                  fz[t] = fma(sc, dz, fz[t]);
                }
              }
            }
          }
        }
      }
      __syncthreads();  // the staged rows (and, after the last, the list) are read
    }
    kept = 0;
  }
  if (live) {
    const long long npts = (long long)nx * ny * nz, pt = ((long long)ix * ny + iy) * nz + iz;
#pragma unroll
    for (int t = 0; t < BP_TYPES; ++t)
      if (t < nt) out[(lt0 + t) * npts + pt] = make_float4((float)e[t], (float)fx[t], (float)fy[t], (float)fz[t]);
  }
}

cudaError_t launch_build_potential(const AttGridGeom& g, const float* rec, int n_rec, const float* pair,
                                   int n_rtypes, int n_ltypes, float cutoff, int outer, float* out,
                                   cudaStream_t st) {
  const int* d = outer ? g.dim2 : g.dim;
  const int tx = (d[0] + 3) / 4, ty = (d[1] + 7) / 8, tz = (d[2] + 7) / 8;
  dim3 grid((unsigned)((long long)tx * ty * tz), (unsigned)((n_ltypes + BP_TYPES - 1) / BP_TYPES));
  build_potential_kernel<<<grid, BP_THREADS, 0, st>>>(g, reinterpret_cast<const float4*>(rec), n_rec,
                                                      reinterpret_cast<const float4*>(pair), n_rtypes, n_ltypes,
                                                      cutoff * cutoff, outer, ty, tz, reinterpret_cast<float4*>(out));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// K4: neighbour lists (test-calc-grid-energy.py:90-103) as CSR
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 1024;

// Grid point and squared distance with every operation rounded on its own
// (no contraction into FMA): the list membership test d^2 <= r^2 is then a
// fixed float32 computation that a host restatement reproduces bit for bit.
__device__ __forceinline__ float coord_of(const AttGridGeom& g, int axis, int i) {
  return __fadd_rn(g.origin[axis], __fmul_rn((float)i, g.spacing));
}

__device__ __forceinline__ float dist2_rn(float x, float y, float z, const float4& r) {
  const float dx = __fsub_rn(x, r.x), dy = __fsub_rn(y, r.y), dz = __fsub_rn(z, r.z);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

__device__ __forceinline__ int3 index_of(const AttGridGeom& g, long long v) {
  const unsigned ny = (unsigned)g.dim[1], nz = (unsigned)g.dim[2];
  if (v <= 0xffffffffLL) {  // 32-bit divisions where they do
    const unsigned w = (unsigned)v, q = w / nz;
    return make_int3((int)(q / ny), (int)(q % ny), (int)(w % nz));
  }
  const long long q = v / nz;
  return make_int3((int)(q / ny), (int)(q % ny), (int)(v % nz));
}

// the bounding box of the consecutive grid points from index a to index b
struct PointBox {
  float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ PointBox box_of(const AttGridGeom& g, const int3& a, const int3& b) {
  const bool plane = a.x == b.x, row = plane && a.y == b.y;
  PointBox q;
  q.lx = coord_of(g, 0, a.x);
  q.hx = coord_of(g, 0, b.x);
  q.ly = coord_of(g, 1, plane ? a.y : 0);
  q.hy = coord_of(g, 1, plane ? b.y : g.dim[1] - 1);
  q.lz = coord_of(g, 2, row ? a.z : 0);
  q.hz = coord_of(g, 2, row ? b.z : g.dim[2] - 1);
  return q;
}
__device__ __forceinline__ bool box_reached(const PointBox& q, const float4& r, float r2) {
  return dist2_rn(nearest_in(r.x, q.lx, q.hx), nearest_in(r.y, q.ly, q.hy), nearest_in(r.z, q.lz, q.hz), r) <= r2;
}

// A block serves NB_POINTS consecutive points, NB_THREADS at a time.
constexpr int NB_THREADS = 512, NB_POINTS = 4096, NB_SUB = NB_POINTS / NB_THREADS;
constexpr int NB_LIST = 1536;  // beads kept by the block's box before its points look at them
constexpr int NB_STEP = 1024;  // beads tested against the box between two barriers

// Calls hit(s, bead, n) for every bead within the radius of this thread's s-th
// point v0 + NB_THREADS * s + thread, in index order; n is what the previous call for
// the point returned (0 at first), and s_n[s][thread] the last one.  The block
// keeps the beads near its points (about 75 of 2500 on the x4 list grid, whose
// blocks are nine rows 100 A long), a warp those near its 32 points (about 11),
// and only these are tested per point.  A warp within one row of z (nearly all)
// has one x and y: fl(fl(dx dx) + fl(dy dy)) is formed once per bead and warp.
template <class Hit>
__device__ __forceinline__ void near_beads(const AttGridGeom& g, const float4* __restrict__ rec, int n_rec, float r2,
                                           long long nvox, unsigned (&s_n)[NB_SUB][NB_THREADS], Hit hit) {
  __shared__ float4 s_rec[NB_LIST];
  __shared__ unsigned short s_idx[NB_LIST];
  __shared__ unsigned s_w[32];
  const long long v0 = (long long)blockIdx.x * NB_POINTS, last = nvox - 1;
  const int lane = threadIdx.x & 31;
  const PointBox block = box_of(g, index_of(g, v0), index_of(g, min(v0 + NB_POINTS - 1, last)));
#pragma unroll
  for (int s = 0; s < NB_SUB; ++s) s_n[s][threadIdx.x] = 0u;
  int kept = 0;
  for (int base = 0; base < n_rec; base += NB_STEP) {
    constexpr int N = NB_STEP / NB_THREADS;
    float4 r[N];
    bool take[N];
    int rank[N], n = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = base + k * NB_THREADS + (int)threadIdx.x;
      take[k] = i < n_rec;
      if (take[k]) r[k] = rec[i];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) take[k] = take[k] && box_reached(block, r[k], r2);
    block_ranks<NB_THREADS>(take, s_w, rank, n);
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (take[k]) {
        s_rec[kept + rank[k]] = r[k];
        s_idx[kept + rank[k]] = (unsigned short)(base + k * NB_THREADS + (int)threadIdx.x);
      }
    kept += n;
    __syncthreads();  // the list written, the warps' counts read
    if (kept == 0 || (kept + NB_STEP <= NB_LIST && base + NB_STEP < n_rec)) continue;
    int3 me = index_of(g, min(v0 + threadIdx.x, last));
    for (int s = 0; s < NB_SUB; ++s) {
      const long long w0 = v0 + s * NB_THREADS + (threadIdx.x & ~31);
      if (w0 > last) break;
      const bool live = w0 + lane <= last;
      const float x = coord_of(g, 0, me.x), y = coord_of(g, 1, me.y), z = coord_of(g, 2, me.z);
      unsigned have = s_n[s][threadIdx.x];
      int3 a;  // this warp's first point
      a.x = __shfl_sync(0xffffffffu, me.x, 0);
      a.y = __shfl_sync(0xffffffffu, me.y, 0);
      if (__all_sync(0xffffffffu, live & (me.x == a.x) & (me.y == a.y))) {
        const float lz = __shfl_sync(0xffffffffu, z, 0), hz = __shfl_sync(0xffffffffu, z, 31);
        for (int c0 = 0; c0 < kept; c0 += 32) {
          const int c = c0 + lane;
          const float4 q = s_rec[min(c, kept - 1)];
          const float dx = __fsub_rn(x, q.x), dy = __fsub_rn(y, q.y);
          const float dxy = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
          const float dn = __fsub_rn(nearest_in(q.z, lz, hz), q.z);
          unsigned m = __ballot_sync(0xffffffffu, c < kept && __fadd_rn(dxy, __fmul_rn(dn, dn)) <= r2);
          while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            const float dz = __fsub_rn(z, __shfl_sync(0xffffffffu, q.z, b));
            if (__fadd_rn(__shfl_sync(0xffffffffu, dxy, b), __fmul_rn(dz, dz)) <= r2) have = hit(s, (int)s_idx[c0 + b], have);
          }
        }
      } else {
        int3 e;  // and its last
        a.z = __shfl_sync(0xffffffffu, me.z, 0);
        e.x = __shfl_sync(0xffffffffu, me.x, 31);
        e.y = __shfl_sync(0xffffffffu, me.y, 31);
        e.z = __shfl_sync(0xffffffffu, me.z, 31);
        const PointBox mine = box_of(g, a, e);
        for (int c0 = 0; c0 < kept; c0 += 32) {
          const int c = c0 + lane;
          unsigned m = __ballot_sync(0xffffffffu, c < kept && box_reached(mine, s_rec[min(c, kept - 1)], r2));
          while (m) {
            const int q = c0 + __ffs(m) - 1;
            m &= m - 1;
            if (live && dist2_rn(x, y, z, s_rec[q]) <= r2) have = hit(s, (int)s_idx[q], have);
          }
        }
      }
      s_n[s][threadIdx.x] = have;
      // the point NB_THREADS further on
      if (w0 + lane + NB_THREADS <= last) {
        me.z += NB_THREADS;
        if (me.z >= g.dim[2]) {
          const int rows = me.z / g.dim[2];
          me.z -= rows * g.dim[2];
          me.y += rows;
          if (me.y >= g.dim[1]) {
            const int planes = me.y / g.dim[1];
            me.y -= planes * g.dim[1];
            me.x += planes;
          }
        }
      } else {
        me = index_of(g, last);
      }
    }
    kept = 0;
    __syncthreads();  // the list is read
  }
}

// count + exclusive scan within each 1024 points; their totals to ws.  2500
// beads, radius 5.2 A, 90.5 M points: 80.5 ms with every bead tested per point,
// 0.97 ms now.
__global__ void __launch_bounds__(NB_THREADS, 3)
nb_count_kernel(AttGridGeom g, const float4* __restrict__ rec, int n_rec, float r2, uint2* __restrict__ hdr,
                unsigned* __restrict__ ws, long long nvox) {
  constexpr int W = NB_THREADS / 32, GROUPS = SCAN_THREADS / NB_THREADS;
  __shared__ unsigned s_n[NB_SUB][NB_THREADS];
  __shared__ unsigned wsum[NB_SUB][W];
  near_beads(g, rec, n_rec, r2, nvox, s_n, [](int, int, unsigned n) { return n + 1u; });
  // scan within the warps, then over the warps of each 1024 points
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned inc[NB_SUB], c[NB_SUB];
#pragma unroll
  for (int s = 0; s < NB_SUB; ++s) {
    c[s] = inc[s] = s_n[s][threadIdx.x];  // (this thread's own)
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, inc[s], off);
      if (lane >= off) inc[s] += t;
    }
    if (lane == 31) wsum[s][w] = inc[s];
  }
  __syncthreads();
  if (threadIdx.x < NB_POINTS / 32) {  // the warps' totals: 32 per 1024 points, one warp's lanes
    const unsigned tot = wsum[threadIdx.x / W][threadIdx.x % W];
    unsigned t = tot;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, t, off);
      if (lane >= off) t += u;
    }
    wsum[threadIdx.x / W][threadIdx.x % W] = t - tot;
    const long long group = (long long)blockIdx.x * (NB_POINTS / SCAN_THREADS) + w;
    if (lane == 31 && group * SCAN_THREADS < nvox) ws[group] = t;
  }
  __syncthreads();
  static_assert(GROUPS * W == 32, "a scan group is 32 warps' points");
#pragma unroll
  for (int s = 0; s < NB_SUB; ++s) {
    const long long v = (long long)blockIdx.x * NB_POINTS + s * NB_THREADS + threadIdx.x;
    if (v < nvox) hdr[v] = make_uint2(wsum[s][w] + inc[s] - c[s], c[s]);
  }
}

// exclusive scan of the block totals (one block, 8 consecutive words per thread and step).
// A word holds 1024 points' entries (at most 1024 x 65 534), so a thread's eight fit in 32
// bits; a step's 8192 words do not (from 512 entries per point on), and the total has to be true
// for the host to refuse lists beyond 32-bit starts: 64 bits from the warp's scan on.
constexpr int SCAN_ITEMS = 8;
__global__ void __launch_bounds__(SCAN_THREADS)
nb_scan_blocks_kernel(unsigned* __restrict__ ws, int nblk, unsigned long long* __restrict__ total) {
  __shared__ unsigned long long wsum[SCAN_THREADS / 32];
  __shared__ unsigned long long carry;
  if (threadIdx.x == 0) carry = 0ull;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < nblk; base += SCAN_THREADS * SCAN_ITEMS) {
    const int i0 = base + (int)threadIdx.x * SCAN_ITEMS;
    unsigned v[SCAN_ITEMS], c = 0u;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      v[k] = i0 + k < nblk ? ws[i0 + k] : 0u;
      c += v[k];
    }
    unsigned long long inc = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += t;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
      unsigned long long s = wsum[lane];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= off) s += t;
      }
      wsum[lane] = s;
    }
    __syncthreads();
    const unsigned long long cb = carry;
    unsigned before = (unsigned)(cb + (w > 0 ? wsum[w - 1] : 0ull) + inc - c);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      if (i0 + k < nblk) ws[i0 + k] = before;
      before += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = cb + wsum[SCAN_THREADS / 32 - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// adds a block's offset to its 1024 headers
__global__ void __launch_bounds__(SCAN_THREADS / 4)
nb_add_kernel(uint2* __restrict__ hdr, const unsigned* __restrict__ ws, long long nvox) {
  const unsigned add = ws[blockIdx.x];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long v = (long long)blockIdx.x * SCAN_THREADS + k * (SCAN_THREADS / 4) + threadIdx.x;
    if (v < nvox) hdr[v].x += add;
  }
}

// The lists, in index order.  The same receptor and points: 120.7 ms with every
// bead tested per point, 1.04 ms now.
__global__ void __launch_bounds__(NB_THREADS, 3)
nb_fill_kernel(AttGridGeom g, const float4* __restrict__ rec, int n_rec, float r2, const uint2* __restrict__ hdr,
               uint16_t* __restrict__ list, long long nvox) {
  __shared__ unsigned s_n[NB_SUB][NB_THREADS];
  const long long v0 = (long long)blockIdx.x * NB_POINTS + threadIdx.x;
  near_beads(g, rec, n_rec, r2, nvox, s_n, [&](int s, int j, unsigned n) {
    const uint2 h = __ldg(hdr + v0 + s * NB_THREADS);
    if (n >= h.y) return n;
    list[h.x + n] = (uint16_t)j;
    return n + 1u;
  });
}

long long nb_workspace_bytes(long long nvox) {
  return ((nvox + SCAN_THREADS - 1) / SCAN_THREADS) * (long long)sizeof(unsigned) + 256;
}

cudaError_t launch_nb_count(const AttGridGeom& g, const float* rec, int n_rec, float radius, uint32_t* hdr,
                            unsigned long long* total, void* ws, cudaStream_t st) {
  const long long nvox = (long long)g.dim[0] * g.dim[1] * g.dim[2];
  const int nblk = (int)((nvox + SCAN_THREADS - 1) / SCAN_THREADS);
  unsigned* w = reinterpret_cast<unsigned*>(ws);
  nb_count_kernel<<<(unsigned)((nvox + NB_POINTS - 1) / NB_POINTS), NB_THREADS, 0, st>>>(g, reinterpret_cast<const float4*>(rec), n_rec, radius * radius,
                                                 reinterpret_cast<uint2*>(hdr), w, nvox);
  nb_scan_blocks_kernel<<<1, SCAN_THREADS, 0, st>>>(w, nblk, total);
  nb_add_kernel<<<nblk, SCAN_THREADS / 4, 0, st>>>(reinterpret_cast<uint2*>(hdr), w, nvox);
  return cudaGetLastError();
}

cudaError_t launch_nb_fill(const AttGridGeom& g, const float* rec, int n_rec, float radius, const uint32_t* hdr,
                           uint16_t* list, cudaStream_t st) {
  const long long nvox = (long long)g.dim[0] * g.dim[1] * g.dim[2];
  nb_fill_kernel<<<(unsigned)((nvox + NB_POINTS - 1) / NB_POINTS), NB_THREADS, 0, st>>>(
      g, reinterpret_cast<const float4*>(rec), n_rec, radius * radius, reinterpret_cast<const uint2*>(hdr), list, nvox);
  return cudaGetLastError();
}

// A quantile of the first `first` non-zero list lengths, linear between the two
// nearest (the record size follows it).  The number of non-zero lists before each
// 1024 points, a histogram of the first ones, its walk: 0.23 ms of 90.5 M points (two
// reads of the headers), where selecting and sorting 16.8 M of them took 1.4 ms.
constexpr int HIST_THREADS = 256, HIST_BINS = 65536, HIST_SMALL = 256;

__global__ void __launch_bounds__(HIST_THREADS)
nb_nonzero_kernel(const uint2* __restrict__ hdr, long long nvox, unsigned* __restrict__ ws) {
  int n = 0;
#pragma unroll
  for (int k = 0; k < SCAN_THREADS / HIST_THREADS; ++k) {
    const long long v = (long long)blockIdx.x * SCAN_THREADS + k * HIST_THREADS + threadIdx.x;
    n += __syncthreads_count(v < nvox && hdr[v].y != 0u);
  }
  if (threadIdx.x == 0) ws[blockIdx.x] = (unsigned)n;
}

__global__ void __launch_bounds__(HIST_THREADS)
nb_hist_kernel(const uint2* __restrict__ hdr, long long nvox, const unsigned* __restrict__ before, int nblk,
               long long first, unsigned* __restrict__ hist) {
  constexpr int N = SCAN_THREADS / HIST_THREADS;
  __shared__ unsigned s_hist[HIST_SMALL];
  __shared__ unsigned s_w[32];
  for (int i = threadIdx.x; i < HIST_SMALL; i += HIST_THREADS) s_hist[i] = 0u;
  __syncthreads();
  for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
    const long long n0 = before[blk];
    if (n0 >= first) break;  // (the later blocks' too)
    unsigned c[N];
    bool take[N];
    int rank[N], n = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const long long v = (long long)blk * SCAN_THREADS + k * HIST_THREADS + threadIdx.x;
      c[k] = v < nvox ? hdr[v].y : 0u;
      take[k] = c[k] != 0u;
      rank[k] = 0;
    }
    if (n0 + SCAN_THREADS > first) block_ranks<HIST_THREADS>(take, s_w, rank, n);  // (block-uniform; the last block)
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (take[k] && n0 + rank[k] < first) {
        if (c[k] < HIST_SMALL) atomicAdd(&s_hist[c[k]], 1u);
        else atomicAdd(hist + min(c[k], (unsigned)HIST_BINS - 1u), 1u);
      }
    if (n0 + SCAN_THREADS > first) __syncthreads();  // s_w may be written again
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HIST_SMALL; i += HIST_THREADS)
    if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
}

__global__ void __launch_bounds__(SCAN_THREADS)
nb_quantile_kernel(const unsigned* __restrict__ hist, const unsigned long long* __restrict__ total, long long first,
                   float q, float* __restrict__ out) {
  constexpr int PER = HIST_BINS / SCAN_THREADS;
  __shared__ unsigned wsum[SCAN_THREADS / 32];
  __shared__ int s_val[2];
  const long long n = min((long long)*total, first);
  if (n <= 0) {
    if (threadIdx.x == 0) *out = 0.f;
    return;
  }
  const float rank = __fmul_rn(q, (float)(n - 1));
  const long long lo = (long long)rank, hi = (long long)ceilf(rank);
  unsigned c = 0;
  const uint4* mine = reinterpret_cast<const uint4*>(hist + threadIdx.x * PER);
#pragma unroll
  for (int i = 0; i < PER / 4; ++i) {
    const uint4 h = __ldg(mine + i);
    c += h.x + h.y + h.z + h.w;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned inc = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += t;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  long long at = inc - c;  // values below this thread's bins
  for (int k = 0; k < w; ++k) at += wsum[k];
  for (int i = 0; i < PER && c; ++i) {
    const unsigned h = hist[threadIdx.x * PER + i];
    if (lo >= at && lo < at + h) s_val[0] = threadIdx.x * PER + i;
    if (hi >= at && hi < at + h) s_val[1] = threadIdx.x * PER + i;
    at += h;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const float a = (float)s_val[0], b = (float)s_val[1], t = rank - (float)lo;
    *out = t < 0.5f ? a + t * (b - a) : b - (b - a) * (1.f - t);
  }
}

// workspace: the scan's words, the number of non-zero lists, the histogram
static long long quantile_words(long long nvox) { return (nvox + SCAN_THREADS - 1) / SCAN_THREADS; }
long long nb_quantile_workspace_bytes(long long nvox) {
  return (quantile_words(nvox) + 3) / 2 * 8 + 24 + (long long)HIST_BINS * 4;
}
cudaError_t launch_nb_quantile(const uint32_t* hdr, long long nvox, float q, long long first, float* out, void* ws,
                               cudaStream_t st) {
  const int nblk = (int)quantile_words(nvox);
  unsigned* words = reinterpret_cast<unsigned*>(ws);
  unsigned long long* total = reinterpret_cast<unsigned long long*>(words + (nblk + 3) / 2 * 2);
  unsigned* hist = reinterpret_cast<unsigned*>((reinterpret_cast<uintptr_t>(total + 1) + 15) & ~(uintptr_t)15);
  const uint2* h = reinterpret_cast<const uint2*>(hdr);
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaMemsetAsync(hist, 0, HIST_BINS * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  nb_nonzero_kernel<<<nblk, HIST_THREADS, 0, st>>>(h, nvox, words);
  nb_scan_blocks_kernel<<<1, SCAN_THREADS, 0, st>>>(words, nblk, total);
  nb_hist_kernel<<<min(nblk, sms * 8), HIST_THREADS, 0, st>>>(h, nvox, words, nblk, first, hist);
  nb_quantile_kernel<<<1, SCAN_THREADS, 0, st>>>(hist, total, first, q, out);
  return cudaGetLastError();
}

// CSR -> fixed-size records {inline entries, u16 count, u32 overflow index}:
// the entries start the record, so that a reader takes eight at a time in
// 16-byte loads.  A thread forms a point's record in registers, 16 bytes at a
// time.  Bound by the records' writes: 90.5 M points, 32-byte records: 7.50 ms
// with 2-byte stores, 0.61 ms with these (2.9 GB written, 1.0 GB read).
template <int RB>
__global__ void __launch_bounds__(256)
nb_pack_kernel(const uint2* __restrict__ hdr, const uint16_t* __restrict__ list, long long nvox,
               uint4* __restrict__ out) {
  constexpr int INL = ATT_NB_INLINE(RB);
  const long long v = (long long)blockIdx.x * 256 + threadIdx.x;
  if (v >= nvox) return;
  const uint2 h = hdr[v];
  const uint16_t* l = list + h.x;
  const unsigned cnt = h.y;
  uint4* r = out + v * (RB / 16);
  auto entry = [&](int i) -> unsigned {  // the i-th u16 of the record
    return i == INL ? min(cnt, 65535u) : (unsigned)i < cnt ? ldg_u16(l + i) : (unsigned)ATT_NB_EMPTY;
  };
#pragma unroll
  for (int q = 0; q < RB / 16; ++q) {
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = q * 8 + k * 2;
      w[k] = i > INL ? h.x + (unsigned)INL : entry(i) | entry(i + 1) << 16;
    }
    r[q] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

cudaError_t launch_nb_pack(const uint32_t* hdr, const uint16_t* list, long long nvox, int rec_bytes, void* out,
                           cudaStream_t st) {
  const uint2* h = reinterpret_cast<const uint2*>(hdr);
  uint4* o = reinterpret_cast<uint4*>(out);
  const unsigned blocks = (unsigned)((nvox + 255) / 256);
  if (rec_bytes == 32) nb_pack_kernel<32><<<blocks, 256, 0, st>>>(h, list, nvox, o);
  else if (rec_bytes == 64) nb_pack_kernel<64><<<blocks, 256, 0, st>>>(h, list, nvox, o);
  else nb_pack_kernel<128><<<blocks, 256, 0, st>>>(h, list, nvox, o);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// K5: dense [T][X][Y][Z][4] -> bricks [T][inner+outer][8 corners]
// ---------------------------------------------------------------------------
// A warp writes the bricks of one row of cells along z; a lane keeps its corner
// and steps 4 cells at a time.  Bound by the writes, which stream past L2 so
// that the dense rows, read 8 times over, stay there: 32 types of 1.40 M + 0.69 M
// cells (8.55 GB) 3.41 ms with an index division per 16 bytes, 1.55 ms now.
constexpr int REPACK_WARPS = 8;
__global__ void __launch_bounds__(REPACK_WARPS * 32)
repack_kernel(const float4* __restrict__ src, int T, int dx, int dy, int dz, long long brick0, long long type_stride,
              float4* __restrict__ dst) {
  const int lane = threadIdx.x & 31, c = lane & 7;
  const long long rows = (long long)T * (dx - 1) * (dy - 1);
  for (long long row = (long long)blockIdx.x * REPACK_WARPS + (threadIdx.x >> 5); row < rows;
       row += (long long)gridDim.x * REPACK_WARPS) {
    const int iy = (int)(row % (dy - 1));
    const long long tx = row / (dy - 1);
    const int ix = (int)(tx % (dx - 1));
    const long long t = tx / (dx - 1);
    const float4* s = src + ((t * dx + ix + (c >> 2)) * dy + iy + ((c >> 1) & 1)) * dz + (c & 1);
    float4* d = dst + (t * type_stride + brick0 + ((long long)ix * (dy - 1) + iy) * (dz - 1)) * 8 + c;
#pragma unroll 4
    for (int iz = lane >> 3; iz < dz - 1; iz += 4) __stcs(d + (long long)iz * 8, __ldg(s + iz));
  }
}

static void repack(const float* src, int T, const int* dim, long long brick0, long long stride, float4* dst,
                   cudaStream_t st) {
  const long long rows = (long long)T * (dim[0] - 1) * (dim[1] - 1);
  const unsigned blocks = (unsigned)min((rows + REPACK_WARPS - 1) / REPACK_WARPS, 1LL << 30);
  repack_kernel<<<blocks, REPACK_WARPS * 32, 0, st>>>(reinterpret_cast<const float4*>(src), T, dim[0], dim[1], dim[2],
                                                      brick0, stride, dst);
}

cudaError_t launch_repack(const AttGridGeom& g, const float* inner, const float* outer, void* bricks,
                          cudaStream_t st) {
  const long long ni = (long long)(g.dim[0] - 1) * (g.dim[1] - 1) * (g.dim[2] - 1);
  const long long no = outer ? (long long)(g.dim2[0] - 1) * (g.dim2[1] - 1) * (g.dim2[2] - 1) : 0;
  float4* dst = reinterpret_cast<float4*>(bricks);
  repack(inner, g.n_types, g.dim, 0, ni + no, dst, st);
  if (outer) repack(outer, g.n_types, g.dim2, ni, ni + no, dst, st);
  return cudaGetLastError();
}

}  // namespace att

// ---------------------------------------------------------------------------
// att_nbgrid_count_noalloc: the neighbour-list count + scan of
// att_nbgrid_count with its scan workspace (one word per 1024 grid points) in
// a fixed device array of this library instead of caller memory, for callers
// that cannot allocate device memory themselves.
// ---------------------------------------------------------------------------
#include <mutex>
#include <stdio.h>

namespace att {
int report_error(int code, const char* msg);
int check_geom(const AttGridGeom* g);  // the validation of att_nbgrid_count (capi.cu)
}

// Fixed scan workspace: 8192 words = 32 KB, i.e. grids of up to 8192 * 1024
// inner points.  Every device that loads the library holds it until exit.
static __device__ __align__(256) unsigned g_nbgrid_scan_ws[ATT_NBGRID_NOALLOC_MAX_VOXELS / 1024];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scan_ws_mutex;
struct ScanWsEntry {
  void* ctx;   // the CUDA context the address belongs to
  void* addr;  // device address of g_nbgrid_scan_ws in that context
};
ScanWsEntry g_scan_ws[kMaxDevices] = {};

// cuCtxGetCurrent through the runtime's driver entry point (no link-time
// dependency on the driver library); NULL when unavailable.
typedef int (*CtxGetCurrentFn)(void**);
CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<CtxGetCurrentFn>(f);
  }();
  return fn;
}

// Device address of the fixed workspace on the current device.  The name
// g_nbgrid_scan_ws in host code is only a host-side stand-in for the symbol;
// the kernel must be given the address that cudaGetSymbolAddress returns with
// that device current.  Looked up on the first call on a device and cached per
// device together with the context it was taken in: after a device reset (or
// with another context current) the stale address is dropped and looked up
// again.  Without a current context handle (none made current yet, or no
// driver entry point) the address is looked up on every call.
int scan_ws_address(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return att::report_error(ATT_E_CUDA, "att_nbgrid_count_noalloc: cudaGetDevice failed");
  if (dev < 0 || dev >= kMaxDevices)
    return att::report_error(ATT_E_UNSUPPORTED, "att_nbgrid_count_noalloc: device index beyond 64");
  void* ctx = nullptr;
  CtxGetCurrentFn get = ctx_get_current();
  const bool have_ctx = get != nullptr && get(&ctx) == 0 && ctx != nullptr;
  std::lock_guard<std::mutex> lock(g_scan_ws_mutex);
  ScanWsEntry& ent = g_scan_ws[dev];
  if (!have_ctx || ent.addr == nullptr || ent.ctx != ctx) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_nbgrid_scan_ws);
    if (e != cudaSuccess || p == nullptr) {
      char msg[256];
      snprintf(msg, sizeof(msg), "att_nbgrid_count_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
               cudaGetErrorString(e));
      return att::report_error(ATT_E_CUDA, msg);
    }
    ent.addr = p;
    ent.ctx = have_ctx ? ctx : nullptr;
  }
  *out = ent.addr;
  return ATT_OK;
}
}  // namespace

extern "C" int att_nbgrid_count_noalloc(const AttGridGeom* geom, const float* rec_dev, int n_rec, float radius,
                                        uint32_t* hdr_dev, unsigned long long* total_dev, void* stream) {
  char msg[256];
  int rc = att::check_geom(geom);  // the same geometry rules as att_nbgrid_count
  if (rc != ATT_OK) return rc;
  const long long nvox = (long long)geom->dim[0] * geom->dim[1] * geom->dim[2];
  if (nvox > ATT_NBGRID_NOALLOC_MAX_VOXELS) {
    snprintf(msg, sizeof(msg),
             "att_nbgrid_count_noalloc: %lld grid points exceed the fixed workspace (at most %lld); "
             "use att_nbgrid_count with a caller-provided workspace",
             nvox, (long long)ATT_NBGRID_NOALLOC_MAX_VOXELS);
    return att::report_error(ATT_E_INVALID, msg);
  }
  if (n_rec < 0 || n_rec >= (int)ATT_NB_EMPTY || (n_rec > 0 && rec_dev == nullptr))
    return att::report_error(ATT_E_INVALID, "att_nbgrid_count_noalloc: receptor beads");
  if (hdr_dev == nullptr || total_dev == nullptr)
    return att::report_error(ATT_E_INVALID, "att_nbgrid_count_noalloc: NULL output");
  if (!(radius >= 0.f)) return att::report_error(ATT_E_INVALID, "att_nbgrid_count_noalloc: radius < 0");
  void* ws = nullptr;
  rc = scan_ws_address(&ws);
  if (rc != ATT_OK) return rc;
  // every workspace word the scan reads is written by the count kernel of the
  // same call first, so nothing has to be cleared between calls
  cudaError_t e = att::launch_nb_count(*geom, rec_dev, n_rec, radius, hdr_dev, total_dev, ws, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    snprintf(msg, sizeof(msg), "att_nbgrid_count_noalloc: %s", cudaGetErrorString(e));
    return att::report_error(ATT_E_CUDA, msg);
  }
  return ATT_OK;
}
