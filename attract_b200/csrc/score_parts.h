// The parts score.cu is compiled in, and what their launches share with the
// kernels: the layout of a warp's shared memory.
#pragma once

#include "common.cuh"

namespace att {

constexpr int SCORE_PARTS = 4;  // 0: the single evaluations, 1: MODE_MIN, 2: MODE_BWD, 3: MODE_QUAT

// the kernel of (mode, lanes per pose, beads per lane), or NULL when the part does not hold the
// mode; chunked: a ligand may have more beads than the team's slots (single evaluations
// of 32 lanes; the other kernels take any)
template <int PART> const void* score_part_kernel(int mode, int S, int K, bool one_grid, bool chunked);
template <int PART> cudaError_t score_part_status(int* out, int clear, cudaStream_t st);
template <int PART> cudaError_t score_part_debug(unsigned long long* out3, int clear, cudaStream_t st);
#define ATT_DECLARE_PART(i_) \
  template <> const void* score_part_kernel<i_>(int, int, int, bool, bool); \
  template <> cudaError_t score_part_status<i_>(int*, int, cudaStream_t); \
  template <> cudaError_t score_part_debug<i_>(unsigned long long*, int, cudaStream_t);
ATT_DECLARE_PART(0) ATT_DECLARE_PART(1) ATT_DECLARE_PART(2) ATT_DECLARE_PART(3)
#undef ATT_DECLARE_PART

// per-bead records shared by the team
struct __align__(16) BeadPos {  // moved bead; w = ligand type (int bits)
  float x, y, z;
  int lt;
};
struct __align__(16) BeadArm {  // lever arm for the torque (Q x) or ligand-frame x (dE/dmat)
  float x, y, z, pad;
};

// shared memory of one warp: per bead slot a 128-B brick, a neighbour-record
// slot of rec_slot bytes, a 16-B moved-bead record and, in the modes that
// accumulate dE/dmat, a 16-B ligand-frame record; the pair buffers of the
// warp's teams (pairs_per_bead(K) u32 words per bead slot, plus S words of
// padding per team so that teams start in different banks).
// A team with more pairs than its buffer holds takes several windows; with
// several beads per lane, 4 words per slot keep a block's shared memory small
// enough for one more block per SM (13 % faster on 40-bead ligands at 2 beads
// per lane, 51 % at 4) while most teams still need a single window.
__host__ __device__ constexpr int pairs_per_bead(int K) { return K == 1 ? 8 : 4; }
__host__ __device__ inline int rec_stride(int rec_slot) { return rec_slot ? rec_slot + 16 : 0; }
__host__ __device__ inline size_t pair_buffer_bytes(int K) { return (size_t)32 * (pairs_per_bead(K) * K + 1) * 4; }
// (the bead arms are held only by the modes that accumulate dE/dmat; the
// others take the lever arm from the bead record)
__host__ __device__ inline size_t warp_smem_bytes(int K, int rec_slot, bool arms = true) {
  return (size_t)32 * K * (128 + rec_stride(rec_slot) + sizeof(BeadPos) + (arms ? sizeof(BeadArm) : 0)) +
         pair_buffer_bytes(K);
}

}  // namespace att
