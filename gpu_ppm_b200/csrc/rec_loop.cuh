// Chunks of ring records in shared memory and the loop in which a CTA's warp sets
// work through them (integrand_nsx_rec_kernel, integrand_bb_rec_kernel).
// The including file provides set_sync, cp_async16 and cp_async_wait_all: device
// code in kernels.cu, host threads in the check of this loop
// (tests/rec_loop_check.cpp).
#pragma once

#include "kernels.cuh"

namespace ppm {
namespace {

// One chunk of a ring's active elements as the deposit needs it, in shared memory
// (read at every step of 32 points: global loads there cost their latency).
struct ChunkCtx {
  double dphi, jofs, l10kT, tE_lo, tE_hi, out_scale, width;  // width: 1 / n_bins
  long long flux_off;
  const int *perm, *cell_first;
  const float* fEs;
  const double* invE;
  unsigned long long* stats;
  float* part;             // the chunk's node sums (stored plainly), or nullptr: added to the flux pool
  int n_act, n_nodes, u_ofs, n_gl, n_fine, n_e, span, iE_min, mode;
  int mono, held;          // phase_o non-decreasing; logT or log g outside the table (points count as clamped)
  int profile, spot, rec;
  int take;                // nodes a set takes at a time (ring records)
  // blackbody: temperature, energies; tasks of per_pass energies, u_mod nodes each; lanes that own energies
  double kT;
  const double* E;
  int per_pass, u_mod, lanes_log;
  float glo[4], ghi[4];    // smallest and largest energy fraction of each slot group
};

// A chunk's tables in shared memory.  Sx: slice row 0.
struct ChunkBufs {
  const unsigned short* j;
  const double *P, *F, *Z, *MU;
  const unsigned short* hidx;
  const float* Sx;
};

// The home-cell kernels' slice image: rows 0..nE-1 start 16-byte aligned after
// room for rows -1 - C .. -1; rows nE .. nE + C follow them.
__host__ __device__ __forceinline__ int slice_row0(int ldS, int C) { return ((C + 1) * ldS + 3) & ~3; }

// State of a chunk slot: the warp sets inside it (low bits) and its flags.
constexpr unsigned kSlotDrain = 1u << 16;    // its chunk has no nodes left to take
constexpr unsigned kSlotLoading = 1u << 17;  // one set is loading its next chunk
constexpr unsigned kSlotDead = 1u << 18;     // no chunk left to load

// One CTA per SM with up to four chunk slots: the warp sets take nodes from any
// loaded chunk; the last set to leave a drained slot loads its next chunk (the
// one with the most work left per slot on it) while the others go on with the
// other slots, so that nobody waits for a chunk's slowest node (three CTAs per SM
// with one chunk each spent 32 % of the warps' time in that wait).
// Work is what a set does with the nodes it took (fill: a loaded chunk's context;
// enter: the set comes to another chunk; nodes: the nodes [u, u + take)).
template <int NTMAX, class Work>
__device__ __forceinline__ void rec_loop(const KernelArgs& a, unsigned char* sm, Work& w) {
  const IntegrandShape& S = a.shape;
  const RingWork& W = a.rings;
  constexpr int kSets = NTMAX / 32;
  __shared__ ChunkCtx s_ctx[kMaxRecSlots];
  __shared__ unsigned s_word[kMaxRecSlots];
  // words a set's leader hands its threads; each is written again only after a set_sync that follows the last read of
  // it (the record has one of its own: s_got is still being read when the loader's leader takes a record)
  __shared__ int s_got[kSets], s_u[kSets], s_rec[kSets];
  __shared__ unsigned long long s_best[kSets];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int n_recs = min(*W.n_recs, W.rec_cap);
  if (n_recs == 0) return;
  const int NS = S.rec_slots;
  if (tid < NS) {
    s_word[tid] = kSlotDrain;
    s_ctx[tid].rec = -1;
  }
  __syncthreads();
  const int per_slot = max(1, nt / w.ST / NS);  // warp sets per slot
  const int a16 = (S.off_F - S.off_P) / 8;      // doubles between the sweep's arrays
  volatile unsigned* const word = s_word;

  // leader of a set: leaves slot sl; true if the set has become the loader of the drained slot
  auto leave = [&](int sl) {
    return atomicSub(&s_word[sl], 1u) == (kSlotDrain | 1u) &&
           atomicCAS(&s_word[sl], kSlotDrain, kSlotLoading) == kSlotDrain;
  };
  constexpr int kExit = -1;  // s_got: a slot to work in, kExit, or -2 - slot to load
  int cur_rec = -1, cur_slot = -1, profile = -1, pref = w.set % NS;
  bool claimed = false;  // (leader) the slot just left is this set's to load
  for (;;) {
    if (w.st == 0) {
      int got = kExit;
      if (claimed) {
        got = -2 - cur_slot;
        claimed = false;
      } else {
        // bounded: a set that finds nothing for a second leaves, the others finish the work
        for (int spin = 0; spin < (1 << 21); ++spin) {
          bool live = false;
          for (int k = 0; k < NS && got == kExit; ++k) {
            int sl = pref + k;
            sl -= sl >= NS ? NS : 0;
            const unsigned v = word[sl];
            if (v & kSlotDead) continue;
            live = true;
            if (v == kSlotDrain) {
              if (atomicCAS(&s_word[sl], kSlotDrain, kSlotLoading) == kSlotDrain) got = -2 - sl;
              continue;
            }
            if (v & (kSlotDrain | kSlotLoading)) continue;
            if (!(atomicAdd(&s_word[sl], 1u) & (kSlotDrain | kSlotLoading | kSlotDead))) {
              __threadfence_block();
              const ChunkCtx& c = s_ctx[sl];
              const int u = atomicAdd(&W.ctr[c.rec].x, c.take);
              if (u < c.n_nodes) {
                s_u[w.set] = u;
                got = sl;
                continue;
              }
              atomicOr(&s_word[sl], kSlotDrain);
            }
            if (leave(sl)) got = -2 - sl;
          }
          if (got != kExit || !live) break;
          __nanosleep(500);
        }
      }
      s_got[w.set] = got;
    }
    set_sync(w.set, w.ST);
    const int got = s_got[w.set];
    if (got == kExit) break;
    if (got < kExit) {
      const int sl = -2 - got;
      int r = -1;
      for (;;) {
        if (s_ctx[sl].rec < 0) {  // the slot's first chunk
          r = (int)((blockIdx.x + (unsigned)sl * gridDim.x) % (unsigned)n_recs);
          if (w.st == 0) atomicAdd(&W.ctr[r].y, 1);
          set_sync(w.set, w.ST);
          break;
        }
        // chunks that nobody has yet, in order
        if (w.st == 0) {
          s_best[w.set] = 0;
          const int first = NS * (int)gridDim.x;  // chunks that are the slots' first ones
          const int nx = first < n_recs ? first + atomicAdd(&W.ctr[W.rec_cap].x, 1) : n_recs;
          s_rec[w.set] = nx < n_recs ? nx : -1;
          if (nx < n_recs) atomicAdd(&W.ctr[nx].y, 1);
        }
        set_sync(w.set, w.ST);
        r = s_rec[w.set];
        if (r >= 0) break;
        // then the one with the most work left per slot on it
        unsigned long long best = 0;
#pragma unroll 4
        for (int q = w.st; q < n_recs; q += w.ST) {
          const int4 t = __ldcg(W.ctr + q);
          const int left = t.z - t.x;
          // (scattered a little, so that slots that look at the same time choose differently)
          const float jitter = 0.5f + (float)(((unsigned)q * 2654435761u + blockIdx.x * 40503u) >> 24) * (1.f / 512.f);
          const float score = (float)left * (float)t.w / (float)(t.y + 1) * jitter;
          const unsigned long long key = ((unsigned long long)__float_as_uint(score) << 32) | (unsigned)q;
          // a chunk whose slots' sets will take the remaining nodes at once is left to them
          best = left > per_slot * t.y / 2 && key > best ? key : best;
        }
        if (best) atomicMax(&s_best[w.set], best);
        set_sync(w.set, w.ST);
        if (s_best[w.set] == 0) break;
        r = (int)(unsigned)s_best[w.set];
        if (w.st == 0) {
          const int y = atomicAdd(&W.ctr[r].y, 1);
          s_rec[w.set] = W.recs[r].n_nodes - __ldcg(&W.ctr[r].x) > per_slot * y / 2 ? 1 : 0;
        }
        set_sync(w.set, w.ST);
        const bool ok = s_rec[w.set] != 0;
        set_sync(w.set, w.ST);
        if (ok) break;
        r = -1;
      }
      if (r < 0) {
        if (w.st == 0) atomicXor(&s_word[sl], kSlotLoading | kSlotDead);
        continue;
      }
      const RingRec q = W.recs[r];
      unsigned char* const dst = sm + (size_t)sl * S.rec_slot_bytes;
      const unsigned char* const img = W.data + (size_t)q.job * W.stride;
      const int n16 = (W.off_slice + W.slice_bytes) >> 4;
      for (int k = w.st; k < n16; k += w.ST) cp_async16(dst + 16 * k, img + 16 * k);
      const int l16 = (q.n_act * W.elem_bytes + 15) >> 4;
      const unsigned char* const list = W.lists + (size_t)q.list * W.elem_bytes;
      for (int k = w.st; k < l16; k += w.ST) cp_async16(dst + 16 * (n16 + k), list + 16 * k);
      if (w.st == 0) {
        const DevProfile& p = a.profiles[q.profile];
        ChunkCtx& c = s_ctx[sl];
        w.fill(c, p, p.spot[q.spot], q);
        // nodes are taken from a chunk's own first one on: chunks that run at the same time add to different bins
        c.u_ofs = (int)((unsigned)q.job * 40503u % (unsigned)c.u_mod);
        c.part = r < W.part_cap ? (float*)W.parts + (size_t)r * W.part_stride : nullptr;
        c.profile = q.profile;
        c.spot = q.spot;
        c.rec = r;
      }
      cp_async_wait_all();
      __threadfence_block();
      set_sync(w.set, w.ST);
      if (w.st == 0) {
        __threadfence_block();
        atomicAnd(&s_word[sl], ~kSlotLoading);
      }
      continue;
    }
    // a node of the chunk in slot `got`
    __threadfence_block();
    cur_slot = pref = got;
    const ChunkCtx& c = s_ctx[got];
    if (c.rec != cur_rec) {
      cur_rec = c.rec;
      if (profile != c.profile) w.count(profile);
      profile = c.profile;
      w.enter(c);
    }
    const unsigned char* const base = sm + (size_t)got * S.rec_slot_bytes;
    const double* P = (const double*)base;
    const ChunkBufs bufs{(const unsigned short*)(base + W.off_slice + W.slice_bytes),
                         P, P + a16, P + 2 * a16, P + 3 * a16, (const unsigned short*)(base + W.off_hidx),
                         (const float*)(base + W.off_slice) + slice_row0(S.ldS, S.cpl)};
    w.nodes(c, bufs, s_u[w.set]);
    __threadfence_block();
    set_sync(w.set, w.ST);
    if (w.st == 0) claimed = leave(got);
  }
  w.count(profile);
}

}  // namespace
}  // namespace ppm
