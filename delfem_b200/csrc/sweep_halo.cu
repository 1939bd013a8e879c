// Range-partitioned ILU triangular sweeps whose level path reads shared
// memory only (schedule modes 9 and 10).
//
// The rows are split among co-resident CTAs as in the range schedule
// (sweep.cu): contiguous ranges of the natural order, or the parts of a row
// partition.  A CTA walks its rows level by level, in rounds of up to
// cw * RPW rows (cw compute warps, RPW rows per warp).  Its warps:
//
//  * Compute warps (1, 2 or 4) take the rows of a round.  A row has B * H
//    lanes: lane (half h, component c) sums component c over the row's blocks
//    h, h + H, ...  All operands are in shared memory: rows of the CTA's own
//    range in its vector slice, rows of other CTAs in a halo area.  After a
//    round the compute warps meet at a named barrier of their own (__syncwarp
//    for a single warp).
//  * One copy warp keeps a ring of stages full: a chunk (a few rounds) is one
//    TMA bulk copy (cp.async.bulk, no multicast), issued as soon as the
//    compute warps have left the chunk that held its stage.
//  * kHaloRhsWarps warps gather a chunk's right-hand sides (and the vector of
//    the fused dot) into the slice, which is laid out in the order the rows
//    are taken, and its round table into a ring.
//  * Halo warps poll the other CTAs' rows in global memory (NaN sentinel = not
//    yet written), a row per lane, in the order the rounds need them, and put
//    them into the halo area, which holds the sentinel until then; a row's last
//    component goes behind a fence and says that the row is there.
//
// What bounds a sweep is the chain of rounds, not bytes.  A round of one warp
// of 1x1 rows takes 92 cycles with nothing but its loads, products, store and
// warp barrier (measured in isolation; 115 with two warps and a named barrier,
// 175 with four), and every other thing a compute warp does per round shows:
// +10 the store to global memory (a fence behind it, for rows of more than one
// component, does not show in a sweep's time), +18 choosing a record for lanes without a
// row, +32 a branch on a row's length, +44 the bookkeeping of stages, +97 a look
// at progress counters, +110 a branch on a NaN among its operands, +150 a
// helper warp at the barrier that does the waiting.  So the compute warps' loop
// is straight-line code with one branch, taken rarely:
//
//  * A lane's part of a row is one record: its K operand offsets, its K blocks'
//    row c, its row of D^-1, padded to an odd number of 16-byte pieces, so 16-
//    byte loads at a record's stride have no bank conflicts and the addresses
//    need no arithmetic.  Lanes with fewer than K blocks read zero blocks
//    against a zero operand kept behind the slice.  Plans whose rows all fit
//    use the kernel without the code for longer rows (EX).
//  * While a round's operands are read, the next round's records are loaded
//    into a second register set (the loop is unrolled over the two sets), and
//    the round table is read two rounds ahead.
//  * A halo row does not depend on the round before, so whether the next
//    round's operands are in is looked at before the barrier, off the chain.
//    The branch is taken if one is missing or at a marked round, where chunks
//    are taken over and handed back.
//
// Every operand is addressed by a precomputed byte offset into X =
// [slice | a zero block | halo area | the dot's vector].  The slice is a ring:
// a row's place is taken over by a later row once no row to come reads it,
// which leaves the room to the stages (a 200x40x40 box in 144 parts has 3,216
// rows in a part and needs 200 places).  The halo area holds every other CTA's
// row that this CTA needs, once; where that leaves too little room it is a ring
// as well (an entry then serves its chunk and the next kHaloReuse, and the copy
// warp puts the sentinel back when it requests the chunk that takes it over).
//
// Progress: a row waits only for rows of lower level; every CTA takes its
// rounds in level order and all CTAs are co-resident (cooperative launch), so
// every wait ends; a halo lane's entries come in the same order.  All waits
// are bounded as well: past the context's limit a wait records
// DFM_WAIT_TIMEOUT and clears the CTA's s_alive; the other warps leave their
// loops, the compute warps stop computing but pass every round's barrier, and
// copies in flight land before the CTA exits.
#include <algorithm>
#include <cstring>
#include <thread>

#include "dfm_internal.h"
#include "sweep.h"
#include "sweep_dev.cuh"

namespace dfm {

constexpr int kHaloMaxStages = 14;
constexpr int kHaloRhsWarps = 2;
constexpr int kHaloMaxWarps = 12;  // compute, copy, right-hand-side and halo warps of a launch
constexpr int kHaloMaxThreads = 32 * kHaloMaxWarps;
constexpr int kHaloMaxCw = 4;
// A chunk closes when a round like its last would take it past kHaloChunkBytes.  Taking a chunk over costs the compute
// warps some 300 cycles, so chunks hold several rounds as long as enough stages fit.
constexpr unsigned kHaloChunkBytes = 24 * 1024;
constexpr unsigned kHaloReuse = 8;  // chunks after its own that may read an entry of a halo ring
constexpr size_t kHaloSmemBudget = 220 * 1024;  // dynamic shared memory per CTA
// A chunk is entered when the two after it are in, and its predecessor's stage is freed then: five chunks must fit so
// that this waits for no copy that was only just requested.
constexpr int kHaloMinStages = 5;
constexpr int kHaloGoodStages = 6;  // enough to cover a copy's latency
constexpr unsigned kHaloChunkRounds = 31;  // and at this many rounds
constexpr unsigned kHaloTable = 512;       // entries of the round-table ring: the rounds of more than kHaloMaxStages chunks
static_assert(kHaloTable > kHaloChunkRounds * (kHaloMaxStages + 2) && (kHaloTable & (kHaloTable - 1)) == 0, "table ring");

// A chunk: [row indices u32, padded to 16 bytes][records per round].
// A record: [K operand offsets u32][K x B values][D^-1 row (forward)][extra blocks: offsets | values].
// A round's table entry: rec, rows: byte offsets in shared memory of its records and row indices; slot: byte
// offset in X of its first row; shape: rows | pieces of a record << 8 | extra blocks per lane << 20 | last round of
// its chunk << 31.
struct HaloRound {
  unsigned rec, slot, rows, shape;
};
constexpr unsigned kHaloMaxPieces = 0xfff, kHaloMaxExtra = 0x7ff, kHaloLast = 0x80000000u;

// Record layout of B x B blocks with KT blocks per lane in registers.
template <int B, int KT, typename TV, bool FWD>
struct HaloRec {
  static constexpr int PO = (4 * KT + 15) / 16;                    // pieces of operand offsets
  static constexpr int VB = (KT * B * (int)sizeof(TV) + 7) & ~7;   // bytes of values
  static constexpr int PV = (VB + (FWD ? 8 * B : 0) + 15) / 16;    // pieces of values and D^-1
  static constexpr int P = (PO + PV) | 1;
};
// Blocks per lane held in registers: a P1 triangle mesh has 3 lower blocks per
// row, a P1 tetrahedral one 7; with 48 / 80 / 144 bytes per record the loads of
// both register sets fit beside each other.
template <int B>
struct HaloK {
  static constexpr int KT = B == 3 ? 4 : 3;
};

DFM_DEVINL int ld_volatile_i(const int* p) { return *reinterpret_cast<const volatile int*>(p); }
DFM_DEVINL void st_volatile_i(int* p, int v) { *reinterpret_cast<volatile int*>(p) = v; }

// the compute warps' barrier
DFM_DEVINL void meet(int ncw) {
  if (ncw > 1) asm volatile("bar.sync 1, %0;" ::"r"(ncw * 32) : "memory");
  else __syncwarp();
}
// one look at a phase, without the suspended wait of try_wait
DFM_DEVINL bool mbar_test(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
      "p;\n}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
DFM_DEVINL void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Spins on cond() until it holds, the CTA is shutting down, or the limit runs
// out (recorded, shutting the CTA down).  NAP: ns to sleep between looks.  Each
// lane leaves by itself: cond() has no vote, and the caller votes on the result.
template <int NAP = 0, typename F>
DFM_DEVINL bool spin_until(F cond, int* s_alive, DevStatus* st, uint64_t wait_ns, int where) {
  if (cond()) return true;
  SpinGuard g(wait_ns);
  for (;;) {
    if (NAP) __nanosleep(NAP);
    if (cond()) return true;
    if (!ld_volatile_i(s_alive)) return false;
    if (g.expired()) {
      raise_error(st, DFM_WAIT_TIMEOUT, where);
      st_volatile_i(s_alive, 0);
      return false;
    }
  }
}

// The partials of (rdot, out) of a backward sweep whose plan has no room for
// rdot: block b sums entries b, b + gridDim, ... in tiles of its threads.
template <int DOT>
__global__ void __launch_bounds__(256)
k_halo_dot(size_t n, const double* __restrict__ rdot, const double* __restrict__ out, double* part,
           const KrylovScalars* sc) {
  if (sc && block_flag(&sc->done)) return;
  double re = 0.0, im = 0.0;
  for (size_t k = blockIdx.x * (size_t)256 + threadIdx.x; k < n; k += (size_t)gridDim.x * 256) {
    if (DOT == 2) {
      const double2 r = reinterpret_cast<const double2*>(rdot)[k], z = reinterpret_cast<const double2*>(out)[k];
      re += r.x * z.x - r.y * z.y;
      im += r.x * z.y + r.y * z.x;
    } else {
      re += rdot[k] * out[k];
    }
  }
  block_partial<256>(re, part);
  if (DOT == 2) block_partial<256>(im, part + kMaxBlocks);
}

// A lane's record and what it needs to finish its row.
template <int B, int KT, typename TV, bool FWD>
struct LaneItem {
  using R = HaloRec<B, KT, TV, FWD>;
  unsigned o[R::PO * 4];
  unsigned w[R::PV * 4];
  unsigned row, slot;  // the row's index in the vectors, its component's offset in X
  bool act, last;      // the lane has a row; the round is its chunk's last
  unsigned extra, rec; // extra blocks per lane, the record's offset (EX only)
  DFM_DEVINL double val(int i) const {
    if constexpr (sizeof(TV) == 8) return __hiloint2double((int)w[2 * i + 1], (int)w[2 * i]);
    else return (double)__uint_as_float(w[i]);
  }
  DFM_DEVINL double dinv(int c) const {
    const int d = R::VB / 4 + 2 * c;
    return __hiloint2double((int)w[d + 1], (int)w[d]);
  }
};

DFM_DEVINL void ld16(unsigned* w, const char* p) {
  const uint4 t = *reinterpret_cast<const uint4*>(p);
  w[0] = t.x;
  w[1] = t.y;
  w[2] = t.z;
  w[3] = t.w;
}

// Loads this lane's record of the round e: rw its row of a round, idx its
// place in the row.  Lanes without a row take the round's first record; so do
// all lanes past the last round, whose entry is the last one's without rows.
template <int B, int H, int KT, typename TV, bool FWD, bool EX>
DFM_DEVINL void item_load(LaneItem<B, KT, TV, FWD>& P, const char* smem, const uint4 e, unsigned rw, unsigned idx,
                          unsigned wrap) {
  using R = HaloRec<B, KT, TV, FWD>;
  P.act = rw < (e.w & 0xffu);
  P.last = (e.w & kHaloLast) != 0;
  const unsigned r = P.act ? rw : 0u, l = P.act ? rw * (B * H) + idx : 0u;
  unsigned rec;
  if (EX) {
    P.extra = (e.w >> 20) & kHaloMaxExtra;
    rec = e.x + l * (16u * ((e.w >> 8) & kHaloMaxPieces));
    P.rec = rec;
  } else {
    rec = e.x + l * (16u * R::P);
  }
#pragma unroll
  for (int p = 0; p < R::PO; p++) ld16(P.o + 4 * p, smem + rec + 16 * p);
#pragma unroll
  for (int p = 0; p < R::PV; p++) ld16(P.w + 4 * p, smem + rec + 16 * (R::PO + p));
  P.row = *reinterpret_cast<const unsigned*>(smem + e.z + 4u * r);
  P.slot = e.y + 8u * (r * B + idx % B);
  if (P.slot >= wrap) P.slot -= wrap;  // the slice is a ring of wrap bytes
}

template <int B>
DFM_DEVINL void ld_operand(double* x, const char* p) {
  if constexpr (B == 1) {
    x[0] = ld_volatile_s(reinterpret_cast<const double*>(p));
  } else if constexpr (B == 2) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    x[0] = t.x;
    x[1] = t.y;
  } else {
#pragma unroll
    for (int c = 0; c < B; c++) x[c] = reinterpret_cast<const double*>(p)[c];
  }
}

// Whether a halo row at offset o has not come yet: its last component, which is stored last, behind a fence.  (Places
// of the CTA's own rows are looked at as well: they hold no sentinel.)  A value read as the same eight bytes that were
// stored is there to stay, so rows of one component need no more; for the others the look is followed by a fence
// before the components are read.
template <int B>
DFM_DEVINL bool halo_missing(const char* smem, unsigned o) {
  return __double2hiint(ld_volatile_s(reinterpret_cast<const double*>(smem + o) + (B - 1))) == (int)(DFM_SENT64 >> 32);
}

template <int B, int H, typename TV, bool FWD, int DOT, bool EX>
__global__ void __launch_bounds__(kHaloMaxThreads, 1)
k_sweep_halo(const HaloChunk* __restrict__ chunks, const HaloCtaDesc* __restrict__ ctas,
             const HaloRound* __restrict__ table,
             const unsigned* __restrict__ rows, const unsigned* __restrict__ hids, const char* __restrict__ blob,
             unsigned stage_bytes, int nstage, unsigned x_bytes, unsigned x_slice, unsigned halo0, unsigned ring,
             unsigned rd_off, int ncw, const double* __restrict__ in, double* out, const double* __restrict__ rdot, double* part,
             KrylovScalars* sc, const double* rr_part, int rr_nparts, DevStatus* st, uint64_t wait_ns) {
  constexpr int KT = HaloK<B>::KT;
  using I = LaneItem<B, KT, TV, FWD>;
  using R = HaloRec<B, KT, TV, FWD>;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr unsigned LR = B * H, RPW = 32u / LR;  // lanes per row, rows per warp
  extern __shared__ __align__(128) char smem[];
  __shared__ int s_alive;
  __shared__ int s_issued;  // chunks whose copy has been requested
  __shared__ int s_armed;   // halo entries that hold the sentinel or their value
  __shared__ unsigned s_copies;              // copies requested in all
  __shared__ unsigned s_rhs[kHaloRhsWarps];  // the first chunk whose phase that warp has not completed
  if (sc) {
    if (block_flag(&sc->done)) return;
    if (FWD && rr_part) {
      const double rr = reduce_partials(rr_part, rr_nparts);
      if (rr * sc->inv0 < sc->tol2) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
          sc->conv = sqrt(rr * sc->inv0);
          sc->conv_it = sc->it;
          sc->done = sc->conv_code;
        }
        return;
      }
    }
  }
  const HaloCtaDesc me = ctas[blockIdx.x];
  const unsigned K = me.nchunk, ns = (unsigned)nstage;
  double* X = reinterpret_cast<double*>(smem);
  char* stages = smem + x_bytes;
  HaloRound* tab = reinterpret_cast<HaloRound*>(stages + (size_t)nstage * stage_bytes);
  uint64_t* landed = reinterpret_cast<uint64_t*>(tab + kHaloTable);
  uint64_t* free_ = landed + kHaloMaxStages;

  if (threadIdx.x < (unsigned)B) X[x_slice + threadIdx.x] = 0.0;  // the operand of padding blocks
  const unsigned armed = min(me.nhalo, ring);
  for (unsigned e = threadIdx.x; e < armed * B; e += blockDim.x) X[halo0 + e] = Sent<double>::value();
  if (threadIdx.x == 0) {
    s_alive = 1;
    s_issued = 0;
    s_armed = (int)armed;
    for (int s = 0; s < nstage; s++) {
      mbar_init(&landed[s], 2);  // the copy's request and the right-hand sides, and the copy's bytes
      mbar_init(&free_[s], 1);
    }
    fence_mbar_init();
  }
  __syncthreads();
  const int warp = (int)(threadIdx.x >> 5);
  const unsigned wl = threadIdx.x & 31u;
  const int nwarps = (int)(blockDim.x >> 5);
  const unsigned wrap = 8u * x_slice;
  double dre = 0.0, dim = 0.0;  // the fused dot

  if (warp < ncw) {
    // ------------------------------------------------------------- compute
    const unsigned idx = wl % LR, base = wl - idx;  // place in the row; the row's first lane
    const unsigned rw = wl < RPW * LR ? (unsigned)warp * RPW + wl / LR : 0xffffu;  // the lane's row of a round
    const bool writes = idx < B;
    double* outc = out + idx % B;
    unsigned k = 0, s = 0;       // the chunk in work, its stage
    unsigned ls = 0, lpar = 0;   // the stage and its phase of the next chunk to wait for
    unsigned q = 0;              // the round
    I P0, P1;
    uint4 e1 = make_uint4(0, 0, 0, 0);
    auto await_chunk = [&] {
      const bool ok =
          __all_sync(FULL, spin_until([&] { return mbar_test(&landed[ls], lpar); }, &s_alive, st, wait_ns, 21));
      if (++ls == ns) {
        ls = 0;
        lpar ^= 1u;
      }
      return ok;
    };
    auto missing = [&](const I& P) {
      bool m = false;
#pragma unroll
      for (int k = 0; k < KT; k++) m |= halo_missing<B>(smem, P.o[k]);
      if (EX)
        for (unsigned k = 0; k < P.extra; k++)
          m |= halo_missing<B>(smem, reinterpret_cast<const unsigned*>(smem + P.rec + 16 * R::P)[k]);
      return m;
    };
    // Waits until no operand of P is missing; the warp leaves together.
    auto await_operands = [&](const I& P) {
      SpinGuard g(wait_ns);
      while (__any_sync(FULL, missing(P))) {
        const bool late = g.expired();
        if ((g.n & 15u) == 0 && __any_sync(FULL, late || !ld_volatile_i(&s_alive))) {
          if (__any_sync(FULL, late)) {
            if (wl == 0) raise_error(st, DFM_WAIT_TIMEOUT, 23);
            st_volatile_i(&s_alive, 0);
          }
          return false;
        }
      }
      return true;
    };
    // Before round q, whose item is P: its operands; after the last round of a chunk (last) its stage is handed back
    // and the chunk after the next waited for: the last round of the next one reads a record and a table entry ahead,
    // which are in those two.  False to stop.
    auto event = [&](const I& P, bool last) {
      bool ok = true;
      if (last) {
        if (threadIdx.x == 0) mbar_arrive(&free_[s]);
        if (++s == ns) s = 0;
        if (++k == K) return false;
        if (k + 2 < K) ok = await_chunk();
      }
      if (ok && __any_sync(FULL, missing(P))) ok = await_operands(P);
      __threadfence_block();
      return ok;
    };
    // round q: C is loaded, N receives round q + 1's record; true if round q + 1 needs event()
    auto body = [&](I& C, I& N) {
      double x[KT][B];
#pragma unroll
      for (int k = 0; k < KT; k++) ld_operand<B>(x[k], smem + C.o[k]);
      const double rhs = *reinterpret_cast<const double*>(smem + C.slot);
      item_load<B, H, KT, TV, FWD, EX>(N, smem, e1, rw, idx, wrap);
      e1 = *reinterpret_cast<const uint4*>(tab + ((q + 2) & (kHaloTable - 1)));
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < KT; k++)
#pragma unroll
        for (int c = 0; c < B; c++) acc += C.val(k * B + c) * x[k][c];
      if (EX && C.extra) {  // rows with more than KT * H blocks: the rest from the stage
        const unsigned* xo = reinterpret_cast<const unsigned*>(smem + C.rec + 16 * R::P);
        const TV* xv = reinterpret_cast<const TV*>(reinterpret_cast<const char*>(xo) + cl_al16(4 * C.extra));
        for (unsigned k = 0; k < C.extra; k++) {
          double y[B];
          ld_operand<B>(y, smem + xo[k]);
#pragma unroll
          for (int c = 0; c < B; c++) acc += (double)xv[k * B + c] * y[c];
        }
      }
#pragma unroll
      for (int o = H / 2; o > 0; o >>= 1) acc += __shfl_sync(FULL, acc, (int)(base + (idx + o * B) % LR));
      const double t = rhs - acc;
      double v = t;
      if (FWD) {
        v = 0.0;
#pragma unroll
        for (int c = 0; c < B; c++) v += C.dinv(c) * (B > 1 ? __shfl_sync(FULL, t, (int)(base + c)) : t);
      }
      if (C.act && writes) {
        *reinterpret_cast<double*>(smem + C.slot) = v;
        st_relaxed(outc + (size_t)C.row * B, v);
        if (DOT == 1) dre += *reinterpret_cast<const double*>(smem + rd_off + C.slot) * v;
        if (DOT == 2) {  // unconjugated: lane 0 holds the real part of z, lane 1 the imaginary one
          const double2 r = *reinterpret_cast<const double2*>(smem + rd_off + (C.slot & ~15u));
          dre += idx ? -(r.y * v) : r.x * v;
          dim += idx ? r.x * v : r.y * v;
        }
      }
      const bool ev = __any_sync(FULL, missing(N)) || C.last;
      if (B > 1) __threadfence_block();
      meet(ncw);
      q++;
      return ev;
    };
    bool go = K > 0;
    for (unsigned j = 0; j < 3 && j < K && go; j++) go = await_chunk();
    if (go) {
      e1 = *reinterpret_cast<const uint4*>(tab);
      item_load<B, H, KT, TV, FWD, EX>(P0, smem, e1, rw, idx, wrap);
      e1 = *reinterpret_cast<const uint4*>(tab + 1);
      go = event(P0, false);
    }
    while (go) {
      if (body(P0, P1) && !event(P1, P0.last)) break;
      if (body(P1, P0) && !event(P0, P1.last)) break;
    }
    // every compute warp passes every round's barrier, stopped or not
    for (; q < me.nround; q++) meet(ncw);
  } else if (warp == ncw) {
    // ---------------------------------------------------------------- copy
    unsigned issued = 0, s = 0, par = 1;  // par: parity of the stage's previous release
    HaloChunk cd = {};
    unsigned at = armed;
    for (unsigned k = 0; k < K; k++) {
      if ((k & 31u) == 0 && k + wl < K) cd = chunks[me.chunk0 + k + wl];
      const unsigned long long o = __shfl_sync(FULL, cd.off, (int)(k & 31u));
      const unsigned nb = __shfl_sync(FULL, cd.bytes, (int)(k & 31u));
      const unsigned need = __shfl_sync(FULL, cd.need, (int)(k & 31u));
      if (k >= ns) {
        const bool ok = spin_until<100>([&] { return mbar_test(&free_[s], par); }, &s_alive, st, wait_ns, 20);
        if (!__all_sync(FULL, ok)) break;
      }
      if (need > at) {  // a ring's entries taken over by this chunk: their last readers are past
        for (unsigned e = at * B + wl; e < need * B; e += 32u) X[halo0 + e % (ring * B)] = Sent<double>::value();
        at = need;
        __syncwarp();
      }
      if (wl == 0) {
        fence_proxy_async_smem();  // the compute warps' reads of the stage precede the copy into it
        mbar_arrive_tx(&landed[s], nb);
        bulk_g2s(stages + (size_t)s * stage_bytes, blob + o, nb, &landed[s]);
        __threadfence_block();
        st_volatile_i(&s_issued, (int)k + 1);
        st_volatile_i(&s_armed, (int)at);
      }
      issued = k + 1;
      if (++s == ns) {
        s = 0;
        par ^= 1u;
      }
    }
    if (wl == 0) s_copies = issued;
  } else if (warp <= ncw + kHaloRhsWarps) {
    // ---------------------------------------- right-hand sides, round table
    // a chunk's descriptor, row indices and right-hand sides are three dependent reads: the descriptor is read two
    // of the warp's chunks ahead and the first rows' indices one ahead
    constexpr unsigned U = B == 1 ? 8 : 4;  // rows in flight per lane
    const HaloChunk* my_chunks = chunks + me.chunk0;
    const unsigned k0 = (unsigned)(warp - ncw - 1), R = x_slice / B;  // rows of the ring
    HaloChunk cd = {}, cd1 = {};
    unsigned r[U];
    auto indices = [&](const HaloChunk& c, unsigned p0, unsigned* i) {
      const unsigned* my_rows = rows + me.row0 + c.pos0 + p0;
#pragma unroll
      for (unsigned u = 0; u < U; u++) i[u] = p0 + 32 * u + wl < c.nrows ? my_rows[32 * u + wl] : 0u;
    };
    if (k0 < K) {
      cd = my_chunks[k0];
      indices(cd, 0, r);
    }
    if (k0 + kHaloRhsWarps < K) cd1 = my_chunks[k0 + kHaloRhsWarps];
    unsigned done = k0;  // the first of this warp's chunks whose phase it has not completed
    for (unsigned k = k0; k < K; k += kHaloRhsWarps) {
      HaloChunk cd2 = {};
      if (k + 2 * kHaloRhsWarps < K) cd2 = my_chunks[k + 2 * kHaloRhsWarps];
      uint4 te = make_uint4(0, 0, 0, 0);
      const unsigned nte = cd.nrounds + (k + 1 == K ? 1u : 0u);  // the entry past the last round comes with it
      if (wl < nte) te = reinterpret_cast<const uint4*>(table)[cd.table0 + wl];
      unsigned r1[U];
      const unsigned first = cd.pos0 % R;
      bool ok = true;
      for (unsigned p0 = 0; p0 < cd.nrows; p0 += 32u * U) {
        if (p0) indices(cd, p0, r);
        double v[U][B], w[U][B];
#pragma unroll
        for (unsigned u = 0; u < U; u++)
          if (p0 + 32 * u + wl < cd.nrows)
#pragma unroll
            for (int c = 0; c < B; c++) {
              v[u][c] = in[(size_t)r[u] * B + c];
              if (DOT) w[u][c] = rdot[(size_t)r[u] * B + c];
            }
        if (p0 == 0) {
          indices(cd1, 0, r1);
          // once the chunk's copy is requested its stage is in its phase, and the rows whose places in the slice and
          // the table it takes are past
          ok = spin_until<100>([&] { return ld_volatile_i(&s_issued) > (int)k; }, &s_alive, st, wait_ns, 24);
          __threadfence_block();
          ok = __all_sync(FULL, ok);
          if (!ok) break;
        }
#pragma unroll
        for (unsigned u = 0; u < U; u++)
          if (p0 + 32 * u + wl < cd.nrows) {
            unsigned at = first + p0 + 32 * u + wl;
            if (at >= R) at -= R;
#pragma unroll
            for (int c = 0; c < B; c++) {
              X[(size_t)at * B + c] = v[u][c];
              if (DOT) reinterpret_cast<double*>(smem + rd_off)[(size_t)at * B + c] = w[u][c];
            }
          }
      }
      if (!ok) break;
      if (wl < nte) reinterpret_cast<uint4*>(tab)[(cd.round0 + wl) & (kHaloTable - 1)] = te;
      __syncwarp();
      __threadfence_block();
      if (wl == 0) mbar_arrive(&landed[k % ns]);
      done = k + kHaloRhsWarps;
      cd = cd1;
      cd1 = cd2;
#pragma unroll
      for (unsigned u = 0; u < U; u++) r[u] = r1[u];
    }
    if (wl == 0) s_rhs[k0] = done;
  } else {
    // ---------------------------------------------------------------- halo
    // a lane takes entries first, first + step, ... and goes on to the next when one is in
    const unsigned step = 32u * (unsigned)(nwarps - ncw - 1 - kHaloRhsWarps), E = me.nhalo;
    const unsigned* my_ids = hids + me.halo0;
    unsigned e = 32u * (unsigned)(warp - ncw - 1 - kHaloRhsWarps) + wl;
    unsigned id = e < E ? my_ids[e] : 0u, id1 = e + step < E ? my_ids[e + step] : 0u;
    SpinGuard g(wait_ns);
    while (__any_sync(FULL, e < E)) {
      bool got = false;
      if (e < E && (ring >= E || (int)e < ld_volatile_i(&s_armed))) {
        const size_t src = (size_t)(id & 0x7fffffffu) * B;
        double v[B];
        got = true;
        if (id & 0x80000000u) {  // an entry of the input vector (merged level pairs)
#pragma unroll
          for (int c = 0; c < B; c++) v[c] = in[src + c];
        } else {
#pragma unroll
          for (int c = 0; c < B; c++) v[c] = ld_relaxed(out + src + c);
#pragma unroll
          for (int c = 0; c < B; c++) got = got && !Sent<double>::is(v[c]);
        }
        if (got) {
          double* h = X + halo0 + (size_t)(ring >= E ? e : e % ring) * B;
          if (ring < E) __threadfence_block();  // the entry was given the sentinel before this
#pragma unroll
          for (int c = 0; c < B; c++) {
            if (B > 1 && c == B - 1) __threadfence_block();  // the last one says that the row is there
            st_volatile_s(h + c, v[c]);
          }
          e += step;
          id = id1;
          id1 = e + step < E ? my_ids[e + step] : 0u;
        }
      }
      if (__any_sync(FULL, got)) {
        g = SpinGuard(wait_ns);
      } else {
        const bool late = g.expired();
        if ((g.n & 15u) == 0 && __any_sync(FULL, late || !ld_volatile_i(&s_alive))) {
          if (__any_sync(FULL, late)) {
            if (wl == 0) raise_error(st, DFM_WAIT_TIMEOUT, 22);
            st_volatile_i(&s_alive, 0);
          }
          break;
        }
      }
    }
  }
  __shared__ double s_w[2][kHaloMaxCw];
  if (DOT && warp < ncw) {  // the CTA's partial: lanes, then compute warps in order
    dre = group_sum<32>(dre);
    dim = group_sum<32>(dim);
    if (wl == 0) {
      s_w[0][warp] = dre;
      s_w[1][warp] = dim;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // The compute warps have waited for every chunk unless the CTA is shutting down.  Then copies may still be in
    // flight; the arrivals that their phases lack are made here, where nobody computes any more, and the copies waited
    // for, with a limit of this wait's own.
    if (!s_alive)
      for (unsigned k = s_copies > ns ? s_copies - ns : 0u; k < s_copies; k++) {
        if (k >= s_rhs[k % kHaloRhsWarps]) mbar_arrive(&landed[k % ns]);
        wait_landed(&landed[k % ns], (k / ns) & 1u, st);
      }
    if (DOT) {
      dre = dim = 0.0;
      for (int w = 0; w < ncw; w++) {
        dre += s_w[0][w];
        dim += s_w[1][w];
      }
      part[blockIdx.x] = dre;
      if (DOT == 2) part[kMaxBlocks + blockIdx.x] = dim;
    }
  }
}

// ------------------------------------------------------- values of a plan
// Fills the records' values (and D^-1 rows, forward) from the factor: a thread
// per packed block, whose recipe (recipe_value, sweep_dev.cuh) says what it
// is; a padding block has none and stays zero.
// Bound by the trips to the factor, so a chunk's blocks are dealt out as one
// list: round after round, a round's ~70 blocks left half of the threads idle
// and each round paid its own trips (factor and apply on the 200x40x40 box
// 2.43 ms, 2.38 ms as it is; ILU(1) on 60x16x16 1.03 -> 0.99 ms).
template <int B, typename TV, bool FWD, bool CPLX>
__global__ void k_gather_halo(const HaloChunk* __restrict__ chunks, unsigned nchunks, int H,
                              const HaloRound* __restrict__ table, const uint4* __restrict__ recipe,
                              const uint4* __restrict__ terms, const double* __restrict__ fdiag,
                              const double* __restrict__ foff, char* blob) {
  constexpr int KT = HaloK<B>::KT;
  using R = HaloRec<B, KT, TV, FWD>;
  constexpr unsigned NONE = 0xffffffffu;
  const unsigned uH = (unsigned)H, LR = B * uH;
  __shared__ unsigned item0[33], row0[33], byte0[33], shape_of[32];  // where each round of the chunk starts
  for (unsigned q = blockIdx.x; q < nchunks; q += gridDim.x) {
    const HaloChunk cd = chunks[q];
    char* base = blob + cd.off;
    char* recs = base + cl_al16(4 * cd.nrows);
    __syncthreads();  // the last chunk's tables are done with
    if (threadIdx.x < 32) {
      const unsigned j = threadIdx.x, shape = j < cd.nrounds ? table[cd.table0 + j].shape : 0u;
      const unsigned n = shape & 0xffu, pieces = (shape >> 8) & kHaloMaxPieces, ke = (shape >> 20) & kHaloMaxExtra;
      unsigned it = n * (KT + ke) * uH, rw = n, by = 16 * pieces * n * LR;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned a = __shfl_up_sync(0xffffffffu, it, o), b = __shfl_up_sync(0xffffffffu, rw, o),
                       c = __shfl_up_sync(0xffffffffu, by, o);
        if (j >= (unsigned)o) it += a, rw += b, by += c;
      }
      if (j == 0) item0[0] = row0[0] = byte0[0] = 0;
      item0[j + 1] = it, row0[j + 1] = rw, byte0[j + 1] = by;
      shape_of[j] = shape;
    }
    __syncthreads();
    auto round_of = [](const unsigned* first, unsigned t) {  // the round whose range has t
      unsigned j = 0;
#pragma unroll
      for (unsigned s = 16; s; s >>= 1)
        if (first[j + s] <= t) j += s;
      return j;
    };
    for (unsigned x = threadIdx.x; x < item0[32]; x += blockDim.x) {
      const uint4 rc = recipe[cd.rec0 + x];
      if (rc.x == NONE && rc.y == rc.z) continue;  // padding
      const unsigned j = round_of(item0, x), t = x - item0[j], shape = shape_of[j];
      const unsigned pieces = (shape >> 8) & kHaloMaxPieces, ke = (shape >> 20) & kHaloMaxExtra;
      const unsigned nb = (KT + ke) * uH;  // packed blocks per row
      const unsigned r = t / nb, b = t - r * nb, half = b % uH, k = b / uH;
      double v[B * B];
      recipe_value<B, CPLX>(rc, terms, fdiag, foff, v);
#pragma unroll
      for (int c = 0; c < B; c++) {
        char* rec = recs + byte0[j] + 16 * (size_t)pieces * (r * LR + half * B + c);
        TV* d = k < (unsigned)KT ? reinterpret_cast<TV*>(rec + 16 * R::PO) + k * B
                                 : reinterpret_cast<TV*>(rec + 16 * R::P + cl_al16(4 * ke)) + (k - KT) * B;
#pragma unroll
        for (int e = 0; e < B; e++) d[e] = (TV)v[c * B + e];
      }
    }
    if (FWD)
      for (unsigned x = threadIdx.x; x < row0[32]; x += blockDim.x) {
        const unsigned j = round_of(row0, x), r = x - row0[j], pieces = (shape_of[j] >> 8) & kHaloMaxPieces;
        double v[B * B];
        load_factor_blk<B, CPLX>(fdiag, reinterpret_cast<const unsigned*>(base)[x], v);
#pragma unroll
        for (int c = 0; c < B; c++) {
          double* d = reinterpret_cast<double*>(recs + byte0[j] + 16 * (size_t)pieces * (r * LR + c) + 16 * R::PO + R::VB);
#pragma unroll
          for (int e = 0; e < B; e++) d[e] = v[c * B + e];
        }
      }
  }
}

int sweep_halo_refresh(dfm_ilu M, SweepPlan* P) {
  const int grid = (int)std::min<unsigned>(P->nchunks, (unsigned)M->ctx->nsm * 8);
  cudaStream_t s = M->ctx->stream;
  const int H = P->lpr;
  const HaloRound* tab = reinterpret_cast<const HaloRound*>(P->d_table);
#define DFM_GATHER(BV, TV, CX)                                                                                       \
  do {                                                                                                               \
    if (P->fwd)                                                                                                      \
      k_gather_halo<BV, TV, true, CX><<<grid, 128, 0, s>>>(P->d_hchunks, P->nchunks, H, tab, P->d_recipe, P->d_terms, \
                                                           M->d_fdiag, M->d_foff, P->d_blob);                    \
    else                                                                                                             \
      k_gather_halo<BV, TV, false, CX><<<grid, 128, 0, s>>>(P->d_hchunks, P->nchunks, H, tab, P->d_recipe,            \
                                                            P->d_terms, M->d_fdiag, M->d_foff, P->d_blob);           \
  } while (0)
  if (M->vt == DFM_COMPLEX) {
    if (P->val_bytes == 8) DFM_GATHER(2, double, true); else DFM_GATHER(2, float, true);
  } else if (P->val_bytes == 8) {
    if (M->b == 1) DFM_GATHER(1, double, false); else if (M->b == 2) DFM_GATHER(2, double, false);
    else DFM_GATHER(3, double, false);
  } else {
    if (M->b == 1) DFM_GATHER(1, float, false); else if (M->b == 2) DFM_GATHER(2, float, false);
    else DFM_GATHER(3, float, false);
  }
#undef DFM_GATHER
  DFM_CUDA_TRY(cudaGetLastError());
  return DFM_OK;
}

// ------------------------------------------------------------------ plan
// One operand of a row: kind 0 = a row of the CTA (v = row), 1 = another
// CTA's output row v, 2 = the input vector's row v (the second level of a
// merged pair reads it in place of the first level's output); with the
// recipe of the packed block.
struct HaloOp {
  unsigned kind, v;
  uint4 rc;
};

struct HaloShape {  // what the byte layout of a plan depends on
  unsigned B, H, KT, PO, P, VB, sv, cap;  // cap: rows of a full round
  // pieces of a record with ke extra blocks
  unsigned pieces(unsigned ke) const {
    const unsigned x = ke ? (cl_al16(4 * ke) + cl_al16(ke * B * sv)) / 16 : 0u;
    return (P + x) | 1u;
  }
};

template <int B, typename TV>
static HaloShape halo_shape_t(unsigned H, bool fwd, unsigned cw) {
  constexpr int KT = HaloK<B>::KT;
  using F = HaloRec<B, KT, TV, true>;
  using W = HaloRec<B, KT, TV, false>;
  const unsigned rpw = 32u / (B * H);
  return {(unsigned)B, H, (unsigned)KT, (unsigned)F::PO, (unsigned)(fwd ? F::P : W::P), (unsigned)F::VB,
          (unsigned)sizeof(TV), cw * rpw};
}
static HaloShape halo_shape(unsigned b, unsigned H, int val_bytes, bool fwd, unsigned cw) {
  if (val_bytes == 8)
    return b == 1 ? halo_shape_t<1, double>(H, fwd, cw)
                  : b == 2 ? halo_shape_t<2, double>(H, fwd, cw) : halo_shape_t<3, double>(H, fwd, cw);
  return b == 1 ? halo_shape_t<1, float>(H, fwd, cw)
                : b == 2 ? halo_shape_t<2, float>(H, fwd, cw) : halo_shape_t<3, float>(H, fwd, cw);
}

// The chunks of one CTA: the blob's bytes, halo row ids, row order, recipes
// and terms with indices of this CTA.  Halo operands are 0x80000000 | entry
// until the ring's size is known.
struct HaloCta {
  std::vector<HaloChunk> chunks;
  std::vector<char> blob;
  std::vector<unsigned> rows, hids;
  std::vector<unsigned> last;  // last chunk that reads a row, by position
  std::vector<HaloRound> table;
  std::vector<uint4> recipe, terms;
  unsigned stage_max = 0;
  bool extras = false;  // a round has rows with more than KT * H blocks
};

// The halo plan of one sweep direction over G CTAs (contiguous ranges of the
// natural order balanced by dependency blocks, or the ILU's row partition),
// for H lanes per component and cw compute warps.
int sweep_halo_plan_build(dfm_ilu M, bool fwd, int G, int val_bytes, SweepPlan* P, int part, bool merge, int lpr,
                          int cw) {
  const unsigned N = M->N;
  const unsigned b = M->vt == DFM_COMPLEX ? 2u : M->b;  // complex scalars as real 2x2 blocks
  if (lpr == 0) lpr = b == 3 ? 2 : 1;
  if (cw == 0) cw = 2;
  const int H = lpr;
  const HaloShape S = halo_shape(b, (unsigned)H, val_bytes, fwd, (unsigned)cw);
  const std::vector<unsigned>& rp = M->A->h_rowptr;
  const std::vector<unsigned>& ci = M->A->h_colind;
  const std::vector<unsigned>& dia = M->h_diaind;
  const std::vector<unsigned>& lev = fwd ? M->lev_f : M->lev_b;
  sweep_plan_free(P);
  if (N >= 0x40000000u) return DFM_ERR_UNSUPPORTED;
  if (part == 2) {
    const int rc = sweep_own_partition(M, (unsigned)G);
    if (rc) return rc;
  }
  const int parts = G;  // as asked for
  if (part == 2) G = (int)M->own_n;
  // cta_of: the CTA of a row; list: the rows CTA by CTA
  std::vector<unsigned> cta_of(N), list(N), range(G + 1, 0);
  if (part) {
    if (part == 1 && ((unsigned)G != M->nparts || M->part_of.size() != N)) return DFM_ERR_INVALID;
    cta_of = part == 1 ? M->part_of : M->own_of;
    for (unsigned i = 0; i < N; i++) range[cta_of[i] + 1]++;
    for (int c = 0; c < G; c++) range[c + 1] += range[c];
    std::vector<unsigned> fill(range.begin(), range.end() - 1);
    for (unsigned i = 0; i < N; i++) list[fill[cta_of[i]]++] = i;
  } else {
    if (G < 1) G = 1;
    if ((unsigned)G > std::max(N, 1u)) G = (int)std::max(N, 1u);
    std::vector<unsigned long long> wpre(N + 1, 0);
    for (unsigned i = 0; i < N; i++) {
      const unsigned nb = fwd ? dia[i] - rp[i] : rp[i + 1] - dia[i];
      wpre[i + 1] = wpre[i] + nb + 1;
    }
    range.assign(G + 1, N);
    range[0] = 0;
    for (int c = 1; c < G; c++) {
      const unsigned long long target = wpre[N] * (unsigned long long)c / (unsigned)G;
      range[c] = (unsigned)(std::lower_bound(wpre.begin(), wpre.end(), target) - wpre.begin());
      range[c] = std::max(range[c], range[c - 1]);
    }
    for (int c = 0; c < G; c++)
      for (unsigned i = range[c]; i < range[c + 1]; i++) {
        cta_of[i] = (unsigned)c;
        list[i] = i;
      }
  }
  constexpr unsigned NONE = 0xffffffffu;
  constexpr unsigned kInput = 0x80000000u;  // halo id of an entry of the input vector
  std::vector<unsigned> slot(N, NONE);  // position of a row in its CTA's slice
  // step of a row: its level, or with merged level pairs its level / 2
  auto step = [&](unsigned i) { return merge ? lev[i] / 2 : lev[i]; };
  // operand codes until the areas' sizes are known: a position of the slice, a halo entry, the zero block
  constexpr unsigned kHalo = 0x80000000u, kZero = 0x7fffffffu;
  struct Round {
    unsigned row0, nrow, K;  // rows of the chunk, blocks per lane
  };
  // the chunks of every CTA; ringed: the halo area cannot hold all entries
  std::vector<HaloCta> ctas;
  // CTAs first, first + by, ...; the CTAs are independent of one another (a row's slot is set and read by its own
  // CTA), so several host threads share them
  auto build_some = [&](int first, int by, bool ringed, unsigned chunk_bytes, unsigned round_bytes) -> int {
    std::vector<unsigned> hpos(N, NONE);                   // scratch: output row -> its halo entry
    std::vector<unsigned> hpos_in(merge ? N : 0u, NONE);   // scratch: the same for input entries
    std::vector<HaloOp> ops;
    std::vector<unsigned> kmap(merge ? N : 0u, NONE);  // scratch: column -> position in ops
    auto slots = [&](unsigned i, unsigned& s0, unsigned& s1) {
      s0 = fwd ? rp[i] : dia[i];
      s1 = fwd ? dia[i] : rp[i + 1];
    };
    // operands of row i of CTA c (the same substitutions as the range plans, sweep.cu)
    auto row_ops = [&](unsigned i, unsigned c, std::vector<uint4>& terms) {
      ops.clear();
      auto opnd = [&](unsigned col, uint4 rc) { return HaloOp{cta_of[col] == c ? 0u : 1u, col, rc}; };
      unsigned s0, s1;
      slots(i, s0, s1);
      if (!(merge && (lev[i] & 1u))) {
        for (unsigned s = s0; s < s1; s++) ops.push_back(opnd(ci[s], make_uint4(s, 0u, 0u, 0u)));
        return;
      }
      // second level of a pair: operands on the first level are substituted
      for (unsigned s = s0; s < s1; s++) {
        const unsigned j = ci[s];
        if (lev[j] + 1 != lev[i]) continue;
        const unsigned t0 = (unsigned)terms.size();
        terms.push_back(make_uint4(s, fwd ? j : NONE, NONE, 0u));  // L_ij D_j^-1  |  U'_ij
        ops.push_back(HaloOp{2u, j, make_uint4(NONE, t0, t0 + 1, 0u)});
      }
      const size_t first_c = ops.size();
      for (unsigned s = s0; s < s1; s++) {
        const unsigned k = ci[s];
        if (lev[k] + 1 == lev[i]) continue;
        kmap[k] = (unsigned)ops.size();
        ops.push_back(opnd(k, make_uint4(s, 0u, 0u, 1u)));
      }
      // fill terms F_ij (D_j^-1) F_jk, grouped per column k
      std::vector<std::vector<uint4>> tl(ops.size() - first_c);
      for (unsigned s = s0; s < s1; s++) {
        const unsigned j = ci[s];
        if (lev[j] + 1 != lev[i]) continue;
        unsigned t0, t1;
        slots(j, t0, t1);
        for (unsigned t = t0; t < t1; t++) {
          const unsigned k = ci[t];
          if (kmap[k] == NONE) {
            kmap[k] = (unsigned)ops.size();
            ops.push_back(opnd(k, make_uint4(NONE, 0u, 0u, 1u)));
            tl.emplace_back();
          }
          tl[kmap[k] - first_c].push_back(make_uint4(s, fwd ? j : NONE, t, 0u));
        }
      }
      for (size_t q = first_c; q < ops.size(); q++) {
        ops[q].rc.y = (unsigned)terms.size();
        for (const uint4& t : tl[q - first_c]) terms.push_back(t);
        ops[q].rc.z = (unsigned)terms.size();
        kmap[ops[q].v] = NONE;
      }
    };
    std::vector<Round> rounds;
    std::vector<unsigned> op0, code;  // operands of the open chunk's rows
    std::vector<uint4> rcs;
    for (int c = first; c < G; c += by) {
      HaloCta& C = ctas[c];
      std::vector<unsigned> todo(list.begin() + range[c], list.begin() + range[c + 1]);
      if (!fwd) std::reverse(todo.begin(), todo.end());
      // level by level; inside a level the longer rows first, so a round's rows need about the same K
      auto klen = [&](unsigned i) {
        unsigned s0, s1;
        slots(i, s0, s1);
        return (s1 - s0 + S.H - 1) / S.H;
      };
      std::stable_sort(todo.begin(), todo.end(), [&](unsigned x, unsigned y) {
        const unsigned lx = step(x), ly = step(y);
        return lx != ly ? lx < ly : klen(x) > klen(y);
      });
      std::vector<unsigned> touched, touched_in;  // rows with a halo entry in hpos / hpos_in
      unsigned pos0 = 0;                          // slice position of the open chunk's first row
      unsigned reuse0 = 0;                        // first halo entry the open chunk may still read in a ring
      auto close = [&]() {
        const unsigned nrow = (unsigned)C.rows.size() - pos0, nround = (unsigned)rounds.size();
        HaloChunk cd = {};
        cd.off = C.blob.size();
        cd.nrows = nrow;
        cd.pos0 = pos0;
        cd.need = (unsigned)C.hids.size();
        cd.rec0 = (unsigned)C.recipe.size();
        cd.round0 = (unsigned)C.table.size();
        cd.nrounds = nround;
        unsigned at = cl_al16(4u * nrow);
        std::vector<HaloRound> tab(nround);  // offsets in the chunk until its stage is known
        for (unsigned j = 0; j < nround; j++) {
          const Round& rd = rounds[j];
          const unsigned ke = rd.K > S.KT ? rd.K - S.KT : 0u;
          const unsigned pieces = S.pieces(ke);
          tab[j] = {at, pos0 + rd.row0, 4u * rd.row0, rd.nrow | (pieces << 8) | (ke << 20)};
          C.extras = C.extras || ke;
          at += 16u * pieces * rd.nrow * S.B * S.H;
        }
        tab[nround - 1].shape |= kHaloLast;
        cd.bytes = at;
        C.blob.resize(C.blob.size() + at, 0);
        char* base = C.blob.data() + cd.off;
        std::memcpy(base, C.rows.data() + pos0, 4 * (size_t)nrow);
        for (unsigned j = 0; j < nround; j++) {
          const Round& rd = rounds[j];
          const unsigned ke = (tab[j].shape >> 20) & kHaloMaxExtra, pieces = (tab[j].shape >> 8) & kHaloMaxPieces;
          const unsigned nb = (S.KT + ke) * S.H;
          for (unsigned r = 0; r < rd.nrow; r++) {
            const unsigned q0 = op0[rd.row0 + r], q1 = op0[rd.row0 + r + 1];
            for (unsigned t = 0; t < nb; t++) {
              const bool pad = q0 + t >= q1;
              C.recipe.push_back(pad ? make_uint4(NONE, 0u, 0u, 0u) : rcs[q0 + t]);
              const unsigned o = pad ? kZero : code[q0 + t], half = t % S.H, k = t / S.H;
              for (unsigned e = 0; e < S.B; e++) {
                char* rec = base + tab[j].rec + 16 * (size_t)pieces * (r * S.B * S.H + half * S.B + e);
                unsigned* d = k < S.KT ? reinterpret_cast<unsigned*>(rec) + k
                                       : reinterpret_cast<unsigned*>(rec + 16 * S.P) + (k - S.KT);
                *d = o;
              }
            }
          }
        }
        C.table.insert(C.table.end(), tab.begin(), tab.end());
        C.stage_max = std::max(C.stage_max, at);
        C.chunks.push_back(cd);
        reuse0 = C.chunks.size() > kHaloReuse ? C.chunks[C.chunks.size() - 1 - kHaloReuse].need : 0u;
        pos0 += nrow;
        rounds.clear();
        op0.assign(1, 0u);
        code.clear();
        rcs.clear();
      };
      op0.assign(1, 0u);
      unsigned bytes = 0;      // of the open chunk
      bool have_ops = false;   // ops holds todo[p]'s operands
      for (size_t p = 0; p < todo.size();) {
        // one round: rows of one step
        const unsigned L = step(todo[p]);
        Round rd = {(unsigned)C.rows.size() - pos0, 0u, 0u};
        while (p < todo.size() && step(todo[p]) == L && rd.nrow < S.cap) {
          const unsigned i = todo[p];
          if (!have_ops) row_ops(i, (unsigned)c, C.terms);
          const unsigned K = std::max(rd.K, ((unsigned)ops.size() + S.H - 1) / S.H);
          have_ops = rd.nrow > 0 && 16u * S.pieces(K > S.KT ? K - S.KT : 0u) * (rd.nrow + 1) * S.B * S.H > round_bytes;
          if (have_ops) break;  // the row starts the next round
          p++;
          for (const HaloOp& o : ops) {
            unsigned cd;
            if (o.kind == 0) {
              cd = slot[o.v];
              C.last[cd] = (unsigned)C.chunks.size();
            } else {
              std::vector<unsigned>& hm = o.kind == 1 ? hpos : hpos_in;
              // fetched once; in a ring again if it was fetched more than kHaloReuse chunks ago
              if (hm[o.v] == NONE || (ringed && hm[o.v] < reuse0)) {
                if (hm[o.v] == NONE) (o.kind == 1 ? touched : touched_in).push_back(o.v);
                hm[o.v] = (unsigned)C.hids.size();
                C.hids.push_back(o.kind == 1 ? o.v : (kInput | o.v));
              }
              cd = kHalo | hm[o.v];
            }
            code.push_back(cd);
            rcs.push_back(o.rc);
          }
          op0.push_back((unsigned)code.size());
          rd.K = K;
          slot[i] = (unsigned)C.rows.size();
          C.rows.push_back(i);
          C.last.push_back((unsigned)C.chunks.size());
          rd.nrow++;
        }
        const unsigned ke = rd.K > S.KT ? rd.K - S.KT : 0u;
        if (ke > kHaloMaxExtra || S.pieces(ke) > kHaloMaxPieces) return DFM_ERR_UNSUPPORTED;
        rounds.push_back(rd);
        const unsigned more = 16u * S.pieces(ke) * rd.nrow * S.B * S.H + 4u * rd.nrow;
        bytes += more;
        if (bytes + more > chunk_bytes || rounds.size() == kHaloChunkRounds || p == todo.size()) {
          close();
          bytes = 0;
        }
      }
      for (unsigned i : touched) hpos[i] = NONE;
      for (unsigned i : touched_in) hpos_in[i] = NONE;
    }
    return DFM_OK;
  };
  auto build = [&](bool ringed, unsigned chunk_bytes, unsigned round_bytes) -> int {
    ctas.assign(G, HaloCta());
    // (a plan of a few thousand rows is built faster than threads are started)
    const int nt = N < 8192 ? 1 : std::min({G, 8, (int)std::max(1u, std::thread::hardware_concurrency())});
    std::vector<int> rc(nt, DFM_ERR_NOMEM);
    auto work = [&](int t) {
      try {
        rc[t] = build_some(t, nt, ringed, chunk_bytes, round_bytes);
      } catch (...) {
      }
    };
    std::vector<std::thread> pool;
    int started = 1;
    try {
      for (; started < nt; started++) pool.emplace_back(work, started);
    } catch (...) {
    }
    work(0);
    for (std::thread& th : pool) th.join();
    for (int t = started; t < nt; t++) work(t);  // shares of threads that could not be started
    for (int r : rc)
      if (r) return r;
    return DFM_OK;
  };
  // Sizes for t stages.  Chunk k is requested when chunk k - t is done.  The slice must hold, beside chunk k's rows,
  // every earlier row that a chunk past k - t reads; a halo ring the entries of the chunks past k - t and of the
  // kHaloReuse before them.
  const size_t bar_bytes = 2 * 8 * (size_t)kHaloMaxStages + 16 * (size_t)kHaloTable;  // barriers, round table
  struct Sizes {
    int ns = 0;
    unsigned slice = 1, ring = 1;  // rows of the slice, entries of the halo area
    size_t halo0 = 0, rd_off = 0, x_bytes = 0, stage = 64;  // element, bytes
  };
  auto sizes_for = [&](int t, bool ringed) {
    Sizes z;
    for (const HaloCta& C : ctas) {
      z.stage = std::max<size_t>(z.stage, C.stage_max);
      const size_t nk = C.chunks.size();
      std::vector<unsigned> low(nk + 1, (unsigned)C.rows.size());  // first position read by chunk j or a later one
      for (size_t p = C.rows.size(); p-- > 0;) low[C.last[p]] = (unsigned)p;
      for (size_t j = nk; j-- > 0;) low[j] = std::min(low[j], low[j + 1]);
      for (size_t k = 0; k < nk; k++) {
        const unsigned end = C.chunks[k].pos0 + C.chunks[k].nrows;
        z.slice = std::max(z.slice, end - low[k >= (size_t)t ? k - t + 1 : 0]);
        const size_t back = (size_t)t + kHaloReuse;
        if (ringed) z.ring = std::max(z.ring, C.chunks[k].need - (k >= back ? C.chunks[k - back].need : 0u));
      }
      if (!ringed) z.ring = std::max(z.ring, (unsigned)C.hids.size());
    }
    z.halo0 = (size_t)z.slice * b + ((b + 1u) & ~1u);  // behind the zero block, at an even element for b = 2
    z.halo0 += z.halo0 & 1u;
    size_t end = (z.halo0 + (size_t)z.ring * b) * 8;
    end += end & 8u;
    if (!fwd && end + 8 * (size_t)z.slice * b + (size_t)t * z.stage + bar_bytes + 128 <= kHaloSmemBudget) {
      z.rd_off = end;
      end += 8 * (size_t)z.slice * b;
    }
    z.x_bytes = (end + 127) & ~(size_t)127;
    if (z.x_bytes + (size_t)t * z.stage + bar_bytes <= kHaloSmemBudget) z.ns = t;
    return z;
  };
  // chunks of several rounds and all halo entries if enough stages fit, else a halo ring, else chunks of one round
  struct Try {
    bool ringed;
    unsigned bytes, round;
  };
  Sizes sz;
  Try built = {}, now = {};
  size_t least = SIZE_MAX;  // bytes that the areas beside the stages take at the least
  auto attempt = [&](const Try& a) -> int {
    now = a;
    const int rc = build(a.ringed, a.bytes, a.round);
    if (rc) return rc;
    Sizes z;
    for (int t = kHaloMaxStages; t >= kHaloMinStages && z.ns == 0; t--) z = sizes_for(t, a.ringed);
    least = std::min(least, z.x_bytes);
    if (z.ns > sz.ns) {
      sz = z;
      built = a;
    }
    return DFM_OK;
  };
  for (const Try& a : {Try{false, kHaloChunkBytes, kChunkMaxBytes}, Try{true, kHaloChunkBytes, kChunkMaxBytes},
                       Try{true, 1u, kChunkMaxBytes}, Try{false, 1u, kChunkMaxBytes}}) {
    if (sz.ns >= kHaloGoodStages) break;
    const int rc = attempt(a);
    if (rc) return rc;
  }
  // Rounds of rows with hundreds of blocks may be what does not fit: smaller ones, down to a row each, as long as the
  // other areas leave room for stages.  (With FP32 values more rows come into a round of the same bytes, so that a plan
  // could be had in FP64 and not in FP32.)
  for (unsigned r = kChunkMaxBytes / 2; sz.ns == 0 && r >= 256 && least + bar_bytes + kHaloMinStages * 1024 <= kHaloSmemBudget;
       r /= 2)
    for (const bool ringed : {true, false}) {
      const int rc = sz.ns ? DFM_OK : attempt({ringed, 1u, r});
      if (rc) return rc;
    }
  if (sz.ns && (now.ringed != built.ringed || now.bytes != built.bytes || now.round != built.round)) {
    const int rc = build(built.ringed, built.bytes, built.round);
    if (rc) return rc;
  }
  if (sz.ns == 0) return DFM_ERR_UNSUPPORTED;
  const int ns = sz.ns;
  const unsigned ring = sz.ring, stage_max = (unsigned)sz.stage;
  const size_t x_bytes = sz.x_bytes, halo0 = sz.halo0, x_slice = (size_t)sz.slice * b;
  size_t nchunks = 0, nrec = 0, nterm = 0, blob_size = 0, nhid = 0, nround = 0;
  for (const HaloCta& C : ctas) {
    nchunks += C.chunks.size();
    nrec += C.recipe.size();
    nterm += C.terms.size();
    blob_size += C.blob.size();
    nhid += C.hids.size();
    nround += C.table.size() + 1;
  }
  if (nround >= 0x80000000ull || nrec >= 0xffffffffull || nterm >= 0xffffffffull || nhid >= 0x80000000ull) return DFM_ERR_UNSUPPORTED;

  std::vector<HaloChunk> chunks;
  chunks.reserve(nchunks);
  std::vector<HaloCtaDesc> desc(G);
  size_t rec0 = 0, term0 = 0, off0 = 0, hid0 = 0, tab0 = 0;
  for (int c = 0; c < G; c++) {
    HaloCta& C = ctas[c];
    desc[c] = {(unsigned)chunks.size(), (unsigned)C.chunks.size(), range[c], (unsigned)C.rows.size(),
               (unsigned)hid0, (unsigned)C.hids.size(), (unsigned)C.table.size(), 0u};
    for (size_t q = 0; q < C.chunks.size(); q++) {
      HaloChunk& cd = C.chunks[q];
      char* base = C.blob.data() + cd.off;
      const unsigned stage = (unsigned)(x_bytes + (q % (size_t)ns) * stage_max);
      for (unsigned j = 0; j < cd.nrounds; j++) {
        HaloRound& rd = C.table[cd.round0 + j];
        const unsigned ke = (rd.shape >> 20) & kHaloMaxExtra, pieces = (rd.shape >> 8) & kHaloMaxPieces;
        const unsigned nrec_j = (rd.shape & 0xffu) * S.B * S.H;
        for (unsigned l = 0; l < nrec_j; l++) {
          char* rec = base + rd.rec + 16 * (size_t)pieces * l;
          auto fix = [&](unsigned* o, unsigned n) {
            for (unsigned t = 0; t < n; t++)
              if (o[t] == kZero) o[t] = (unsigned)(8 * x_slice);
              else if (o[t] & kHalo) o[t] = (unsigned)((halo0 + (size_t)((o[t] & ~kHalo) % ring) * b) * 8);
              else o[t] = 8u * b * (o[t] % sz.slice);
          };
          fix(reinterpret_cast<unsigned*>(rec), S.KT);
          fix(reinterpret_cast<unsigned*>(rec + 16 * S.P), ke);
        }
        rd.slot = 8u * b * (rd.slot % sz.slice);
        rd.rec += stage;
        rd.rows += stage;
      }
      cd.off += off0;
      cd.rec0 += (unsigned)rec0;
      cd.table0 = (unsigned)tab0 + cd.round0;
      chunks.push_back(cd);
    }
    if (!C.table.empty()) {  // past the last round: its records, no rows
      C.table.push_back(C.table.back());
      C.table.back().shape &= ~(0xffu | kHaloLast);
    }
    for (uint4& r : C.recipe) {
      r.y += (unsigned)term0;
      r.z += (unsigned)term0;
    }
    rec0 += C.recipe.size();
    term0 += C.terms.size();
    off0 += C.blob.size();
    hid0 += C.hids.size();
    tab0 += C.table.size();
  }
  P->G = G;
  for (const HaloCta& C : ctas) P->extras = P->extras || C.extras;
  P->fwd = fwd;
  P->halo = true;
  P->nchunks = (unsigned)chunks.size();
  P->stage_bytes = stage_max;
  P->x_bytes = (unsigned)x_bytes;
  P->x_slice = (unsigned)x_slice;
  P->halo0 = (unsigned)halo0;
  P->rd_off = (unsigned)sz.rd_off;
  P->ring = ring;
  for (const HaloCta& C : ctas) {
    P->ringed = P->ringed || C.hids.size() > ring;
    P->part_rows = std::max(P->part_rows, (unsigned)C.rows.size());
  }
  P->val_bytes = val_bytes;
  P->vec_bytes = 8;
  P->nstage = ns;
  P->smem = x_bytes + (size_t)ns * stage_max + bar_bytes;
  P->lpr = lpr;
  P->cw = cw;
  P->hw = 4;
  cudaStream_t s = M->ctx->stream;
  // one allocation: the blob, then the arrays (16-byte aligned); the arrays go over in one copy from `host`, the blob
  // CTA by CTA
  size_t at = (blob_size + 255) & ~(size_t)255;
  const size_t arrays0 = at;
  auto place = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 15) & ~(size_t)15;
    return o;
  };
  const size_t o_chunks = place(sizeof(HaloChunk) * chunks.size()), o_ctas = place(sizeof(HaloCtaDesc) * G);
  const size_t o_table = place(sizeof(HaloRound) * nround), o_rows = place(sizeof(unsigned) * N);
  const size_t o_hids = place(sizeof(unsigned) * nhid), o_rec = place(sizeof(uint4) * nrec);
  const size_t o_terms = place(sizeof(uint4) * nterm);
  std::vector<char> host(at - arrays0 + 16);
  auto put = [&](size_t o, const void* src, size_t bytes) {
    if (bytes) std::memcpy(host.data() + (o - arrays0), src, bytes);
  };
  put(o_chunks, chunks.data(), sizeof(HaloChunk) * chunks.size());
  put(o_ctas, desc.data(), sizeof(HaloCtaDesc) * G);
  rec0 = term0 = off0 = hid0 = tab0 = 0;
  for (int c = 0; c < G; c++) {
    const HaloCta& C = ctas[c];
    put(o_rec + sizeof(uint4) * rec0, C.recipe.data(), sizeof(uint4) * C.recipe.size());
    put(o_terms + sizeof(uint4) * term0, C.terms.data(), sizeof(uint4) * C.terms.size());
    put(o_hids + sizeof(unsigned) * hid0, C.hids.data(), sizeof(unsigned) * C.hids.size());
    put(o_table + sizeof(HaloRound) * tab0, C.table.data(), sizeof(HaloRound) * C.table.size());
    put(o_rows + sizeof(unsigned) * range[c], C.rows.data(), sizeof(unsigned) * C.rows.size());
    rec0 += C.recipe.size();
    term0 += C.terms.size();
    hid0 += C.hids.size();
    tab0 += C.table.size();
  }
  DFM_CUDA_TRY(cudaMalloc(&P->d_arena, at + 16));
  P->d_blob = P->d_arena;
  P->d_hchunks = reinterpret_cast<HaloChunk*>(P->d_arena + o_chunks);
  P->d_ctas = reinterpret_cast<HaloCtaDesc*>(P->d_arena + o_ctas);
  P->d_table = P->d_arena + o_table;
  P->d_rows = reinterpret_cast<unsigned*>(P->d_arena + o_rows);
  P->d_hids = reinterpret_cast<unsigned*>(P->d_arena + o_hids);
  P->d_recipe = reinterpret_cast<uint4*>(P->d_arena + o_rec);
  P->d_terms = reinterpret_cast<uint4*>(P->d_arena + o_terms);
  DFM_CUDA_TRY(cudaMemcpyAsync(P->d_arena + arrays0, host.data(), at - arrays0, cudaMemcpyHostToDevice, s));
  off0 = 0;
  for (const HaloCta& C : ctas) {
    if (!C.blob.empty())
      DFM_CUDA_TRY(cudaMemcpyAsync(P->d_blob + off0, C.blob.data(), C.blob.size(), cudaMemcpyHostToDevice, s));
    off0 += C.blob.size();
  }
  P->part = part;
  P->parts = parts;
  P->merged = merge;
  DFM_CUDA_TRY(cudaStreamSynchronize(s));
  P->valid = true;
  P->stale = true;
  return DFM_OK;
}

// ---------------------------------------------------------------- launch
template <int B, int H, typename TV, bool FWD, int DK, bool EX>
static cudaError_t launch_halo(dfm_ilu M, const SweepPlan* P, const double* in, double* out, const double* rdot,
                               double* part, KrylovScalars* sc, const double* rr_part, int rr_n) {
  dfm_ctx c = M->ctx;
  // the launch holds kHaloMaxWarps warps; more halo warps than fit bring nothing
  const int ncw = P->cw, nhw = std::min(P->hw, kHaloMaxWarps - 1 - kHaloRhsWarps - P->cw);
  if (ncw < 1 || ncw > kHaloMaxCw || nhw < 1) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P->G);
  cfg.blockDim = dim3(32 * (ncw + 1 + kHaloRhsWarps + nhw));
  cfg.dynamicSmemBytes = P->smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto go = [&](auto fn) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P->smem);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, fn, (const HaloChunk*)P->d_hchunks, (const HaloCtaDesc*)P->d_ctas,
                              (const HaloRound*)P->d_table,
                              (const unsigned*)P->d_rows, (const unsigned*)P->d_hids, (const char*)P->d_blob,
                              P->stage_bytes, P->nstage, P->x_bytes, P->x_slice, P->halo0, P->ring, P->rd_off, ncw,
                              in, out,
                              rdot, part, sc, rr_part, rr_n, c->d_status, (uint64_t)c->wait_ns);
  };
  // forward sweeps carry no fused dot; backward ones take it when asked
  if constexpr (FWD) {
    return go(k_sweep_halo<B, H, TV, true, 0, EX>);
  } else {
    if (part && P->rd_off) return go(k_sweep_halo<B, H, TV, false, DK, EX>);
    if (part) {  // no room for rdot: a pass of its own
      const cudaError_t e = go(k_sweep_halo<B, H, TV, false, 0, EX>);
      if (e != cudaSuccess) return e;
      k_halo_dot<DK><<<P->G, 256, 0, c->stream>>>((size_t)M->N * (DK == 2 ? 1 : B), rdot, out, part, sc);
      return cudaGetLastError();
    }
    return go(k_sweep_halo<B, H, TV, false, 0, EX>);
  }
}

template <int B, typename TV, bool FWD, int DK>
static cudaError_t launch_halo_lanes(dfm_ilu M, const SweepPlan* P, const double* in, double* out, const double* rdot,
                                     double* part, KrylovScalars* sc, const double* rr_part, int rr_n) {
#define DFM_HALO_H(HV)                                                                                       \
  return P->extras ? launch_halo<B, HV, TV, FWD, DK, true>(M, P, in, out, rdot, part, sc, rr_part, rr_n)     \
                   : launch_halo<B, HV, TV, FWD, DK, false>(M, P, in, out, rdot, part, sc, rr_part, rr_n)
  switch (P->lpr) {
    case 1: DFM_HALO_H(1);
    case 2: DFM_HALO_H(2);
    case 4: DFM_HALO_H(4);
    default:  // 8 lanes run when a caller asks for them: the kernel for rows of any length alone
      return launch_halo<B, 8, TV, FWD, DK, true>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
  }
#undef DFM_HALO_H
}

template <typename TV, bool FWD>
static cudaError_t launch_halo_b(dfm_ilu M, const SweepPlan* P, const double* in, double* out, const double* rdot,
                                 double* part, KrylovScalars* sc, const double* rr_part, int rr_n) {
  if (M->vt == DFM_COMPLEX) return launch_halo_lanes<2, TV, FWD, 2>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
  switch (M->b) {
    case 1: return launch_halo_lanes<1, TV, FWD, 1>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
    case 2: return launch_halo_lanes<2, TV, FWD, 1>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
    default: return launch_halo_lanes<3, TV, FWD, 1>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
  }
}

cudaError_t sweep_halo_launch(dfm_ilu M, bool fwd, const SweepPlan* P, const double* in, double* out,
                              const double* rdot, double* part, KrylovScalars* sc, const double* rr_part, int rr_n,
                              bool f32) {
  if (f32)
    return fwd ? launch_halo_b<float, true>(M, P, in, out, rdot, part, sc, rr_part, rr_n)
               : launch_halo_b<float, false>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
  return fwd ? launch_halo_b<double, true>(M, P, in, out, rdot, part, sc, rr_part, rr_n)
             : launch_halo_b<double, false>(M, P, in, out, rdot, part, sc, rr_part, rr_n);
}

}  // namespace dfm
