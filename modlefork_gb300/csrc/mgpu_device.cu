// mgpu_device.cu - sm_103a kernels of the loop-extrusion epoch engine.
//
// One thread block simulates one cell (Simulation::simulate_one_cell, src/libmodle/cpu/
// simulation.cpp:1056-1152): 1 to 16 worker warps by the number of LEFs, and one or two producer
// warps that generate the cell's random numbers.  The cell's state is structure-of-arrays of
// 32-bit words; the host plans which per-LEF arrays fit in the cell's shared memory and places
// the rest in a per-cell global scratch slot (large chromosomes).  The barrier track and its integer
// thresholds are read-only in global memory and shared by every cell of the chromosome.
// The kernel is persistent: each block pulls cell indices from a global work counter.
//
// Why a block per cell.  An epoch is about twenty dependent sweeps over the LEFs or barriers.  With one
// warp per cell a sweep of 2,000 LEFs is 63 dependent rounds of loads, shared memory holds at most a
// dozen such warps per SM, and an instruction issued on 10 % of cycles.  With 16 warps a sweep is
// two or four rounds, the arrays stay in shared memory, and a sweep costs about one barrier.  152 cells
// of 73 Mbp (1,460 LEFs) took 843 ms with a warp per cell, 147-165 now; 24 chromosomes of 40-110 Mbp x 24 cells
// 1.29 s and 0.29; 2 x 1024 cells of 20 Mbp (an instruction-fetch-bound load: several small blocks per SM
// in different steps) 1.2-1.34 s and 0.57-0.63.  Cells of a few dozen LEFs get a warp or two (workers_for): there the
// barriers would cost more than the rounds they save.
//
// Draw order.  Every random number of the reference comes from one sequential
// Xoshiro256++ stream per cell, consumed in a data-dependent order.  The producer warps keep a
// ring of draws in shared memory filled ahead of the workers: each of their P lanes generates
// RNG_S consecutive draws per refill and then advances its private state by (P - 1) * RNG_S steps with
// a GF(2) jump table (the state transition of xoshiro is linear), so the ring always holds the
// exact stream.  A jump costs as much as 50 draws and has a long latency, which is why it runs
// beside the epoch loop instead of inside it.  The workers acquire the ring's fill position
// (rng_ensure) and release the draws they are done with after a barrier (rng_publish); every wait
// is bounded and ends the cell with a status.
//
// Every step of the epoch runs block-parallel with the exact draw order:
//  * steps whose items take one draw each (binding, barrier steps, release, LEF-BAR and LEF-LEF
//    trials) give every item the draw at its offset from a block-wide scan;
//  * items that may take more draws (ziggurat wedges and tails, rejected contact attempts,
//    failed bypass trials in a chain of secondary collisions) are evaluated speculatively at
//    the offsets they would have if every earlier item took its usual count; the offsets are then
//    corrected from the items that deviate, or the workers resume after the first of them;
//  * sequential sweeps are replaced by closed forms: rank_lefs by a merge of the units that moved
//    into the still-sorted order of the others, the adjustment of moves by walks from the units that push a
//    neighbour, the LEF-BAR and primary LEF-LEF sweeps by searches over the ranked positions.
// Where a closed form's precondition does not hold (full ties in the ranking, a chain that
// reaches a chromosome end, unsorted caller input), the step falls back to an exact restatement run
// by one warp or one thread, so results never depend on the fast path.
//
// Floating point.  The file is compiled with --fmad=false so every double multiply and add
// is rounded separately, like the reference's x86-64 build; bernoulli and
// generate_canonical comparisons are exact integer thresholds computed on the host.

#include <cuda_runtime.h>

#include <cstdio>

#include "cppsort_emul.h"
#include "mgpu_internal.h"
#define MGPU_ZIG_TABLE_QUAL __device__ const
#include "ziggurat_tables.h"

namespace mgpu {

#define MGPU_ITER_LIMIT 100000000ull
#define FULL 0xFFFFFFFFu

__device__ __forceinline__ u64 rotl64(u64 x, int k) { return (x << k) | (x >> (64 - k)); }

__device__ __forceinline__ u64 xo_next(u64* s) {
  const u64 result = rotl64(s[0] + s[3], 23) + s[0];
  const u64 t = s[1] << 17;
  s[2] ^= s[0];
  s[3] ^= s[1];
  s[1] ^= s[2];
  s[0] ^= s[3];
  s[2] ^= t;
  s[3] = rotl64(s[3], 45);
  return result;
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__device__ __forceinline__ u32 ln() { return threadIdx.x & 31u; }

__device__ __forceinline__ u64 pos64(u32 v) { return v == UNBOUND ? ~0ull : (u64)v; }

// exclusive prefix sum over the warp; *total receives the sum of all lanes
__device__ __forceinline__ u32 warp_excl_scan(u32 v, u32* total) {
  u32 x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u32 y = __shfl_up_sync(FULL, x, d);
    if ((int)ln() >= d) x += y;
  }
  if (total) *total = __shfl_sync(FULL, x, 31);
  return x - v;
}

// Cell scalars (the same for every thread, kept in shared memory so thread 0's serial code can update
// them; a value thread 0 writes is read by the others only after a barrier).
// Per-launch profile counters (cycles per step and fallback counts), summed over cells.  The two refill
// counters stay 0: the producer warps refill the ring beside the epoch.
enum : u32 {
  PF_BURNIN = 0, PF_BIND, PF_RANK, PF_CONTACTS, PF_MOVES, PF_ADJUST, PF_BARRIERS, PF_BOUNDARIES,
  PF_LEF_BAR, PF_PRIMARY, PF_CORRECT, PF_SECONDARY, PF_FIX, PF_EXTRUDE_RELEASE, PF_TRACE, PF_TOTAL,
  PF_RANK_FALLBACK, PF_ADJUST_FALLBACK, PF_CHAIN_SERIAL, PF_CONTACT_SERIAL, PF_FIX_FALLBACK,
  PF_REFILLS, PF_STALE_REFILLS, PF_EPOCHS, PF_RANK_PDQ, PF_RANK_PASS, PF_RANK_BLOCK, PF_RANK_MERGE,
  PF_RANK_SERIAL, PF_RANK_SPLIT, PF_COUNT = 32
};

struct Scalars {
  u64 rpos;        // next draw to consume (stream index)
  u64 canon[4];    // xoshiro state at the start of the stream
  u32 gpos;        // draws generated so far (modulo 2^32): producers release, workers acquire
  u32 rpub;        // draws the workers are done with (modulo 2^32): thread 0 releases
  u32 stop, pgo;   // end of the cell; the producers' decision to refill
  u32 status;
  u64 epoch, num_burnin_epochs, num_active, num_contacts;
  u32 burnin_completed, flag;
  u64 missed, lef_epochs, sort_fallbacks;
  u64 n5, n3;
  u32 hist_size, hist_head;
  u64 bc0, bc1, bc2;  // broadcast slots for lane 0 results
  u64 nrec;           // model-state records written for this cell
  u64* prof;          // profile counters of the launch (device memory) or null
  u64 mark;           // clock of the last profile mark
};
static_assert(sizeof(Scalars) <= CELL_HEADER_BYTES, "scalars do not fit the cell header");

constexpr u32 MAX_TIES = 64;     // full ties among the units of one ranking that still form the sequence
constexpr u32 TRIAL_WORDS = 65;  // outcomes of up to 2048 draws, and a word read past them

// Scratch of the block-wide steps.
struct BlockTmp {
  u32 cnt[2][32];       // scan2
  u32 tab[16][32];      // gen_moves_dir: per warp and entry lane, leaving position | normals << 16
  u64 wmax[16];         // rank_dir_block
  u32 rem[16], rembase[16];
  u32 nrem, ntie, tie2;
  u32 tierank[MAX_TIES];
  u32 dev[16], okm[16], dus[16];  // sample_contacts
  u32 trial[TRIAL_WORDS];  // secondary_dir_block
  u32 used, qend, nr, nf, released, missed, flag, total;
  u64 sum;
  ulonglong2 zt[128];   // normal ziggurat per layer: {draws below this are accepted, width * 2^60}
  ulonglong2 ln[128];   // logarithm by table: {1 / c * 2^64, ln c * 2^63} for the 128 parts c of [1, 2)
  float2 zy[128];       // and the density at its lower and upper edge: {y_i, y_{i+1} - y_i}
};

// Pointers of one cell (lives in shared memory; identical for every thread).
struct Cell {
  Scalars* sc;
  u64* ring;
  u32 T;      // worker threads (0: no producers, one thread generates its own draws)
  u32 rmask;  // ring capacity - 1
  u32 lim;    // draws the producers always provide beyond the last published position
  u32 off[NARR], bst_off;  // offsets of the arrays in dynamic shared memory (all_smem)
  u32 all_smem;            // every array lives there
  u32 *rev, *fwd, *rr, *fr, *rm, *fm, *rc, *fc, *sr, *sf, *tmp, *bep;
  u32* bst;
  double *hcfx, *havg;
  const DevBarrier* bar;
  const uint2* bpf;  // {pos, flags}
  u32 nb;
  const ulonglong2* jt;
  u32* band;
};

// The cell a block is working on.  Shared variables of the translation unit, so that every function
// addresses them directly: passed by reference they become generic pointers, and each access to a
// per-LEF array then starts with a dependent load of its pointer.
__shared__ Cell g_c;
__shared__ Scalars g_sc;
__shared__ BlockTmp g_bt;
__shared__ __align__(16) KParams g_P;
extern __shared__ __align__(16) char dyn_smem[];  // the PRNG ring, then what the plan placed on chip

// A per-LEF array of 32-bit words: an offset into dynamic shared memory when the plan placed every
// array there (SM), which the compiler turns into shared-memory accesses with 32-bit addresses,
// otherwise a generic pointer (shared memory or the block's global slot).
template <bool SM>
struct Arr;
template <>
struct Arr<true> {
  u32 off;
  template <class I>
  __device__ __forceinline__ u32& operator[](I i) const {
    return *reinterpret_cast<u32*>(dyn_smem + off + 4u * (u32)i);
  }
  __device__ __forceinline__ u64& at64(u32 i) const { return *reinterpret_cast<u64*>(dyn_smem + off + 8u * i); }
  __device__ __forceinline__ Arr operator+(u32 k) const { return Arr{off + 4u * k}; }
};
template <>
struct Arr<false> {
  u32* p;
  template <class I>
  __device__ __forceinline__ u32& operator[](I i) const {
    return p[(u32)i];
  }
  __device__ __forceinline__ u64& at64(u32 i) const { return reinterpret_cast<u64*>(p)[i]; }
  __device__ __forceinline__ Arr operator+(u32 k) const { return Arr{p + k}; }
};

// What a step reads of the cell, loaded once at its start (fields it does not use cost nothing).
template <bool SM>
struct View {
  u32 T, rmask, lim, nb;
  Arr<SM> rev, fwd, rr, fr, rm, fm, rc, fc, sr, sf, tmp, bep, bst;
  const DevBarrier* bar;
  const uint2* bpf;
  u32* band;
  __device__ __forceinline__ View()
      : T(g_c.T), rmask(g_c.rmask), lim(g_c.lim), nb(g_c.nb), bar(g_c.bar), bpf(g_c.bpf), band(g_c.band) {
    if constexpr (SM) {
      rev.off = g_c.off[ARR_REV];
      fwd.off = g_c.off[ARR_FWD];
      rr.off = g_c.off[ARR_RR];
      fr.off = g_c.off[ARR_FR];
      rm.off = g_c.off[ARR_RM];
      fm.off = g_c.off[ARR_FM];
      rc.off = g_c.off[ARR_RC];
      fc.off = g_c.off[ARR_FC];
      sr.off = g_c.off[ARR_SR];
      sf.off = g_c.off[ARR_SF];
      tmp.off = g_c.off[ARR_TMP];
      bep.off = g_c.off[ARR_BEP];
      bst.off = g_c.bst_off;
    } else {
      rev.p = g_c.rev;
      fwd.p = g_c.fwd;
      rr.p = g_c.rr;
      fr.p = g_c.fr;
      rm.p = g_c.rm;
      fm.p = g_c.fm;
      rc.p = g_c.rc;
      fc.p = g_c.fc;
      sr.p = g_c.sr;
      sf.p = g_c.sf;
      tmp.p = g_c.tmp;
      bep.p = g_c.bep;
      bst.p = g_c.bst;
    }
  }
};

// Position and flags of barrier i through the read-only data path (8 bytes per barrier, so the
// sweeps over the barrier track stay in cache).
__device__ __forceinline__ u32 bar_pos(const uint2* bpf, u32 i) { return __ldg(&bpf[i].x); }
__device__ __forceinline__ u32 bar_flags(const uint2* bpf, u32 i) { return __ldg(&bpf[i].y); }
template <class A>
__device__ __forceinline__ bool bar_active(const A& bst, u32 i) {
  return (bst[i >> 5] >> (i & 31)) & 1u;
}

// ---------------------------------------------------------------------------------------
// PRNG ring
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ u32 ld_acquire(const u32* p) {
  u32 v;
  asm volatile("ld.acquire.cta.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(u32* p, u32 v) {
  asm volatile("st.release.cta.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ u64 global_ns() {
  u64 t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier of the cell's worker warps (the producer warps do not take part).
__device__ __forceinline__ void wsync(u32 T) { asm volatile("barrier.sync 1, %0;" ::"r"(T) : "memory"); }
// The same, returning whether any worker thread passed a true predicate.
__device__ __forceinline__ bool wsync_or(u32 T, bool p) {
  u32 r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.red.or.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((u32)p), "r"(T)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void set_status(Cell& c, u32 st) {
  if (c.sc->status == DEV_OK) c.sc->status = st;
}

__device__ __forceinline__ void xo_jump(u64* s, const ulonglong2* jt) {
  u64 n0 = 0, n1 = 0, n2 = 0, n3 = 0;
#pragma unroll 8
  for (int c = 0; c < 64; ++c) {
    const u32 v = (u32)(s[c >> 4] >> ((c & 15) * 4)) & 15u;
    const ulonglong2* e = jt + 2 * (c * 16 + v);
    const ulonglong2 e0 = __ldg(e), e1 = __ldg(e + 1);
    n0 ^= e0.x;
    n1 ^= e0.y;
    n2 ^= e1.x;
    n3 ^= e1.y;
  }
  s[0] = n0;
  s[1] = n1;
  s[2] = n2;
  s[3] = n3;
}

// Body of the producer warps for one cell: whenever a refill fits beside the unconsumed draws,
// each lane writes its next RNG_S draws and jumps over the other lanes' (see the file header).
// Returns when the workers set sc->stop, or after 20 s without a consumer (which then runs into
// its own limit in rng_wait).
__device__ __noinline__ void rng_produce(Cell& c) {
  Scalars* sc = c.sc;
  const u32 pl = threadIdx.x - c.T, P = blockDim.x - c.T;
  const u32 block = P * RNG_S, mask = c.rmask;
  u64 s[4];
  for (int k = 0; k < 4; ++k) s[k] = sc->canon[k];
  for (u32 t = 0; t < pl * RNG_S; ++t) xo_next(s);
  u64* ring = c.ring;
  const ulonglong2* jt = c.jt;
  u32 g = 0;
  for (;;) {
    if (pl == 0) {
      u32 go = 1;
      u64 t0 = 0;
      for (;;) {
        if (ld_acquire(&sc->stop)) {
          go = 0;
          break;
        }
        if (g - ld_acquire(&sc->rpub) <= block) break;
        __nanosleep(100);
        const u64 t = global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > 20000000000ull) {
          go = 0;
          break;
        }
      }
      sc->pgo = go;
    }
    asm volatile("barrier.sync 2, %0;" ::"r"(P) : "memory");
    if (!sc->pgo) return;
    const u32 at = g + pl * RNG_S;
#pragma unroll 4
    for (u32 k = 0; k < (u32)RNG_S; ++k) ring[(at + k) & mask] = xo_next(s);
    g += block;
    asm volatile("barrier.sync 2, %0;" ::"r"(P) : "memory");
    if (pl == 0) st_release(&sc->gpos, g);
    xo_jump(s, jt);  // overlaps with the consumers
  }
}

// Wait for the producers (at most 2 s, then the cell is abandoned with a status).
__device__ __noinline__ void rng_wait(Cell& c, u32 rp, u32 n) {
  const u64 t0 = global_ns();
  while (ld_acquire(&c.sc->gpos) - rp < n) {
    if (*(volatile u32*)&c.sc->status == DEV_ERR_RNG) return;
    __nanosleep(20);
    if (global_ns() - t0 > 2000000000ull) {
      c.sc->status = DEV_ERR_RNG;
      return;
    }
  }
}

// Every worker thread that reads draws [rp, rp + n) calls this first (n <= c.lim minus the draws
// consumed since the last rng_publish).
__device__ __forceinline__ void rng_ensure(u64 rp, u32 n) {
  if (ld_acquire(&g_sc.gpos) - (u32)rp < n) rng_wait(g_c, (u32)rp, n);
}

// Thread 0, after a wsync that follows every read of the draws before rp: record the position
// and hand the ring space back to the producers.
__device__ __forceinline__ void rng_publish(u64 rp) {
  if (threadIdx.x == 0) {
    g_sc.rpos = rp;
    st_release(&g_sc.rpub, (u32)rp);
  }
}

__device__ __forceinline__ u64 ring_at(u32 rmask, u64 k) {
  return *reinterpret_cast<const u64*>(dyn_smem + 8u * ((u32)k & rmask));
}

// Thread 0 only (the other workers wait at a barrier): next draw of the stream.  Without
// producer warps (c.T == 0, the sampler probe) the thread generates it itself.
__device__ __noinline__ u64 rng_serial(Cell& c) {
  Scalars* sc = c.sc;
  if ((u32)sc->rpos == ld_acquire(&sc->gpos)) {
    if (c.T == 0) {
      c.ring[sc->gpos & c.rmask] = xo_next(sc->canon);
      sc->gpos++;
    } else {
      rng_wait(c, (u32)sc->rpos, 1);
    }
  }
  const u64 v = c.ring[(u32)sc->rpos & c.rmask];
  sc->rpos++;
  if (c.T) st_release(&sc->rpub, (u32)sc->rpos);
  return v;
}

// Profile mark (all workers call it): adds the cycles since the previous mark to step k.  Out of line,
// as everything the epoch loop does in many places: with several cells on an SM, each in another step,
// the loop's code competes for the instruction caches.
__device__ __noinline__ void prof_mark(u32 k) {
  if (threadIdx.x != 0 || !g_sc.prof) return;
  const u64 t = clock64();
  if (k < PF_COUNT) {
    atomicAdd((unsigned long long*)&g_sc.prof[k], (unsigned long long)(t - g_sc.mark));
    atomicAdd((unsigned long long*)&g_sc.prof[PF_TOTAL], (unsigned long long)(t - g_sc.mark));
  }
  g_sc.mark = t;
}
__device__ __noinline__ void prof_add(u32 k, u64 v) {
  if (threadIdx.x == 0 && g_sc.prof) atomicAdd((unsigned long long*)&g_sc.prof[k], (unsigned long long)v);
}

// ---------------------------------------------------------------------------------------
// Serial distributions (thread 0).  Boost.Random 1.79 semantics, see the oracle for the
// line-by-line restatement; thresholds replace bernoulli / canonical comparisons.
// ---------------------------------------------------------------------------------------

__device__ __noinline__ u64 s_uniform_int(Cell& c, u64 a, u64 b) {
  const u64 range = b - a;
  if (range == 0) return a;
  if (range == ~0ull) return rng_serial(c) + a;
  u64 bucket = ~0ull / (range + 1);
  if (~0ull % (range + 1) == range) ++bucket;
#pragma unroll 1
  for (u64 it = 0; it < 1000; ++it) {
    const u64 r = rng_serial(c) / bucket;
    if (r <= range) return a + r;
  }
  set_status(c, DEV_ERR_ITER_LIMIT);
  return a;
}

__device__ __forceinline__ bool s_trial(Cell& c, const Trial& t) {
  if (t.always) return true;
  if (!t.draws) return false;
  return rng_serial(c) <= t.thr;
}

__device__ __forceinline__ double u01_of(u64 u) { return (double)u * (1.0 / 18446744073709551616.0); }

__device__ __noinline__ double s_uniform01(Cell& c) {
#pragma unroll 1
  for (int it = 0; it < 1000; ++it) {
    const double r = u01_of(rng_serial(c));
    if (r < 1.0) return r;
  }
  set_status(c, DEV_ERR_ITER_LIMIT);
  return 0.0;
}

__device__ __forceinline__ double canonical_of(u64 u) {
  double r = (double)u / 18446744073709551616.0;
  if (r == 1.0) r -= 1.1102230246251565e-16;  // DBL_EPSILON / 2
  return r;
}

// generate_int_float_pair<double, 8>
__device__ __forceinline__ double ifp_fraction(u64 u) {
  u &= ~(1ull << 11);
  return (double)(u >> 8) * (1.0 / 72057594037927936.0);
}

// Draw sources of the samplers below.  SerialSrc is thread 0's view of the cell's stream; RingSrc
// is one lane's view of the pre-generated ring starting at a given stream position, which
// reports exhaustion instead of generating.
struct SerialSrc {
  Cell& c;
  u32 n;
  __device__ bool next(u64& u) {
    u = rng_serial(c);
    ++n;
    return true;
  }
};

struct RingSrc {
  u32 mask, pos, end;
  u32 n;
  __device__ bool next(u64& u) {
    if (pos == end) return false;
    u = *reinterpret_cast<const u64*>(dyn_smem + 8u * (pos & mask));
    ++pos;
    ++n;
    return true;
  }
};

// Sampler results: 0 = value produced, 1 = the source ran dry, 2 = iteration limit.
enum { SMP_OK = 0, SMP_DRY = 1, SMP_LIMIT = 2 };

// y < exp(a) for a <= 0, decided exactly: a float estimate of exp(a) settles it unless y lies
// within 1e-5 (relative) of the estimate, whose error is below 1e-6; only then is the double
// exp evaluated.
__device__ __forceinline__ bool below_exp(double y, double a) {
  const float ef = expf((float)a);
  const double d = y - (double)ef;
  if (fabs(d) > 1e-5 * (double)ef) return d < 0;
  return y < exp(a);
}

// uniform_01<double> on one draw per attempt (values equal to 1 are rejected)
template <class Src>
__device__ int uniform01_t(Src& g, double& r) {
#pragma unroll 1
  for (int it = 0; it < 1000; ++it) {
    u64 u;
    if (!g.next(u)) return SMP_DRY;
    r = u01_of(u);
    if (r < 1.0) return SMP_OK;
  }
  return SMP_LIMIT;
}

// unit_exponential_distribution: 256-layer ziggurat with the shift-on-layer-0 tail
template <class Src>
__device__ int unit_exponential_t(Src& g, double& out) {
  double shift = 0;
#pragma unroll 1
  for (int it = 0; it < 100000; ++it) {
    u64 u;
    if (!g.next(u)) return SMP_DRY;
    const int i = (int)(u & 0xFF);
    const double x = ifp_fraction(u) * mgpu_zig_exp_x[i];
    if (x < mgpu_zig_exp_x[i + 1]) {
      out = shift + x;
      return SMP_OK;
    }
    if (i == 0) {
      shift += mgpu_zig_exp_x[1];
    } else {
      double y01;
      const int r = uniform01_t(g, y01);
      if (r) return r;
      const double y = mgpu_zig_exp_y[i] + y01 * (mgpu_zig_exp_y[i + 1] - mgpu_zig_exp_y[i]);
      if (below_exp(y, -x)) {
        out = x + shift;
        return SMP_OK;
      }
    }
  }
  return SMP_LIMIT;
}

// tail of the normal ziggurat (Marsaglia's method with two exponentials)
template <class Src>
__device__ int normal_tail_t(Src& g, double& out) {
  const double tail_start = mgpu_zig_normal_x[1];
#pragma unroll 1
  for (int it = 0; it < 100000; ++it) {
    double e1, e2;
    int r = unit_exponential_t(g, e1);
    if (r) return r;
    r = unit_exponential_t(g, e2);
    if (r) return r;
    const double x = e1 / tail_start;
    const double y = e2 / 1.0;
    if (2 * y > x * x) {
      out = x + tail_start;
      return SMP_OK;
    }
  }
  return SMP_LIMIT;
}

// unit_normal_distribution: 128-layer ziggurat, sign from bit 0 of the layer byte
template <class Src>
__device__ int unit_normal_t(Src& g, double& out) {
#pragma unroll 1
  for (int it = 0; it < 100000; ++it) {
    u64 u;
    if (!g.next(u)) return SMP_DRY;
    const int ii = (int)(u & 0xFF);
    const int sign = (ii & 1) * 2 - 1;
    const int i = ii >> 1;
    const double x = ifp_fraction(u) * mgpu_zig_normal_x[i];
    if (x < mgpu_zig_normal_x[i + 1]) {
      out = x * sign;
      return SMP_OK;
    }
    if (i == 0) {
      double t;
      const int r = normal_tail_t(g, t);
      if (r) return r;
      out = t * sign;
      return SMP_OK;
    }
    double y01;
    const int r = uniform01_t(g, y01);
    if (r) return r;
    const double y = mgpu_zig_normal_y[i] + y01 * (mgpu_zig_normal_y[i + 1] - mgpu_zig_normal_y[i]);
    if (below_exp(y, -(x * x / 2))) {
      out = x * sign;
      return SMP_OK;
    }
  }
  return SMP_LIMIT;
}

__device__ __noinline__ double s_unit_exponential(Cell& c) {
  SerialSrc g{c, 0};
  double v = 0.0;
  if (unit_exponential_t(g, v) != SMP_OK) set_status(c, DEV_ERR_ITER_LIMIT);
  return v;
}

__device__ __noinline__ double s_unit_normal(Cell& c) {
  SerialSrc g{c, 0};
  double v = 0.0;
  if (unit_normal_t(g, v) != SMP_OK) set_status(c, DEV_ERR_ITER_LIMIT);
  return v;
}

__device__ const double kLogFactorial[10] = {0.0,
                                             0.0,
                                             0.69314718055994529,
                                             1.7917594692280550,
                                             3.1780538303479458,
                                             4.7874917427820458,
                                             6.5792512120101012,
                                             8.5251613610654147,
                                             10.604602902745251,
                                             12.801827480081469};

__device__ __noinline__ u64 s_poisson(Cell& c, const KParams& P) {
  const double mean = P.pois_mean;
  if (mean < 10) {
    double p = P.pois_exp_mean;
    u64 x = 0;
    double u = s_uniform01(c);
#pragma unroll 1
    while (u > p) {
      u = u - p;
      ++x;
      p = mean * p / (double)x;
      if (x > MGPU_ITER_LIMIT) {
        set_status(c, DEV_ERR_ITER_LIMIT);
        break;
      }
    }
    return x;
  }
  const double smu = P.pois_smu, b = P.pois_b, a = P.pois_a, inv_alpha = P.pois_inv_alpha,
               v_r = P.pois_v_r;
#pragma unroll 1
  for (int it = 0; it < 100000; ++it) {
    double u;
    double v = s_uniform01(c);
    if (v <= 0.86 * v_r) {
      u = v / v_r - 0.43;
      return (u64)floor((2 * a / (0.5 - fabs(u)) + b) * u + mean + 0.445);
    }
    if (v >= v_r) {
      u = s_uniform01(c) - 0.5;
    } else {
      u = v / v_r - 0.93;
      u = ((u < 0) ? -0.5 : 0.5) - u;
      v = s_uniform01(c) * v_r;
    }
    const double us = 0.5 - fabs(u);
    if (us < 0.013 && v > us) continue;
    const double k = floor((2 * a / us + b) * u + mean + 0.43);
    v = v * inv_alpha / (a / (us * us) + b);
    const double log_sqrt_2pi = 0.91893853320467267;
    if (k >= 10) {
      if (log(v * smu) <= (k + 0.5) * log(mean / k) - mean - log_sqrt_2pi + k -
                              (1 / 12. - (1 / 360. - 1 / (1260. * k * k)) / (k * k)) / k) {
        return (u64)k;
      }
    } else if (k >= 0) {
      if (log(v) <= k * log(mean) - mean - kLogFactorial[(int)k]) return (u64)k;
    }
  }
  set_status(c, DEV_ERR_ITER_LIMIT);
  return 0;
}

__device__ const double kBinomialFc[10] = {0.08106146679532726, 0.04134069595540929,
                                           0.02767792568499834, 0.02079067210376509,
                                           0.01664469118982119, 0.01387612882307075,
                                           0.01189670994589177, 0.01041126526197209,
                                           0.009255462182712733, 0.008330563433362871};

__device__ double binomial_fc(i64 k) {
  if (k < 10) return kBinomialFc[k];
  const double ikp1 = 1.0 / (double)(k + 1);
  return (1.0 / 12 - (1.0 / 360 - (1.0 / 1260) * (ikp1 * ikp1)) * (ikp1 * ikp1)) * ikp1;
}

__device__ __noinline__ i64 s_binomial(Cell& c, const KParams& P, i64 t_, double p_) {
  const double p = (0.5 < p_) ? (1 - p_) : p_;
  const i64 t = t_;
  const i64 m = (i64)((t + 1) * p);
  if (m < 11) {
    const double q_n = ((u64)t == P.spe) ? P.bin_q_n : pow((1 - p), (double)t);
    const double pp = (0.5 < p_) ? (1 - p_) : p_;
    const double q = 1 - pp;
    const double s = pp / q;
    const double a = (t + 1) * s;
    double r = q_n;
    double u = s_uniform01(c);
    i64 x = 0;
#pragma unroll 1
    while (u > r) {
      u = u - r;
      ++x;
      const double r1 = ((a / x) - s) * r;
      if (r1 < 2.220446049250313e-16 && r1 < r) break;
      r = r1;
    }
    return (0.5 < p_) ? t_ - x : x;
  }
  const double r = p / (1 - p);
  const double nr = (t + 1) * r;
  const double npq = t * p * (1 - p);
  const double sqrt_npq = sqrt(npq);
  const double b = 1.15 + 2.53 * sqrt_npq;
  const double a = -0.0873 + 0.0248 * b + 0.01 * p;
  const double cc = t * p + 0.5;
  const double alpha = (2.83 + 5.1 / b) * sqrt_npq;
  const double v_r = 0.92 - 4.2 / b;
  const double u_rv_r = 0.86 * v_r;
  i64 res = 0;
  bool done = false;
#pragma unroll 1
  for (int it = 0; it < 100000 && !done; ++it) {
    double u;
    double v = s_uniform01(c);
    if (v <= u_rv_r) {
      u = v / v_r - 0.43;
      res = (i64)floor((2 * a / (0.5 - fabs(u)) + b) * u + cc);
      done = true;
      break;
    }
    if (v >= v_r) {
      u = s_uniform01(c) - 0.5;
    } else {
      u = v / v_r - 0.93;
      u = ((u < 0) ? -0.5 : 0.5) - u;
      v = s_uniform01(c) * v_r;
    }
    const double us = 0.5 - fabs(u);
    const i64 k = (i64)floor((2 * a / us + b) * u + cc);
    if (k < 0 || k > t) continue;
    v = v * alpha / (a / (us * us) + b);
    const double km = fabs((double)(k - m));
    if (km <= 15) {
      double f = 1;
      if (m < k) {
        i64 i = m;
        do {
          ++i;
          f = f * (nr / i - r);
        } while (i != k);
      } else if (m > k) {
        i64 i = k;
        do {
          ++i;
          v = v * (nr / i - r);
        } while (i != m);
      }
      if (v <= f) {
        res = k;
        done = true;
      }
      continue;
    }
    v = log(v);
    const double rho = (km / npq) * (((km / 3. + 0.625) * km + 1. / 6) / npq + 0.5);
    const double tt = -km * km / (2 * npq);
    if (v < tt - rho) {
      res = k;
      done = true;
      continue;
    }
    if (v > tt + rho) continue;
    const i64 nm = t - m + 1;
    const double h = (m + 0.5) * log((m + 1) / (r * nm)) + binomial_fc(m) + binomial_fc(t - m);
    const i64 nk = t - k + 1;
    if (v <= h + (t + 1) * log((double)nm / nk) + (k + 0.5) * log(nk * r / (k + 1)) -
                 binomial_fc(k) - binomial_fc(t - k)) {
      res = k;
      done = true;
    }
  }
  if (!done) set_status(c, DEV_ERR_ITER_LIMIT);
  return (0.5 < p_) ? t_ - res : res;
}

__device__ __noinline__ double s_gev(Cell& c, const KParams& P) {
  const double u = canonical_of(rng_serial(c));
  if (P.gev_xi == 0.0) return (P.gev_mu - P.gev_sigma) * log(-log(u));
  return P.gev_mu + (P.gev_sigma * (1.0 - pow(-log(u), P.gev_xi))) / P.gev_xi;
}


// ---------------------------------------------------------------------------------------
// Serial restatements (thread 0): the exact fallbacks of the warp-parallel steps.  They and the
// serial samplers are kept out of line: the epoch loop's code is large enough that, with eight
// or more cells per SM, instruction fetch stalls grow with its size.
// ---------------------------------------------------------------------------------------

// rank_lefs for one direction (simulation.cpp:402-487): split_sort (or pdq_sort at epoch 0)
// by position, then runs of equal positions insertion-sorted by binding epoch (ascending
// for rev units, descending for fwd units).
__device__ __noinline__ void rank_dir_serial(Cell& c, u32 dir, u32 n, bool partially_sorted) {
  u32* R = dir ? c.fr : c.rr;
  const u32* pos = dir ? c.fwd : c.rev;
  const KeyCmp cmp{pos};
  if (partially_sorted) {
    split_sort(R, n, c.tmp, cmp);
  } else {
    pdq_sort(R, 0, n, cmp);
  }
#pragma unroll 1
  for (u32 i = 1; i < n; ++i) {
    if (pos[R[i - 1]] == pos[R[i]]) {
      const u32 begin = i - 1;
#pragma unroll 1
      for (; i < n; ++i) {
        if (pos[R[i - 1]] != pos[R[i]]) break;
      }
      if (dir) {
        ins_sort(R, begin, i, KeyCmpRev{c.bep});
      } else {
        ins_sort(R, begin, i, KeyCmp{c.bep});
      }
    }
  }
}

// adjust_moves_of_consecutive_extr_units (simulation.cpp:343-399), one direction; lane 0
__device__ __noinline__ void adjust_dir_serial(Cell& c, const KParams& P, u32 dir, u32 n) {
  if (n == 0) return;
  const u64 start = P.start, end = P.end;
  if (dir == 0) {
#pragma unroll 1
    for (u32 i = n - 1; i > 0; --i) {
      const u32 i1 = c.rr[i - 1], i2 = c.rr[i];
      if (c.bep[i1] != UNBOUND && c.bep[i2] != UNBOUND) {
        const u64 r1 = pos64(c.rev[i1]), r2 = pos64(c.rev[i2]);
        const u64 m1 = c.rm[i1], m2 = c.rm[i2];
        if (r1 <= start + m1 || r2 <= start + m2) continue;
        const u64 pos1 = r1 - m1, pos2 = r2 - m2;
        if (pos2 <= pos1) c.rm[i1] = (u32)(m1 + (pos1 - pos2) + 1);
      }
    }
  } else {
#pragma unroll 1
    for (u32 i = 1; i < n; ++i) {
      const u32 i1 = c.fr[i - 1], i2 = c.fr[i];
      if (c.bep[i1] != UNBOUND && c.bep[i2] != UNBOUND) {
        const u64 f1 = pos64(c.fwd[i1]), f2 = pos64(c.fwd[i2]);
        const u64 m1 = c.fm[i1], m2 = c.fm[i2];
        if (f1 + m1 > end - 1 || f2 + m2 > end - 1) continue;
        const u64 pos1 = f1 + m1, pos2 = f2 + m2;
        if (pos1 >= pos2) c.fm[i2] = (u32)(m2 + (pos1 - pos2) + 1);
      }
    }
  }
}

// compute_lef_lef_collision_pos (simulation.cpp:514-542).  The reference rounds the double
// fwd_move * (delta / rel); for moves that add up to less than 46340 bp its error is below 2^-35
// while a value that is not exactly halfway between two integers is at least 1 / (2 rel) > 2^-17
// away from one, so the rounded quotient of 32-bit integers is the same number.  Only an exact
// half, whose side the doubles' rounding decides, and longer moves are evaluated in doubles (a
// division takes some 30 instructions on a pipe that runs at 1/64 of the FP32 rate).
__device__ __forceinline__ void lef_lef_collision_pos(u64 rev_pos, u64 fwd_pos, u64 rev_move,
                                                      u64 fwd_move, u64& p_rev, u64& p_fwd) {
  const u64 rel = rev_move + fwd_move, delta = rev_pos - fwd_pos;
  u64 off = 0;
  bool exact = true;
  if (rel - 1 < 46339 && delta <= rel) {
    const u32 num = 2 * (u32)fwd_move * (u32)delta + (u32)rel, den = 2 * (u32)rel;  // below 2^32
    const u32 q = num / den;
    exact = q * den == num;
    off = q;
  }
  if (exact) {
    const double t = (double)delta / (double)rel;
    off = (u64)round((double)fwd_move * t);
  }
  const u64 cp = fwd_pos + off;
  if (cp == fwd_pos) {
    p_rev = cp + 1;
    p_fwd = cp;
  } else {
    p_rev = cp;
    p_fwd = cp - 1;
  }
}

// detect_units_at_chrom_boundaries (simulation_detect_collisions.cpp:30-125); lane 0.  The
// loops stop at the first unit that is neither at nor about to reach a chromosome end.
template <class C>
__device__ void detect_boundaries_serial(const C& c, const KParams& P, u32 n, u64& n5, u64& n3) {
  n5 = 0;
  n3 = 0;
  const u64 start = P.start, end = P.end;
  const u64 first_fwd_pos = pos64(c.fwd[c.fr[0]]);
  u32 last_rev = UNBOUND;
#pragma unroll 1
  for (u32 k = n; k > 0; --k) {
    if (c.bep[c.rr[k - 1]] != UNBOUND) {
      last_rev = c.rr[k - 1];
      break;
    }
  }
  if (last_rev == UNBOUND) {
    set_status(g_c, DEV_ERR_BAD_STATE);
    last_rev = c.rr[0];
  }
  const u64 last_rev_pos = pos64(c.rev[last_rev]);
#pragma unroll 1
  for (u32 i = 0; i < n; ++i) {
    const u32 idx = c.rr[i];
    const u64 pos = pos64(c.rev[idx]);
    const u64 mv = c.rm[idx];
    if (pos == start) {
      ++n5;
      c.rc[idx] = cw_make(5, EV_COLLISION | EV_CHROM_BOUNDARY);
    } else if (pos > first_fwd_pos) {
      break;
    } else if (pos - mv == start) {
      c.rc[idx] = cw_make(5, EV_COLLISION | EV_CHROM_BOUNDARY);
      ++n5;
      break;
    }
  }
#pragma unroll 1
  for (u32 i = n - 1; i > 0; --i) {
    const u32 idx = c.fr[i];
    const u64 pos = pos64(c.fwd[idx]);
    const u64 mv = c.fm[idx];
    if (c.bep[idx] == UNBOUND) {
      ++n3;
      continue;
    }
    if (pos == end - 1) {
      ++n3;
      c.fc[idx] = cw_make(3, EV_COLLISION | EV_CHROM_BOUNDARY);
    } else if (pos < last_rev_pos) {
      break;
    } else if (pos + mv == end - 1) {
      c.fc[idx] = cw_make(3, EV_COLLISION | EV_CHROM_BOUNDARY);
      ++n3;
      break;
    }
  }
}


// detect_lef_bar_collisions (simulation_detect_collisions.cpp:128-252); lane 0
__device__ __noinline__ void detect_lef_bar_serial(Cell& c, const KParams& P, u32 n, u64 n5, u64 n3) {
  u64 j = min(n5, n5 - 1);
  u32 unit_idx = c.rr[j];
  u64 unit_pos = pos64(c.rev[unit_idx]);
  bool rev_done = false;
#pragma unroll 1
  for (u32 i = 0; i < c.nb && !rev_done; ++i) {
    if (!bar_active(c.bst, i)) continue;
    const u32 dir = bar_flags(c.bpf, i) & BF_DIR_MASK;
    const Trial& tr = P.lef_bar[dir == MGPU_DIR_REV ? 0 : 1];
    const u64 bpos = bar_pos(c.bpf, i);
#pragma unroll 1
    while (unit_pos <= bpos) {
      if (++j == n) {
        rev_done = true;
        break;
      }
      unit_idx = c.rr[j];
      unit_pos = pos64(c.rev[unit_idx]);
    }
    if (rev_done) break;
    if (c.bep[unit_idx] != UNBOUND) {
      const u64 delta = unit_pos - bpos;
      if (delta > 0 && delta <= c.rm[unit_idx] && s_trial(c, tr)) {
        c.rc[unit_idx] = cw_make(i, EV_COLLISION | EV_LEF_BAR);
      }
    }
  }
  j = n - min(n3, n3 - 1);
  unit_idx = c.fr[--j];
  unit_pos = pos64(c.fwd[unit_idx]);
#pragma unroll 1
  for (u64 i = (u64)c.nb - 1; i != ~0ull; --i) {
    if (!bar_active(c.bst, (u32)i)) continue;
    const u32 dir = bar_flags(c.bpf, i) & BF_DIR_MASK;
    const Trial& tr = P.lef_bar[dir == MGPU_DIR_FWD ? 0 : 1];
    const u64 bpos = bar_pos(c.bpf, i);
#pragma unroll 1
    while (unit_pos >= bpos) {
      if (--j == ~0ull) return;
      unit_idx = c.fr[j];
      unit_pos = pos64(c.fwd[unit_idx]);
    }
    if (c.bep[unit_idx] != UNBOUND) {
      const u64 delta = bpos - unit_pos;
      if (delta > 0 && delta <= c.fm[unit_idx] && s_trial(c, tr)) {
        c.fc[unit_idx] = cw_make((u32)i, EV_COLLISION | EV_LEF_BAR);
      }
    }
  }
}

template <class C>
__device__ __forceinline__ u64 barrier_pos_checked(const C& c, u32 idx) {
  if (idx >= c.nb) {
    set_status(g_c, DEV_ERR_BAD_STATE);
    return 0;
  }
  return bar_pos(c.bpf, idx);
}

// The collision words of one tested primary pair (simulation_detect_collisions.cpp:344-399).
template <class C>
__device__ __forceinline__ void primary_pair_update(const C& c, u32 rev_idx, u32 fwd_idx, u64 rev_pos,
                                                    u64 fwd_pos, u64 rmv, u64 fmv) {
  u64 cpr, cpf;
  lef_lef_collision_pos(rev_pos, fwd_pos, rmv, fmv, cpr, cpf);
  const u32 rcol = c.rc[rev_idx], fcol = c.fc[fwd_idx];
  if (!cw_occurred(rcol) && !cw_occurred(fcol)) {
    c.rc[rev_idx] = cw_make(fwd_idx, EV_COLLISION | EV_PRIMARY);
    c.fc[fwd_idx] = cw_make(rev_idx, EV_COLLISION | EV_PRIMARY);
  } else if (cw_occurred(rcol) && !cw_occurred(fcol)) {
    const u64 bpos = barrier_pos_checked(c, cw_idx(rcol));
    if (cpf > bpos) {
      c.rc[rev_idx] = cw_make(fwd_idx, EV_COLLISION | EV_PRIMARY);
      c.fc[fwd_idx] = cw_make(rev_idx, EV_COLLISION | EV_PRIMARY);
    } else {
      c.fc[fwd_idx] = cw_make(rev_idx, EV_COLLISION | EV_PRIMARY);
    }
  } else if (!cw_occurred(rcol) && cw_occurred(fcol)) {
    const u64 bpos = barrier_pos_checked(c, cw_idx(fcol));
    c.rc[rev_idx] = cw_make(fwd_idx, EV_COLLISION | EV_PRIMARY);
    if (cpr < bpos) c.fc[fwd_idx] = cw_make(rev_idx, EV_COLLISION | EV_PRIMARY);
  }
}

// detect_primary_lef_lef_collisions (simulation_detect_collisions.cpp:255-401); lane 0
__device__ __noinline__ void detect_primary_serial(Cell& c, const KParams& P, u32 n, u64 n5, u64 n3) {
  if (n5 == n || n3 == n) return;
  u64 i1 = 0, j1 = n5;
  const u64 i2 = n - min(n3, n3 - 1);
  const u64 j2 = n;
#pragma unroll 1
  for (u64 it = 0; it < 4ull * n + 16; ++it) {
    u32 rev_idx = c.rr[j1];
    u64 rev_pos = pos64(c.rev[rev_idx]);
    u32 fwd_idx = c.fr[i1];
    u64 fwd_pos = pos64(c.fwd[fwd_idx]);
#pragma unroll 1
    while (rev_pos <= fwd_pos) {
      if (++j1 == j2) return;
      rev_idx = c.rr[j1];
      rev_pos = pos64(c.rev[rev_idx]);
    }
#pragma unroll 1
    while (fwd_pos < rev_pos) {
      if (++i1 == i2) return;
      fwd_idx = c.fr[i1];
      fwd_pos = pos64(c.fwd[fwd_idx]);
    }
    fwd_idx = c.fr[min(i1, i1 - 1)];
    fwd_pos = pos64(c.fwd[fwd_idx]);
    const u64 delta = rev_pos - fwd_pos;
    const u64 rmv = c.rm[rev_idx], fmv = c.fm[fwd_idx];
    if (delta > 0 && delta < rmv + fmv && s_trial(c, P.lef_lef)) {
      primary_pair_update(c, rev_idx, fwd_idx, rev_pos, fwd_pos, rmv, fmv);
    }
  }
  set_status(c, DEV_ERR_ITER_LIMIT);
}

// process_secondary_lef_lef_collisions (simulation_detect_collisions.cpp:404-518); lane 0
__device__ __noinline__ void process_secondary_serial(Cell& c, const KParams& P, u32 n, u64 n5, u64 n3) {
#pragma unroll 1
  for (u64 i = max((u64)1, n5); i < n; ++i) {
    const u32 idx1 = c.rr[i - 1];
    if (!cw_occurred(c.rc[idx1])) continue;
    const u32 idx2 = c.rr[i];
    if (cw_occurred(c.rc[idx2])) continue;
    const u64 pos1 = pos64(c.rev[idx1]), pos2 = pos64(c.rev[idx2]);
    const u64 move1 = c.rm[idx1], move2 = c.rm[idx2];
    if (pos2 - move2 <= pos1 - move1) {
      if (s_trial(c, P.lef_lef)) {
        c.rc[idx2] = cw_make(idx1, EV_COLLISION | EV_SECONDARY);
        const u64 mv = pos2 - (pos1 - move1);
        c.rm[idx2] = (u32)min(mv, mv - 1);
      } else {
        c.rc[idx2] = cw_make(idx1, EV_SECONDARY);
      }
    }
  }
  u64 i = n - min(n3, n3 - 1) - 1;
#pragma unroll 1
  for (; i > 0 && i != ~0ull; --i) {
    const u32 idx2 = c.fr[i];
    if (!cw_occurred(c.fc[idx2])) continue;
    const u32 idx1 = c.fr[i - 1];
    if (cw_occurred(c.fc[idx1])) continue;
    const u64 pos1 = pos64(c.fwd[idx1]), pos2 = pos64(c.fwd[idx2]);
    const u64 move1 = c.fm[idx1], move2 = c.fm[idx2];
    if (pos1 + move1 >= pos2 + move2) {
      if (s_trial(c, P.lef_lef)) {
        c.fc[idx1] = cw_make(idx2, EV_COLLISION | EV_SECONDARY);
        const u64 mv = (pos2 + move2) - pos1;
        c.fm[idx1] = (u32)min(mv, mv - 1);
      } else {
        c.fc[idx1] = cw_make(idx2, EV_SECONDARY);
      }
    }
  }
}

// One rev candidate of fix_secondary_lef_lef_collisions (simulation_detect_collisions.cpp:556-605).
template <class C>
__device__ __forceinline__ void fix_rev_at(const C& c, u64 start, u64 i) {
  const u32 idx2 = c.rr[i];
  const u32 idx1 = c.rr[i - 1];
  const u64 pos1 = pos64(c.rev[idx1]) - c.rm[idx1];
  const u64 r2 = pos64(c.rev[idx2]);
  c.rm[idx2] = (r2 > pos1 + 1) ? (u32)(r2 - (pos1 + 1)) : 0u;
  c.rc[idx2] = cw_make(idx1, EV_COLLISION | EV_SECONDARY);
  const u64 p1 = pos64(c.rev[idx1]), p2 = r2;
  c.rev[idx1] = (u32)min(pos64(c.fwd[idx1]), p2);
  c.rev[idx2] = (u32)min(pos64(c.fwd[idx2]), p1);
  u32 t = c.rc[idx1];
  c.rc[idx1] = c.rc[idx2];
  c.rc[idx2] = t;
  t = c.rm[idx1];
  c.rm[idx1] = c.rm[idx2];
  c.rm[idx2] = t;
  c.rr[i - 1] = idx2;
  c.rr[i] = idx1;
  c.rm[idx2] = (u32)min(pos64(c.rev[idx2]) - start, (u64)c.rm[idx2]);
  c.rm[idx1] = (u32)min(pos64(c.rev[idx1]) - start, (u64)c.rm[idx1]);
}

// One fwd candidate (simulation_detect_collisions.cpp:608-646).
template <class C>
__device__ __forceinline__ void fix_fwd_at(const C& c, u64 end, u64 i) {
  const u32 idx1 = c.fr[i];
  const u32 idx2 = c.fr[i + 1];
  const u64 f1 = pos64(c.fwd[idx1]);
  const u64 pos2 = pos64(c.fwd[idx2]) + c.fm[idx2];
  c.fm[idx1] = (pos2 > f1 + 1) ? (u32)(pos2 - (f1 + 1)) : 0u;
  c.fc[idx1] = cw_make(idx2, EV_COLLISION | EV_SECONDARY);
  const u64 p1 = f1, p2 = pos64(c.fwd[idx2]);
  c.fwd[idx1] = (u32)max(pos64(c.rev[idx1]), p2);
  c.fwd[idx2] = (u32)max(pos64(c.rev[idx2]), p1);
  u32 t = c.fc[idx1];
  c.fc[idx1] = c.fc[idx2];
  c.fc[idx2] = t;
  t = c.fm[idx1];
  c.fm[idx1] = c.fm[idx2];
  c.fm[idx2] = t;
  c.fr[i] = idx2;
  c.fr[i + 1] = idx1;
  c.fm[idx2] = (u32)min(end - 1 - pos64(c.fwd[idx2]), (u64)c.fm[idx2]);
  c.fm[idx1] = (u32)min(end - 1 - pos64(c.fwd[idx1]), (u64)c.fm[idx1]);
}

// fix_secondary_lef_lef_collisions (simulation_detect_collisions.cpp:520-647); lane 0
__device__ __noinline__ void fix_secondary_serial(Cell& c, const KParams& P, u32 n, u64 n5, u64 n3) {
  const u64 num_active_fwd = n - min(n3, n3 - 1);
#pragma unroll 1
  for (u64 i = max((u64)1, n5); i < n; ++i) {
    if (cw_avoided_as(c.rc[c.rr[i]], EV_SECONDARY)) fix_rev_at(c, P.start, i);
  }
#pragma unroll 1
  for (u64 i = 0; i + 1 < num_active_fwd; ++i) {
    if (cw_avoided_as(c.fc[c.fr[i]], EV_SECONDARY)) fix_fwd_at(c, P.end, i);
  }
}


// ---------------------------------------------------------------------------------------
// Block-parallel steps (the cell's worker threads, uniform control flow).  Each step takes the
// stream position rp and returns the position after it; every step ends with a wsync after which
// the state it wrote is visible to all workers.
// ---------------------------------------------------------------------------------------

// Exclusive counts of two flags per thread over the window's items in order (item h of thread t is
// item h * T + t): where this thread's flags fall, and how many there are.  One wsync; successive
// calls alternate buf.
struct Scan2 {
  u32 off0, off1, total;
};
template <bool SM>
__device__ __forceinline__ Scan2 scan2(u32 buf, bool f0, bool f1) {
  const View<SM> c;
  const unsigned m0 = __ballot_sync(FULL, f0), m1 = __ballot_sync(FULL, f1);
  const u32 w = threadIdx.x >> 5, l = ln();
  u32* cnt = g_bt.cnt[buf];
  if (l == 0) {
    cnt[w] = __popc(m0);
    cnt[16 + w] = __popc(m1);
  }
  wsync(c.T);
  const u32 v = (l & 15u) < (c.T >> 5) ? cnt[l] : 0u;
  const u32 before = (l & 15u) < w ? v : 0u;
  const u32 b0 = __reduce_add_sync(FULL, l < 16 ? before : 0u);
  const u32 b1 = __reduce_add_sync(FULL, l < 16 ? v : before);
  Scan2 r;
  r.total = __reduce_add_sync(FULL, v);
  r.off0 = b0 + __popc(m0 & lanemask_lt());
  r.off1 = b1 + __popc(m1 & lanemask_lt());
  return r;
}

// floor(a / b), and the bucket width of a uniform_int over [0, range]: a 64-bit division is about 70
// instructions, so the steps share one copy.
__device__ __noinline__ u64 div64(u64 a, u64 b) { return a / b; }
__device__ __forceinline__ u64 bucket_of(u64 range) {
  const u64 q = div64(~0ull, range + 1);
  return ~0ull - q * (range + 1) == range ? q + 1 : q;
}

// The same for one flag per thread.
struct Scan1 {
  u32 off, total;
};
template <bool SM>
__device__ __forceinline__ Scan1 scan1(u32 T, u32 buf, bool f) {
  const unsigned m = __ballot_sync(FULL, f);
  const u32 w = threadIdx.x >> 5, l = ln();
  u32* cnt = g_bt.cnt[buf];
  if (l == 0) cnt[w] = __popc(m);
  wsync(T);
  const u32 v = l < (T >> 5) ? cnt[l] : 0u;
  Scan1 r;
  r.total = __reduce_add_sync(FULL, v);
  r.off = __reduce_add_sync(FULL, l < w ? v : 0u) + __popc(m & lanemask_lt());
  return r;
}

// ExtrusionBarriers::init_states (extrusion_barriers.cpp:220-231)
template <bool SM>
__device__ __noinline__ u64 barriers_init(u64 rp) {
  const View<SM> c;
  const u32 T = c.T;
  u32 buf = 0;
#pragma unroll 1
  for (u32 base = 0; base < c.nb; base += T) {
    const u32 i = base + threadIdx.x;
    const bool need = i < c.nb && (bar_flags(c.bpf, i) & BF_OCC_DRAWS);
    const Scan2 sc2 = scan2<SM>(buf, need, false);
    rng_publish(rp);
    buf ^= 1;
    rng_ensure(rp, T);
    const bool occ = need && ring_at(c.rmask, rp + sc2.off0) <= c.bar[i].t_occ;
    const unsigned om = __ballot_sync(FULL, occ);
    if (ln() == 0 && i < c.nb) c.bst[i >> 5] = om;
    rp += sc2.total;
  }
  wsync(c.T);
  rng_publish(rp);
  return rp;
}

// ExtrusionBarriers::next_state (extrusion_barriers.cpp:145-161): one draw per barrier.
template <bool SM>
__device__ __noinline__ u64 barriers_next(u64 rp) {
  const View<SM> c;
  const u32 T = c.T, nb = c.nb;
  const uint2* __restrict__ bpf = c.bpf;
  const DevBarrier* __restrict__ bar = c.bar;
#pragma unroll 1
  for (u32 base = 0; base < nb; base += 2 * T) {
    rng_ensure(rp, 2 * T);
    u32 f[2];
    u64 thr[2];
    bool st[2];
#pragma unroll
    for (u32 h = 0; h < 2; ++h) {
      const u32 i = base + h * T + threadIdx.x, ic = i < nb ? i : 0u;
      st[h] = i < nb && ((c.bst[i >> 5] >> ln()) & 1u);
      f[h] = __ldg(&bpf[ic].y);
      thr[h] = st[h] ? __ldg(&bar[ic].t_act) : __ldg(&bar[ic].t_ina);
    }
    __syncwarp();
#pragma unroll
    for (u32 h = 0; h < 2; ++h) {
      const u32 k = h * T + threadIdx.x, i = base + k;
      const bool above = ring_at(c.rmask, rp + k) >= thr[h];
      const bool nst = st[h] ? !(!(f[h] & BF_ACT_NEVER) && above) : !(f[h] & BF_INA_NEVER) && above;
      const unsigned m = __ballot_sync(FULL, i < nb && nst);
      if (ln() == 0 && i < nb) c.bst[i >> 5] = m;
    }
    rp += min(2 * T, nb - base);
    wsync(c.T);
    rng_publish(rp);
  }
  return rp;
}

// select_lefs_to_bind + bind_lefs (simulation_impl.hpp:28-89): one uniform_int draw per
// selected LEF in index order.  Selection: mode 0 = unbound LEFs (the epoch loop), 1 =
// nonzero entries of mask, 2 = every LEF (an empty mask in the reference).  The selected LEFs are
// compacted first: they are a few per cent of all, and each takes a 64-bit division.
template <bool SM>
__device__ __noinline__ u64 bind_lefs(u64 rp, u32 n, u32 epoch, int mode,
                                      const u64* mask) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  const auto list = c.tmp;
  u32 nsel = 0, buf = 0;
#pragma unroll 1
  for (u32 base = 0; base < n; base += 2 * T) {
    const u32 i0 = base + threadIdx.x, i1 = i0 + T;
    const bool f0 = i0 < n && (mode == 0 ? c.bep[i0] == UNBOUND : (mode == 1 ? mask[i0] != 0 : true));
    const bool f1 = i1 < n && (mode == 0 ? c.bep[i1] == UNBOUND : (mode == 1 ? mask[i1] != 0 : true));
    const Scan2 s = scan2<SM>(buf, f0, f1);
    buf ^= 1;
    if (f0) list[nsel + s.off0] = i0;
    if (f1) list[nsel + s.off1] = i1;
    nsel += s.total;
  }
  wsync(c.T);
#pragma unroll 1
  for (u32 q = 0; q < nsel; q += T) {
    const u32 cnt = min(T, nsel - q);
    rng_ensure(rp, cnt);
    const bool mine = threadIdx.x < cnt;
    u64 r = 0;
    bool ok = true;
    if (mine) {
      r = div64(ring_at(c.rmask, rp + threadIdx.x), P.pos_bucket);
      ok = r <= P.pos_range;
    }
    if (wsync_or(c.T, !ok)) {
      // a bucket rejection: the rest one by one with the exact number of draws
      if (threadIdx.x == 0) {
#pragma unroll 1
        for (u32 j = q; j < nsel; ++j) {
          const u64 pos = s_uniform_int(g_c, P.wstart, (u64)P.wend - 1);
          c.rev[list[j]] = (u32)pos;
          c.fwd[list[j]] = (u32)pos;
          c.bep[list[j]] = epoch;
        }
      }
      wsync(c.T);
      return g_sc.rpos;
    }
    rp += cnt;
    rng_publish(rp);
    if (mine) {
      const u32 i = list[q + threadIdx.x], pos = (u32)(P.wstart + r);
      c.rev[i] = pos;
      c.fwd[i] = pos;
      c.bep[i] = epoch;
    }
  }
  wsync(c.T);
  return rp;
}
// Ranking key of a unit: position, then binding epoch ascending (rev) or descending (fwd).
__device__ __forceinline__ u64 rank_key(const Cell& c, u32 dir, u32 idx) {
  const u32 p = dir ? c.fwd[idx] : c.rev[idx];
  const u32 e = dir ? ~c.bep[idx] : c.bep[idx];
  return ((u64)p << 32) | e;
}

// Warp bitonic sort of the index block a[0..m) by the 64-bit keys hi[k] << 32 | lo[k] stored
// beside it (a, hi and lo move together).  Only ascending comparators are used (each merge
// starts by comparing mirror pairs), so the virtual +inf padding up to a power of two never
// moves and needs no storage.  Block sizes and strides are powers of two, so the comparator
// indexes are shifts and masks.
__device__ void bitonic_keyed(u32* a, u32* hi, u32* lo, u32 m) {
  u32 lg = 0;
#pragma unroll 1
  while ((1u << lg) < m) ++lg;
  const u32 ncmp = (1u << lg) >> 1;  // comparators per stage
  auto cmpx = [&](u32 i, u32 j) {
    if (j >= m) return;
    const u64 ki = ((u64)hi[i] << 32) | lo[i], kj = ((u64)hi[j] << 32) | lo[j];
    if (ki > kj) {
      hi[i] = (u32)(kj >> 32);
      lo[i] = (u32)kj;
      hi[j] = (u32)(ki >> 32);
      lo[j] = (u32)ki;
      const u32 x = a[i];
      a[i] = a[j];
      a[j] = x;
    }
  };
#pragma unroll 1
  for (u32 s = 1; s <= lg; ++s) {
    // merge into sorted blocks of 2^s: mirror pairs, then strides 2^(s-2) .. 1
#pragma unroll 1
    for (u32 t = ln(); t < ncmp; t += 32) {
      const u32 base = (t >> (s - 1)) << s, off = t & ((1u << (s - 1)) - 1u);
      cmpx(base + off, base + (1u << s) - 1u - off);
    }
    __syncwarp();
#pragma unroll 1
    for (int q = (int)s - 2; q >= 0; --q) {
#pragma unroll 1
      for (u32 t = ln(); t < ncmp; t += 32) {
        const u32 i = ((t >> q) << (q + 1)) | (t & ((1u << q) - 1u));
        cmpx(i, i + (1u << q));
      }
      __syncwarp();
    }
  }
}

// Lane 0: insertion-sort the run of equal positions around a[t-1], a[t] by binding epoch
// (ascending for rev units, descending for fwd units), as the tie fix of rank_lefs does
// (simulation.cpp:446-485).  Returns the end of the run.
__device__ __noinline__ u32 tie_fix_run(const Cell& c, u32 dir, u32* a, u32 t, u32 len) {
  const u32* pos = dir ? c.fwd : c.rev;
  const u32 p = pos[a[t]];
  u32 lo = t - 1, hi = t + 1;
#pragma unroll 1
  while (lo > 0 && pos[a[lo - 1]] == p) --lo;
#pragma unroll 1
  while (hi < len && pos[a[hi]] == p) ++hi;
  if (dir) {
    ins_sort(a, lo, hi, KeyCmpRev{c.bep});
  } else {
    ins_sort(a, lo, hi, KeyCmp{c.bep});
  }
  return hi;
}

// rank_lefs for one direction when the previous order is reused (split_sort,
// simulation.cpp:427-435, then the tie fix :446-485), warp-parallel and exact.
//
// split_sort makes one pass that keeps a non-decreasing stack K of the input (a smaller
// element pops the stack top and both leave), pdq-sorts the removed elements B in the order the
// pass's swaps leave them, and merges K and B stably.  The tie fix then orders runs of equal
// positions by binding epoch.  The result is the stable sort of K followed by B by the key
// (position, epoch): the order is unique except among full ties (equal position and epoch),
// which keep K's order, then B's order after pdq_sort.
//
// Here the pass runs 32 elements at a time: the lanes up to the first one below its
// predecessor (or below the stack top) are pushed together, and each pop is an event.  The
// removed block only changes by events (top prepended, reader appended) and by pushes (each
// rotates it left by one), so every removed element's final slot follows from the event list.
// B is sorted by key with a warp bitonic sort; only if B holds full ties is it pdq-sorted
// exactly on lane 0.  Returns false (R untouched) for n < 2 or n > 65535.
//
// Scratch: the stack K in sr, the input positions and later B in tmp, and the event lists in
// rm, fm and sf.  The move arrays are dead from binding until the moves are generated (the
// callers that keep them restore them), and every event removes one input element, so n
// entries per list always suffice.
__device__ __noinline__ bool rank_dir_split(Cell& c, u32 dir, u32 n) {
  if (n < 2 || n > 0xFFFFu) return false;
  u32* R = dir ? c.fr : c.rr;
  const u32* pos = dir ? c.fwd : c.rev;
  u32* K = c.sr;
  const u32 EMAX = n;
  u32* ev_q = c.rm;  // pushes since the previous event; later (q mod k_prev) | k_prev << 16
  u32* ev_top = c.fm;
  u32* ev_rd = c.sf;
  u32* B = c.tmp;
  const u32 lane = ln();
  u64 tprof = clock64();
  // positions in input order, gathered up front with independent loads (B is written to tmp
  // only after the pass)
  {
    const u32* __restrict__ Rr = R;
    const u32* __restrict__ pr = pos;
    u32* __restrict__ V = c.tmp;
#pragma unroll 1
    for (u32 r = lane; r < n; r += 32) V[r] = pr[Rr[r]];
  }
  __syncwarp();
  const u32* V = c.tmp;
  const u32 first = R[0];
  if (lane == 0) K[0] = first;
  u32 m = 0, T = V[0], E = 0, q = 0;
#pragma unroll 1
  for (u32 base = 1; base < n; base += 32) {
    const u32 r = base + lane;
    const u32 nvalid = min(32u, n - base);
    const bool valid = lane < nvalid;
    const u32 idx = valid ? R[r] : 0;
    const u32 v = valid ? V[r] : 0;
    const u32 vprev = __shfl_up_sync(FULL, v, 1);
    const bool pre_ok = lane == 0 || v >= vprev;
    u32 start = 0;
#pragma unroll 1
    while (start < nvalid) {
      const bool ok = lane == start ? v >= T : pre_ok;
      const unsigned fail = __ballot_sync(FULL, !ok && lane >= start && valid);
      const u32 f = fail ? (u32)(__ffs(fail) - 1) : nvalid;
      if (lane >= start && lane < f) K[m + 1 + lane - start] = idx;
      if (f > start) {
        m += f - start;
        if (E) q += f - start;
        T = __shfl_sync(FULL, v, f - 1);
      }
      if (f == nvalid) break;
      const u32 rd = __shfl_sync(FULL, idx, f);
      if (E >= EMAX) return false;
      __syncwarp();
      u32 top = UNBOUND;
      if (m > 0) {
        top = K[m];
        --m;
        T = pos[K[m]];
      }
      if (lane == 0) {
        ev_q[E] = q;
        ev_top[E] = top;
        ev_rd[E] = rd;
      }
      ++E;
      q = 0;
      start = f + 1;
    }
  }
  __syncwarp();
  {
    const u64 t = clock64();
    prof_add(PF_RANK_PASS, t - tprof);
    tprof = t;
  }
  const u32 ns = m + 1;
  // block size before each event, and the rotation it saw since the previous event
  u32 kacc = 0;
#pragma unroll 1
  for (u32 b = 0; b < E; b += 32) {
    const u32 j = b + lane;
    const bool vj = j < E;
    const u32 sz = vj ? (ev_top[j] != UNBOUND ? 2u : 1u) : 0u;
    u32 tot;
    const u32 ex = warp_excl_scan(sz, &tot);
    if (vj) {
      const u32 kprev = kacc + ex;
      const u32 qm = kprev ? ev_q[j] % kprev : 0u;
      ev_q[j] = qm | (kprev << 16);
    }
    kacc += tot;
  }
  const u32 kE = kacc;
  __syncwarp();
  // final slot of every removed element
  const u32 qfm = kE ? q % kE : 0u;
#pragma unroll 1
  for (u32 b = 0; b < E; b += 32) {
    const u32 j = b + lane;
    const bool vj = j < E;
    const u32 top = vj ? ev_top[j] : UNBOUND;
    const u32 rd = vj ? ev_rd[j] : 0u;
    const u32 kj = vj ? (ev_q[j] >> 16) + (top != UNBOUND ? 2u : 1u) : 1u;
    u32 it = 0, ir = kj - 1;
#pragma unroll 1
    for (u32 jj = b + 1; jj < E; ++jj) {
      const u32 w = ev_q[jj];
      const bool pop = ev_top[jj] != UNBOUND;
      if (jj > j) {
        const u32 qm = w & 0xFFFFu, kk = w >> 16;
        it = it >= qm ? it - qm : it + kk - qm;
        ir = ir >= qm ? ir - qm : ir + kk - qm;
        if (pop) {
          ++it;
          ++ir;
        }
      }
    }
    it = it >= qfm ? it - qfm : it + kE - qfm;
    ir = ir >= qfm ? ir - qfm : ir + kE - qfm;
    if (vj) {
      if (top != UNBOUND) B[it] = top;
      B[ir] = rd;
    }
  }
  __syncwarp();
  // sort B by key (the events are dead: sf, rm and fm are free); the keys are loaded once and
  // sorted alongside the indices, so the network compares values already in memory.  Measured
  // on the genome workload, sorting every block this way beats handing large blocks (or, as
  // split_sort's event list once had to, whole ranks) to lane 0's serial sorts.
  u32* Bs = c.sf;
  u32* Kh = c.rm;  // position
  u32* Kl = c.fm;  // binding epoch (complemented for fwd units)
  bool full_tie = false;
#pragma unroll 1
  for (u32 t = lane; t < kE; t += 32) {
    const u32 idx = B[t];
    const u64 k = rank_key(c, dir, idx);
    Bs[t] = idx;
    Kh[t] = (u32)(k >> 32);
    Kl[t] = (u32)k;
  }
  __syncwarp();
  bitonic_keyed(Bs, Kh, Kl, kE);
#pragma unroll 1
  for (u32 t = lane + 1; t < kE; t += 32) full_tie |= Kh[t - 1] == Kh[t] && Kl[t - 1] == Kl[t];
  const u32* Bf = Bs;
  if (__any_sync(FULL, full_tie)) {
    prof_add(PF_RANK_PDQ, 1);
    if (lane == 0) {
      pdq_sort(B, 0, kE, KeyCmp{pos});
#pragma unroll 1
      for (u32 t = 1; t < kE; ++t) {
        if (pos[B[t - 1]] == pos[B[t]]) t = tie_fix_run(c, dir, B, t, kE);
      }
    }
    __syncwarp();
    Bf = B;
  }
  {
    const u64 t = clock64();
    prof_add(PF_RANK_BLOCK, t - tprof);
    tprof = t;
  }
  // tie fix of K: runs of equal positions whose epochs are out of order (each element's key is
  // read once; the previous element's comes from the adjacent lane or the previous chunk)
  u64 kprev = ns ? rank_key(c, dir, K[0]) : 0;
#pragma unroll 1
  for (u32 base = 1; base < ns; base += 32) {
    const u32 t = base + lane;
    const u64 kt = t < ns ? rank_key(c, dir, K[t]) : ~0ull;
    u64 k0 = __shfl_up_sync(FULL, kt, 1);
    if (lane == 0) k0 = kprev;
    kprev = __shfl_sync(FULL, kt, 31);
    const bool bad = t < ns && (k0 >> 32) == (kt >> 32) && k0 > kt;
    unsigned bm = __ballot_sync(FULL, bad);
    if (bm) {
      if (lane == 0) {
#pragma unroll 1
        while (bm) {
          const u32 t0 = base + (u32)(__ffs(bm) - 1);
          const u32 hi = tie_fix_run(c, dir, K, t0, ns);
          const u32 last = hi - 1 - base;  // bits up to the run's end are done
          bm = last >= 31 ? 0u : bm & ~((2u << last) - 1u);
        }
      }
      __syncwarp();
      // a fixed run may reach the chunk's end: carry the key now at its last slot
      const u32 tl = min(base + 31, ns - 1);
      kprev = rank_key(c, dir, K[tl]);
    }
  }
  // merge, K first among equal keys.  u_j = #K with key <= key(B_j) (binary search; K is
  // sorted by key), so B_j lands at j + u_j and K_i at i + #{j : u_j <= i}; u is
  // non-decreasing in j, so one pass over K with a pointer into u counts the latter.
  u32* U = Bf == Bs ? B : Bs;  // the dead one of the two B buffers
#pragma unroll 1
  for (u32 j = lane; j < kE; j += 32) {
    const u32 idx = Bf[j];
    const u64 key = rank_key(c, dir, idx);
    u32 lo = 0, hi = ns;
#pragma unroll 1
    while (lo < hi) {
      const u32 mid = (lo + hi) >> 1;
      if (rank_key(c, dir, K[mid]) <= key) lo = mid + 1; else hi = mid;
    }
    U[j] = lo;
    R[j + lo] = idx;
  }
  __syncwarp();
  u32 jb = 0;  // B elements with u_j below the chunk
#pragma unroll 1
  for (u32 base = 0; base < ns; base += 32) {
    const u32 i = base + lane;
    u32 cnt = jb, j = jb;
#pragma unroll 1
    for (; j < kE; ++j) {
      const u32 uj = U[j];
      if (uj >= base + 32) break;
      cnt += uj <= i ? 1u : 0u;
    }
    if (i < ns) R[i + cnt] = K[i];
    jb = j;
  }
  __syncwarp();
  prof_add(PF_RANK_MERGE, clock64() - tprof);
  return true;
}

__device__ __forceinline__ u64 max64(u64 a, u64 b) { return a > b ? a : b; }

// Whether the kept unit of rank r and the one of rank r - 1, which it ties with in position and epoch,
// surely stay in this order in the reference.  Its split_sort keeps a stack: an element below the top
// leaves together with the top, the others are pushed; what stays keeps its order, even in a tie.  So
// the pair's order is certain when neither can have left:
//  * later pops reach rank r only if they outnumber the pushes after it.  Every pop needs a removed unit
//    (one below its predecessors, or one bound this epoch that the next unit pops), so with the k-th
//    removed unit after r at rank q_k, q_k - r >= 2 k + 2 for all k keeps a push in front of each pop;
//  * the units themselves pop something only if a removed unit before them is still on the stack, and each
//    of those is popped by one unit after it: (r - 1) - p_j >= 2 j + 2 for the j-th one before;
//  * except that the bottom of the stack is never popped: rank 0 has to be a kept unit.
template <class A>
__device__ __noinline__ bool tie_keeps_order(const A& kmask, u32 nch, u32 r) {
  const u32 a = r - 1;
  if (r == 0 || !(kmask[0] & 1u) || !((kmask[a >> 5] >> (a & 31)) & 1u)) return false;
  u32 k = 0;
#pragma unroll 1
  for (u32 ch = r >> 5; ch < nch; ++ch) {
    u32 gone = ~kmask[ch];
    if (ch == r >> 5) gone &= (r & 31) == 31 ? 0u : ~0u << ((r & 31) + 1);
#pragma unroll 1
    for (; gone; gone &= gone - 1) {
      const u32 q = ch * 32 + (u32)(__ffs(gone) - 1);
      if (q - r < 2 * ++k + 2) return false;
    }
  }
  k = 0;
#pragma unroll 1
  for (u32 ch = a >> 5; ch != ~0u; --ch) {
    u32 gone = ~kmask[ch];
    if (ch == a >> 5) gone &= (1u << (a & 31)) - 1u;
#pragma unroll 1
    for (; gone; gone &= ~(1u << (31 - __clz(gone)))) {
      const u32 q = ch * 32 + 31 - __clz(gone);
      if (a - q < 2 * ++k + 2) return false;
    }
  }
  return true;
}

// Which ranks stay on the stack of the reference's split_sort, one warp: a bit mask, from the positions in
// rank order.  The pass runs 32 elements at a time as in rank_dir_split; the stack holds ranks.
template <bool SM>
__device__ __noinline__ void split_mask(u32 n, const Arr<SM> pos, const Arr<SM> stack, const Arr<SM> kmask) {
  const u32 lane = ln();
#pragma unroll 1
  for (u32 ch = lane; ch < (n + 31) >> 5; ch += 32) kmask[ch] = n - ch * 32 >= 32 ? FULL : (1u << (n & 31)) - 1u;
  if (lane == 0) stack[0] = 0;
  u32 m = 0, T = pos[0];
#pragma unroll 1
  for (u32 base = 1; base < n; base += 32) {
    const u32 r = base + lane, nvalid = min(32u, n - base);
    const bool valid = lane < nvalid;
    const u32 v = valid ? pos[r] : 0;
    const u32 vprev = __shfl_up_sync(FULL, v, 1);
    const bool pre_ok = lane == 0 || v >= vprev;
    u32 start = 0;
#pragma unroll 1
    while (start < nvalid) {
      const bool ok = lane == start ? v >= T : pre_ok;
      const unsigned fail = __ballot_sync(FULL, !ok && lane >= start && valid);
      const u32 f = fail ? (u32)(__ffs(fail) - 1) : nvalid;
      if (lane >= start && lane < f) stack[m + 1 + lane - start] = r;
      if (f > start) {
        m += f - start;
        T = __shfl_sync(FULL, v, f - 1);
      }
      if (f == nvalid) break;
      __syncwarp();
      const u32 rd = base + f, top = stack[m];
      if (m > 0) {
        --m;
        T = pos[stack[m]];
      }
      if (lane == 0) {
        kmask[rd >> 5] &= ~(1u << (rd & 31));
        if (m > 0 || stack[0] != top) kmask[top >> 5] &= ~(1u << (top & 31));
      }
      start = f + 1;
    }
  }
  __syncwarp();
}

enum : u32 { RANK_DONE = 0, RANK_TIE = 1, RANK_MANY = 2 };  // rank_dir_block's outcome

// rank_lefs for one direction with the previous order reused, by all workers.
//
// Unless two units share position and binding epoch (a full tie), the reference's order (split_sort,
// then the tie fix) is simply the order by that key, whatever the way it is sorted.  So the units are
// split into those that still form a non-decreasing sequence and the few that do not: the units bound
// this epoch and every other one below the running maximum of the rest.  The few are sorted by key
// (runs of 32 in registers, then each finds its place in the other runs by binary search) and merged
// back by rank.  R stays untouched when a full tie turns up whose order is not certain
// (tie_keeps_order, RANK_TIE) or when too many units moved (RANK_MANY); n is 2 to 65535.  With exact, the kept units are those the
// reference's own pass keeps (split_mask): then ties among them and with a removed unit have the
// order the stable merge gives them, and only a tie between two removed units is left to
// rank_dir_split.
//
// Phases, each ended by a wsync; warp w owns a contiguous range of the ranks:
//  1 keys in rank order to rm / fm, and their maximum per warp;
//  2 running maximum; the removed units' keys to the 64-bit array in sr / sf, with index and
//    rank packed in tmp; a bit mask of the kept ranks at the end of sf;
//  3 runs of 32 removed units sorted in registers;
//  4 each removed unit's place among the removed (pairwise searches) and among the kept;
//  5 the new order, written to rm; 6 copied to R.
template <bool SM>
__device__ __noinline__ u32 rank_dir_block(u32 dir, u32 n, u32 epoch, bool exact) {
  const View<SM> c;
  const u32 T = c.T, W = T >> 5, w = threadIdx.x >> 5, lane = ln();
  const auto R = dir ? c.fr : c.rr;
  const auto pos = dir ? c.fwd : c.rev;
  const auto bep = c.bep;
  const auto kh = c.rm;
  const auto kl = c.fm;
  const auto bk = c.sr;  // as 64-bit words
  const u32 nch = (n + 31) >> 5;
  const auto kmask = c.sf + (n - nch);
  const u32 maxb = n / 3;
  const auto bp = c.tmp, sr0 = c.tmp + maxb, sfin = c.tmp + 2 * maxb;
  const u32 ch0 = w * nch / W, ch1 = (w + 1) * nch / W;
  const u32 newlo = dir ? ~epoch : epoch;
  u32 mh = 0, ml = 0;  // this lane's largest key
#pragma unroll 1
  for (u32 ch = ch0; ch < ch1; ++ch) {
    const u32 r = ch * 32 + lane;
    if (r < n) {
      const u32 idx = R[r];
      const u32 p = pos[idx], e = bep[idx], lo = dir ? ~e : e;
      kh[r] = p;
      kl[r] = lo;
      if (lo != newlo && (p > mh || (p == mh && lo > ml))) {
        mh = p;
        ml = lo;
      }
    }
  }
  const u32 wh = __reduce_max_sync(FULL, mh);
  const u64 mx = ((u64)wh << 32) | __reduce_max_sync(FULL, mh == wh ? ml : 0u);
  if (lane == 0) g_bt.wmax[w] = mx;
  if (threadIdx.x == 0) {
    g_bt.nrem = 0;
    g_bt.ntie = 0;
    g_bt.tie2 = 0;
  }
  wsync(c.T);
  if (exact) {
    if (w == 0) split_mask<SM>(n, kh, c.sr, kmask);
    wsync(c.T);
    // maxima of the kept units
    u64 kmx = 0;
#pragma unroll 1
    for (u32 ch = ch0; ch < ch1; ++ch) {
      const u32 r = ch * 32 + lane;
      if ((kmask[ch] >> lane) & 1u) kmx = max64(kmx, ((u64)kh[r] << 32) | kl[r]);
    }
#pragma unroll 1
    for (int d = 16; d > 0; d >>= 1) kmx = max64(kmx, __shfl_xor_sync(FULL, kmx, d));
    if (lane == 0) g_bt.wmax[w] = kmx;
    wsync(c.T);
  }
  u64 carry = lane < w ? g_bt.wmax[lane] : 0;
#pragma unroll 1
  for (int d = 8; d > 0; d >>= 1) carry = max64(carry, __shfl_xor_sync(FULL, carry, d));
  carry = __shfl_sync(FULL, carry, 0);
  u32 removed = 0;
#pragma unroll 1
  for (u32 ch = ch0; ch < ch1; ++ch) {
    const u32 r = ch * 32 + lane;
    const bool valid = r < n;
    const u32 hi = valid ? kh[r] : 0u, lo = valid ? kl[r] : 0u;
    const bool old = exact ? (kmask[ch] >> lane) & 1u : valid && lo != newlo;
    // running maximum of the old units before this one: by position alone unless positions repeat
    u32 x = old ? hi : 0;
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
      const u32 y = __shfl_up_sync(FULL, x, d);
      if ((int)lane >= d) x = max(x, y);
    }
    const u32 px = __shfl_up_sync(FULL, x, 1);
    const u32 eh = max(lane == 0 ? 0u : px, (u32)(carry >> 32));
    bool keep = old && hi > eh;
    u64 excl;
    const u64 key = ((u64)hi << 32) | lo;
    if (!exact && !__any_sync(FULL, old && hi == eh)) {
      // the maximum's epoch is that of the last unit kept before
      const unsigned kb = __ballot_sync(FULL, keep), before = kb & lanemask_lt();
      const u32 el = __shfl_sync(FULL, lo, before ? 31 - __clz(before) : 0);
      excl = ((u64)eh << 32) | (before ? el : (u32)carry);
      const u32 top = __shfl_sync(FULL, lo, kb ? 31 - __clz(kb) : 0);
      const u32 th = __shfl_sync(FULL, hi, kb ? 31 - __clz(kb) : 0);
      if (kb) carry = ((u64)th << 32) | top;
    } else {
      u64 z = old ? key : 0;
#pragma unroll 1
      for (int d = 1; d < 32; d <<= 1) {
        const u64 y = __shfl_up_sync(FULL, z, d);
        if ((int)lane >= d) z = max64(z, y);
      }
      excl = __shfl_up_sync(FULL, z, 1);
      excl = lane == 0 ? carry : max64(excl, carry);
      keep = old && key >= excl;
      if (exact && keep != old) g_bt.tie2 = 1;  // equal positions out of epoch order
      if (!exact && keep && key == excl) {
        const u32 q = atomicAdd(&g_bt.ntie, 1u);
        if (q < MAX_TIES) g_bt.tierank[q] = r;
      }
      carry = max64(carry, __shfl_sync(FULL, z, 31));
    }
    const bool rem = valid && !keep;
    const unsigned km = __ballot_sync(FULL, keep), rmk = __ballot_sync(FULL, rem);
    if (lane == 0) kmask[ch] = km;
    if (rmk) {
      u32 q = 0;
      if (lane == 0) q = atomicAdd(&g_bt.nrem, (u32)__popc(rmk));
      q = __shfl_sync(FULL, q, 0) + __popc(rmk & lanemask_lt());
      if (rem) {
        kh[r] = (u32)(excl >> 32);
        kl[r] = (u32)excl;
        if (q < maxb) {
          bk.at64(q) = key;
          bp[q] = R[r] | (r << 16);
        }
      }
      removed += __popc(rmk);
    }
  }
  if (lane == 0) g_bt.rem[w] = removed;
  wsync(c.T);
  const u32 m = g_bt.nrem;
  const u32 nt = g_bt.ntie;
  if (m > maxb) return RANK_MANY;
  if (nt > MAX_TIES) return RANK_TIE;
#pragma unroll 1
  for (u32 q = threadIdx.x; q < nt; q += T)
    if (!tie_keeps_order(kmask, nch, g_bt.tierank[q])) g_bt.tie2 = 1;
  // 3: runs of 32
  if (w == W - 1) {  // removed units before each warp's range
    u32 v = lane < W ? g_bt.rem[lane] : 0u;
    const u32 ex = warp_excl_scan(v, nullptr);
    if (lane < W) g_bt.rembase[lane] = ex;
  }
#pragma unroll 1
  for (u32 run = w; run * 32 < m; run += W) {
    const u32 q = run * 32 + lane;
    u64 key = q < m ? bk.at64(q) : ~0ull;
    u32 pl = q < m ? bp[q] : 0u;
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll 1
      for (int j = k >> 1; j > 0; j >>= 1) {
        const u64 ok = __shfl_xor_sync(FULL, key, j);
        const u32 op = __shfl_xor_sync(FULL, pl, j);
        const bool up = (lane & k) == 0 || k == 32;
        const bool lower = (lane & j) == 0;
        const bool take = (lower == up) ? ok < key : ok > key;
        if (take) {
          key = ok;
          pl = op;
        }
      }
    }
    const u64 prev = __shfl_up_sync(FULL, key, 1);
    if (q < m) {
      bk.at64(q) = key;
      bp[q] = pl;
      if (lane > 0 && prev == key) g_bt.tie2 = 1;
    }
  }
  wsync(c.T);
  // 4: places
#pragma unroll 1
  for (u32 q = threadIdx.x; q < m; q += T) {
    const u64 key = bk.at64(q);
    const u32 my = q >> 5;
    u32 rank = q & 31u;
#pragma unroll 1
    for (u32 s0 = 0; s0 < m; s0 += 32) {
      if ((s0 >> 5) == my) continue;
      const u32 len = min(32u, m - s0);
      u32 lo = 0, hi = len;
#pragma unroll 1
      while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (bk.at64(s0 + mid) < key) lo = mid + 1; else hi = mid;
      }
      if (lo < len && bk.at64(s0 + lo) == key) g_bt.tie2 = 1;
      rank += lo;
    }
    const u32 khi = (u32)(key >> 32), klo = (u32)key;
    u32 lo = 0, hi = n;  // first rank whose running maximum is >= key
#pragma unroll 1
    while (lo < hi) {
      const u32 mid = (lo + hi) >> 1;
      const u32 h = kh[mid];
      if (h < khi || (h == khi && kl[mid] < klo + ((exact && klo != ~0u) ? 1u : 0u))) lo = mid + 1; else hi = mid;
    }
    u32 before = m;  // removed units at ranks below lo
    if (lo < n) {
      if (kh[lo] == khi && kl[lo] == klo) g_bt.tie2 = 1;  // exact: passed above
      const u32 ch = lo >> 5, ow = ((ch + 1) * W - 1) / nch;
      before = g_bt.rembase[ow];
#pragma unroll 1
      for (u32 k = ow * nch / W; k < ch; ++k) before += 32 - __popc(kmask[k]);
      before += (lo & 31u) - __popc(kmask[ch] & ((1u << (lo & 31u)) - 1u));
    }
    sr0[rank] = lo;
    sfin[rank] = (bp[q] & 0xFFFFu) | ((rank + lo - before) << 16);
  }
  wsync(c.T);
  if (g_bt.tie2) return RANK_TIE;
  // 5: the new order
  const auto O = c.rm;
#pragma unroll 1
  for (u32 q = threadIdx.x; q < m; q += T) {
    const u32 v = sfin[q];
    O[v >> 16] = v & 0xFFFFu;
  }
  {
    u32 j;  // removed units that go before this warp's range
    {
      const u32 r0 = ch0 * 32;
      u32 lo = 0, hi = m;
#pragma unroll 1
      while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (sr0[mid] < r0) lo = mid + 1; else hi = mid;
      }
      j = lo;
    }
    u32 rb = g_bt.rembase[w];
#pragma unroll 1
    for (u32 ch = ch0; ch < ch1; ++ch) {
      const u32 r = ch * 32 + lane;
      const u32 km = kmask[ch];
      u32 ins = j;
#pragma unroll 1
      for (; j < m; ++j) {
        const u32 at = sr0[j];
        if (at >= ch * 32 + 32) break;
        ins += at <= r ? 1u : 0u;
      }
      if ((km >> lane) & 1u) O[r - rb - (lane - __popc(km & lanemask_lt())) + ins] = R[r];
      rb += 32 - __popc(km);
    }
  }
  wsync(c.T);
#pragma unroll 1
  for (u32 r = threadIdx.x; r < n; r += T) R[r] = O[r];
  wsync(c.T);
  return RANK_DONE;
}

// Sort of all units of one direction by key, by all workers: a bitonic network of ascending comparators
// (see bitonic_keyed) on keys in rm / fm and indices in tmp.  Returns false, R untouched, on a full tie.
template <bool SM>
__device__ __noinline__ bool rank_dir_all(u32 dir, u32 n) {
  const View<SM> c;
  const u32 T = c.T;
  const auto R = dir ? c.fr : c.rr;
  const auto pos = dir ? c.fwd : c.rev;
  const auto hi = c.rm, lo = c.fm, ix = c.tmp;
#pragma unroll 1
  for (u32 r = threadIdx.x; r < n; r += T) {
    const u32 u = R[r], e = c.bep[u];
    ix[r] = u;
    hi[r] = pos[u];
    lo[r] = dir ? ~e : e;
  }
  wsync(T);
  u32 lg = 0;
#pragma unroll 1
  while ((1u << lg) < n) ++lg;
  const u32 ncmp = (1u << lg) >> 1;
#pragma unroll 1
  for (u32 s = 1; s <= lg; ++s) {
#pragma unroll 1
    for (int q = (int)s - 1; q >= 0; --q) {
#pragma unroll 1
      for (u32 t = threadIdx.x; t < ncmp; t += T) {
        u32 i, j;
        if (q == (int)s - 1) {  // mirror pairs
          const u32 base = (t >> q) << s, off = t & ((1u << q) - 1u);
          i = base + off;
          j = base + (1u << s) - 1u - off;
        } else {
          i = ((t >> q) << (q + 1)) | (t & ((1u << q) - 1u));
          j = i + (1u << q);
        }
        if (j >= n) continue;
        const u32 hi_i = hi[i], hi_j = hi[j], lo_i = lo[i], lo_j = lo[j];
        if (hi_i > hi_j || (hi_i == hi_j && lo_i > lo_j)) {
          hi[i] = hi_j;
          hi[j] = hi_i;
          lo[i] = lo_j;
          lo[j] = lo_i;
          const u32 x = ix[i];
          ix[i] = ix[j];
          ix[j] = x;
        }
      }
      wsync(T);
    }
  }
  bool tie = false;
#pragma unroll 1
  for (u32 r = threadIdx.x + 1; r < n; r += T) tie |= hi[r - 1] == hi[r] && lo[r - 1] == lo[r];
  if (wsync_or(T, tie)) return false;
#pragma unroll 1
  for (u32 r = threadIdx.x; r < n; r += T) R[r] = ix[r];
  wsync(T);
  return true;
}

// The incremental merge; after a full tie the merge on the reference's own kept units; a sort of all
// units when many moved (a young cell binds most of its units in one epoch) and for the first epoch;
// and where ties are left to pdq_sort's element moves, one warp's exact emulation or, without a previous
// order, the serial restatement.  sort_fallbacks counts the directions without a reusable order.
template <bool SM>
__device__ __noinline__ void rank_lefs(u32 n, u32 epoch, bool partially_sorted) {
  const View<SM> c;
  const KParams& P = g_P;
  const bool serial = P.debug_flags & DBG_SERIAL_RANK;
  const bool fast = partially_sorted && !serial && n >= 2 && n <= 0xFFFFu;
#pragma unroll 1
  for (u32 dir = 0; dir < 2; ++dir) {
    if (fast) {
      u32 got = rank_dir_block<SM>(dir, n, epoch, false);
      if (got == RANK_DONE) continue;
      wsync(c.T);  // the scratch is written again
      if (got == RANK_TIE) {
        got = rank_dir_block<SM>(dir, n, epoch, true);
        if (got == RANK_DONE) continue;
        wsync(c.T);
      }
      if (got == RANK_MANY && rank_dir_all<SM>(dir, n)) continue;
      prof_add(PF_RANK_SPLIT, 1);
      if (threadIdx.x < 32) rank_dir_split(g_c, dir, n);
      wsync(c.T);
    } else {
      prof_add(PF_RANK_FALLBACK, 1);
      if (threadIdx.x == 0) g_sc.sort_fallbacks++;
      if (serial || !rank_dir_all<SM>(dir, n)) {
        if (threadIdx.x == 0) rank_dir_serial(g_c, dir, n, partially_sorted);
        wsync(c.T);
      }
    }
  }
}

// positions in rank order: sr[k] = rev[rr[k]], sf[k] = fwd[fr[k]]
template <bool SM>
__device__ __noinline__ void gather_ranked(u32 n) {
  const View<SM> c;
  const auto rr = c.rr;
  const auto fr = c.fr;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
  const auto sr = c.sr;
  const auto sf = c.sf;
#pragma unroll 1
  for (u32 k = threadIdx.x; k < n; k += c.T) {
    sr[k] = rev[rr[k]];
    sf[k] = fwd[fr[k]];
  }
  wsync(c.T);
}

// One draw of the moves' normal distribution and the move it gives: v = round(max(0, z * sd + mean)).
// The reference evaluates this in doubles; here the ziggurat's comparison is an integer threshold on
// the draw (zt[i].x) and the move is computed in 32.32 fixed point from the layer's width (zt[i].y =
// x_i * 2^60) and sd * 2^36.  Both the doubles' rounding and the fixed point's are below 8 units of
// 2^-32 for the parameters MoveSpec marks as fixed, so the rounded move is the reference's unless the value
// lies within 16 units of a half: then, for the tail layer, and where the wedge test is closer than
// the single-precision estimate resolves, the draw is evaluated in doubles by unit_normal_t.
// The FP64 pipe of sm_103a runs at 1/64 of the FP32 rate: with doubles alone the moves of a
// 2,500-LEF cell kept it busy for about a third of the epoch.
__device__ __noinline__ int move_exact(RingSrc& g, const MoveSpec& ms, u32* v, bool* range) {
  double z = 0.0;
  const int st = unit_normal_t(g, z);
  const double d = round(fmax(0.0, z * ms.sd + ms.mean));
  *range = d > 4294967295.0;
  *v = (u32)(u64)d;
  return st;
}

__device__ __forceinline__ int move_sample(RingSrc& g, const MoveSpec& ms, u32* v, bool* range) {
  *range = false;
  if (ms.fixed) {
#pragma unroll 1
    for (int it = 0; it < 64; ++it) {
      const RingSrc here = g;  // an attempt of the sampler carries nothing from the one before
      u64 u;
      if (!g.next(u)) return SMP_DRY;
      const u32 ii = (u32)u & 0xFFu, i = ii >> 1;
      const u64 m = (u & ~(1ull << 11)) >> 8;
      const ulonglong2 e = g_bt.zt[i];
      const u64 t = __umul64hi(m << 8, e.y);  // x * 2^60
      bool acc = m < e.x, exact = false;
      if (!acc) {
        u64 u2 = 0;
        if (i == 0) {
          exact = true;
        } else if (!g.next(u2)) {
          return SMP_DRY;
        } else if (u2 >= ~0ull << 12) {
          exact = true;  // uniform_01 may round to 1 and be drawn again
        } else {
          const float x = (float)(u32)(t >> 32) * 0x1p-28f;
          const float ef = expf(-0.5f * x * x);
          const float2 y = g_bt.zy[i];
          const float d = y.x + (float)(u32)(u2 >> 32) * 0x1p-32f * y.y - ef;
          exact = fabsf(d) <= 2e-5f * ef;
          acc = d < 0.0f;
        }
      }
      if (acc && !exact) {
        const i64 wq = (i64)__umul64hi(t, ms.sdq);
        const i64 q = (ii & 1u) ? ms.meanq + wq : ms.meanq - wq;
        if (q <= -16) {
          *v = 0;
          return SMP_OK;
        }
        const u32 frac = (u32)q - 0x80000000u;
        exact = frac + 16u <= 32u;
        if (!exact) {
          *v = (u32)((q + 0x80000000ll) >> 32);
          return SMP_OK;
        }
      }
      if (exact) {
        g = here;
        return move_exact(g, ms, v, range);
      }
    }
  }
  return move_exact(g, ms, v, range);
}

// generate_moves_helper (simulation.cpp:264-290) for one direction: move = round(max(0,
// normal(mean, sd))) for every bound LEF in index order, unbound ones get 0.
//
// The normals are variable-length (a ziggurat wedge takes a second draw, the tail takes
// exponentials), so the workers evaluate a window of T candidate starts at once: thread k runs the
// whole sampler as if a normal started at stream position rp + k.  The real starts form the chain
// s0 = 0, s(j+1) = s(j) + len(s(j)).  Each warp tabulates, for every lane it could be entered at, the
// number of normals starting inside it and where the chain leaves it; after one wsync every warp
// composes the tables of the warps before it and marks its starts.  A window serves about T normals, in stream order, to the next LEFs in index order.
template <bool SM>
__device__ __noinline__ u64 gen_moves_dir(u64 rp, const Arr<SM> mv, u32 n, const MoveSpec& spec) {
  const View<SM> c;
  const u32 T = c.T, w = threadIdx.x >> 5, lane = ln();
  const MoveSpec ms = spec;
  if (ms.constant) {
#pragma unroll 1
    for (u32 i = threadIdx.x; i < n; i += T) mv[i] = c.bep[i] == UNBOUND ? 0u : (u32)ms.move_int;
    wsync(c.T);
    return rp;
  }
  // items: the bound LEFs in index order (a compacted list only when some are unbound)
  u32 nb = n;
  bool unb = false;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += T) unb |= c.bep[i] == UNBOUND;
  const bool all = !wsync_or(c.T, unb);
  if (!all) {
    nb = 0;
    u32 buf = 0;
#pragma unroll 1
    for (u32 base = 0; base < n; base += T) {
      const u32 i = base + threadIdx.x;
      const bool need = i < n && c.bep[i] != UNBOUND;
      const Scan2 s = scan2<SM>(buf, need, false);
      buf ^= 1;
      if (i < n && !need) mv[i] = 0;
      if (need) c.tmp[nb + s.off0] = i;
      nb += s.total;
    }
    wsync(c.T);
  }
  const u32 DRY = 0x4000u;
  u32 t0 = 0;
#pragma unroll 1
  while (t0 < nb) {
    // warps of the window: those that serve the remaining normals, and one for longer ones
    const u32 W = min(T >> 5, (nb - t0 + 31) / 32 + 1), span = 32 * W;
    u32 v = 0, len = 1;
    bool range = false;
    int st = SMP_OK;
    unsigned dm = 0;
    u32 step = 0;
    if (w < W) {
    rng_ensure(rp, span + 64);
    RingSrc g{c.rmask, (u32)rp + threadIdx.x, (u32)rp + span + 64, 0};
    st = move_sample(g, ms, &v, &range);
    len = g.n;
    // Per entry lane: where the chain leaves the warp (32 + the lane it enters the next one at, or
    // DRY + the lane whose sampler ran dry) and how many normals start before that.  Almost every
    // normal takes one draw, so the chain only bends at the few lanes of dm, taken from the last.
    dm = __ballot_sync(FULL, st != SMP_OK || len != 1);
    step = st == SMP_OK ? lane + len : DRY;
    u32 leave = 32, cnt = 32 - lane;
#pragma unroll 1
    for (unsigned r = dm; r;) {
      const u32 d = 31 - __clz(r);
      r &= ~(1u << d);
      const u32 q = __shfl_sync(FULL, step, d);
      const u32 l2 = __shfl_sync(FULL, leave, q & 31u), c2 = __shfl_sync(FULL, cnt, q & 31u);
      if (lane <= d) {
        leave = q == DRY ? DRY + d : (q < 32 ? l2 : q);
        cnt = d - lane + (q == DRY ? 0u : (q < 32 ? c2 + 1 : 1u));
      }
    }
    g_bt.tab[w][lane] = leave | (cnt << 16);
    }
    wsync(c.T);
    // Entry lane of every warp (lane k of each warp holds warp k's): all zero unless a normal straddles
    // two warps, so start there and repeat until the entries agree with the warps before.
    u32 e = 0, t = 0;
    bool odd = false;
#pragma unroll 1
    for (;;) {
      t = lane < W ? g_bt.tab[lane][e & 31u] : 32u;
      odd = lane < W && ((t & 0xFFFFu) >= 64 || e >= 32);
      u32 ne = __shfl_up_sync(FULL, (t & 0xFFFFu) - 32, 1);
      if (lane == 0) ne = 0;
      const bool same = lane >= W || ne == e;
      e = ne;
      if (__any_sync(FULL, odd) || __all_sync(FULL, same)) break;
    }
    u32 base, my_e, my_base, used;
    if (!__any_sync(FULL, odd)) {
      const u32 ex = warp_excl_scan(lane < W ? t >> 16 : 0u, &base);
      my_base = __shfl_sync(FULL, ex, w);
      my_e = w < W ? __shfl_sync(FULL, e, w) : 64u;
      used = span + __shfl_sync(FULL, (t & 0xFFFFu) - 32, W - 1);
    } else {
      // a normal of more than 32 draws or a dry sampler: follow the entries one by one
      u32 en = 0;
      bool dry = false;
      base = my_base = 0;
      my_e = 64;
      used = 0;
#pragma unroll 1
      for (u32 k = 0; k < W; ++k) {
        if (en >= 32) {
          en -= 32;
          continue;
        }
        if (k == w) {
          my_e = en;
          my_base = base;
        }
        const u32 v2 = g_bt.tab[k][en];
        base += v2 >> 16;
        const u32 q = v2 & 0xFFFFu;
        if (q & DRY) {
          dry = true;
          used = k * 32 + (q & 31u);  // the window ends before the sampler that ran dry
          break;
        }
        en = q - 32;
      }
      if (!dry) used = span + en;
    }
    const u32 served = min(base, nb - t0);
    if (my_e < 32) {
      u32 vis = 0;  // lanes a normal starts at
#pragma unroll 1
      for (u32 q = my_e; q < 32;) {
        const unsigned r = dm >> q << q;
        const u32 d = r ? (u32)(__ffs(r) - 1) : 31u;
        vis |= (0xFFFFFFFFu << q) & (0xFFFFFFFFu >> (31 - d));
        if (!r) break;
        q = __shfl_sync(FULL, step, d);
      }
      const u32 ord = my_base + __popc(vis & lanemask_lt());
      if (((vis >> lane) & 1u) && st == SMP_OK && ord < served) {
        if (range) set_status(g_c, DEV_ERR_MOVE_RANGE);
        mv[all ? t0 + ord : c.tmp[t0 + ord]] = v;
        if (ord == served - 1) g_bt.used = threadIdx.x + len;
      }
    }
    wsync(c.T);
    if (served == 0) {
      // the first normal needs more draws than the window holds: take it serially
      if (threadIdx.x == 0) {
        g_sc.rpos = rp;
        const double zz = s_unit_normal(g_c);
        const double d = round(fmax(0.0, zz * ms.sd + ms.mean));
        if (d > 4294967295.0) set_status(g_c, DEV_ERR_MOVE_RANGE);
        mv[all ? t0 : c.tmp[t0]] = (u32)(u64)d;
      }
      wsync(c.T);
      rp = g_sc.rpos;
      ++t0;
      continue;
    }
    if (served < base) used = g_bt.used;
    rp += used;
    rng_publish(rp);
    t0 += served;
  }
  wsync(c.T);
  return rp;
}

// adjust_moves_of_consecutive_extr_units (simulation.cpp:343-399).
// rev: with t_k = pos_k - move_k the reference goes down the ranks and sets T_k = min(t_k, T_{k+1} - 1)
// when the pair links (both bound, t_k > start, T_{k+1} > start), else T_k = t_k.  Every unit whose lower
// neighbour it pushes starts a walk down the ranks that carries its target, one less per rank, until a
// unit is clear of it; the walks meet in an atomic maximum of the moves, so each unit ends with the
// smallest target that reaches it.  Pushed units are few and their walks short, so almost all threads
// only compare two neighbours.  fwd units mirror this upwards.  A linked pair whose pushing target lies
// beyond the chromosome end is skipped by the reference: that rejects the result (serial restatement).
// out holds the moves in rank order.
template <class A>
__device__ __forceinline__ bool adjust_pushes(u32 dir, const A& S, const A& out, u32 k, u32 i) {
  // unit of rank k against the unit i it would push, on the moves before any push
  return dir ? (u64)S[k] + out[k] >= (u64)S[i] + out[i] : (i64)S[k] - out[k] <= (i64)S[i] - out[i];
}

template <bool SM>
__device__ __noinline__ bool adjust_walk(u32 dir, u32 n, u32 k, const Arr<SM> out) {
  const View<SM> c;
  const KParams& P = g_P;
  const auto R = dir ? c.fr : c.rr;
  const auto S = dir ? c.sf : c.sr;
  const auto M = dir ? c.fm : c.rm;  // the moves before any push
  const i64 lim = dir ? (i64)P.end - 1 : (i64)P.start;
  const u32 src = R[k];
  if (c.bep[src] == UNBOUND) return true;
  i64 T = dir ? (i64)pos64(S[k]) + M[src] : (i64)pos64(S[k]) - M[src];
#pragma unroll 1
  for (u32 i = dir ? k + 1 : k - 1; i < n; i += dir ? 1u : ~0u) {  // below rank 0 wraps past n
    const u32 u = R[i];
    if (c.bep[u] == UNBOUND) break;
    const i64 p = (i64)pos64(S[i]);
    const i64 t = dir ? p + M[u] : p - M[u];
    if (dir ? t > lim : t <= lim) break;
    if (dir ? T > lim : T <= lim) return false;
    if (dir ? T < t : T > t) break;
    T += dir ? 1 : -1;
    atomicMax(&out[i], (u32)(dir ? T - p : p - T));
  }
  return true;
}

// The walks of all units that push a neighbour.  Returns (to every worker) false when the result is rejected.
template <bool SM>
__device__ __noinline__ bool adjust_pushed(u32 n, const Arr<SM> out_r, const Arr<SM> out_f) {
  const View<SM> c;
  const Arr<SM> S[2] = {c.sr, c.sf}, out[2] = {out_r, out_f};
  bool bad = false;
  // 32 items per thread and direction at a time: a bit for each unit that pushes
#pragma unroll 1
  for (u32 base = 0; base < n; base += 32 * c.T) {
    u32 push[2] = {0, 0};
#pragma unroll
    for (u32 dir = 0; dir < 2; ++dir) {
      u32 b = 0;
#pragma unroll 1
      for (u32 k = base + threadIdx.x; b < 32 && k < n; k += c.T, ++b) {
        const bool end = dir ? k + 1 >= n : k == 0;
        if (!end && adjust_pushes(dir, S[dir], out[dir], k, dir ? k + 1 : k - 1)) push[dir] |= 1u << b;
      }
    }
    // comparisons before walks: a later group of a large cell compares moves already pushed, which only
    // adds sources whose own, unpushed targets stop at once
    if (wsync_or(c.T, (push[0] | push[1]) != 0)) {
#pragma unroll
      for (u32 dir = 0; dir < 2; ++dir) {
#pragma unroll 1
        for (u32 r = push[dir]; r; r &= r - 1)
          bad |= !adjust_walk<SM>(dir, n, base + threadIdx.x + (u32)(__ffs(r) - 1) * c.T, out[dir]);
      }
    }
  }
  return !wsync_or(c.T, bad);
}

// Ranked positions (sr, sf), adjusted and, with clamp, clamped moves (clamp_moves,
// simulation.cpp:325-340) in three sweeps; zeroes the collision words, one of whose arrays is its
// scratch: callers that keep the words restore them.
template <bool SM>
__device__ __noinline__ void place_moves(u32 n, bool clamp) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  const auto rr = c.rr;
  const auto fr = c.fr;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
  const auto rm = c.rm;
  const auto fm = c.fm;
  const auto out_r = c.tmp;
  const auto out_f = c.rc;
#pragma unroll 1
  for (u32 k = threadIdx.x; k < n; k += T) {
    const u32 ru = rr[k], fu = fr[k];
    c.sr[k] = rev[ru];
    c.sf[k] = fwd[fu];
    out_r[k] = rm[ru];
    out_f[k] = fm[fu];
  }
  wsync(c.T);
  const bool serial = (P.debug_flags & DBG_SERIAL_ADJUST) || !adjust_pushed<SM>(n, out_r, out_f);
  if (serial) {
    prof_add(PF_ADJUST_FALLBACK, 1);
    if (threadIdx.x == 0) {
      adjust_dir_serial(g_c, P, 0, n);
      adjust_dir_serial(g_c, P, 1, n);
    }
    wsync(c.T);
  }
  const u64 start = P.start, end = P.end;
#pragma unroll 1
  for (u32 k = threadIdx.x; k < n; k += T) {
    const u32 ru = rr[k], fu = fr[k];
    u64 mr = serial ? rm[ru] : out_r[k], mf = serial ? fm[fu] : out_f[k];
    if (clamp && c.bep[ru] != UNBOUND) mr = min(mr, pos64(c.sr[k]) - start);
    if (clamp && c.bep[fu] != UNBOUND) mf = min(mf, end - pos64(c.sf[k]) - 1);
    rm[ru] = (u32)mr;
    fm[fu] = (u32)mf;
    c.rc[k] = 0;
    c.fc[k] = 0;
  }
  wsync(c.T);
}

// clamp_moves (simulation.cpp:325-340)
template <bool SM>
__device__ __noinline__ void clamp_moves(u32 n) {
  const View<SM> c;
  const KParams& P = g_P;
  const auto bep = c.bep;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
  const auto rm = c.rm;
  const auto fm = c.fm;
  const u64 start = P.start, end = P.end;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    if (bep[i] == UNBOUND) continue;
    const u64 rmv = min((u64)rm[i], pos64(rev[i]) - start);
    const u64 fmv = min((u64)fm[i], end - pos64(fwd[i]) - 1);
    rm[i] = (u32)rmv;
    fm[i] = (u32)fmv;
  }
  wsync(c.T);
}

// ranked positions sorted (non-decreasing)?  Needed by the closed forms below; the epoch loop
// always satisfies it, caller-provided ranks may not.
template <bool SM>
__device__ __noinline__ bool ranked_sorted(u32 n) {
  const View<SM> c;
  bool bad = false;
#pragma unroll 1
  for (u32 k = threadIdx.x + 1; k < n; k += c.T) bad |= c.sr[k - 1] > c.sr[k] || c.sf[k - 1] > c.sf[k];
  return !wsync_or(c.T, bad);
}

// Bucket index over a sorted array of ranked positions (unbound units, UNBOUND, at the tail):
// T[b] = #{k : key[k] < start + (b << shift)} for b in [0, nbk], with shift chosen so that
// nbk + 1 <= n (about one key per bucket).  lower_bound(x) then starts from T[b(x)] and scans a
// few keys instead of a binary search over the whole array.
template <bool SM>
struct BucketIndex {
  Arr<SM> key, T;
  u32 n, start, shift, nbk;
  bool table;
};

// first k in [0, n) with key[k] >= x
template <bool SM>
__device__ __noinline__ u32 lower_bound(const BucketIndex<SM> ix, u32 x) {
  if (!ix.table) {  // n too small for a table
    u32 lo = 0, hi = ix.n;
#pragma unroll 1
    while (lo < hi) {
      const u32 mid = (lo + hi) >> 1;
      if (ix.key[mid] >= x) hi = mid; else lo = mid + 1;
    }
    return lo;
  }
  if (x <= ix.start) return 0;
  u32 k = ix.T[min((x - ix.start) >> ix.shift, ix.nbk)];
#pragma unroll 1
  while (k < ix.n && ix.key[k] < x) ++k;
  return k;
}

// Collective; T needs n entries.
template <bool SM>
__device__ __forceinline__ BucketIndex<SM> build_bucket_index(const Arr<SM> key, u32 n, u32 start, u32 end,
                                                               const Arr<SM> T) {
  const View<SM> c;
  BucketIndex<SM> ix{key, T, n, start, 0, 0, false};
  if (n < 8 || end <= start) return ix;
  const u32 range = end - start;
  // smallest shift with (range >> shift) + 2 <= n
  u32 shift = 0;
  {
    const int d = __clz(n - 2) - __clz(range);
    shift = d > 0 ? (u32)d : 0u;
    if (shift && (range >> (shift - 1)) + 2 <= n) --shift;
#pragma unroll 1
    while ((range >> shift) + 2 > n) ++shift;
  }
  const u32 nbk = range >> shift;
#pragma unroll 1
  for (u32 k = threadIdx.x; k <= n; k += c.T) {
    u32 bmin = 0, bmax = nbk;
    if (k > 0) {
      const u32 lo = key[k - 1];
      bmin = lo == UNBOUND ? nbk + 1 : ((lo - start) >> shift) + 1;
    }
    if (k < n) {
      const u32 hi = key[k];
      if (hi != UNBOUND) bmax = min(nbk, (hi - start) >> shift);
    }
#pragma unroll 1
    for (u32 b = bmin; b <= bmax; ++b) T[b] = k;
  }
  wsync(c.T);
  ix.table = true;
  ix.shift = shift;
  ix.nbk = nbk;
  return ix;
}

// Bernoulli trial of one thread with the draw at its offset (or none).
__device__ __forceinline__ bool trial_needs_draw(const Trial& t) { return !t.always && t.draws; }
__device__ __forceinline__ bool trial_outcome(const Trial& t, u64 u) {
  if (t.always) return true;
  if (!t.draws) return false;
  return u <= t.thr;
}

// detect_lef_bar_collisions (simulation_detect_collisions.cpp:128-252) for one direction.  For
// an occupied barrier the reference's sweep tests the first rev unit (in rank order, from
// index max(n5 - 1, 0)) strictly downstream of it and the last fwd unit strictly upstream of
// it (up to index n - max(n3 - 1, 0) - 1): searches over the ranked positions.  Trials draw in
// barrier order (ascending for rev units, descending for fwd units), and a unit hit by several
// barriers keeps the last successful one in that order: the largest barrier index for rev units,
// the smallest for fwd units, which an atomic maximum on the unit's word resolves.  Until the
// closing sweep of detect_lef_bar_block a hit is stored under an event code above every other
// (EV_HIT), fwd units with the complemented index.
constexpr u32 EV_HIT = EV_COLLISION | EV_CHROM_BOUNDARY | EV_LEF_BAR;

template <bool SM>
__device__ __noinline__ u64 detect_lef_bar_dir(u64 rp, u32 dir, u32 n, u32 n5, u32 n3) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  const auto R = dir ? c.fr : c.rr;
  const auto S = dir ? c.sf : c.sr;
  const auto bep = c.bep;
  const auto M = dir ? c.fm : c.rm;
  const auto C = dir ? c.fc : c.rc;
  // rev: first k >= j0 with S[k] > bpos; fwd: last k <= jtop with S[k] < bpos
  const u32 j0 = min(n5, n5 - 1);
  const u32 jtop = (n - min(n3, n3 - 1)) - 1;
  const BucketIndex<SM> ix = build_bucket_index<SM>(S, n, (u32)P.start, (u32)P.end, c.tmp);
  u32 buf = 0;
#pragma unroll 1
  for (u32 base = 0; base < c.nb; base += T) {
    rng_ensure(rp, T);
    const u32 o = base + threadIdx.x;
    bool cand = false, drawn = false;
    u32 bi = 0, unit = 0, ti = 0;
    if (o < c.nb) {
      const u32 i = dir ? c.nb - 1 - o : o;
      if (bar_active(c.bst, i)) {
        const uint2 pf = __ldg(&c.bpf[i]);
        u32 k = lower_bound<SM>(ix, dir ? pf.x : pf.x + 1);
        bool ok;
        if (dir == 0) {
          k = max(j0, k);
          ok = k < n;
        } else {
          k = min(jtop + 1, k);
          ok = k > 0;
          --k;
        }
        if (ok) {
          const u32 u = R[k], kpos = S[k];
          if (bep[u] != UNBOUND) {
            const u64 delta = dir ? (u64)pf.x - kpos : (u64)kpos - pf.x;
            if (delta > 0 && delta <= M[u]) {
              cand = true;
              bi = i;
              unit = u;
              ti = (pf.y & BF_DIR_MASK) == (dir ? MGPU_DIR_FWD : MGPU_DIR_REV) ? 0u : 1u;
              drawn = trial_needs_draw(P.lef_bar[ti]);
            }
          }
        }
      }
    }
    const Scan1 s = scan1<SM>(T, buf, drawn);
    rng_publish(rp);  // the draws of the windows before
    buf ^= 1;
    if (cand && trial_outcome(P.lef_bar[ti], drawn ? ring_at(c.rmask, rp + s.off) : 0))
      atomicMax(&C[unit], cw_make(dir ? CW_IDX_MASK - bi : bi, EV_HIT));
    rp += s.total;
  }
  wsync(c.T);
  rng_publish(rp);
  return rp;
}

template <bool SM>
__device__ __noinline__ u64 detect_lef_bar_block(u64 rp, u32 n, u32 n5, u32 n3) {
  const View<SM> c;
  rp = detect_lef_bar_dir<SM>(rp, 0, n, n5, n3);
  rp = detect_lef_bar_dir<SM>(rp, 1, n, n5, n3);
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    const u32 r = c.rc[i], f = c.fc[i];
    if (cw_event(r) == EV_HIT) c.rc[i] = cw_make(cw_idx(r), EV_COLLISION | EV_LEF_BAR);
    if (cw_event(f) == EV_HIT) c.fc[i] = cw_make(CW_IDX_MASK - cw_idx(f), EV_COLLISION | EV_LEF_BAR);
  }
  wsync(c.T);
  return rp;
}

// No caller-provided collision word uses the sweep's own code (the epoch loop writes none).
template <bool SM>
__device__ __noinline__ bool words_plain(u32 n) {
  const View<SM> c;
  bool bad = false;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) bad |= cw_event(c.rc[i]) == EV_HIT || cw_event(c.fc[i]) == EV_HIT;
  return !wsync_or(c.T, bad);
}

// detect_primary_lef_lef_collisions (simulation_detect_collisions.cpp:255-401).
// With cnt(j) = number of fwd units (rank < i2) strictly before rev unit j, the sweep tests
// exactly the rev units j >= n5 with cnt(j) > cnt(j - 1) (cnt(n5 - 1) := 0) and cnt(j) < i2,
// each against the fwd unit of rank cnt(j) - 1.  Tested pairs are disjoint, so their
// collision words are updated independently; trials draw in ascending j.
template <bool SM>
__device__ __noinline__ u64 detect_primary_block(u64 rp, u32 n, u32 n5, u32 n3) {
  const View<SM> c;
  const KParams& P = g_P;
  if (n5 == n || n3 == n) return rp;
  const u32 T = c.T;
  const u32 i2 = (n - min(n3, n3 - 1));
  // bucket index over the fwd ranked positions (this step can also run on its own)
  const BucketIndex<SM> ixf = build_bucket_index<SM>(c.sf, n, (u32)P.start, (u32)P.end, c.tmp);
  u32 buf = 0;
#pragma unroll 1
  for (u32 base = n5; base < n; base += T) {
    rng_ensure(rp, T);
    const u32 j = base + threadIdx.x;
    const bool valid = j < n;
    const u32 pr = valid ? c.sr[j] : 0u;
    u32 cnt = 0;
    if (valid) cnt = min(i2, lower_bound<SM>(ixf, pr));  // first i < i2 with sf[i] >= rev position
    u32 prev = __shfl_up_sync(FULL, cnt, 1);
    if (ln() == 0 && valid) prev = j == n5 ? 0u : min(i2, lower_bound<SM>(ixf, c.sr[j - 1]));
    bool cand = false, drawn = false;
    u32 ru = 0, fu = 0, pf = 0, rmv = 0, fmv = 0;
    if (valid && cnt > prev && cnt < i2) {
      ru = c.rr[j];
      fu = c.fr[cnt - 1];
      pf = c.sf[cnt - 1];
      rmv = c.rm[ru];
      fmv = c.fm[fu];
      const u64 delta = pos64(pr) - pos64(pf);
      cand = delta > 0 && delta < (u64)rmv + fmv;
      drawn = cand && trial_needs_draw(P.lef_lef);
    }
    const Scan1 sc = scan1<SM>(T, buf, drawn);
    rng_publish(rp);
    buf ^= 1;
    if (cand && trial_outcome(P.lef_lef, drawn ? ring_at(c.rmask, rp + sc.off) : 0))
      primary_pair_update(c, ru, fu, pos64(pr), pos64(pf), rmv, fmv);
    rp += sc.total;
  }
  wsync(c.T);
  rng_publish(rp);
  return rp;
}

// correct_moves_for_lef_bar_collisions (simulation_correct_moves.cpp:20-51)
template <bool SM>
__device__ __noinline__ void correct_lef_bar(u32 n) {
  const View<SM> c;
  const auto rc = c.rc;
  const auto fc = c.fc;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
  const auto rm = c.rm;
  const auto fm = c.fm;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    const u32 r = rc[i], f = fc[i];
    if (cw_occurred_as(r, EV_LEF_BAR)) rm[i] = (u32)(pos64(rev[i]) - bar_pos(c.bpf, cw_idx(r)) - 1);
    if (cw_occurred_as(f, EV_LEF_BAR)) fm[i] = (u32)(bar_pos(c.bpf, cw_idx(f)) - pos64(fwd[i]) - 1);
  }
  wsync(c.T);
}

// correct_moves_for_primary_lef_lef_collisions (simulation_correct_moves.cpp:54-122): the
// pairs it visits are disjoint, so both passes are parallel.
template <bool SM>
__device__ __noinline__ void correct_primary(u32 n) {
  const View<SM> c;
  // detect_primary pairs each fwd unit with at most one rev unit, so visiting the units in
  // index order instead of rank order changes nothing
#pragma unroll 1
  for (u32 rev_idx = threadIdx.x; rev_idx < n; rev_idx += c.T) {
    const u32 r = c.rc[rev_idx];
    if (!cw_occurred_as(r, EV_PRIMARY)) continue;
    const u32 fwd_idx = cw_idx(r);
    const u32 f = c.fc[fwd_idx];
    if (cw_occurred_as(f, EV_PRIMARY)) {
      const u64 rp = pos64(c.rev[rev_idx]), fp = pos64(c.fwd[fwd_idx]);
      u64 p1, p2;
      lef_lef_collision_pos(rp, fp, c.rm[rev_idx], c.fm[fwd_idx], p1, p2);
      c.rm[rev_idx] = (u32)(rp - p1);
      c.fm[fwd_idx] = (u32)(p2 - fp);
    } else if (cw_occurred_as(f, EV_LEF_BAR)) {
      c.rm[rev_idx] = (u32)(pos64(c.rev[rev_idx]) - (pos64(c.fwd[fwd_idx]) + c.fm[fwd_idx]) - 1);
    }
  }
  wsync(c.T);
#pragma unroll 1
  for (u32 fwd_idx = threadIdx.x; fwd_idx < n; fwd_idx += c.T) {
    const u32 f = c.fc[fwd_idx];
    if (!cw_occurred_as(f, EV_PRIMARY)) continue;
    const u32 rev_idx = cw_idx(f);
    if (cw_occurred_as(c.rc[rev_idx], EV_LEF_BAR)) {
      c.fm[fwd_idx] = (u32)((pos64(c.rev[rev_idx]) - c.rm[rev_idx]) - pos64(c.fwd[fwd_idx]) - 1);
    }
  }
  wsync(c.T);
}

// Both corrections in one sweep, as the epoch loop needs them: a pair's partner that a barrier stopped
// takes its corrected move from the barrier's position instead of waiting for it to be written, and of a
// primary pair the rev unit's thread writes both moves.
template <bool SM>
__device__ __noinline__ void correct_moves(u32 n) {
  const View<SM> c;
  const auto rc = c.rc;
  const auto fc = c.fc;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
  const auto rm = c.rm;
  const auto fm = c.fm;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    const u32 r = rc[i], f = fc[i];
    if (cw_occurred_as(r, EV_LEF_BAR)) {
      rm[i] = (u32)(pos64(rev[i]) - bar_pos(c.bpf, cw_idx(r)) - 1);
    } else if (cw_occurred_as(r, EV_PRIMARY)) {
      const u32 j = cw_idx(r);
      const u32 g = fc[j];
      if (cw_occurred_as(g, EV_PRIMARY)) {
        const u64 rp = pos64(rev[i]), fp = pos64(fwd[j]);
        u64 p1, p2;
        lef_lef_collision_pos(rp, fp, rm[i], fm[j], p1, p2);
        rm[i] = (u32)(rp - p1);
        fm[j] = (u32)(p2 - fp);
      } else if (cw_occurred_as(g, EV_LEF_BAR)) {
        const u32 mj = (u32)(bar_pos(c.bpf, cw_idx(g)) - pos64(fwd[j]) - 1);
        rm[i] = (u32)(pos64(rev[i]) - (pos64(fwd[j]) + mj) - 1);
      }
    }
    if (cw_occurred_as(f, EV_LEF_BAR)) {
      fm[i] = (u32)(bar_pos(c.bpf, cw_idx(f)) - pos64(fwd[i]) - 1);
    } else if (cw_occurred_as(f, EV_PRIMARY)) {
      const u32 j = cw_idx(f);
      const u32 g = rc[j];
      if (cw_occurred_as(g, EV_LEF_BAR)) {
        const u32 mj = (u32)(pos64(rev[j]) - bar_pos(c.bpf, cw_idx(g)) - 1);
        fm[i] = (u32)((pos64(rev[j]) - mj) - pos64(fwd[i]) - 1);
      }
    }
  }
  wsync(c.T);
}

// process_secondary_lef_lef_collisions (simulation_detect_collisions.cpp:404-518).
// A stalled unit followed (rev: in rank order; fwd: in reverse rank order) by free units
// starts a chain: each free unit whose target passes its stalled predecessor's target draws a
// bypass trial; success stalls it one bp behind (extending the chain), failure marks it
// avoided and ends the chain.  Chains lie between units that were stalled on entry, so they
// are disjoint and one thread walks one chain.  A chain of at most one trial always takes the
// same number of draws, so only a longer chain that fails before its last trial shifts the chains
// after it: one warp settles the offsets of all chains of a round from those few, then every
// chain is walked with its draws.
enum ChainMode { CHAIN_COUNT = 0, CHAIN_RING = 1, CHAIN_SERIAL = 2 };

template <int MODE, class C>
__device__ __forceinline__ u32 chain_walk(const C& c, const Trial& tr, u32 dir, u32 n, i64 k, u64 at) {
  const auto R = dir ? c.fr : c.rr;
  const auto M = dir ? c.fm : c.rm;
  const auto W = dir ? c.fc : c.rc;
  const auto S = dir ? c.sf : c.sr;
  const i64 step = dir ? -1 : 1;
  const i64 stop = dir ? -1 : (i64)n;
  u32 idx_prev = R[k - step];
  u64 tprev = dir ? pos64(S[k - step]) + M[idx_prev] : pos64(S[k - step]) - M[idx_prev];
  u32 trials = 0;
#pragma unroll 1
  for (; k != stop; k += step) {
    const u32 idx = R[k];
    if (cw_occurred(W[idx])) break;  // stalled on entry: the next chain starts after it
    const u64 p = pos64(S[k]);
    const u64 m = M[idx];
    if (!(dir ? (p + m >= tprev) : (p - m <= tprev))) break;
    bool ok;
    if (tr.always) {
      ok = true;
    } else if (!tr.draws) {
      ok = false;
    } else {
      u64 u = 0;
      if (MODE == CHAIN_RING) u = ring_at(c.rmask, at++);
      if (MODE == CHAIN_SERIAL) u = rng_serial(g_c);
      ok = MODE == CHAIN_COUNT || u <= tr.thr;
    }
    ++trials;
    if (!ok) {
      if (MODE != CHAIN_COUNT) W[idx] = cw_make(idx_prev, EV_SECONDARY);
      break;
    }
    const u64 mv = dir ? (tprev - p) : (p - tprev);
    const u64 m2 = min(mv, mv - 1);
    if (MODE != CHAIN_COUNT) {
      W[idx] = cw_make(idx_prev, EV_COLLISION | EV_SECONDARY);
      M[idx] = (u32)m2;
    }
    tprev = dir ? p + m2 : p - m2;
    idx_prev = idx;
  }
  return trials;
}

template <bool SM>
__device__ __noinline__ void chains_serial(u32 dir, u32 n, const Arr<SM> starts, u32 q0, u32 q1) {
  const View<SM> c;
#pragma unroll 1
  for (u32 q = q0; q < q1; ++q) chain_walk<CHAIN_SERIAL>(c, g_P.lef_lef, dir, n, starts[q], 0);
}

template <bool SM>
__device__ __noinline__ u64 secondary_dir_block(u64 rp, u32 dir, u32 n, u32 n5, u32 n3) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  const auto R = dir ? c.fr : c.rr;
  const auto C = dir ? c.fc : c.rc;
  // chain starts (index of the first free unit): rev: k in [max(1, n5), n) with R[k-1]
  // stalled and R[k] free, ascending; fwd: k = i - 1 for i in [1, itop] with R[i] stalled
  // and R[k] free, in descending i.  Each start pairs with its own stalled unit: at most n / 2.
  const auto starts = c.tmp;
  const i64 itop = (i64)(n - min(n3, n3 - 1)) - 1;
  const u32 k0 = max(1u, n5);
  const u32 items = dir ? (itop > 0 ? (u32)itop : 0u) : (n > k0 ? n - k0 : 0u);
  if (threadIdx.x == 0) g_bt.total = 0;
  u32 nst = 0, buf = 0;
#pragma unroll 1
  for (u32 base = 0; base < items; base += 2 * T) {
    bool st[2];
    u32 at[2];
#pragma unroll
    for (u32 h = 0; h < 2; ++h) {
      const u32 o = base + h * T + threadIdx.x;
      st[h] = false;
      at[h] = 0;
      if (o < items) {
        const u32 k = dir ? (u32)itop - o - 1 : k0 + o;      // the free unit
        const u32 kp = dir ? k + 1 : k - 1;                  // the stalled one
        st[h] = cw_occurred(C[R[kp]]) && !cw_occurred(C[R[k]]);
        at[h] = k;
      }
    }
    const Scan2 s = scan2<SM>(buf, st[0], st[1]);
    buf ^= 1;
    if (st[0]) starts[nst + s.off0] = at[0];
    if (st[1]) starts[nst + s.off1] = at[1];
    nst += s.total;
  }
  wsync(c.T);
  if (nst == 0) return rp;
  const auto lens = c.tmp + nst;  // trials of each chain if all succeed, then its first draw's offset
#pragma unroll 1
  for (u32 q = threadIdx.x; q < nst; q += T) {
    const u32 L = chain_walk<CHAIN_COUNT>(c, P.lef_lef, dir, n, starts[q], 0);
    lens[q] = L;
    atomicAdd(&g_bt.total, L);
  }
  wsync(c.T);
  const bool draws = trial_needs_draw(P.lef_lef);
  const u64 thr = P.lef_lef.thr;
  // draws of one round at most
  const u32 lim = min(min(c.lim, 32 * TRIAL_WORDS - 32), (g_bt.total + 31) & ~31u);
  u32 q0 = 0;
#pragma unroll 1
  while (q0 < nst) {
    // outcomes of the next lim draws as trials, one bit each
    if (draws) {
      rng_ensure(rp, lim);
#pragma unroll 1
      for (u32 k = threadIdx.x; k < lim; k += T) {  // whole warps: lim is a multiple of 32
        const unsigned m = __ballot_sync(FULL, ring_at(c.rmask, rp + k) <= thr);
        if (ln() == 0) g_bt.trial[k >> 5] = m;
      }
      wsync(c.T);
    }
    if (threadIdx.x < 32) {
      u32 off = 0, q = q0;
#pragma unroll 1
      for (; q < nst; q += 32) {
        const u32 ci = q + ln();
        const u32 L = ci < nst && draws ? lens[ci] : 0u;
        u32 tot;
        u32 o = off + warp_excl_scan(L, &tot);
        if (off + tot > lim) break;
        u32 fixed = 0;  // lanes whose offset is settled
#pragma unroll 1
        for (;;) {
          bool dev = false;
          u32 used = L;
          if (L >= 2 && ln() >= fixed) {
            // trials until the first failure: 32 outcomes from bit o, more only in a very long chain
            u32 k = 0;
#pragma unroll 1
            for (;;) {
              const u32 at = o + k;
              const u32 bits = ~__funnelshift_r(g_bt.trial[at >> 5], g_bt.trial[(at >> 5) + 1], at & 31u);
              const u32 f = bits ? (u32)(__ffs(bits) - 1) : 32u;
              k += f;
              if (f < 32 || k >= L) break;
            }
            used = min(L, k + 1);
            dev = used < L;
          }
          const unsigned dm = __ballot_sync(FULL, dev);
          if (!dm) break;
          const u32 f = (u32)(__ffs(dm) - 1);
          const u32 d = __shfl_sync(FULL, L - used, f);
          if (ln() > f) o -= d;
          tot -= d;
          fixed = f + 1;
        }
        if (ci < nst) lens[ci] = o;
        off += tot;
      }
      if (ln() == 0) {
        g_bt.qend = min(q, nst);
        g_bt.used = off;
      }
    }
    wsync(c.T);
    const u32 q1 = g_bt.qend, used = g_bt.used;
    if (q1 == q0) {
      // 32 chains that might outrun the ring: walk them one by one
      prof_add(PF_CHAIN_SERIAL, 1);
      const u32 qe = min(q0 + 32, nst);
      if (threadIdx.x == 0) chains_serial<SM>(dir, n, starts, q0, qe);
      wsync(c.T);
      rp = g_sc.rpos;
      q0 = qe;
      continue;
    }
#pragma unroll 1
    for (u32 q = q0 + threadIdx.x; q < q1; q += T)
      chain_walk<CHAIN_RING>(c, P.lef_lef, dir, n, starts[q], rp + lens[q]);
    rp += used;
    q0 = q1;
    wsync(c.T);
    rng_publish(rp);
  }
  wsync(c.T);
  return rp;
}

// fix_secondary_lef_lef_collisions: candidates (units marked avoided) are never
// adjacent in rank order (the unit before a rev candidate, after a fwd candidate, is stalled),
// so each is an independent swap of two neighbours.
template <bool SM>
__device__ __noinline__ bool fix_secondary_block(u32 n, u32 n5, u32 n3) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  const u32 k0 = max(1u, n5);
  const u32 naf = (n - min(n3, n3 - 1));
  if (threadIdx.x == 0) g_bt.nr = g_bt.nf = 0;
  wsync(c.T);
  // candidate ranks: rev [k0, n), fwd [0, naf - 1); rev list from the front of tmp, fwd list from its end
  const auto list = c.tmp;
  bool adj = false;
#pragma unroll 1
  for (u32 k = k0 + threadIdx.x; k < n; k += T) {
    if (!cw_avoided_as(c.rc[c.rr[k]], EV_SECONDARY)) continue;
    if (k > k0 && cw_avoided_as(c.rc[c.rr[k - 1]], EV_SECONDARY)) adj = true;
    const u32 s = atomicAdd(&g_bt.nr, 1u);
    if (s < n) list[s] = k;
  }
  wsync(c.T);
  const u32 nr = g_bt.nr;
#pragma unroll 1
  for (u32 k = threadIdx.x; k + 1 < naf; k += T) {
    if (!cw_avoided_as(c.fc[c.fr[k]], EV_SECONDARY)) continue;
    if (k > 0 && cw_avoided_as(c.fc[c.fr[k - 1]], EV_SECONDARY)) adj = true;
    const u32 s = atomicAdd(&g_bt.nf, 1u);
    if (nr + s < n) list[nr + s] = k;
  }
  if (wsync_or(c.T, adj)) return false;
  const u32 nf = g_bt.nf;
  if (nr + nf > n) return false;
#pragma unroll 1
  for (u32 t = threadIdx.x; t < nr; t += T) fix_rev_at(c, P.start, list[t]);
  wsync(c.T);
#pragma unroll 1
  for (u32 t = threadIdx.x; t < nf; t += T) fix_fwd_at(c, P.end, list[nr + t]);
  wsync(c.T);
  return true;
}

// process_collisions (simulation.cpp:925-955) in the reference's order.
// sorted_ranks: the ranked positions are known to be sorted (the epoch loop ranks them itself);
// otherwise (caller state) they are checked and unsorted ones take the serial restatement.
template <bool SM>
__device__ __noinline__ u64 process_collisions(u64 rp, u32 n, bool fix,
                                               bool sorted_ranks = false) {
  const View<SM> c;
  const KParams& P = g_P;
  const bool serial = (P.debug_flags & DBG_SERIAL_COLLISIONS) || !(sorted_ranks || (ranked_sorted<SM>(n) && words_plain<SM>(n)));
  if (threadIdx.x == 0) {
    u64 n5, n3;
    detect_boundaries_serial(c, P, n, n5, n3);
    g_sc.n5 = n5;
    g_sc.n3 = n3;
  }
  wsync(c.T);
  prof_mark(PF_BOUNDARIES);
  const u32 n5 = (u32)g_sc.n5, n3 = (u32)g_sc.n3;
  if (serial) {
    if (threadIdx.x == 0) {
      detect_lef_bar_serial(g_c, P, n, n5, n3);
      detect_primary_serial(g_c, P, n, n5, n3);
    }
    wsync(c.T);
    rp = g_sc.rpos;
  } else {
    rp = detect_lef_bar_block<SM>(rp, n, n5, n3);
    prof_mark(PF_LEF_BAR);
    rp = detect_primary_block<SM>(rp, n, n5, n3);
  }
  prof_mark(PF_PRIMARY);
  if (sorted_ranks) {
    correct_moves<SM>(n);
  } else {
    correct_lef_bar<SM>(n);
    correct_primary<SM>(n);
  }
  prof_mark(PF_CORRECT);
  if (serial) {
    if (threadIdx.x == 0) process_secondary_serial(g_c, P, n, n5, n3);
    wsync(c.T);
    rp = g_sc.rpos;
  } else {
    // chains read ranked positions; secondary moves only change moves and words
    rp = secondary_dir_block<SM>(rp, 0, n, n5, n3);
    rp = secondary_dir_block<SM>(rp, 1, n, n5, n3);
  }
  prof_mark(PF_SECONDARY);
  if (fix) {
    if (serial || !fix_secondary_block<SM>(n, n5, n3)) {
      prof_add(PF_FIX_FALLBACK, 1);
      if (threadIdx.x == 0) fix_secondary_serial(g_c, P, n, n5, n3);
      wsync(c.T);
    }
  }
  prof_mark(PF_FIX);
  return rp;
}

// extrude (simulation.cpp:489-512)
template <bool SM>
__device__ __noinline__ void extrude(u32 n) {
  const View<SM> c;
  const auto bep = c.bep;
  const auto rm = c.rm;
  const auto fm = c.fm;
  const auto rev = c.rev;
  const auto fwd = c.fwd;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    if (bep[i] == UNBOUND) continue;
    rev[i] -= rm[i];
    fwd[i] += fm[i];
  }
  wsync(c.T);
}

// release_lefs (simulation.cpp:544-592): one draw per bound LEF with p > 0; with move, after extrude
// (simulation.cpp:489-512) of the units that stay.  bt->released counts the released units (reset by
// the caller that wants it).
template <bool SM>
__device__ __noinline__ u64 release_lefs(u64 rp, u32 n, bool completed, bool move = false) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T;
  u32 buf = 0;
#pragma unroll 1
  for (u32 base = 0; base < n; base += T) {
    rng_ensure(rp, T);
    const u32 i = base + threadIdx.x;
    const bool bound = i < n && c.bep[i] != UNBOUND;
    u64 thr = 0;
    bool need = false;
    if (bound) {
      const u32 r = c.rc[i], f = c.fc[i];
      u32 nh = 0;
      if (cw_occurred_as(r, EV_LEF_BAR) && (bar_flags(c.bpf, cw_idx(r)) & BF_DIR_MASK) == MGPU_DIR_REV) ++nh;
      if (cw_occurred_as(f, EV_LEF_BAR) && (bar_flags(c.bpf, cw_idx(f)) & BF_DIR_MASK) == MGPU_DIR_FWD) ++nh;
      const Trial& tr = P.release[completed ? 1 : 0][nh];
      need = tr.draws;
      thr = tr.thr;
    }
    const Scan1 s = scan1<SM>(T, buf, need);
    rng_publish(rp);
    buf ^= 1;
    const bool rel = need && ring_at(c.rmask, rp + s.off) <= thr;
    if (rel) {
      c.rev[i] = UNBOUND;
      c.fwd[i] = UNBOUND;
      c.bep[i] = UNBOUND;
    } else if (move && bound) {
      c.rev[i] -= c.rm[i];
      c.fwd[i] += c.fm[i];
    }
    const unsigned m = __ballot_sync(FULL, rel);
    if (m && ln() == 0) atomicAdd(&g_bt.released, (u32)__popc(m));
    rp += s.total;
  }
  wsync(c.T);
  rng_publish(rp);
  return rp;
}

// Sum of n non-negative doubles with the rounding of the loop s = s + t[i], by one warp, in integers.
// While s stays inside one binade, adding t adds t rounded to a multiple of that binade's unit in the
// last place, unless t lies exactly halfway between two multiples (then the parity of s decides).
// So a group of terms adds as integers; a term that carries s out of the binade, or is an exact
// half, is added in double precision, and the group goes on after it.  (A loop of double additions
// waits about 60 cycles for each.)
__device__ __forceinline__ u64 ulp_multiple(double t, u32 e, bool* stop) {
  const u64 b = (u64)__double_as_longlong(t);
  const u32 te = (u32)(b >> 52);
  if (b == 0) return 0;
  if (te == 0 || te > e) {  // denormal, or above s
    *stop = true;
    return 0;
  }
  const u32 sh = e - te;
  const u64 m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  if (sh == 0) return m;
  if (sh > 53) return 0;  // below half a unit
  const u64 half = 1ull << (sh - 1), rem = m & (2 * half - 1);
  if (rem == half) *stop = true;
  return (m >> sh) + (rem > half ? 1 : 0);
}

template <bool SM>
__device__ __noinline__ double ordered_sum(u32 n) {
  const View<SM> c;
  const auto t = c.sr;
  const u32 lane = ln();
  const u64 MANT = 0xFFFFFFFFFFFFFull, TOP = 1ull << 53;
  double s = 0.0;
  u32 i = 0;
  if (n <= 64) {  // the first terms leave a binade each, so a short sum is cheaper as it stands (20 LEFs: 2,700 cycles)
#pragma unroll 1
    for (; i < n; ++i) s = s + __longlong_as_double((i64)t.at64(i));
    return s;
  }
#pragma unroll 1
  while (i < n) {
    u64 sb = (u64)__double_as_longlong(s);
    u32 e = (u32)(sb >> 52);
    // four terms per lane while none of them needs care
    const u32 cnt = min(n - i, 128u);
    {
      bool stop = e == 0;
      u64 part = 0;
#pragma unroll
      for (u32 h = 0; h < 4; ++h) {
        const u32 k = 32 * h + lane;
        if (k < cnt) part += ulp_multiple(__longlong_as_double((i64)t.at64(i + k)), e, &stop);
      }
      if (!__any_sync(FULL, stop)) {
        // part < 2^55: three partial sums of at most 21 bits per lane
        const u64 total = (u64)__reduce_add_sync(FULL, (u32)part & 0x1FFFFFu) +
                          ((u64)__reduce_add_sync(FULL, (u32)(part >> 21) & 0x1FFFFFu) << 21) +
                          ((u64)__reduce_add_sync(FULL, (u32)(part >> 42)) << 42);
        const u64 mant = (sb & MANT) | (1ull << 52);
        if (mant + total < TOP) {
          s = __longlong_as_double((i64)((sb & ~MANT) | ((mant + total) & MANT)));
          i += cnt;
          continue;
        }
      }
    }
#pragma unroll 1
    for (u32 k0 = 0; k0 < cnt; k0 += 32) {
      const u32 m = min(32u, cnt - k0);
      const double mine = lane < m ? __longlong_as_double((i64)t.at64(i + k0 + lane)) : 0.0;
      u32 from = 0;  // terms [from, m) of the 32 are still to be added
#pragma unroll 1
      while (from < m) {
        sb = (u64)__double_as_longlong(s);
        e = (u32)(sb >> 52);
        bool stop = false;
        u64 r = 0;
        if (lane >= from && lane < m) {
          r = ulp_multiple(mine, e, &stop);
          stop |= e == 0;
        }
        u64 x = r;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const u64 y = __shfl_up_sync(FULL, x, d);
          if ((int)lane >= d) x += y;
        }
        const u64 mant = (sb & MANT) | (1ull << 52);
        const unsigned bad = __ballot_sync(FULL, stop || (lane >= from && mant + x >= TOP));
        const u32 f = bad ? (u32)(__ffs(bad) - 1) : 31u;
        const u64 upto = __shfl_sync(FULL, bad ? x - r : x, f);
        if (e != 0) s = __longlong_as_double((i64)((sb & ~MANT) | ((mant + upto) & MANT)));
        if (!bad) break;
        s = s + __shfl_sync(FULL, mine, f);
        from = f + 1;
      }
    }
    i += cnt;
  }
  return s;
}

// compute_loop_size_stats + evaluate_burnin (simulation.cpp:957-1025).  Loop sizes are
// integers below 2^32, so the reference's double sum is exact and the mean is computed from an
// integer sum; the sum of squared deviations keeps the reference's left-to-right rounding
// (ordered_sum).
template <bool SM>
__device__ __noinline__ bool burnin_stats(u32 n) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 cap = P.hist_cap;
  if (n == 0) {
    if (threadIdx.x == 0) {
      g_sc.hist_size = 0;
      g_sc.hist_head = 0;
    }
    wsync(c.T);
    return false;
  }
  if (threadIdx.x == 0) g_bt.sum = 0;
  wsync(c.T);
  u64 part = 0;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) part += pos64(c.fwd[i]) - pos64(c.rev[i]);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(FULL, part, d);
  if (ln() == 0) atomicAdd((unsigned long long*)&g_bt.sum, (unsigned long long)part);
  wsync(c.T);
  const double mean = (double)g_bt.sum / (double)n;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    const double d = (double)(pos64(c.fwd[i]) - pos64(c.rev[i])) - mean;
    c.sr.at64(i) = (u64)__double_as_longlong(d * d);  // sr and sf are adjacent: n doubles
  }
  wsync(c.T);
  if (threadIdx.x < 32) {
    const double ssd = ordered_sum<SM>(n);
    if (ln() == 0) {
      const double sd = sqrt(ssd / (double)n);
      if (g_sc.hist_size == cap) {
        g_sc.hist_head = (g_sc.hist_head + 1) % cap;
        g_sc.hist_size--;
      }
      const u32 slot = (g_sc.hist_head + g_sc.hist_size) % cap;
      g_c.havg[slot] = mean;
      g_c.hcfx[slot] = sd / mean;
      g_sc.hist_size++;
    }
    __syncwarp();
    bool done = false;
    if (g_sc.hist_size == cap) {
      // evaluate_burnin's smoothed-dip ratio: window pairs (i1, i2) = (k + 1, k + 1 + w) for
      // k < cap - w - 1, one window per lane, each window summed in the reference's order
      const u32 w = P.smooth_w;
      const u32 head = g_sc.hist_head;
      auto ratio = [&](const double* d) {
        u32 nd = 0;
#pragma unroll 1
        for (u32 i1 = 1 + ln(); i1 + w < cap; i1 += 32) {
          const u32 i2 = i1 + w;
          double a1 = 0.0, a2 = 0.0;
          u32 k = head + i1 - 1;
          if (k >= cap) k -= cap;
#pragma unroll 1
          for (u32 t = 0; t < w; ++t) {
            a1 = a1 + d[k];
            if (++k == cap) k = 0;
          }
          k = head + i1;
          if (k >= cap) k -= cap;
#pragma unroll 1
          for (u32 t = 0; t < w; ++t) {
            a2 = a2 + d[k];
            if (++k == cap) k = 0;
          }
          const double n1 = a1 / (double)(i2 - i1), n2 = a2 / (double)(i2 - i1);
          nd += (n1 > n2) ? 1u : 0u;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nd += __shfl_xor_sync(FULL, nd, o);
        return (double)nd / (double)((u64)cap - w - nd);
      };
      const double r1 = ratio(g_c.hcfx);
      if (r1 >= 0.95 && r1 <= 1.05) {
        const double r2 = ratio(g_c.havg);
        done = r2 >= 0.95 && r2 <= 1.05;
      }
    }
    if (ln() == 0) g_bt.flag = done ? 1 : 0;
  }
  wsync(c.T);
  return g_bt.flag != 0;
}

// run_burnin (simulation.cpp:1027-1054)
template <bool SM>
__device__ __noinline__ u64 run_burnin(u64 rp) {
  const View<SM> c;
  const KParams& P = g_P;
#pragma unroll 1
  for (u64 it = 0; it < MGPU_ITER_LIMIT; ++it) {
    const bool active = g_sc.num_active == P.nlefs;
    wsync(c.T);  // thread 0 changes num_active below
    bool done = false;
    if (active) done = burnin_stats<SM>(P.nlefs);
    if (threadIdx.x == 0) {
      ++g_sc.num_burnin_epochs;
      if (!active) {
        const u64 k = s_poisson(g_c, P);
        g_sc.num_active = min(g_sc.num_active + k, (u64)P.nlefs);
      } else {
        done = done && (g_sc.epoch > P.min_burnin);
        if (!done && g_sc.epoch >= P.max_burnin) done = true;
        g_sc.burnin_completed = done ? 1 : 0;
      }
    }
    wsync(c.T);
    rp = g_sc.rpos;
    if (g_sc.num_active != 0) return rp;
  }
  if (threadIdx.x == 0) set_status(g_c, DEV_ERR_ITER_LIMIT);
  wsync(c.T);
  return rp;
}

// ContactMatrixDense::increment (contact_matrix_dense_safe_impl.hpp:52-87); returns whether
// the contact fell outside the band (missed update).
template <class C>
__device__ __forceinline__ bool band_increment(const C& c, const KParams& P, u64 row, u64 col) {
  u64 i, j;
  if (row > col) {
    i = row - col;
    j = row;
  } else {
    i = col - row;
    j = col;
  }
  if (i >= P.nrows) return true;
  if (c.band) atomicAdd(&c.band[j * P.nrows + i], 1u);
  return false;
}

// genextreme noise of one draw (register_contacts.cpp:48-64)
__device__ __noinline__ double gev_noise(u64 u) {
  const KParams& P = g_P;
  const double l = -log(canonical_of(u));
  if (P.gev_xi == 0.0) return (P.gev_mu - P.gev_sigma) * log(l);
  return P.gev_mu + (P.gev_sigma * (1.0 - pow(l, P.gev_xi))) / P.gev_xi;
}

// The same in fixed point, 2^-25 bp: n = base + scale * L * (e^y - 1) / y with L = ln(-ln u) and
// y = xi * L.  The positions that follow from it are only needed as whole base pairs, so the caller
// takes gev_noise when the fixed-point value is too close to one to tell.  CUDA's double log and pow
// take some 250 instructions on the FP64 pipe (1/64 of the FP32 rate); this takes about 110 integer
// ones.  Logarithms: x = c (1 + r) with |r| < 2^-8 from a table of 128 parts, and the series of
// ln(1 + r) to r^5; absolute error below 2^-44.  Error of n: |scale| * 2^-44 / -ln u, and the caller's
// margin is 2^-13 for |scale| < 2^15 and -ln u >= 2^-15.  Returns false outside that range.
__device__ __forceinline__ i64 ln_mantissa(u64 m) {  // m = x * 2^63, x in [1, 2): ln x * 2^63
  const ulonglong2 e = g_bt.ln[(m >> 56) & 127u];
  const i64 r = (i64)(__umul64hi(m, e.x) - (1ull << 63));
  const i32 r39 = (i32)(r >> 24), r32 = r39 >> 7;
  const i32 a = (1 << 30) - __mulhi(r32, 858993459);  // 1/4 - r/5
  const i32 b = 1431655765 - __mulhi(r32, a);         // 1/3 - r (..)
  const u32 q = (u32)((1 << 30) - (__mulhi(r32, b) >> 1));  // (1/2 - r (..)) * 2^31
  const u32 r2 = (u32)((u64)((i64)r39 * r39) >> 32);  // r^2 * 2^46
  return (i64)e.y + r - (i64)(((u64)r2 * q) >> 14);
}

__device__ __noinline__ bool gev_fixed(u64 u, i64* n) {
  const KParams& P = g_P;
  const u64 LN2_57 = 0x162E42FEFA39EF3ull;  // ln 2 * 2^57
  const u32 lz = u ? (u32)__clzll((i64)u) : 63u;
  const i64 e = (i64)((u64)(1 + lz) * LN2_57) - (ln_mantissa(u << lz) >> 6);
  if (u == 0 || e < (1ll << 42)) return false;
  const u32 lz2 = (u32)__clzll(e);
  const i64 L = (6 - (i64)lz2) * (i64)LN2_57 + (ln_mantissa((u64)e << lz2) >> 6);
  const bool neg = L < 0;
  const u64 aL = (u64)(neg ? -L : L);
  const u64 t = __umul64hi(aL, P.gev_scale);  // |scale L| * 2^25
  const u64 y = __umul64hi(aL, P.gev_xiq);    // |y| * 2^57
  const i64 half = (i64)(__umul64hi(t << 20, y) >> 14);  // |scale L| |y| / 2
  const bool yneg = neg != (P.gev_xi < 0.0f);
  const float yf = (float)(u32)(y >> 26) * 0x1p-31f, ys = yneg ? -yf : yf;
  const float tf = (float)(u32)(t >> 12) * 0x1p-13f;
  const float more = tf * (yf * yf * (1.0f / 6.0f + ys * (1.0f / 24.0f + ys * (1.0f / 120.0f))));
  const i64 mag = (i64)t + (yneg ? -half : half) + (i64)(i32)(more * 0x1p25f);
  *n = P.gev_base + (neg != (P.gev_scale_neg != 0) ? -mag : mag);
  return true;
}

// The whole base pairs that a contact's noised positions rev - noise(u1) and fwd + noise(u2) fall into.
__device__ __forceinline__ void noised_positions(u64 rev, u64 fwd, u64 u1, u64 u2, i64* ia, i64* ib) {
  i64 n1, n2;
  bool exact = !g_P.gev_fixed || !gev_fixed(u1, &n1) || !gev_fixed(u2, &n2);
  if (!exact) {
    const i64 a = ((i64)rev << 25) - n1, d = ((i64)fwd << 25) + n2;
    const u32 near = 1u << 12, one = 1u << 25;  // fractions within 2^-13 of a whole number
    exact = (((u32)a + near) & (one - 1)) <= 2 * near || (((u32)d + near) & (one - 1)) <= 2 * near;
    *ia = a >> 25;
    *ib = d >> 25;
  }
  if (exact) {
    // positions outside [0, 2^32) fail a contact's bounds in any case
    *ia = (i64)floor(fmin(fmax((double)rev - gev_noise(u1), -1.0), 4294967296.0));
    *ib = (i64)floor(fmin(fmax((double)fwd + gev_noise(u2), -1.0), 4294967296.0));
  }
}

// One contact attempt read from draws at `at` (register_contacts.cpp:129-198).  Returns the
// draws it takes; *ok tells whether it registers a contact; *regular is false when the attempt
// hit a bucket rejection (exact handling needs the serial path).
template <bool SM>
__device__ __forceinline__ u32 contact_attempt(u64 at, bool tad,
                                               u64 na, u64 lbucket, bool* ok, bool* regular,
                                               u64* row, u64* col) {
  const View<SM> c;
  const KParams& P = g_P;
  *ok = false;
  *regular = true;
  const u64 start = (u64)P.wstart + 1, end = (u64)P.wend - 1;
  u32 used = 0;
  const u64 li = div64(ring_at(c.rmask, at + used++), lbucket);
  if (li > na - 1) {
    *regular = false;
    return used;
  }
  if (c.bep[li] == UNBOUND) return used;
  const u64 rp = pos64(c.rev[li]), fp = pos64(c.fwd[li]);
  if (!(rp > start && rp < end && fp > start && fp < end)) return used;
  // whole base pairs of the two noised positions
  i64 ia = (i64)rp, ib = (i64)fp;
  if (P.noisify) {
    const u64 u1 = ring_at(c.rmask, at + used), u2 = ring_at(c.rmask, at + used + 1);
    used += 2;
    noised_positions(rp, fp, u1, u2, &ia, &ib);
  }
  const i64 p1 = min(ia, ib), p2 = max(ia, ib);
  if (!(p1 >= (i64)start && p2 < (i64)end)) return used;
  if (!tad) {
    *row = ((u32)p1 - (u32)start) / P.bin;
    *col = ((u32)p2 - (u32)start) / P.bin;
    *ok = true;
    return used;
  }
  const u64 q1 = (u64)p1, q2 = (u64)p2;
  const u64 range = q2 - q1;
  u64 p11 = q1, p22 = q1;
  if (range != 0) {
    const u64 bucket = bucket_of(range);
    const u64 r1 = div64(ring_at(c.rmask, at + used++), bucket);
    if (r1 > range) {
      *regular = false;
      return used;
    }
    const u64 r2 = div64(ring_at(c.rmask, at + used++), bucket);
    if (r2 > range) {
      *regular = false;
      return used;
    }
    p11 = q1 + r1;
    p22 = q1 + r2;
  }
  *row = ((u32)p11 - (u32)start) / P.bin;
  *col = ((u32)p22 - (u32)start) / P.bin;
  *ok = true;
  return used;
}

// Thread 0: one contact attempt with serial draws (the exact path for rejections).
// register_1d_lef_occupancy (register_contacts.cpp:200-232): one count in each of the two bins
__device__ __forceinline__ void occ_increment(const KParams& P, u64 i1, u64 i2) {
  if (!P.occ) return;
  if (i1 < P.occ_bins) atomicAdd(&P.occ[i1], 1ull);
  if (i2 < P.occ_bins) atomicAdd(&P.occ[i2], 1ull);
}

// One attempt of register_contacts_loop / _tad (register_contacts.cpp:129-198) or, with occ, of
// register_1d_lef_occupancy (the loop attempt with the 1D counters as its sink); thread 0.
__device__ __noinline__ void contact_attempt_serial(Cell& c, const KParams& P, bool tad, u64 na, bool* ok, bool* miss,
                                       bool occ = false) {
  *ok = false;
  *miss = false;
  const u64 start = (u64)P.wstart + 1, end = (u64)P.wend - 1;
  const u64 li = s_uniform_int(c, 0, na - 1);
  if (c.bep[li] == UNBOUND) return;
  const u64 rp = pos64(c.rev[li]), fp = pos64(c.fwd[li]);
  if (!(rp > start && rp < end && fp > start && fp < end)) return;
  const double n1 = P.noisify ? s_gev(c, P) : 0.0;
  const double a = (double)rp - n1;
  const double n2 = P.noisify ? s_gev(c, P) : 0.0;
  const double b = (double)fp + n2;
  const double p1 = fmin(a, b), p2 = fmax(a, b);
  if (!(p1 >= (double)start && p2 >= (double)start && p1 < (double)end && p2 < (double)end)) return;
  if (occ) {
    occ_increment(P, ((u64)p1 - start) / P.bin, ((u64)p2 - start) / P.bin);
  } else if (!tad) {
    *miss = band_increment(c, P, ((u64)p1 - start) / P.bin, ((u64)p2 - start) / P.bin);
  } else {
    const u64 p11 = s_uniform_int(c, (u64)p1, (u64)p2);
    const u64 p22 = s_uniform_int(c, (u64)p1, (u64)p2);
    *miss = band_increment(c, P, (p11 - start) / P.bin, (p22 - start) / P.bin);
  }
  *ok = true;
}

// sample_and_register_contacts (register_contacts.cpp:94-198): attempts are evaluated up to T at a
// time at the offsets they would have if each took the usual number of draws (1 for the LEF,
// 2 for the noise, 2 more for a TAD contact).  The workers commit up to the first attempt that
// took a different number (a LEF or position outside the bounds, a zero-width TAD range) and
// resume after it; an attempt that hit a uniform_int bucket rejection is redone serially.
template <bool SM>
__device__ __noinline__ u64 sample_contacts(u64 rp, u64 target) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 T = c.T, W = T >> 5, w = threadIdx.x >> 5, lane = ln();
  u64 num = P.spe;
  if (P.density_positive) num = min(num, target - g_sc.num_contacts);
  if (num == 0) return rp;
  if (threadIdx.x == 0) {
    u64 n_loop;
    if (P.ratio_mode == 0) {
      n_loop = num;
    } else if (P.ratio_mode == 1) {
      n_loop = 0;
    } else {
      n_loop = (u64)s_binomial(g_c, P, (i64)num, P.p_loop);
    }
    g_sc.bc0 = n_loop;
    g_bt.missed = 0;
  }
  wsync(c.T);
  rp = g_sc.rpos;
  const u64 n_loop = g_sc.bc0;
  const u64 na = g_sc.num_active;
  const u64 lbucket = bucket_of(na - 1);
  u64 budget = 1000 * num + 1000000;  // attempts before giving up (see DEV_ERR_NO_BOUND_LEF)
  u32 missed = 0;
  const int passes = P.track_occ ? 3 : 2;  // loop, TAD, then the 1D occupancy
#pragma unroll 1
  for (int pass = 0; pass < passes; ++pass) {
    const bool tad = pass == 1, occ = pass == 2;
    u64 todo = occ ? num : (tad ? num - n_loop : n_loop);
    const u32 nominal = 1 + (P.noisify ? 2 : 0) + (tad ? 2 : 0);
    const u32 most = min(T, c.lim / nominal);
#pragma unroll 1
    while (todo != 0) {
      if (budget < T) {
        if (threadIdx.x == 0) {
          rng_publish(rp);
          set_status(g_c, DEV_ERR_NO_BOUND_LEF);
        }
        wsync(c.T);
        return rp;
      }
      // a few attempts more than contacts are wanted, in whole warps
      const u32 active = (u32)min((u64)most, (u64)((todo + todo / 16 + 32) & ~31ull));
      budget -= active;
      rng_ensure(rp, active * nominal);
      bool ok = false, regular = true;
      u64 row = 0, col = 0;
      u32 used = nominal;
      if (threadIdx.x < active)
        used = contact_attempt<SM>(rp + (u64)threadIdx.x * nominal, tad, na, lbucket, &ok, &regular, &row, &col);
      const bool deviates = !regular || used != nominal;
      const unsigned dm = __ballot_sync(FULL, deviates), om = __ballot_sync(FULL, ok);
      const u32 fl = dm ? (u32)(__ffs(dm) - 1) : 0u;
      const u32 fu = __shfl_sync(FULL, used | (regular ? 0x80000000u : 0u), fl);
      if (lane == 0) {
        g_bt.dev[w] = dm;
        g_bt.okm[w] = om;
        g_bt.dus[w] = fu;
      }
      wsync(c.T);
      // first deviating attempt f, its draws, and the commit limit: attempts [0, lim) are exact
      const u32 myd = lane < W ? g_bt.dev[lane] : 0u;
      const unsigned dw = __ballot_sync(FULL, myd != 0);
      u32 f = active, f_used = nominal;
      bool f_regular = false;
      if (dw) {
        const u32 fw = (u32)(__ffs(dw) - 1);
        f = fw * 32 + (u32)(__ffs(__shfl_sync(FULL, myd, fw)) - 1);
        const u32 v = g_bt.dus[fw];
        f_used = v & 0x7FFFFFFFu;
        f_regular = (v & 0x80000000u) != 0;
      }
      u32 lim = f_regular ? f + 1 : f;
      // contacts among them; the todo-th success ends the pass
      u32 okw = lane < W ? g_bt.okm[lane] : 0u;
      if (lim <= lane * 32) okw = 0;
      else if (lim < lane * 32 + 32) okw &= (1u << (lim - lane * 32)) - 1u;
      u32 total;
      const u32 ex = warp_excl_scan(__popc(okw), &total);
      if ((u64)total >= todo) {
        const u32 want = (u32)todo;  // total <= T
        const unsigned hit = __ballot_sync(FULL, ex < want && ex + __popc(okw) >= want);
        const u32 hw = (u32)(__ffs(hit) - 1);
        unsigned mm = __shfl_sync(FULL, okw, hw);
        const u32 skip = want - 1 - __shfl_sync(FULL, ex, hw);
#pragma unroll 1
        for (u32 t = 0; t < skip; ++t) mm &= mm - 1;
        lim = hw * 32 + (u32)__ffs(mm);
        total = want;
      }
      if (ok && threadIdx.x < lim) {
        if (occ) {
          occ_increment(P, row, col);
        } else if (band_increment(c, P, row, col)) {
          ++missed;
        }
      }
      if (lim) rp += (u64)(lim - 1) * nominal + (lim - 1 == f ? f_used : nominal);
      todo -= total;
      wsync(c.T);  // the draws are read and bt may be written again
      rng_publish(rp);
      if (todo != 0 && lim == f && f < active) {
        // attempt f could not be evaluated from the ring: run it serially
        prof_add(PF_CONTACT_SERIAL, 1);
        if (threadIdx.x == 0) {
          bool sok, smiss;
          contact_attempt_serial(g_c, P, tad, na, &sok, &smiss, occ);
          g_sc.bc1 = sok ? 1 : 0;
          if (smiss) g_sc.missed++;
        }
        wsync(c.T);
        rp = g_sc.rpos;
        if (g_sc.bc1) todo -= 1;
        wsync(c.T);
      }
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) missed += __shfl_xor_sync(FULL, missed, d);
  if (lane == 0 && missed) atomicAdd(&g_bt.missed, missed);
  wsync(c.T);
  if (threadIdx.x == 0) {
    g_sc.missed += g_bt.missed;
    g_sc.num_contacts += num;
  }
  wsync(c.T);
  return rp;
}

// sample_and_register_contacts with serial draws (lane 0): the exact path behind the
// DBG_SERIAL_CONTACTS switch.
__device__ __noinline__ void sample_contacts_serial(Cell& c, const KParams& P, u64 target) {
  Scalars* sc = c.sc;
  u64 num = P.spe;
  if (P.density_positive) num = min(num, target - sc->num_contacts);
  if (num == 0) return;
  u64 n_loop;
  if (P.ratio_mode == 0) {
    n_loop = num;
  } else if (P.ratio_mode == 1) {
    n_loop = 0;
  } else {
    n_loop = (u64)s_binomial(c, P, (i64)num, P.p_loop);
  }
  u64 budget = 1000 * num + 1000000;
  const int passes = P.track_occ ? 3 : 2;  // loop, TAD, then the 1D occupancy
#pragma unroll 1
  for (int pass = 0; pass < passes; ++pass) {
    u64 todo = pass == 0 ? n_loop : (pass == 1 ? num - n_loop : num);
#pragma unroll 1
    while (todo != 0) {
      if (--budget == 0 || sc->status != DEV_OK) {
        set_status(c, DEV_ERR_NO_BOUND_LEF);
        return;
      }
      bool ok, miss;
      contact_attempt_serial(c, P, pass == 1, sc->num_active, &ok, &miss, pass == 2);
      if (miss) sc->missed++;
      if (ok) --todo;
    }
  }
  sc->num_contacts += num;
}

// ---------------------------------------------------------------------------------------
// Trace, cell setup and the epoch loop (simulation.cpp:1056-1152)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ u64 mix64(u64 z) {
  z ^= z >> 30;
  z *= 0xbf58476d1ce4e5b9ull;
  z ^= z >> 27;
  z *= 0x94d049bb133111ebull;
  z ^= z >> 31;
  return z;
}

// mgpu_state_digest of the cell's state, and the full arrays when requested.
template <bool SM>
__device__ __noinline__ void trace_record(const DevTrace& T, u64 rec) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 nl = P.nlefs;
  const bool full = rec < T.max_records;
  u64 part = 0;
  if (threadIdx.x == 0) g_bt.sum = 0;
  wsync(c.T);
#pragma unroll 1
  for (u32 i = threadIdx.x; i < nl; i += c.T) {
    const u64 v[9] = {pos64(c.rev[i]), pos64(c.fwd[i]), pos64(c.bep[i]), c.rr[i], c.fr[i],
                      c.rm[i], c.fm[i], cw_to_ref(c.rc[i]), cw_to_ref(c.fc[i])};
    u64 h = mix64((u64)i * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull);
#pragma unroll 1
    for (int k = 0; k < 9; ++k) h = mix64(h ^ v[k]);
    part += h;
    if (full) {
      const u64 o = rec * nl + i;
      if (T.rev_pos) T.rev_pos[o] = v[0];
      if (T.fwd_pos) T.fwd_pos[o] = v[1];
      if (T.binding_epoch) T.binding_epoch[o] = v[2];
      if (T.rev_rank) T.rev_rank[o] = v[3];
      if (T.fwd_rank) T.fwd_rank[o] = v[4];
      if (T.rev_move) T.rev_move[o] = v[5];
      if (T.fwd_move) T.fwd_move[o] = v[6];
      if (T.rev_collision) T.rev_collision[o] = v[7];
      if (T.fwd_collision) T.fwd_collision[o] = v[8];
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(FULL, part, off);
  if (ln() == 0) atomicAdd((unsigned long long*)&g_bt.sum, (unsigned long long)part);
  wsync(c.T);
  if (threadIdx.x == 0) {
      mgpu_trace_header h;
    h.epoch = g_sc.epoch;
    h.num_active_lefs = g_sc.num_active;
    h.burnin_completed = g_sc.burnin_completed;
    h.num_burnin_epochs = g_sc.num_burnin_epochs;
    h.num_contacts = g_sc.num_contacts;
    h.rng_draws = g_sc.rpos;
    h.n5prime = g_sc.n5;
    h.n3prime = g_sc.n3;
    h.digest = g_bt.sum;
    if (T.all_headers && rec < T.max_epochs) T.all_headers[rec] = h;
    if (full && T.headers) T.headers[rec] = h;
  }
  wsync(c.T);
}

// Lay out one cell: each per-LEF array, the barrier bits and the burn-in history either in dynamic
// shared memory behind the ring or in the block's global scratch slot, as the plan in g_P places them.
// Thread 0; the caller's barrier follows.
__device__ void carve(char* gslot, const DevChrom& ch, const ulonglong2* jt, u32* band) {
  if (threadIdx.x != 0) return;
  Cell& c = g_c;
  const KParams& P = g_P;
  const u32 workers = P.workers, pw = producer_warps(workers);
  c.sc = &g_sc;
  c.T = workers * 32;
  c.lim = pw * 32 * RNG_S;
  c.rmask = 2 * c.lim - 1;
  c.ring = reinterpret_cast<u64*>(dyn_smem);
  c.hcfx = reinterpret_cast<double*>((P.hist_smem ? dyn_smem : gslot) + P.hist_off);
  c.havg = c.hcfx + P.hist_cap;
  c.bst = reinterpret_cast<u32*>((P.bst_smem ? dyn_smem : gslot) + P.bst_off);
  c.bst_off = P.bst_off;
  u32** arr[NARR] = {&c.rev, &c.fwd, &c.rr, &c.fr, &c.rm, &c.fm, &c.rc, &c.fc, &c.sr, &c.sf, &c.tmp, &c.bep};
  for (u32 k = 0; k < NARR; ++k) {
    char* base = ((P.arr_smem >> k) & 1u) ? dyn_smem : gslot;
    *arr[k] = reinterpret_cast<u32*>(base + P.arr_off[k]);
    c.off[k] = P.arr_off[k];
  }
  c.all_smem = P.arr_smem == (1u << NARR) - 1 && P.bst_smem;
  c.bar = ch.barriers;
  c.bpf = ch.pos_flags;
  c.nb = ch.nbarriers;
  c.jt = jt + (u64)(pw - 1) * 2 * JUMP_TABLE_ENTRIES;
  c.band = band;
}

// Launch parameters into shared memory (the caller's barrier follows).
__device__ __forceinline__ void load_plan(const KParams& P) {
  const u32* src = reinterpret_cast<const u32*>(&P);
  u32* dst = reinterpret_cast<u32*>(&g_P);
  for (u32 w = threadIdx.x; w < sizeof(KParams) / 4; w += blockDim.x) dst[w] = src[w];
}

// The normal ziggurat's fixed-point layers (after the two jump tables) into the block's scratch.
__device__ __forceinline__ void load_layers(const ulonglong2* jt) {
#pragma unroll 1
  for (u32 i = threadIdx.x; i < 128; i += blockDim.x) {
    g_bt.zt[i] = jt[4 * JUMP_TABLE_ENTRIES + i];
    g_bt.ln[i] = jt[4 * JUMP_TABLE_ENTRIES + NORMAL_LAYERS + i];
    const double y0 = mgpu_zig_normal_y[i], y1 = mgpu_zig_normal_y[i + 1];
    g_bt.zy[i] = make_float2((float)y0, (float)(y1 - y0));
  }
}

__device__ __noinline__ void cell_reset(u64 seed) {
  Cell& c = g_c;
  const u32 nl = g_P.nlefs;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < nl; i += blockDim.x) {
    c.rev[i] = UNBOUND;
    c.fwd[i] = UNBOUND;
    c.bep[i] = UNBOUND;
    c.rr[i] = i;
    c.fr[i] = i;
    c.rm[i] = 0;
    c.fm[i] = 0;
    c.rc[i] = 0;
    c.fc[i] = 0;
  }
#pragma unroll 1
  for (u32 w = threadIdx.x; w < (c.nb + 31) / 32; w += blockDim.x) c.bst[w] = 0;
  if (threadIdx.x == 0) {
    Scalars* sc = &g_sc;
    u64 st = seed;  // SplitMix64 seeding (random.hpp:26-30)
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      u64 z = (st += 0x9e3779b97f4a7c15ull);
      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
      z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
      sc->canon[k] = z ^ (z >> 31);
    }
    sc->rpos = 0;
    sc->gpos = sc->rpub = 0;
    sc->stop = 0;
    sc->nrec = 0;
    sc->status = DEV_OK;
    sc->epoch = 0;
    sc->num_burnin_epochs = 0;
    sc->num_active = 0;
    sc->num_contacts = 0;
    sc->burnin_completed = 0;
    sc->missed = 0;
    sc->lef_epochs = 0;
    sc->sort_fallbacks = 0;
    sc->n5 = sc->n3 = 0;
    sc->hist_size = 0;
    sc->hist_head = 0;
    sc->bc0 = sc->bc1 = sc->bc2 = 0;
    sc->prof = g_P.prof;
  }
}

// Simulation::dump_stats (simulation.cpp:1166-1224): the epoch's model-state record, taken after
// extrude and before release_lefs; the loop-size mean is exact (an integer sum below 2^53).
// Warp 0; the caller's barrier follows.
template <bool SM>
__device__ __noinline__ void log_model_state(u32 n, u64 cell) {
  const View<SM> c;
  const KParams& P = g_P;
  if (!P.records || g_sc.nrec >= P.rec_max || threadIdx.x >= 32) return;
  u32 st_rev = 0, st_fwd = 0, st_both = 0, lb = 0, pri = 0, sec = 0;
  u64 loop = 0;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += 32) {
    const u32 r = c.rc[i], f = c.fc[i];
    const bool sr = cw_occurred(r), sf = cw_occurred(f);
    st_rev += sr;
    st_fwd += sf;
    st_both += sr && sf;
    lb += cw_occurred_as(r, EV_LEF_BAR) + cw_occurred_as(f, EV_LEF_BAR);
    pri += cw_occurred_as(r, EV_PRIMARY) + cw_occurred_as(f, EV_PRIMARY);
    sec += cw_occurred_as(r, EV_SECONDARY) + cw_occurred_as(f, EV_SECONDARY);
    loop += pos64(c.fwd[i]) - pos64(c.rev[i]);
  }
  u32 occ = 0;
#pragma unroll 1
  for (u32 w = threadIdx.x; w < (c.nb + 31) / 32; w += 32) occ += __popc(c.bst[w]);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    st_rev += __shfl_xor_sync(FULL, st_rev, d);
    st_fwd += __shfl_xor_sync(FULL, st_fwd, d);
    st_both += __shfl_xor_sync(FULL, st_both, d);
    lb += __shfl_xor_sync(FULL, lb, d);
    pri += __shfl_xor_sync(FULL, pri, d);
    sec += __shfl_xor_sync(FULL, sec, d);
    loop += __shfl_xor_sync(FULL, loop, d);
    occ += __shfl_xor_sync(FULL, occ, d);
  }
  if (ln() == 0) {
    mgpu_epoch_record* r = P.records + cell * P.rec_max + g_sc.nrec;
    r->epoch = g_sc.epoch;
    r->cell = cell;
    r->burnin = g_sc.burnin_completed ? 0 : 1;
    r->barriers_occupied = occ;
    r->nbarriers = c.nb;
    r->num_lefs = n;
    r->stalled_rev = st_rev;
    r->stalled_fwd = st_fwd;
    r->stalled_both = st_both;
    r->lef_bar = lb;
    r->lef_lef_primary = pri;
    r->lef_lef_secondary = sec;
    r->avg_loop_size = n ? (double)loop / (double)n : 0.0;
    g_sc.nrec++;
  }
  __syncwarp();
}

// The epoch loop of one cell (simulation.cpp:1056-1152), run by the worker threads.
template <bool SM>
__device__ __noinline__ void run_cell(u64 target, u64 target_epochs, const DevTrace* trace,
                                      mgpu_cell_stats* stats, u64 cell) {
  const View<SM> c;
  const KParams& P = g_P;
  const u32 nl = P.nlefs;
  u64 rp = barriers_init<SM>(0);
  if (P.skip_burnin && threadIdx.x == 0) {
    g_sc.num_active = nl;
    g_sc.burnin_completed = 1;
  }
  wsync(c.T);
#pragma unroll 1
  for (u64 guard = 0; guard < MGPU_ITER_LIMIT; ++guard) {
    const bool go = P.contact_mode ? (g_sc.num_contacts < target)
                                   : (g_sc.epoch - g_sc.num_burnin_epochs < target_epochs);
    if (!go) break;
    prof_mark(PF_COUNT);
    if (!g_sc.burnin_completed) rp = run_burnin<SM>(rp);
    prof_mark(PF_BURNIN);
    const u32 n = (u32)g_sc.num_active;
    const u32 epoch = (u32)g_sc.epoch;
    const bool completed = g_sc.burnin_completed != 0;
    if (threadIdx.x == 0) g_sc.lef_epochs += n;
    rp = bind_lefs<SM>(rp, n, epoch, 0, nullptr);
    prof_mark(PF_BIND);
    rank_lefs<SM>(n, epoch, epoch != 0);
    prof_mark(PF_RANK);
    if (completed) {
      if (P.debug_flags & DBG_SERIAL_CONTACTS) {
        if (threadIdx.x == 0) sample_contacts_serial(g_c, P, target);
        wsync(c.T);
        rp = g_sc.rpos;
      } else {
        rp = sample_contacts<SM>(rp, target);
      }
        prof_mark(PF_CONTACTS);
      if (target != 0 && g_sc.num_contacts >= target) {
        break;
      }
      if (g_sc.status != DEV_OK) break;
      wsync(c.T);  // no worker writes a status before all have read it
    }
    rp = gen_moves_dir<SM>(rp, c.rm, n, P.rev_move[completed]);
    rp = gen_moves_dir<SM>(rp, c.fm, n, P.fwd_move[completed]);
    prof_mark(PF_MOVES);
    place_moves<SM>(n, true);
    prof_mark(PF_ADJUST);
    rp = barriers_next<SM>(rp);
    prof_mark(PF_BARRIERS);
    rp = process_collisions<SM>(rp, n, true, true);
    if (P.log_state) {  // the record is taken between the two
      extrude<SM>(n);
      log_model_state<SM>(n, cell);
      wsync(c.T);
    }
    rp = release_lefs<SM>(rp, n, completed, !P.log_state);
    prof_mark(PF_EXTRUDE_RELEASE);
    if (trace) trace_record<SM>(*trace, g_sc.epoch);
    const bool failed = g_sc.status != DEV_OK;
    wsync(c.T);
    if (threadIdx.x == 0) g_sc.epoch++;
    wsync(c.T);
    prof_mark(PF_TRACE);
    prof_add(PF_EPOCHS, 1);
    if (failed) break;
  }
  if (threadIdx.x == 0) {
    if (P.rec_count) P.rec_count[cell] = g_sc.nrec;
    if (trace && trace->num_recorded) *trace->num_recorded = g_sc.epoch;
    if (stats) {
      stats->epochs = g_sc.epoch;
      stats->burnin_epochs = g_sc.num_burnin_epochs;
      stats->contacts = g_sc.num_contacts;
      stats->missed_updates = g_sc.missed;
      stats->lef_epochs = g_sc.lef_epochs;
      stats->rng_draws = rp;
      stats->sort_fallbacks = g_sc.sort_fallbacks;
      stats->status = g_sc.status;
    }
  }
}

// One cell on the whole block: reset, then the workers run the epoch loop while the producers
// generate its draws.
__device__ __forceinline__ void block_cell(const CellTask& task, u64 target_epochs, const DevTrace* trace,
                                           mgpu_cell_stats* stats, u64 cell) {
  cell_reset(task.seed);
  __syncthreads();
  if (threadIdx.x < g_c.T) {
    if (g_c.all_smem) {
      run_cell<true>(task.target_contacts, target_epochs, trace, stats, cell);
    } else {
      run_cell<false>(task.target_contacts, target_epochs, trace, stats, cell);
    }
    wsync(g_c.T);
    if (threadIdx.x == 0) st_release(&g_sc.stop, 1);
  } else {
    rng_produce(g_c);
  }
  __syncthreads();
}

// Next index of the launch's work queue, the same for the whole block.
__device__ __forceinline__ u32 next_cell(u32* work, u32* slot) {
  if (threadIdx.x == 0) *slot = atomicAdd(work, 1u);
  __syncthreads();
  const u32 cell = *slot;
  __syncthreads();
  return cell;
}

__global__ void __launch_bounds__(MAX_BLOCK_THREADS) simulate_kernel(const __grid_constant__ KParams P, DevChrom ch,
                                                                     const CellTask* tasks, u64 ncells,
                                                                     u64 target_epochs, u32* band, u64* missed,
                                                                     mgpu_cell_stats* stats,
                                                                     const __grid_constant__ DevTrace trace,
                                                                     u32 tracing, const ulonglong2* jt, u32* work,
                                                                     char* gscratch) {
  __shared__ u32 slot;
  load_layers(jt);
  load_plan(P);
  __syncthreads();
  carve(gscratch + (u64)blockIdx.x * P.slot_bytes, ch, jt, band);
  for (;;) {
    const u32 cell = next_cell(work, &slot);
    if (cell >= ncells) break;
    block_cell(tasks[cell], target_epochs, tracing ? &trace : nullptr, stats ? stats + cell : nullptr, cell);
    if (threadIdx.x == 0 && missed) atomicAdd((unsigned long long*)missed, (unsigned long long)g_sc.missed);
  }
}

// Batched persistent kernel: cells of many chromosomes or windows in one work queue.  Each
// task names its plan (parameters, layout, barrier track, band); a block copies the plan's
// parameters into shared memory when its next cell belongs to another plan than the last.
__global__ void __launch_bounds__(MAX_BLOCK_THREADS) simulate_batch_kernel(const BatchPlan* plans,
                                                                           const BatchTask* tasks, u64 ntasks,
                                                                           u64 slot_bytes, mgpu_cell_stats* stats,
                                                                           const ulonglong2* jt, u32* work,
                                                                           char* gscratch) {
  __shared__ u32 slot;
  load_layers(jt);
  u32 cur = 0xFFFFFFFFu;
  for (;;) {
    const u32 cell = next_cell(work, &slot);
    if (cell >= ntasks) break;
    const BatchTask t = tasks[cell];
    const BatchPlan& pl = plans[t.plan];
    if (t.plan != cur) {
      load_plan(pl.P);
      __syncthreads();
      carve(gscratch + (u64)blockIdx.x * slot_bytes, pl.ch, jt, pl.band);
      __syncthreads();
      cur = t.plan;
    }
    const CellTask ct{t.seed, t.target_contacts};
    block_cell(ct, pl.target_epochs, nullptr, stats ? stats + cell : nullptr, cell);
    if (threadIdx.x == 0 && pl.missed) atomicAdd(pl.missed, (unsigned long long)g_sc.missed);
  }
}

// One step of the epoch loop on the state in g_c (mgpu_run_phase).
template <bool SM>
__device__ __noinline__ void run_phase(int phase, u32 n, const u64* bind_mask, u64 epoch, bool completed,
                                       u32 partially_sorted, u32 init_ranks, u32 adjust) {
  const View<SM> c;
  const KParams& P = g_P;
  const bool fast = !(P.debug_flags & DBG_SERIAL_COLLISIONS);
  u64 rp = 0;
  switch (phase) {
    case MGPU_PHASE_BIND:
      rp = bind_lefs<SM>(rp, n, (u32)epoch, bind_mask ? 1 : 2, bind_mask);
      rank_lefs<SM>(n, (u32)epoch, epoch != 0);
      break;
    case MGPU_PHASE_RANK:
      if (init_ranks) {
#pragma unroll 1
        for (u32 i = threadIdx.x; i < n; i += c.T) {
          c.rr[i] = i;
          c.fr[i] = i;
        }
        wsync(c.T);
      }
      rank_lefs<SM>(n, (u32)epoch, partially_sorted != 0);
      break;
    case MGPU_PHASE_ADJUST_AND_CLAMP:
      place_moves<SM>(n, true);
      break;
    case MGPU_PHASE_GENERATE_MOVES:
      rp = gen_moves_dir<SM>(rp, c.rm, n, P.rev_move[completed]);
      rp = gen_moves_dir<SM>(rp, c.fm, n, P.fwd_move[completed]);
      if (adjust) place_moves<SM>(n, true);
      else clamp_moves<SM>(n);
      break;
    case MGPU_PHASE_PROCESS_COLLISIONS:
      gather_ranked<SM>(n);
      rp = process_collisions<SM>(rp, n, false);
      break;
    case MGPU_PHASE_FIX_SECONDARY:
      if (threadIdx.x == 0) fix_secondary_serial(g_c, P, n, 0, 0);
      break;
    case MGPU_PHASE_DETECT_LEF_BAR:
      gather_ranked<SM>(n);
      if (ranked_sorted<SM>(n) && words_plain<SM>(n) && fast) {
        rp = detect_lef_bar_block<SM>(rp, n, 0, 0);
      } else if (threadIdx.x == 0) {
        detect_lef_bar_serial(g_c, P, n, 0, 0);
      }
      break;
    case MGPU_PHASE_LEF_LEF:
      gather_ranked<SM>(n);
      if (ranked_sorted<SM>(n) && fast) {
        rp = detect_primary_block<SM>(rp, n, 0, 0);
        correct_primary<SM>(n);
        rp = secondary_dir_block<SM>(rp, 0, n, 0, 0);
        rp = secondary_dir_block<SM>(rp, 1, n, 0, 0);
      } else {
        if (threadIdx.x == 0) detect_primary_serial(g_c, P, n, 0, 0);
        wsync(c.T);
        correct_primary<SM>(n);
        if (threadIdx.x == 0) process_secondary_serial(g_c, P, n, 0, 0);
      }
      break;
    case MGPU_PHASE_DETECT_PRIMARY:
      gather_ranked<SM>(n);
      if (ranked_sorted<SM>(n) && fast) {
        rp = detect_primary_block<SM>(rp, n, 0, 0);
      } else if (threadIdx.x == 0) {
        detect_primary_serial(g_c, P, n, 0, 0);
      }
      break;
    case MGPU_PHASE_DETECT_BOUNDARIES:
      if (threadIdx.x == 0) {
        u64 n5, n3;
        detect_boundaries_serial(c, P, n, n5, n3);
        g_sc.n5 = n5;
        g_sc.n3 = n3;
      }
      break;
    case MGPU_PHASE_CORRECT_LEF_BAR:
      correct_lef_bar<SM>(n);
      break;
    case MGPU_PHASE_CORRECT_PRIMARY:
      correct_primary<SM>(n);
      break;
    case MGPU_PHASE_EXTRUDE:
      extrude<SM>(n);
      break;
    case MGPU_PHASE_RELEASE:
      rp = release_lefs<SM>(rp, n, completed);
      break;
    case MGPU_PHASE_BARRIER_NEXT:
      rp = barriers_next<SM>(rp);
      break;
    case MGPU_PHASE_BARRIER_INIT:
      rp = barriers_init<SM>(rp);
      break;
    default:
      break;
  }
  wsync(c.T);
}

// One step of the epoch loop on caller state (mgpu_run_phase).
__global__ void __launch_bounds__(MAX_BLOCK_THREADS) phase_kernel(const __grid_constant__ KParams P, DevChrom ch, int phase,
                                                   u32 n, u64* arrays, u64* bind_mask,
                                                   uint8_t* barrier_state, u64 epoch,
                                                   u32 burnin_completed, u32 partially_sorted,
                                                   u32 init_ranks, u32 adjust, u64* prng,
                                                   u64* outs, const ulonglong2* jt, char* gslot) {
  load_layers(jt);
  load_plan(P);
  __syncthreads();
  carve(gslot, ch, jt, nullptr);
  __syncthreads();
  Cell& c = g_c;
  u64* A[9];
#pragma unroll 1
  for (int k = 0; k < 9; ++k) A[k] = arrays + (u64)k * n;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += blockDim.x) {
    c.rev[i] = A[0][i] == ~0ull ? UNBOUND : (u32)A[0][i];
    c.fwd[i] = A[1][i] == ~0ull ? UNBOUND : (u32)A[1][i];
    c.bep[i] = A[2][i] == ~0ull ? UNBOUND : (u32)A[2][i];
    c.rr[i] = (u32)A[3][i];
    c.fr[i] = (u32)A[4][i];
    c.rm[i] = (u32)A[5][i];
    c.fm[i] = (u32)A[6][i];
    c.rc[i] = cw_from_ref(A[7][i]);
    c.fc[i] = cw_from_ref(A[8][i]);
  }
#pragma unroll 1
  for (u32 w = threadIdx.x; w < (c.nb + 31) / 32; w += blockDim.x) {
    u32 bits = 0;
#pragma unroll 1
    for (u32 b = 0; b < 32; ++b) {
      const u32 i = w * 32 + b;
      if (i < c.nb && barrier_state && barrier_state[i]) bits |= 1u << b;
    }
    c.bst[w] = bits;
  }
  u64 init_state[4];
#pragma unroll 1
  for (int k = 0; k < 4; ++k) init_state[k] = prng[k];
  if (threadIdx.x == 0) {
    Scalars* sc = &g_sc;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) sc->canon[k] = prng[k];
    sc->rpos = 0;
    sc->gpos = sc->rpub = 0;
    sc->stop = 0;
    sc->status = DEV_OK;
    sc->epoch = epoch;
    sc->num_active = n;
    sc->burnin_completed = burnin_completed;
    sc->sort_fallbacks = 0;
    sc->n5 = sc->n3 = 0;
    sc->prof = nullptr;
    g_bt.released = 0;
  }
  __syncthreads();
  if (threadIdx.x >= c.T) {
    rng_produce(g_c);
    return;
  }
  const bool completed = burnin_completed != 0;
  if (g_c.all_smem) {
    run_phase<true>(phase, n, bind_mask, epoch, completed, partially_sorted, init_ranks, adjust);
  } else {
    run_phase<false>(phase, n, bind_mask, epoch, completed, partially_sorted, init_ranks, adjust);
  }
  // rank_lefs uses the move arrays as scratch, place_moves the collision words: the caller's stay as they were
  const bool moves_kept = phase == MGPU_PHASE_BIND || phase == MGPU_PHASE_RANK;
  const bool words_kept = phase == MGPU_PHASE_ADJUST_AND_CLAMP || phase == MGPU_PHASE_GENERATE_MOVES;
#pragma unroll 1
  for (u32 i = threadIdx.x; i < n; i += c.T) {
    A[0][i] = pos64(c.rev[i]);
    A[1][i] = pos64(c.fwd[i]);
    A[2][i] = pos64(c.bep[i]);
    A[3][i] = c.rr[i];
    A[4][i] = c.fr[i];
    if (!moves_kept) {
      A[5][i] = c.rm[i];
      A[6][i] = c.fm[i];
    }
    if (!words_kept) {
      A[7][i] = cw_to_ref(c.rc[i]);
      A[8][i] = cw_to_ref(c.fc[i]);
    }
  }
#pragma unroll 1
  for (u32 i = threadIdx.x; i < c.nb; i += c.T) {
    if (barrier_state) barrier_state[i] = bar_active(c.bst, i) ? 1 : 0;
  }
  if (threadIdx.x == 0) {
    st_release(&c.sc->stop, 1);
    // the caller's PRNG advanced by exactly the number of draws consumed
    u64 st[4] = {init_state[0], init_state[1], init_state[2], init_state[3]};
#pragma unroll 1
    for (u64 k = 0; k < c.sc->rpos; ++k) xo_next(st);
#pragma unroll 1
    for (int k = 0; k < 4; ++k) prng[k] = st[k];
    outs[0] = c.sc->n5;
    outs[1] = c.sc->n3;
    outs[2] = g_bt.released;
    outs[3] = c.sc->status;
  }
}

// ---------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------
static int cuda_fail(cudaError_t e, const char* what, char* errbuf, int errlen) {
  if (e == cudaSuccess) return MGPU_OK;
  if (errbuf) snprintf(errbuf, errlen, "%s: %s", what, cudaGetErrorString(e));
  return MGPU_ERR_CUDA;
}

// Largest dynamic shared memory a block of either kernel may request: the device's opt-in
// limit minus the kernels' static shared memory.
u64 max_smem_per_block() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  u64 stat = 0;
  cudaFuncAttributes a{};
  if (cudaFuncGetAttributes(&a, simulate_kernel) == cudaSuccess) stat = a.sharedSizeBytes;
  if (cudaFuncGetAttributes(&a, phase_kernel) == cudaSuccess && a.sharedSizeBytes > stat) stat = a.sharedSizeBytes;
  if (cudaFuncGetAttributes(&a, simulate_batch_kernel) == cudaSuccess && a.sharedSizeBytes > stat)
    stat = a.sharedSizeBytes;
  cudaGetLastError();
  return (u64)v > stat ? (u64)v - stat : 0;
}

u64 resident_cells(const KParams& P, u64 ncells) {
  // tuning switches carried in the debug flags: bits 8-15 carveout percent, 16-23 cells per SM
  const u32 carveout = (P.debug_flags >> 8) & 0xFFu, max_per_sm = (P.debug_flags >> 16) & 0xFFu;
  cudaFuncSetAttribute(simulate_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                       carveout ? (int)carveout : -1);
  cudaGetLastError();
  // The attribute is a per-function permission shared by every thread and context of the
  // process, so it is always set to the device limit: lowering it for one launch would make a
  // concurrent launch with a larger plan fail.
  if (cudaFuncSetAttribute(simulate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)max_smem_per_block()) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, simulate_kernel, (int)block_threads(P.workers),
                                                    P.smem_bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (max_per_sm && per_sm > (int)max_per_sm) per_sm = (int)max_per_sm;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  u64 grid = (u64)sms * (u64)(per_sm > 0 ? per_sm : 1);
  return grid < ncells ? grid : ncells;
}

int launch_simulate(const KParams& P, const DevChrom& ch, const CellTask* tasks, u64 ncells,
                    u64 target_epochs, u32* band, u64* missed, mgpu_cell_stats* stats,
                    const DevTrace* trace, const void* jump_table, u32* work_counter,
                    char* gscratch, u64 gscratch_bytes, void* stream, char* errbuf, int errlen) {
  int rc = cuda_fail(cudaFuncSetAttribute(simulate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)max_smem_per_block()),
                     "cudaFuncSetAttribute", errbuf, errlen);
  if (rc) return rc;
  u64 grid = resident_cells(P, ncells);
  if (grid == 0) return MGPU_OK;
  if (P.slot_bytes && gscratch_bytes / P.slot_bytes < grid) grid = gscratch_bytes / P.slot_bytes;
  if (grid == 0) {
    if (errbuf) snprintf(errbuf, errlen, "global scratch too small for one cell");
    return MGPU_ERR_INTERNAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  rc = cuda_fail(cudaMemsetAsync(work_counter, 0, sizeof(u32), st), "memset", errbuf, errlen);
  if (rc) return rc;
  DevTrace tr{};
  u32 tracing = 0;
  if (trace) {
    tr = *trace;
    tracing = 1;
  }
  simulate_kernel<<<(unsigned)grid, block_threads(P.workers), P.smem_bytes, st>>>(P, ch, tasks, ncells, target_epochs, band,
                                                             missed, stats, tr, tracing,
                                                             (const ulonglong2*)jump_table, work_counter,
                                                             gscratch);
  return cuda_fail(cudaGetLastError(), "simulate_kernel launch", errbuf, errlen);
}

u64 resident_batch_cells(u32 workers, u32 smem_bytes, u64 ntasks, u32 carveout_pct, u32 max_per_sm) {
  if (cudaFuncSetAttribute(simulate_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)max_smem_per_block()) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  // shared memory / L1 split preference (a tuning switch; -1 lets the CUDA driver choose)
  cudaFuncSetAttribute(simulate_batch_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                       carveout_pct ? (int)carveout_pct : -1);
  cudaGetLastError();
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, simulate_batch_kernel, (int)block_threads(workers),
                                                    smem_bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (max_per_sm && per_sm > (int)max_per_sm) per_sm = (int)max_per_sm;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (max_per_sm && per_sm > (int)max_per_sm) per_sm = (int)max_per_sm;
  const u64 grid = (u64)sms * (u64)(per_sm > 0 ? per_sm : 1);
  return grid < ntasks ? grid : ntasks;
}

int launch_simulate_batch(const BatchPlan* plans, const BatchTask* tasks, u64 ntasks, u32 workers, u32 smem_bytes,
                          u64 slot_bytes, mgpu_cell_stats* stats, const void* jump_table, u32* work_counter,
                          char* gscratch, u64 gscratch_bytes, u32 carveout_pct, u32 max_per_sm, void* stream,
                          char* errbuf, int errlen) {
  u64 grid = resident_batch_cells(workers, smem_bytes, ntasks, carveout_pct, max_per_sm);
  if (grid == 0) return ntasks ? MGPU_ERR_CUDA : MGPU_OK;
  if (slot_bytes && gscratch_bytes / slot_bytes < grid) grid = gscratch_bytes / slot_bytes;
  if (grid == 0) {
    if (errbuf) snprintf(errbuf, errlen, "global scratch too small for one cell");
    return MGPU_ERR_INTERNAL;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc = cuda_fail(cudaMemsetAsync(work_counter, 0, sizeof(u32), st), "memset", errbuf, errlen);
  if (rc) return rc;
  simulate_batch_kernel<<<(unsigned)grid, block_threads(workers), smem_bytes, st>>>(plans, tasks, ntasks, slot_bytes, stats,
                                                                 (const ulonglong2*)jump_table, work_counter,
                                                                 gscratch);
  return cuda_fail(cudaGetLastError(), "simulate_batch_kernel launch", errbuf, errlen);
}

int launch_phase(const KParams& P, const DevChrom& ch, int phase, u64 n, u64* arrays,
                 u64* bind_mask, uint8_t* barrier_state, u64 epoch, u32 burnin_completed,
                 u32 partially_sorted, u32 init_ranks, u32 adjust, u64* prng_state, u64* outs,
                 const void* jump_table, char* gscratch, void* stream, char* errbuf, int errlen) {
  int rc = cuda_fail(cudaFuncSetAttribute(phase_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)max_smem_per_block()),
                     "cudaFuncSetAttribute", errbuf, errlen);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  phase_kernel<<<1, block_threads(P.workers), P.smem_bytes, st>>>(P, ch, phase, (u32)n, arrays, bind_mask, barrier_state, epoch,
                                            burnin_completed, partially_sorted, init_ranks, adjust,
                                            prng_state, outs, (const ulonglong2*)jump_table, gscratch);
  return cuda_fail(cudaGetLastError(), "phase_kernel launch", errbuf, errlen);
}

// ---------------------------------------------------------------------------------------
// Probes of the device's floating-point library (test hooks): the samplers of the epoch loop
// run on whole seeded streams, and the transcendental functions on caller arguments, so that
// the test-suite can compare them with the host's libm (glibc, the reference's) bit for bit.
// ---------------------------------------------------------------------------------------

// One block per stream (grid-stride): thread 0 draws `per` samples of one distribution from the
// Xoshiro256++ state states[4 s .. 4 s + 3] through the same serial samplers the epoch loop
// uses, writes them to out[s * per ..] and the number of raw draws taken to draws[s].
__global__ void __launch_bounds__(32) sampler_probe_kernel(const __grid_constant__ KParams P, int kind,
                                                           const u64* states, u64 nstreams, u64 per,
                                                           double a0, double a1, double* out, u64* draws) {
  __shared__ Scalars sc;
  constexpr u32 PROBE_RING = 16;
  __shared__ u64 ring[PROBE_RING];
  if (threadIdx.x != 0) return;
  for (u64 s = blockIdx.x; s < nstreams; s += gridDim.x) {
    Cell c{};
    c.sc = &sc;
    c.ring = ring;
    c.rmask = PROBE_RING - 1;
    sc.rpos = 0;
    sc.gpos = 0;
    sc.status = DEV_OK;
    sc.prof = nullptr;
    for (int k = 0; k < 4; ++k) sc.canon[k] = states[4 * s + k];
    for (u64 i = 0; i < per; ++i) {
      double v = 0.0;
      switch (kind) {
        case 0: v = s_unit_normal(c) * a1 + a0; break;
        case 1: v = s_unit_exponential(c); break;
        case 2: v = (double)s_poisson(c, P); break;
        case 3: v = (double)s_binomial(c, P, (i64)a0, a1); break;
        case 4: v = s_gev(c, P); break;
        default: break;
      }
      out[s * per + i] = v;
    }
    draws[s] = sc.status == DEV_OK ? sc.rpos : ~0ull;
  }
}

// The same for what the epoch's parallel steps evaluate themselves: kind 5 the moves of P.rev_move[0]
// (move_sample), kind 6 the whole base pairs of 2^31 - noise and 2^31 + noise in turn (noised_positions), one
// draw each.  A ring of the stream's draws in shared memory, as the producer warps keep one.
constexpr u32 PROBE_DRAWS = 512;
__global__ void __launch_bounds__(32) step_probe_kernel(const __grid_constant__ KParams P, int kind, const u64* states,
                                                        u64 nstreams, u64 per, double* out, u64* draws,
                                                        const ulonglong2* jt) {
  load_layers(jt);
  load_plan(P);
  __syncthreads();
  if (threadIdx.x != 0) return;
  u64* ring = reinterpret_cast<u64*>(dyn_smem);
  for (u64 s = blockIdx.x; s < nstreams; s += gridDim.x) {
    u64 st[4];
    for (int k = 0; k < 4; ++k) st[k] = states[4 * s + k];
    u64 pos = 0, filled = 0;
    bool ok = true;
    for (u64 i = 0; i < per; ++i) {
      for (; filled - pos < PROBE_DRAWS / 2; ++filled) ring[filled & (PROBE_DRAWS - 1)] = xo_next(st);
      double r = 0.0;
      if (kind == 5) {
        RingSrc g{PROBE_DRAWS - 1, (u32)pos, (u32)filled, 0};
        u32 v = 0;
        bool range = false;
        ok &= move_sample(g, g_P.rev_move[0], &v, &range) == SMP_OK;
        pos += g.n;
        r = range ? -1.0 : (double)v;
      } else {
        const u64 u = ring[pos & (PROBE_DRAWS - 1)];
        ++pos;
        i64 ia, ib;
        noised_positions(1ull << 31, 1ull << 31, u, u, &ia, &ib);
        r = (double)((i & 1) ? ib : ia);
      }
      out[s * per + i] = r;
    }
    draws[s] = ok ? pos : ~0ull;
  }
}

// out[i] = f(x[i], y[i]) for f = 0: log x, 1: exp x, 2: pow(x, y), 3: the GEV noise of
// register_contacts.cpp:48-64 from u = x (mu, sigma, xi), 4: below_exp(x, y) as 0 or 1.
__global__ void libm_probe_kernel(int kind, const double* x, const double* y, u64 n, double mu, double sigma,
                                  double xi, double* out) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    const double a = x[i];
    double r = 0.0;
    switch (kind) {
      case 0: r = log(a); break;
      case 1: r = exp(a); break;
      case 2: r = pow(a, y[i]); break;
      case 3: r = xi == 0.0 ? (mu - sigma) * log(-log(a)) : mu + (sigma * (1.0 - pow(-log(a), xi))) / xi; break;
      case 4: r = below_exp(a, y[i]) ? 1.0 : 0.0; break;
      default: break;
    }
    out[i] = r;
  }
}

int launch_sampler_probe(const KParams& P, int kind, const u64* states, u64 nstreams, u64 per, double a0,
                         double a1, double* out, u64* draws, void* stream, char* errbuf, int errlen) {
  if (nstreams == 0) return MGPU_OK;
  const u64 blocks = nstreams < 65535 ? nstreams : 65535;
  sampler_probe_kernel<<<(unsigned)blocks, 32, 0, (cudaStream_t)stream>>>(P, kind, states, nstreams, per, a0, a1,
                                                                          out, draws);
  return cuda_fail(cudaGetLastError(), "sampler_probe_kernel launch", errbuf, errlen);
}

int launch_step_probe(const KParams& P, int kind, const u64* states, u64 nstreams, u64 per, double* out, u64* draws,
                      const void* tables, void* stream, char* errbuf, int errlen) {
  if (nstreams == 0) return MGPU_OK;
  const u64 blocks = nstreams < 65535 ? nstreams : 65535;
  step_probe_kernel<<<(unsigned)blocks, 32, PROBE_DRAWS * sizeof(u64), (cudaStream_t)stream>>>(
      P, kind, states, nstreams, per, out, draws, (const ulonglong2*)tables);
  return cuda_fail(cudaGetLastError(), "step_probe_kernel launch", errbuf, errlen);
}

int launch_libm_probe(int kind, const double* x, const double* y, u64 n, double mu, double sigma, double xi,
                      double* out, void* stream, char* errbuf, int errlen) {
  if (n == 0) return MGPU_OK;
  const u64 blocks = (n + 255) / 256 < 152 * 16 ? (n + 255) / 256 : 152 * 16;
  libm_probe_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(kind, x, y, n, mu, sigma, xi, out);
  return cuda_fail(cudaGetLastError(), "libm_probe_kernel launch", errbuf, errlen);
}

// ---------------------------------------------------------------------------------------
// Fixed scratch of the allocation-free entry point (one array per device, part of the module)
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[MGPU_NOALLOC_SCRATCH_BYTES];

__global__ void pack_tasks_kernel(const u64* seeds, const u64* targets, u64 n, CellTask* tasks) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    tasks[i].seed = seeds[i];
    tasks[i].target_contacts = targets[i];
  }
}

int noalloc_scratch_address(void** ptr, char* errbuf, int errlen) {
  return cuda_fail(cudaGetSymbolAddress(ptr, g_noalloc_scratch), "cudaGetSymbolAddress", errbuf, errlen);
}

int launch_pack_tasks(const u64* seeds, const u64* targets, u64 n, CellTask* tasks, void* stream,
                      char* errbuf, int errlen) {
  if (n == 0) return MGPU_OK;
  const u64 blocks = (n + 255) / 256;
  pack_tasks_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(seeds, targets, n, tasks);
  return cuda_fail(cudaGetLastError(), "pack_tasks_kernel launch", errbuf, errlen);
}

}  // namespace mgpu

