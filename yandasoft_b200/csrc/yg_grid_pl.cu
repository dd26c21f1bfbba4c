// Plane-major gridding: k_grid_pl and its halo sum.
//
// GridKernel::grid (GridKernel.cc:57-97) over records ordered by tile, CF
// block, position in the tile and oversampling offset: consecutive samples
// then mostly share their footprint (4 to 6 samples per cell and CF plane on
// hour-long tracks at 5 to 10 s), so the running sums of a footprint live in
// registers while only the CF matrix changes from sample to sample.
#include <algorithm>
#include <atomic>

#include "yg_cf.h"
#include "yg_grid_pl.h"
#include "yg_internal.h"
#include "yg_ring.cuh"

namespace yg {

namespace {

struct GridPlArgs {
  const int4* items;
  const int4* rec;           // plane-major records
  const float2* svis;        // weighted visibilities, [sample][npol]
  int npol, pcf;
  const float2* cf;          // packed W x W matrices
  const long long* cfoff;    // per matrix: its first element
  int W, W2;
  int stride;                // elements from one matrix of a block to the next
  int fs;                    // matrices of a CF block
  int P;                     // padded tile side, T + 2 Smax
  int groups, nw;            // groups of nw tap warps (blockIdx.y: the part of the residues)
  int stage_bytes, nstages, block_bytes;
  int fetch_off;             // the producer's fetch area, from the ring on
  int item0;                 // first item of this launch
  float2* scratch;           // [item - item0][group] slots of P x P cells x NPOL
  long long slot;            // elements of a slot
  int pol0;
  DevError* err;
};

// groups that work on an item of n samples (a power of two up to groups):
// every group has a slot of its own to clear and to sum, so one is worth
// having for 128 samples and more
constexpr int kMaxGroups = 4;
__host__ __device__ __forceinline__ int item_groups(int n, int groups) {
  int g = 1;
  while (2 * g <= groups && n >= 256 * g) g *= 2;
  return g;
}

// a * b + c on both halves of a register pair (one issue slot)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}

// predicated vector reductions (no result) of 8 and 16 bytes
__device__ __forceinline__ void red2(float2* g, float2 v, bool go) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p red.global.add.v2.f32 [%0], {%1, %2};\n}\n" ::"l"(g),
               "f"(v.x), "f"(v.y), "r"(go ? 1u : 0u)
               : "memory");
}
__device__ __forceinline__ void red4(float2* g, float2 v, float2 w, bool go) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n @p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n}\n" ::"l"(g),
      "f"(v.x), "f"(v.y), "f"(w.x), "f"(w.y), "r"(go ? 1u : 0u)
      : "memory");
}

// Running sums of one footprint cell, NPOL polarisations.  Several
// polarisations share the swapped tap (-cy, cx); a single one keeps the sums
// of vx c and vy c apart until they leave the registers, which spares it.
template <int NPOL>
struct CellSum {
  float2 s[NPOL];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int p = 0; p < NPOL; ++p) s[p] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(const float4 (&v)[NPOL], float2 c) {
    const float2 cs = make_float2(-c.y, c.x);
#pragma unroll
    for (int p = 0; p < NPOL; ++p)
      s[p] = fma2(make_float2(v[p].x, v[p].y), c, fma2(make_float2(v[p].z, v[p].w), cs, s[p]));
  }
  // adds the sums to their cell where go is set and starts anew there
  // (predicated, not branched: the slots of a thread stay independent)
  __device__ __forceinline__ void flush(float2* g, bool go) {
#pragma unroll
    for (int p = 0; p < NPOL; p += 2) red4(g + p, s[p], s[p + 1], go);
  }
  __device__ __forceinline__ void restart(bool go) {
#pragma unroll
    for (int p = 0; p < NPOL; ++p) s[p] = go ? make_float2(0.f, 0.f) : s[p];
  }
};

template <>
struct CellSum<1> {
  float2 x, y;
  __device__ __forceinline__ void clear() { x = y = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void add(const float4 (&v)[1], float2 c) {
    x = fma2(make_float2(v[0].x, v[0].y), c, x);
    y = fma2(make_float2(v[0].z, v[0].w), c, y);
  }
  __device__ __forceinline__ void flush(float2* g, bool go) { red2(g, make_float2(x.x - y.y, x.y + y.x), go); }
  __device__ __forceinline__ void restart(bool go) {
    x = go ? make_float2(0.f, 0.f) : x;
    y = go ? make_float2(0.f, 0.f) : y;
  }
};

// copies of 4, 8 or 16 bytes from global to shared memory that the issuing
// thread waits for by groups
template <int N>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// What the producer fetches ahead: kAhead windows of 32 samples, each lane its
// own sample (records twice as far).
constexpr int kAhead = 3;

template <int NPOL>
struct Fetch {
  int4 rec[2 * kAhead][32];
  float2 vis[kAhead][32][NPOL];
  long long off[kAhead][32];                     // unstaged CF: first element of the sample's matrix
};

// The weighted visibilities in the cube's own order, a sample's polarisations
// together: each polarisation plane is read in coalesced runs and a sample's
// 8 npol bytes are written in one piece, so that the producers of k_grid_pl,
// who pick samples in sorted order, touch one sector per sample.  Their random
// reads of the cube itself (a sector per polarisation) took 6.6 ms of DRAM
// time for 4.4e7 samples x 4; this pass takes 0.5 ms and leaves 2.7.
template <int NPOL>
__global__ void __launch_bounds__(256) k_weigh_cube(VisArgs v, float2* __restrict__ out) {
  const unsigned n = (unsigned)(v.nrow * (long long)v.nchan);   // plans hold fewer than 2^31 samples
  const unsigned nr = (unsigned)v.nrow;
  const bool data = !v.psf && !v.pcf;
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    float pr = 1.f, pi = 0.f, m = 1.f;
    if (v.mfs || (v.delay && data)) {
      const unsigned chan = s / nr;
      if (v.mfs) m = v.mfs[chan];
      if (v.delay && data) phasor(v.freq[chan], v.delay[s - chan * nr], &pr, &pi);
    }
    float2 o[NPOL];
#pragma unroll
    for (int p = 0; p < NPOL; ++p) {
      const size_t i = s + (size_t)n * p;
      const float wt = v.noise ? noise_weight(v.noise[i].x) : 1.f;
      o[p] = weigh(v, data ? v.vis[i] : make_float2(0.f, 0.f), wt, pr, pi, m);
    }
    float2* d = out + (size_t)s * NPOL;
    if (NPOL % 2 == 0) {
#pragma unroll
      for (int p = 0; p < NPOL; p += 2)
        reinterpret_cast<float4*>(d)[p / 2] = make_float4(o[p].x, o[p].y, o[(p + 1) % NPOL].x, o[(p + 1) % NPOL].y);
    } else {
#pragma unroll
      for (int p = 0; p < NPOL; ++p) d[p] = o[p];
    }
  }
}

// One CTA per work item.  The CTA's tap warps form groups; a group takes whole
// segments (up to 32 samples of one CF block) in turn, and its nw warps share
// every sample's W x W taps: thread t owns the residues k = t + 32 nw q of the
// footprint, (x mod W, y mod W) = (k mod W, k / W) with W the exact CF width,
// so no lane works on padding beyond the last 32 nw SL - W^2 and no two threads
// of a group ever touch one cell.  Each slot's sums stay in registers while
// its cell stays the same (the producer marks runs of samples with one
// footprint, inside which there is nothing but CF loads and multiply-adds) and
// go to the group's slot of the scratch tile as one vector reduction when a
// sample moves the slot to another cell, and at the start of every segment: a
// crowded cell's thousands of samples come one after the other here, and sums
// of like terms round the same way each time (2e7 samples on 1024^2: 1.7e-5
// of the grid in one running sum, against 6e-6 of the CF-major order and
// 1.5e-7 in sums of at most 32).  A slot is touched by one thread per cell, in program
// order, so the sums are the same from run to run.  Moving is
// predicated, not branched: a step of one cell moves some lane of nearly every
// slot (with a branch per slot a run cost 1000 cycles more, 6 ms of 20).
//
// Bound by the latency of a sample's taps and of the moves at 8 to 16 tap
// warps per SM, then by L2 bandwidth where the taps come from there.  Per
// launch, before (k_grid with its gather and inverse permutation) and now with
// k_weigh_cube: 4.4e7 samples x 4, W 13: 42.6 -> 11.8 ms; 2.1e7 x 4, W 19:
// 70.4 -> 12.6; 1.6e6 x 1, W 49: 6.3 -> 4.3; 2.8e6 x 2, W 7: 2.5 -> 0.4.
//
// The last warp is the producer: it decodes the records, fetches the weighted
// visibilities of its samples (k_weigh_cube's) some windows ahead and fills
// the ring of segments; stage s belongs to the group that takes segment s
// (the ring depth is a multiple of the groups), which alone waits for it and
// releases it.  STAGED: a block of CF matrices (all oversampling offsets of a
// plane) is brought into shared memory by one bulk copy when every segment of
// the previous block is consumed.  Otherwise the taps are read through L1 / L2
// (grid_pl_block says when).
template <int NPOL, int SL, bool STAGED>
__global__ void __launch_bounds__(NPOL == 1 ? 416 : (SL <= 4 ? 288 : 256), NPOL == 1 ? 1 : 2)
    k_grid_pl(const __grid_constant__ GridPlArgs a) {
  // samples in flight per thread, as registers allow
  constexpr int UNROLL = NPOL == 4 && SL > 3 ? 1 : (NPOL == 1 && SL <= 4 ? 4 : 2);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const float2* block = reinterpret_cast<const float2*>(smem_raw);
  unsigned char* ring = smem_raw + (STAGED ? a.block_bytes : 0);
  const int SB = a.stage_bytes;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(ring + (size_t)a.nstages * SB);
  unsigned long long* empty = full + a.nstages;
  unsigned long long* blockbar = empty + a.nstages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntap = a.groups * a.nw;              // tap warps
  const int4 it = a.items[a.item0 + blockIdx.x];
  const int G = item_groups(it.z - it.y, a.groups);
  const int NST = a.nstages / G * G;
  float2* slots = a.scratch + (size_t)blockIdx.x * a.groups * a.slot;
  if (threadIdx.x == 0) {
    for (int q = 0; q < NST; ++q) {
      mbar_init(&full[q], 1);
      mbar_init(&empty[q], a.nw);
    }
    mbar_init(blockbar, 1);
    mbar_fence_init();
  }
  if (gridDim.y == 1) {   // (several parts share slots that are cleared beforehand)
    const long long n4 = G * a.slot / 2;
    float4* z = reinterpret_cast<float4*>(slots);
    for (long long i = threadIdx.x; i < n4; i += blockDim.x) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  const int W = a.W;
  if (warp == ntap) {
    // ---- producer
    const unsigned fm = 0xffffffffu;
    // coordinates below 2^16 (a record holds no more) divide exactly by W
    // through this reciprocal: the product is at least k for x = k W and below
    // k + 1 for x = k W + W - 1 (every x and W checked, W up to 1032)
    const float rW = __frcp_rn((float)W) * (1.f + 1e-6f);
    int seg = 0, cur = -1, nblock = 0, why = 1;
    bool ok = true;
    // The samples lie anywhere behind their records, a microsecond away: each
    // lane copies its own into shared memory kAhead windows ahead
    Fetch<NPOL>& f = *reinterpret_cast<Fetch<NPOL>*>(ring + a.fetch_off);
    auto fetch_rec = [&](int w) {
      const int i = it.y + 32 * w + lane;
      if (i < it.z) copy_async<16>(&f.rec[w % (2 * kAhead)][lane], a.rec + i);
    };
    auto fetch = [&](int w) {
      if (it.y + 32 * w + lane >= it.z) return;
      const int k = w % kAhead;
      const int4 r = f.rec[w % (2 * kAhead)][lane];
      if (!STAGED) copy_async<8>(&f.off[k][lane], a.cfoff + r.z);
      const float2* src = a.svis + (size_t)(unsigned)r.w * a.npol + a.pol0;
      copy_async<NPOL == 1 ? 8 : 16>(&f.vis[k][lane][0], src);
      if (NPOL == 4) copy_async<16>(&f.vis[k][lane][NPOL / 2], src + 2);
    };
    auto acquire = [&](int stage) -> bool {
      bool okw = true;
      if (seg >= NST && lane == 0) okw = mbar_wait(&empty[stage], (unsigned)((seg / NST) - 1) & 1u);
      return __shfl_sync(fm, okw ? 1 : 0, 0) != 0;
    };
    const int nwin_all = (it.z - it.y + 31) / 32;
    for (int w = 0; w < 2 * kAhead; ++w) fetch_rec(w);
    copy_commit();
    copy_wait<0>();
    for (int w = 0; w < kAhead; ++w) {
      fetch(w);
      copy_commit();
    }
    for (int w = 0; w < nwin_all && ok; ++w) {
      // the groups of the last kAhead - 1 windows may still be on their way
      copy_wait<kAhead - 1>();
      const int base = it.y + 32 * w, k = w % kAhead;
      const int nwin = min(32, it.z - base);
      const int4 r = lane < nwin ? f.rec[w % (2 * kAhead)][lane] : make_int4(-1, 0, -1, -1);
      const int blk = r.z >= 0 ? r.z / a.fs : -1;
      const int px0 = r.x & 0xffff, py0 = (r.x >> 16) & 0xffff;
      // segments start where the CF block changes, runs where the footprint does
      const int bprev = __shfl_up_sync(fm, blk, 1), xprev = __shfl_up_sync(fm, r.x, 1);
      const unsigned heads0 = __ballot_sync(fm, lane < nwin && (lane == 0 || (STAGED && bprev != blk)));
      const unsigned runs = __ballot_sync(fm, lane == 0 || xprev != r.x) | heads0;
      unsigned heads = heads0;
      while (heads) {
        const int h = __ffs(heads) - 1;
        const unsigned rest = heads & (heads - 1);
        const int h2 = rest ? __ffs(rest) - 1 : nwin;
        heads = rest;
        const int stage = seg % NST;
        if (!acquire(stage)) {
          ok = false;
          break;
        }
        unsigned char* sp = ring + (size_t)stage * SB;
        if (lane >= h && lane < h2) {
          const unsigned after = lane < 31 ? runs >> (lane + 1) : 0u;
          const int end = min(h2, after ? lane + __ffs(after) : 32);
          reinterpret_cast<int4*>(sp)[lane - h] =
              make_int4(px0 + a.P * py0,
                        (px0 - W * (int)((float)px0 * rW)) | ((py0 - W * (int)((float)py0 * rW)) << 16),
                        STAGED ? (r.z - blk * a.fs) * a.stride : (int)f.off[k][lane], end - lane);
          // (vx, vx, vy, vy) per polarisation: the multipliers of (cx, cy) and
          // (-cy, cx); the preconditioner's conjugate CF half negates the
          // imaginary multiplier (its values are real)
          const bool conj = a.pcf && r.y < 0;
          float4* vs = reinterpret_cast<float4*>(sp + kSeg * 16);
#pragma unroll
          for (int p = 0; p < NPOL; ++p) {
            const float2 x = f.vis[k][lane][p];
            vs[(lane - h) * NPOL + p] = make_float4(x.x, conj ? -x.x : x.x, x.y, x.y);
          }
        }
        const int b = __shfl_sync(fm, blk, h);
        bool okp = true;
        if (STAGED && b != cur) {
          // the block buffer is free once every group has consumed its last segment
          if (lane == 0) {
            for (int q = 1; q <= G && q <= seg && okp; ++q)
              okp = mbar_wait(&empty[(seg - q) % NST], (unsigned)((seg - q) / NST) & 1u);
            if (okp) {
              const unsigned bytes = (unsigned)a.fs * a.stride * (unsigned)sizeof(float2);
              fence_proxy_async_smem();
              mbar_expect_tx(blockbar, bytes);
              bulk_g2s(smem_raw, a.cf + a.cfoff[(size_t)b * a.fs], bytes, blockbar);
            }
          }
          okp = __shfl_sync(fm, okp ? 1 : 0, 0) != 0;
          if (!okp) {
            ok = false;
            why = 3;
            break;
          }
          cur = b;
          ++nblock;
        }
        if (lane == 0) {
          int* hdr = reinterpret_cast<int*>(sp + SB - 16);
          hdr[0] = h2 - h;
          hdr[1] = nblock - 1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[stage]);
        ++seg;
      }
      fetch(w + kAhead);
      fetch_rec(w + 2 * kAhead);
      copy_commit();
    }
    copy_wait<0>();
    // one terminal segment per group
    for (int q = 0; q < G && ok; ++q) {
      const int stage = seg % NST;
      ok = acquire(stage);
      if (ok && lane == 0) {
        reinterpret_cast<int*>(ring + (size_t)stage * SB + SB - 16)[0] = -1;
        mbar_arrive(&full[stage]);
      }
      ++seg;
    }
    if (!ok && lane == 0) {
      raise_error(a.err, YG_ERR_TIMEOUT, timeout_where(2, why, seg, blockIdx.x));
      // no copy may be in flight when the CTA exits
      if (STAGED && nblock > 0) mbar_wait(blockbar, (unsigned)(nblock - 1) & 1u);
    }
  } else if (warp / a.nw < G) {
    // ---- tap warps
    const int g = warp / a.nw;
    const int nthr = 32 * a.nw;
    const int t = threadIdx.x - g * nthr;
    float2* tile = slots + (size_t)g * a.slot;
    // per slot: its residue (x | y << 16) and the cell of its running sums, the
    // one cell of the residue class inside the current footprint
    int res[SL], cell[SL];
    CellSum<NPOL> acc[SL];
    int nlive = 0;                                // slots below W^2
#pragma unroll
    for (int q = 0; q < SL; ++q) {
      const int k = (blockIdx.y * SL + q) * nthr + t;
      nlive += k < a.W2 ? 1 : 0;
      const int rx = (k < a.W2 ? k : 0) % W, ry = (k < a.W2 ? k : 0) / W;
      res[q] = rx | (ry << 16);
      cell[q] = rx + a.P * ry;
      acc[q].clear();
    }
    int cur = -1;
    for (int seg = g;; seg += G) {
      const int stage = seg % NST;
      if (!mbar_wait(&full[stage], (unsigned)(seg / NST) & 1u)) {
        if (lane == 0) raise_error(a.err, YG_ERR_TIMEOUT, timeout_where(2, 2, seg, blockIdx.x));
        break;
      }
      const unsigned char* sp = ring + (size_t)stage * SB;
      const int cnt = reinterpret_cast<const volatile int*>(sp + SB - 16)[0];
      if (cnt < 0) break;
      if (STAGED) {
        const int nb = reinterpret_cast<const volatile int*>(sp + SB - 16)[1];
        if (nb != cur) {
          if (!mbar_wait(blockbar, (unsigned)nb & 1u)) {
            if (lane == 0) raise_error(a.err, YG_ERR_TIMEOUT, timeout_where(2, 2, seg, blockIdx.x));
            break;
          }
          cur = nb;
        }
      }
      const int4* __restrict__ recs = reinterpret_cast<const int4*>(sp);
      const float4* __restrict__ vs = reinterpret_cast<const float4*>(sp + kSeg * 16);
      const float2* __restrict__ cfb = STAGED ? block : a.cf;
      int l = 0;
      while (l < cnt) {
        const int4 r = recs[l];
        const int mx = r.y & 0xffff, my = r.y >> 16;
        int tap[SL];
#pragma unroll
        for (int q = 0; q < SL; ++q) {
          int jx = (res[q] & 0xffff) - mx, jy = (res[q] >> 16) - my;
          jx += jx < 0 ? W : 0;
          jy += jy < 0 ? W : 0;
          tap[q] = jx + W * jy;
          const int now = r.x + jx + a.P * jy;
          const bool moved = now != cell[q] || l == 0;
          acc[q].flush(tile + cell[q] * NPOL, moved && q < nlive);
          acc[q].restart(moved);
          cell[q] = now;
        }
        const int end = l + r.w;
#pragma unroll(UNROLL)
        for (; l < end; ++l) {
          const float2* __restrict__ cm = cfb + recs[l].z;
          float4 vv[NPOL];
#pragma unroll
          for (int p = 0; p < NPOL; ++p) vv[p] = vs[l * NPOL + p];
          float2 c[SL];
#pragma unroll
          for (int q = 0; q < SL; ++q) c[q] = STAGED ? cm[tap[q]] : __ldg(cm + tap[q]);
#pragma unroll
          for (int q = 0; q < SL; ++q) acc[q].add(vv, c[q]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
    }
#pragma unroll
    for (int q = 0; q < SL; ++q)
      acc[q].flush(tile + cell[q] * NPOL, q < nlive);
  }
}

struct GridCfArgs {
  const int4* items;
  const int4* rec;           // CF-major records
  const float2* svis;        // weighted visibilities, [sample][npol]
  int npol, pcf, pol0;
  const float2* cf;
  const long long* cfoff;
  int W, P;
  int Wx, nres;              // residue modulus along x (W rounded up to 8), Wx x W residues
  int nw;                    // tap warps
  int cf_bytes;              // CFS: one matrix, rounded up to 16 bytes
  int stage_bytes, nstages, fetch_off;
  float2* scratch;           // [item] P x P cells x NPOL
  long long slot;
  DevError* err;
};

// GridKernel::grid over the CF-major records, every cell's sum in the order of
// its samples: the sums of k_grid bit for bit (it adds zero taps besides).  One
// CTA per work item; thread t of the tap warps owns the residues k = t + 32 nw q
// of the footprint, rows modulo the exact CF width W and columns, with staged
// CFs, modulo W rounded up to 8 (k_grid: both up to 16, 1.2 to 5 times the
// taps), so no two threads touch one cell, and eight lanes of a row always lie
// on eight different 16-byte banks (modulo W itself a footprint's wrap puts two
// lanes on one: 35.7 instead of 30.0 ms at W 13, 4 polarisations, 4.4e7
// samples; unstaged, the latency of the taps hides it and the idle lanes of the
// rounding cost more: 7.4 against 11.9 ms at W 67 to 73).  The
// shared-memory tile holds two polarisations of a cell together (a plane of
// 16-byte cells per pair: neighbouring lanes on neighbouring banks); all slots of a thread are loaded before any is
// stored.  CFS: a segment is up to 32 samples of one CF matrix, brought into
// its stage by one bulk copy; otherwise 32 samples of any, the taps through
// L1 / L2 (matrices too large to stage beside the tile, and oversampling so
// fine that hardly two samples share one).
// Bound by shared memory (16 NPOL + 8 bytes per tap) and the latency from one
// sample's stores to the next one's loads.  Per launch, k_grid with its gather
// and inverse permutation, and now with k_weigh_cube: W 13, 4.4e7 samples x 4:
// 42.6 -> 30.5 ms; W 19, 2.1e7 x 4: 70.4 -> 30.8; W 49, 1.6e6 x 1: 6.3 -> 4.6;
// W 67 to 73, 1.5e6 x 1: 14.1 -> 7.4; W 7, 2.8e6 x 2: 2.5 -> 1.6.
template <int NPOL, int SL, bool CFS>
__global__ void __launch_bounds__(544, 1) k_grid_cf(const __grid_constant__ GridCfArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2* tile = reinterpret_cast<float2*>(smem_raw);
  unsigned char* ring = smem_raw + (((size_t)a.slot * sizeof(float2) + 127) & ~(size_t)127);
  const int SB = a.stage_bytes, NST = a.nstages;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(ring + (size_t)NST * SB);
  unsigned long long* empty = full + NST;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int4 it = a.items[blockIdx.x];
  __shared__ int s_abort;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int q = 0; q < NST; ++q) {
      mbar_init(&full[q], 1);
      mbar_init(&empty[q], a.nw);
    }
    mbar_fence_init();
  }
  const int n4 = (int)(a.slot / 2);
  for (int i = threadIdx.x; i < n4; i += blockDim.x)
    reinterpret_cast<float4*>(tile)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  const int W = a.W;
  const int rec_at = CFS ? a.cf_bytes : 0, vis_at = rec_at + kSeg * 16;
  if (warp == a.nw) {
    // ---- producer (as k_grid_pl's)
    const unsigned fm = 0xffffffffu;
    const int Wx = a.Wx;
    const float rW = __frcp_rn((float)W) * (1.f + 1e-6f), rWx = __frcp_rn((float)Wx) * (1.f + 1e-6f);
    Fetch<NPOL>& f = *reinterpret_cast<Fetch<NPOL>*>(ring + a.fetch_off);
    auto fetch_rec = [&](int w) {
      const int i = it.y + 32 * w + lane;
      if (i < it.z) copy_async<16>(&f.rec[w % (2 * kAhead)][lane], a.rec + i);
    };
    auto fetch = [&](int w) {
      if (it.y + 32 * w + lane >= it.z) return;
      const int k = w % kAhead;
      const int4 r = f.rec[w % (2 * kAhead)][lane];
      copy_async<8>(&f.off[k][lane], a.cfoff + r.z);
      const float2* src = a.svis + (size_t)(unsigned)r.w * a.npol + a.pol0;
      copy_async<NPOL == 1 ? 8 : 16>(&f.vis[k][lane][0], src);
      if (NPOL == 4) copy_async<16>(&f.vis[k][lane][NPOL / 2], src + 2);
    };
    const int nwin_all = (it.z - it.y + 31) / 32;
    for (int w = 0; w < 2 * kAhead; ++w) fetch_rec(w);
    copy_commit();
    copy_wait<0>();
    for (int w = 0; w < kAhead; ++w) {
      fetch(w);
      copy_commit();
    }
    int seg = 0;
    bool ok = true;
    auto acquire = [&](int stage) -> bool {
      bool okw = true;
      if (seg >= NST && lane == 0) okw = mbar_wait(&empty[stage], (unsigned)((seg / NST) - 1) & 1u);
      return __shfl_sync(fm, okw ? 1 : 0, 0) != 0;
    };
    for (int w = 0; w < nwin_all && ok; ++w) {
      copy_wait<kAhead - 1>();
      const int nwin = min(32, it.z - it.y - 32 * w), k = w % kAhead;
      const int4 r = lane < nwin ? f.rec[w % (2 * kAhead)][lane] : make_int4(-1, 0, -1, -1);
      const long long off = lane < nwin ? f.off[k][lane] : 0;
      const int px0 = r.x & 0xffff, py0 = (r.x >> 16) & 0xffff;
      const int zprev = __shfl_up_sync(fm, r.z, 1);
      unsigned heads = __ballot_sync(fm, lane < nwin && (lane == 0 || (CFS && zprev != r.z)));
      while (heads) {
        const int h = __ffs(heads) - 1;
        const unsigned rest = heads & (heads - 1);
        const int h2 = rest ? __ffs(rest) - 1 : nwin;
        heads = rest;
        const int stage = seg % NST;
        if (!acquire(stage)) {
          ok = false;
          break;
        }
        unsigned char* sp = ring + (size_t)stage * SB;
        if (lane >= h && lane < h2) {
          reinterpret_cast<int4*>(sp + rec_at)[lane - h] =
              make_int4(px0 + a.P * py0,
                        (px0 - Wx * (int)((float)px0 * rWx)) | ((py0 - W * (int)((float)py0 * rW)) << 16),
                        CFS ? 0 : (int)off, 0);
          const bool conj = a.pcf && r.y < 0;
          float4* vs = reinterpret_cast<float4*>(sp + vis_at);
#pragma unroll
          for (int p = 0; p < NPOL; ++p) {
            const float2 x = f.vis[k][lane][p];
            vs[(lane - h) * NPOL + p] = make_float4(x.x, conj ? -x.x : x.x, x.y, x.y);
          }
        }
        const long long o = __shfl_sync(fm, off, h);
        if (lane == 0) reinterpret_cast<int*>(sp + SB - 16)[0] = h2 - h;
        __syncwarp();
        if (lane == 0) {
          if (CFS) {
            fence_proxy_async_smem();
            mbar_expect_tx(&full[stage], (unsigned)a.cf_bytes);
            bulk_g2s(sp, a.cf + o, (unsigned)a.cf_bytes, &full[stage]);
          } else {
            mbar_arrive(&full[stage]);
          }
        }
        ++seg;
      }
      fetch(w + kAhead);
      fetch_rec(w + 2 * kAhead);
      copy_commit();
    }
    copy_wait<0>();
    if (ok && acquire(seg % NST)) {
      if (lane == 0) {
        reinterpret_cast<int*>(ring + (size_t)(seg % NST) * SB + SB - 16)[0] = -1;
        mbar_arrive(&full[seg % NST]);
      }
    } else if (lane == 0) {
      raise_error(a.err, YG_ERR_TIMEOUT, timeout_where(1, 1, seg, blockIdx.x));
      s_abort = 1;
      // no copy may be in flight when the CTA exits
      if (CFS)
        for (int q = 0; q < NST && q < seg; ++q) mbar_wait(&full[q], (unsigned)((seg - q + NST - 1) / NST - 1) & 1u);
    }
  } else {
    // ---- tap warps
    const int nthr = 32 * a.nw, t = threadIdx.x;
    const int P2 = a.P * a.P, Wx = a.Wx;
    int rx[SL], ry[SL];
    bool live[SL];
#pragma unroll
    for (int q = 0; q < SL; ++q) {
      const int k = q * nthr + t;
      live[q] = k < a.nres;
      rx[q] = live[q] ? k % Wx : 0;
      ry[q] = live[q] ? k / Wx : 0;
    }
    for (int seg = 0;; ++seg) {
      const int stage = seg % NST;
      if (!mbar_wait(&full[stage], (unsigned)(seg / NST) & 1u)) {
        if (lane == 0) raise_error(a.err, YG_ERR_TIMEOUT, timeout_where(1, 2, seg, blockIdx.x));
        s_abort = 1;
        break;
      }
      const unsigned char* sp = ring + (size_t)stage * SB;
      const int cnt = *reinterpret_cast<const volatile int*>(sp + SB - 16);
      if (cnt < 0) break;
      const float2* __restrict__ cfs = reinterpret_cast<const float2*>(sp);
      const int4* __restrict__ recs = reinterpret_cast<const int4*>(sp + rec_at);
      const float4* __restrict__ vs = reinterpret_cast<const float4*>(sp + vis_at);
      float2* __restrict__ g_s = tile;
      float4* __restrict__ g4 = reinterpret_cast<float4*>(tile);
#pragma unroll(SL* NPOL <= 8 ? 2 : 1)
      for (int l = 0; l < cnt; ++l) {
        const int4 r = recs[l];
        const int mx = r.y & 0xffff, my = r.y >> 16;
        float4 vv[NPOL];
#pragma unroll
        for (int p = 0; p < NPOL; ++p) vv[p] = vs[l * NPOL + p];
        float2 c[SL];
        int cell[SL];
        bool on[SL];
#pragma unroll
        for (int q = 0; q < SL; ++q) {
          int jx = rx[q] - mx, jy = ry[q] - my;
          jx += jx < 0 ? Wx : 0;
          jy += jy < 0 ? W : 0;
          const int tap = jx + W * jy;
          on[q] = live[q] && (!CFS || jx < W);
          if (CFS) {
            c[q] = make_float2(0.f, 0.f);
            if (on[q]) c[q] = cfs[tap];
          } else {
            c[q] = __ldg(a.cf + r.z + tap);
          }
          cell[q] = r.x + jx + a.P * jy;
        }
        float2 g[SL][NPOL];
#pragma unroll
        for (int q = 0; q < SL; ++q) {
          if (!on[q]) continue;
          if (NPOL == 1) {
            g[q][0] = g_s[cell[q]];
          } else {
#pragma unroll
            for (int p = 0; p < NPOL; p += 2) {
              const float4 w = g4[cell[q] + p / 2 * P2];
              g[q][p] = make_float2(w.x, w.y);
              g[q][(p + 1) % NPOL] = make_float2(w.z, w.w);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < SL; ++q) {
          const float2 cs = make_float2(-c[q].y, c[q].x);
#pragma unroll
          for (int p = 0; p < NPOL; ++p)
            g[q][p] = fma2(make_float2(vv[p].x, vv[p].y), c[q], fma2(make_float2(vv[p].z, vv[p].w), cs, g[q][p]));
        }
#pragma unroll
        for (int q = 0; q < SL; ++q) {
          if (!on[q]) continue;
          if (NPOL == 1) {
            g_s[cell[q]] = g[q][0];
          } else {
#pragma unroll
            for (int p = 0; p < NPOL; p += 2)
              g4[cell[q] + p / 2 * P2] =
                  make_float4(g[q][p].x, g[q][p].y, g[q][(p + 1) % NPOL].x, g[q][(p + 1) % NPOL].y);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
    }
  }
  __syncthreads();
  if (s_abort) return;
  float4* out = reinterpret_cast<float4*>(a.scratch + (size_t)blockIdx.x * a.slot);
  const float4* t4 = reinterpret_cast<const float4*>(tile);
  if (NPOL == 4) {
    for (int i = threadIdx.x; i < n4; i += blockDim.x) out[i] = t4[(i >> 1) + (i & 1) * a.P * a.P];
  } else {
    for (int i = threadIdx.x; i < n4; i += blockDim.x) out[i] = t4[i];
  }
}

// grid[cell] += sum over the slots whose padded tile covers the cell, in a
// fixed order (neighbouring tiles, their items, their groups).  One thread per
// cell for all polarisations (a slot keeps a cell's polarisations together);
// blockIdx.x is the (grid plane / channel, tile), blockIdx.y the CTA's share of
// its cells.  Bound by latency where the items of a short track crowd into few
// tiles: a cell's loads from consecutive items, and from an item's groups, do
// not wait for one another, and several CTAs share a tile where there are few
// (1.2e6 samples x 1 in 1296 items of 94^2 cells, 576 tiles: one slot per item
// 0.79 ms in a loop of one load at a time, 0.23 with loads in flight, 0.074
// shared; k_halo_sum of the same items 0.25.  Up to four slots per item: 1.03,
// 0.92, 0.29).
struct HaloPlArgs {
  const int* item_base;      // per tile: first item
  const int* nit;            // per tile: number of items
  const int4* items;
  const float2* scratch;
  float2* grid;              // ngc planes of (nx, ny, npol) per grid plane
  int nx, ny, npol, nchan_img, pol0;
  int tile, ntx, nty;
  long long ntiles;
  int smax, P, groups;
  int item0, item1;          // items whose slots the scratch holds
  long long slot;
  int npass;                 // passes of NPOL polarisations from pol0 on,
  long long pass_slots;      // elements from one pass's slots to the next's
};

// a cell's polarisations
template <int NPOL>
__device__ __forceinline__ void load_cell(const float2* __restrict__ s, float2 (&v)[NPOL]) {
  if (NPOL == 1) {
    v[0] = s[0];
  } else {
#pragma unroll
    for (int p = 0; p < NPOL; p += 2) {
      const float4 q = *reinterpret_cast<const float4*>(s + p);
      v[p] = make_float2(q.x, q.y);
      v[p + 1 < NPOL ? p + 1 : p] = make_float2(q.z, q.w);
    }
  }
}

template <int NPOL, bool GROUPS>
__global__ void __launch_bounds__(256) k_halo_pl(const __grid_constant__ HaloPlArgs a) {
  const long long tid = blockIdx.x;               // over ngc * ntiles
  const long long gc = tid / a.ntiles;
  const int t = (int)(tid % a.ntiles);
  const int tx = t % a.ntx, ty = t / a.ntx;
  const int R = (a.smax + a.tile - 1) / a.tile;   // neighbour reach in tiles
  const int side = 2 * R + 1;
  bool mine = false;
  for (int q = threadIdx.x; q < side * side; q += blockDim.x) {
    const int ax = tx + q % side - R, ay = ty + q / side - R;
    if (ax < 0 || ay < 0 || ax >= a.ntx || ay >= a.nty) continue;
    const long long nt = gc * a.ntiles + ax + (long long)a.ntx * ay;
    const int b = a.item_base[nt], m = a.nit[nt];
    if (m > 0 && b < a.item1 && b + m > a.item0) mine = true;
  }
  if (!__syncthreads_or(mine)) return;            // no neighbouring tile holds data
  const int gind = (int)(gc / a.nchan_img), ichan = (int)(gc % a.nchan_img);
  const size_t plane_cells = (size_t)a.nx * a.ny;
  const int T = a.tile;
  for (int pass = 0; pass < a.npass; ++pass)
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < T * T; c += gridDim.y * blockDim.x) {
    const int x = tx * T + c % T, y = ty * T + c / T;
    if (x >= a.nx || y >= a.ny) continue;
    float2 sum[NPOL];
#pragma unroll
    for (int p = 0; p < NPOL; ++p) sum[p] = make_float2(0.f, 0.f);
    bool hit = false;
    for (int dy = -R; dy <= R; ++dy) {
      const int ay = ty + dy;
      if (ay < 0 || ay >= a.nty) continue;
      const int py = y - (ay * T - a.smax);
      if (py < 0 || py >= a.P) continue;
      for (int dx = -R; dx <= R; ++dx) {
        const int ax = tx + dx;
        if (ax < 0 || ax >= a.ntx) continue;
        const int px = x - (ax * T - a.smax);
        if (px < 0 || px >= a.P) continue;
        const long long nt = gc * a.ntiles + ax + (long long)a.ntx * ay;
        const int b = a.item_base[nt];
        const int j0 = max(b, a.item0), j1 = min(b + a.nit[nt], a.item1);
        hit = hit || j0 < j1;
        const float2* s = a.scratch + pass * a.pass_slots + (size_t)(j0 - a.item0) * a.groups * a.slot + ((size_t)px + (size_t)a.P * py) * NPOL;
        if (!GROUPS) {
#pragma unroll 4
          for (int j = j0; j < j1; ++j, s += a.slot) {
            float2 v[NPOL];
            load_cell<NPOL>(s, v);
#pragma unroll
            for (int p = 0; p < NPOL; ++p) {
              sum[p].x += v[p].x;
              sum[p].y += v[p].y;
            }
          }
        } else {
#pragma unroll(NPOL == 4 ? 1 : 2)
          for (int j = j0; j < j1; ++j, s += a.groups * a.slot) {
            const int4 it = a.items[j];
            const int G = item_groups(it.z - it.y, a.groups);
            float2 v[kMaxGroups][NPOL], isum[NPOL];   // the item's groups first, then the items
#pragma unroll
            for (int g = 0; g < kMaxGroups; ++g)
              if (g < G) load_cell<NPOL>(s + g * a.slot, v[g]);
#pragma unroll
            for (int p = 0; p < NPOL; ++p) {
              isum[p] = v[0][p];
#pragma unroll
              for (int g = 1; g < kMaxGroups; ++g) {
                if (g >= G) continue;
                isum[p].x += v[g][p].x;
                isum[p].y += v[g][p].y;
              }
              sum[p].x += isum[p].x;
              sum[p].y += isum[p].y;
            }
          }
        }
      }
    }
    if (hit) {
      float2* g = a.grid + (size_t)gind * plane_cells * a.npol * a.nchan_img +
                  plane_cells * (a.pol0 + pass * NPOL + (size_t)a.npol * ichan) + x + (size_t)a.nx * y;
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        float2 o = g[p * plane_cells];
        o.x += sum[p].x;
        o.y += sum[p].y;
        g[p * plane_cells] = o;
      }
    }
  }
}

// a CF table of which L2 (126 MB) holds little beside the rest, and samples per
// CF plane below which a tile holds hardly two of one matrix
constexpr long long kBigTable = 32ll << 20, kSparsePlane = 4000;

// Shared memory of a CTA, and what two CTAs of one SM may each take of it.
constexpr size_t kSmemOne = 227 * 1024;
constexpr size_t kSmemTwo = 113 * 1024;
constexpr size_t kSmemThree = 75 * 1024 - 128;

struct Shape {
  int sl = 0, nw = 0, parts = 1, groups = 1, nstages = 0;
  size_t smem = 0;
};

size_t fetch_bytes(int npol) {
  return npol == 1 ? sizeof(Fetch<1>) : (npol == 2 ? sizeof(Fetch<2>) : sizeof(Fetch<4>));
}

int stage_bytes(int npol) { return (kSeg * 16 + kSeg * npol * 16 + 16 + 127) / 128 * 128; }

size_t block_bytes(int W, int fs) { return ((size_t)fs * ((W * W + 1) & ~1) * sizeof(float2) + 127) & ~(size_t)127; }

// Slots per thread, warps per group and parts for the W^2 residues.  Few slots
// and many warps hide the latency of a sample's taps, many slots share its
// record and visibilities among more of them.  Measured, ms of k_grid_pl
// (slots: 2 / 3 / 4 / 6): 4 polarisations, 4.4e7 samples, W 13: 13.9 / 11.2 /
// 13.8 / 12.7; 2.1e7 samples, W 19: - / 12.3 / 14.3 / 13.7; two polarisations,
// W 7 (2 / 4): 0.40 / 0.52; W 39 (2 / 4 / 8): 1.27 / 1.37 / 1.53; one
// polarisation, W 49 (4 / 8 / 12): 4.5 / 4.3 / 5.8.  Residues beyond the warps
// of a CTA go to further CTAs of the same item.  More than four groups cost
// more in slots to clear and sum than they hide (W 7: halo sum 0.28 -> 0.39).
Shape shape_for(int W, int npol, size_t block) {
  const int wslots = (W * W + 31) / 32;
  Shape s;
  if (npol == 4) s.sl = wslots <= 2 ? 2 : 3;
  else if (npol == 2) s.sl = wslots <= 48 ? 2 : (wslots <= 96 ? 4 : 8);
  else s.sl = wslots <= 2 ? 2 : (wslots <= 16 ? 4 : 8);
  const int maxw = npol == 1 ? 12 : (s.sl <= 4 ? 8 : 7);
  s.parts = (wslots + s.sl * maxw - 1) / (s.sl * maxw);
  s.nw = (wslots + s.sl * s.parts - 1) / (s.sl * s.parts);
  while (s.groups < kMaxGroups && 2 * s.groups * s.nw <= std::min(maxw, 8)) s.groups *= 2;
  const size_t fixed = block + 64 + fetch_bytes(npol), stage = stage_bytes(npol) + 16;
  const size_t budget = fixed + 2 * s.groups * stage <= kSmemTwo ? kSmemTwo : kSmemOne;
  s.nstages = fixed < budget ? (int)std::min<size_t>(16, (budget - fixed) / stage) / s.groups * s.groups : 0;
  if (s.nstages < std::max(2, s.groups)) {
    s.sl = 0;
    return s;
  }
  s.smem = fixed + s.nstages * stage;
  return s;
}

template <int NPOL, int SL, bool STAGED>
cudaError_t launch(const GridPlArgs& a, const Shape& s, int nitems, cudaStream_t st) {
  auto k = k_grid_pl<NPOL, SL, STAGED>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  if (e != cudaSuccess) return e;
  k<<<dim3(nitems, s.parts), 32 * (s.groups * s.nw + 1), s.smem, st>>>(a);
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

template <bool STAGED>
cudaError_t launch_any(const GridPlArgs& a, const Shape& s, int npol, int nitems, cudaStream_t st) {
  switch (npol * 100 + s.sl) {
    case 102: return launch<1, 2, STAGED>(a, s, nitems, st);
    case 104: return launch<1, 4, STAGED>(a, s, nitems, st);
    case 108: return launch<1, 8, STAGED>(a, s, nitems, st);
    case 202: return launch<2, 2, STAGED>(a, s, nitems, st);
    case 204: return launch<2, 4, STAGED>(a, s, nitems, st);
    case 208: return launch<2, 8, STAGED>(a, s, nitems, st);
    case 402: return launch<4, 2, STAGED>(a, s, nitems, st);
    case 403: return launch<4, 3, STAGED>(a, s, nitems, st);
    default: return cudaErrorInvalidConfiguration;
  }
}

int weigh_cube(const Plan& pl, const VisArgs& v, DevBuf& svis, cudaStream_t st) {
  if (svis.ensure_headroom((size_t)pl.nsamples * v.npol * sizeof(float2)) != cudaSuccess) return YG_ERR_CUDA;
  const unsigned blocks = (unsigned)std::max(1ll, std::min((pl.nsamples + 255) / 256, 148ll * 32));
  switch (v.npol) {
    case 1: k_weigh_cube<1><<<blocks, 256, 0, st>>>(v, svis.as<float2>()); break;
    case 2: k_weigh_cube<2><<<blocks, 256, 0, st>>>(v, svis.as<float2>()); break;
    case 3: k_weigh_cube<3><<<blocks, 256, 0, st>>>(v, svis.as<float2>()); break;
    default: k_weigh_cube<4><<<blocks, 256, 0, st>>>(v, svis.as<float2>()); break;
  }
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError() == cudaSuccess ? YG_OK : YG_ERR_CUDA;
}

HaloPlArgs halo_args(const Plan& pl, const VisArgs& v, float2* grid, int nx, int ny, int nchan_img, int groups,
                     long long slot) {
  HaloPlArgs h{};
  h.item_base = pl.itembase.as<int>();
  h.nit = pl.nit.as<int>();
  h.items = pl.items.as<int4>();
  h.grid = grid;
  h.nx = nx;
  h.ny = ny;
  h.npol = v.npol;
  h.nchan_img = nchan_img;
  h.tile = pl.tile;
  h.ntx = pl.ntx;
  h.nty = pl.nty;
  h.ntiles = (long long)pl.ntx * pl.nty;
  h.smax = pl.smax;
  h.P = pl.pad;
  h.groups = groups;
  h.slot = slot;
  h.npass = 1;
  return h;
}

template <int NPOL>
void launch_halo(const HaloPlArgs& h, dim3 blocks, cudaStream_t st) {
  if (h.groups > 1) k_halo_pl<NPOL, true><<<blocks, 256, 0, st>>>(h);
  else k_halo_pl<NPOL, false><<<blocks, 256, 0, st>>>(h);
}

int halo_sum(const HaloPlArgs& h, int npa, unsigned ntiles, cudaStream_t st) {
  // a few hundred large tiles would leave the chip idle: several CTAs share one
  const unsigned share = std::max(1u, std::min({8u, 148u * 16 / ntiles, (unsigned)h.tile * h.tile / 512}));
  const dim3 blocks(ntiles, share);
  switch (npa) {
    case 1: launch_halo<1>(h, blocks, st); break;
    case 2: launch_halo<2>(h, blocks, st); break;
    default: launch_halo<4>(h, blocks, st); break;
  }
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError() == cudaSuccess ? YG_OK : YG_ERR_CUDA;
}

// polarisations per pass: the most whose groups fit
int pols_per_pass(int W, int npol, size_t block) {
  for (int c : {4, 2, 1})
    if (npol % c == 0 && shape_for(W, c, block).sl) return c;
  return 0;
}

}  // namespace

int grid_pl_block(const CFView& cf, int os, int cf_mode, int npol) {
  if (cf.varsup || cf.maxsize <= 0 || npol > 4 || (cf.maxsize & 1) == 0 || cf.maxsize > 1023) return 0;
  if ((long long)cf.ncf * (cf.maxsize * cf.maxsize + 1) > 0x7fffffffll) return 0;   // 32-bit matrix offsets
  // Staged where all offsets of a plane leave room for two CTAs per SM (13-wide
  // CFs at oversample 8: 11.3 ms staged, 12.3 through L2).  Larger blocks
  // (one CTA per SM, or the offsets of one v offset at a time, whose samples
  // no longer come in runs) lose to L2: 19-wide at oversample 8 12.4 against
  // 13.0 and 18.2 ms, 49-wide at oversample 4 4.3 against 5.7.  So do tables
  // with many matrices per plane (oversample above 8) or planes per channel
  // and beam, where a block serves a few samples of a tile.
  if (os <= 8 && cf_mode != CF_MODE_AW && block_bytes(cf.maxsize, os * os) + 26 * 1024 <= kSmemTwo) return os * os;
  return -os * os;
}

int plan_grid_pl(const Plan& pl, const VisArgs& v, const CFView& cf, float2* grid, int nx, int ny, int nchan_img,
                 DevBuf& scratch, DevBuf& svis, DevError* err, cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1) {
  const bool staged = pl.pl_fs > 0;
  const int fs = staged ? pl.pl_fs : -pl.pl_fs;
  const int W = cf.maxsize;
  const size_t block = staged ? block_bytes(W, fs) : 0;
  const int npa = pols_per_pass(W, v.npol, block);
  if (npa == 0) return YG_ERR_UNSUPPORTED;
  const Shape s = shape_for(W, npa, block);
  const int P = pl.pad;
  GridPlArgs g;
  g.items = pl.items.as<int4>();
  g.rec = pl.rec_pos.as<int4>();
  g.npol = v.npol;
  g.pcf = v.pcf;
  g.cf = cf.data;
  g.cfoff = cf.off;
  g.W = W;
  g.W2 = W * W;
  g.stride = (W * W + 1) & ~1;
  g.fs = fs;
  g.P = P;
  g.groups = s.groups;
  g.nw = s.nw;
  g.stage_bytes = stage_bytes(npa);
  g.nstages = s.nstages;
  g.fetch_off = (s.nstages * (g.stage_bytes + 16) + 8 + 15) & ~15;
  g.block_bytes = (int)block;
  g.slot = ((long long)P * P * npa + 1) & ~1ll;
  g.err = err;
  // scratch for kScratch bytes of slots at a time, or for 1184 items (eight per
  // SM) where those are more: launches over consecutive items, each followed by
  // its halo sum
  constexpr size_t kScratch = (size_t)4 << 30;
  const size_t per_item = (size_t)s.groups * g.slot * sizeof(float2);
  const int batch = (int)std::min<long long>(pl.nitems, std::max<long long>(1184, (long long)(kScratch / per_item)));
  if (scratch.ensure_headroom(per_item * batch) != cudaSuccess) return YG_ERR_CUDA;
  g.scratch = scratch.as<float2>();
  int rc = weigh_cube(pl, v, svis, st);
  if (rc) return rc;
  g.svis = svis.as<float2>();
  HaloPlArgs h = halo_args(pl, v, grid, nx, ny, nchan_img, s.groups, g.slot);
  h.scratch = g.scratch;
  if (pl.ntiles_total > 0x7fffffffll) return YG_ERR_UNSUPPORTED;
  const unsigned nblocks = (unsigned)pl.ntiles_total;
  if (ev0) cudaEventRecord(ev0, st);
  for (int pol0 = 0; pol0 < v.npol; pol0 += npa) {
    for (int i0 = 0; i0 < pl.nitems; i0 += batch) {
      const int n = std::min(batch, pl.nitems - i0);
      g.pol0 = pol0;
      g.item0 = i0;
      if (s.parts > 1 && cudaMemsetAsync(scratch.p, 0, per_item * n, st) != cudaSuccess) return YG_ERR_CUDA;
      const cudaError_t e = staged ? launch_any<true>(g, s, npa, n, st) : launch_any<false>(g, s, npa, n, st);
      if (e == cudaErrorInvalidConfiguration) return YG_ERR_UNSUPPORTED;
      if (e != cudaSuccess) return YG_ERR_CUDA;
      if (ev1 && i0 + n >= pl.nitems && pol0 + npa >= v.npol) cudaEventRecord(ev1, st);
      h.pol0 = pol0;
      h.item0 = i0;
      h.item1 = i0 + n;
      rc = halo_sum(h, npa, nblocks, st);
      if (rc) return rc;
    }
  }
  return YG_OK;
}

namespace {

struct CfShape {
  int npa = 0, sl = 0, nw = 0, nstages = 0, stage = 0;
  bool cfs = false;
  size_t smem = 0;
};

int cf_stage_bytes(int cf_b, int npa) { return (cf_b + kSeg * 16 + kSeg * npa * 16 + 16 + 127) / 128 * 128; }

// Slots per thread and warps for the residues: two slots share a sample's
// record and visibilities (W 13: 30.0 ms with two, 31.0 with one, 34.5 with
// three; W 19: 30.6 / 32.9 / 35.9), one where that leaves fewer than three
// warps (W 7: 1.6 / 1.9 ms), more where the warps would not fit.
bool cf_threads(int nres, int npa, int ctas, CfShape* s) {
  static const int cands[5] = {1, 2, 4, 8, 12};
  const int wslots = (nres + 31) / 32;
  for (int sl : cands) {
    if ((npa >= 2 && sl > 4) || (sl == 1 && wslots > 4)) continue;
    const int nw = (wslots + sl - 1) / sl;
    if (nw > 16 || nw * ctas > 48) continue;
    s->sl = sl;
    s->nw = nw;
    return true;
  }
  return false;
}

// As many polarisations per pass as fit at all (W 19: four with one CTA per SM
// 30.6 ms, two passes of two with two CTAs 35.8), then staged before unstaged
// CFs (W 49: 4.6 against 5.0 ms), then as many CTAs per SM as fit.  `few`
// (oversampling above 8): unstaged, hardly two samples share a matrix (W 7:
// 1.6 against 3.8 ms).
CfShape cf_shape(int W, int P, int npol, bool few) {
  const int cf_b = (W * W * 8 + 15) / 16 * 16;
  for (int npa : {4, 2, 1}) {
    if (npol % npa) continue;
    for (int mode = 0; mode < 6; ++mode) {
      const bool cfs = mode < 3;
      if (few && cfs) continue;
      const int ctas = 3 - mode % 3;
      const size_t budget = ctas == 3 ? kSmemThree : (ctas == 2 ? kSmemTwo : kSmemOne);
      CfShape s;
      s.npa = npa;
      s.cfs = cfs;
      s.stage = cf_stage_bytes(cfs ? cf_b : 0, npa);
      const size_t slot = (((size_t)P * P * npa + 1) & ~(size_t)1) * sizeof(float2);
      const size_t fixed = slot + 448 + fetch_bytes(npa);   // (with roundings and the kernel's static shared memory)
      const int want = cfs && cf_b > 8192 ? 2 : 4;
      if (fixed + want * (size_t)(s.stage + 16) > budget) continue;
      if (!cf_threads((cfs ? (W + 7) / 8 * 8 : W) * W, npa, ctas, &s)) continue;
      s.nstages = (int)std::min<size_t>(8, (budget - fixed) / (s.stage + 16));
      // what the kernel addresses: its static shared memory comes on top of the
      // dynamic size, which must leave it its part of the budget (a ring that
      // fills the budget to the byte would not launch: W 75, tile 56)
      s.smem = (slot + 127) / 128 * 128 + s.nstages * (size_t)(s.stage + 16) + fetch_bytes(npa);
      return s;
    }
  }
  return CfShape{};
}

template <int NPOL, int SL, bool CFS>
cudaError_t launch_cf(const GridCfArgs& a, const CfShape& s, int nitems, cudaStream_t st) {
  auto k = k_grid_cf<NPOL, SL, CFS>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  if (e != cudaSuccess) return e;
  k<<<nitems, 32 * (s.nw + 1), s.smem, st>>>(a);
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

template <bool CFS>
cudaError_t launch_cf_any(const GridCfArgs& a, const CfShape& s, int nitems, cudaStream_t st) {
  switch (s.npa * 100 + s.sl) {
    case 101: return launch_cf<1, 1, CFS>(a, s, nitems, st);
    case 102: return launch_cf<1, 2, CFS>(a, s, nitems, st);
    case 104: return launch_cf<1, 4, CFS>(a, s, nitems, st);
    case 108: return launch_cf<1, 8, CFS>(a, s, nitems, st);
    case 112: return launch_cf<1, 12, CFS>(a, s, nitems, st);
    case 201: return launch_cf<2, 1, CFS>(a, s, nitems, st);
    case 202: return launch_cf<2, 2, CFS>(a, s, nitems, st);
    case 204: return launch_cf<2, 4, CFS>(a, s, nitems, st);
    case 401: return launch_cf<4, 1, CFS>(a, s, nitems, st);
    case 402: return launch_cf<4, 2, CFS>(a, s, nitems, st);
    case 404: return launch_cf<4, 4, CFS>(a, s, nitems, st);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace

// Where k_grid (padded to Wp, CFs through a ring) is the faster of the two, per
// launch, k_grid / k_grid_cf in ms:
// - just below 48, where eight slots a thread or a polarisation per pass leave
//   k_grid_cf short of warps and the padding is thin (1.8e6 samples, W 47: one
//   polarisation 3.6 / 4.1, two 5.9 / 8.3, four 11.7 / 16.7; W 43, one 3.7 /
//   4.1, but two, in one pass of four slots, 2.06 / 1.89 at 6e5 samples; from
//   49 on k_grid pads to 64: W 49 6.3 / 4.6);
// - tables of tens of MB with few samples per plane, whose segments are hardly
//   longer than a sample (AWProject, 25344 matrices, 1.2e6 samples), at widths
//   that fill k_grid's rows: W 13, two polarisations 1.16 / 1.32, four 1.41 /
//   1.81, but one, with the sums after it, 1.69 / 1.58; W 31, one 2.26 / 2.48,
//   two 3.02 / 3.30, but four 5.4 / 4.4; other widths the other way (W 29, two
//   3.02 / 2.46; W 7, two 1.00 / 0.89).
bool grid_cf_takes(const CFView& cf, int tile, int npol, int os, long long n) {
  const int W = cf.maxsize;
  if (cf.varsup || W <= 0 || (W & 1) == 0 || W > 1023 || npol > 4) return false;
  const long long elems = (long long)cf.ncf * (W * W + 1);
  if (elems > 0x7fffffffll) return false;
  const CfShape s = cf_shape(W, tile + W - 1, npol, os > 8);
  if (!s.npa) return false;
  const bool sparse = elems * 8 > kBigTable && n < kSparsePlane * (cf.ncf / (os * os));
  const bool thin = (s.sl >= 8 && W > 40 && W < 48) ||
                    (sparse && ((W >= 13 && W < 16 && npol >= 2) || (W == 31 && npol <= 2)));
  return !thin || grid_ring_pols(cf, tile, npol) == 0;
}

// k_grid_pl lives from samples of a CF plane that share their footprint; where
// they do not, a move and mostly a matrix from beyond L1 per sample cost more
// than the CF-major kernels' passes.  Grid passes, CF-major / plane-major in ms,
// AWProject with 48 channels x 33 planes, 40 integrations of 5 s (1.2e6
// samples), every 36th / 9th / 4th / 1st of a track, that is 1.05 / 1.58 / 3.0 /
// 9.1 samples per plane and cell:
//   W 47 to 37, one polarisation  4.6/8.3   3.2/4.0   3.1/3.0   3.0/2.1
//               two               6.5/9.4   4.2/4.3   4.2/3.4   3.9/2.6
//   W 29,       one               2.8/3.9   2.5/3.1   2.4/2.4   2.2/1.9
//               two               3.0/3.3   2.7/2.7   2.8/2.1   2.5/1.7
//               four              4.7/5.3   4.2/4.1   4.0/3.2   3.9/2.5
//   W 25,       one               2.3/2.9   2.1/2.4   2.0/2.0   1.9/1.6
//               two               2.8/2.8   2.6/2.3   2.4/1.9   2.3/1.5
//   W 13,       one               1.6/1.9   1.4/1.6   1.3/1.4   1.3/1.2
//               two               1.8/1.4   1.8/1.3   1.7/1.2   1.7/1.1
// The size of the table hardly matters (24 channels, half of it: the same
// ratios).  Where the CF-major kernel needs several passes it loses throughout
// (W 39, four 8.5/7.6 to 7.3/3.3), as it does with many samples to a plane.
bool grid_pl_asks(const CFView& cf, int tile, int npol, int os, long long n) {
  const int W = cf.maxsize, pl_pols = pols_per_pass(W, npol, 0);
  // (asking costs 30 us: 15,000 samples, 0.49 -> 0.52 ms per grid call, to
  // choose between kernels of 0.08 ms)
  if (n < (1 << 16) || n >= kSparsePlane * (cf.ncf / (os * os))) return false;
  if (pl_pols == 1) return W > 9;
  if (W <= 25) return false;
  const int cf_pols = grid_cf_takes(cf, tile, npol, os, n) ? cf_shape(W, tile + W - 1, npol, os > 8).npa
                                                           : grid_ring_pols(cf, tile, npol);
  return cf_pols >= pl_pols;
}

bool grid_pl_better(const CFView& cf, int tile, int npol, int os, long long n, double per_cell) {
  return !grid_pl_asks(cf, tile, npol, os, n) || per_cell >= (pols_per_pass(cf.maxsize, npol, 0) == 1 ? 3.0 : 2.0);
}

int plan_grid_cf(const Plan& pl, const VisArgs& v, const CFView& cf, float2* grid, int nx, int ny, int nchan_img,
                 int os, DevBuf& scratch, DevBuf& svis, DevError* err, cudaStream_t st, cudaEvent_t ev0,
                 cudaEvent_t ev1) {
  const int W = cf.maxsize, P = pl.pad;
  const CfShape s = cf_shape(W, P, v.npol, os > 8);
  if (!s.npa) return YG_ERR_UNSUPPORTED;
  GridCfArgs g;
  g.items = pl.items.as<int4>();
  g.rec = pl.rec.as<int4>();
  g.npol = v.npol;
  g.pcf = v.pcf;
  g.cf = cf.data;
  g.cfoff = cf.off;
  g.W = W;
  g.Wx = s.cfs ? (W + 7) / 8 * 8 : W;
  g.nres = g.Wx * W;
  g.P = P;
  g.nw = s.nw;
  g.cf_bytes = (W * W * 8 + 15) / 16 * 16;
  g.stage_bytes = s.stage;
  g.nstages = s.nstages;
  g.fetch_off = (s.nstages * (s.stage + 16) + 15) & ~15;
  g.slot = ((long long)P * P * s.npa + 1) & ~1ll;
  g.err = err;
  // a halo sum after every pass, while its slots are in L2; where nearly all
  // tiles are empty (w-stacks of a short chunk), one sum over all passes, each
  // with slots of its own: 46,000 tiles, 594 items, three passes 0.42 -> 0.35 ms
  // per grid call, but 841 tiles, 1439 items 5.00 -> 5.09
  const int npass = v.npol / s.npa;
  const bool once = pl.ntiles_total > 16ll * pl.nitems;
  const long long pass_slots = once ? pl.nitems * g.slot : 0;
  if (scratch.ensure_headroom((size_t)(once ? npass : 1) * pl.nitems * g.slot * sizeof(float2)) != cudaSuccess)
    return YG_ERR_CUDA;
  int rc = weigh_cube(pl, v, svis, st);
  if (rc) return rc;
  g.svis = svis.as<float2>();
  HaloPlArgs h = halo_args(pl, v, grid, nx, ny, nchan_img, 1, g.slot);
  h.scratch = scratch.as<float2>();
  h.item1 = pl.nitems;
  h.npass = once ? npass : 1;
  h.pass_slots = pass_slots;
  if (pl.ntiles_total > 0x7fffffffll) return YG_ERR_UNSUPPORTED;
  if (ev0) cudaEventRecord(ev0, st);
  for (int pass = 0; pass < npass; ++pass) {
    g.pol0 = pass * s.npa;
    g.scratch = scratch.as<float2>() + pass * pass_slots;
    const cudaError_t e = s.cfs ? launch_cf_any<true>(g, s, pl.nitems, st) : launch_cf_any<false>(g, s, pl.nitems, st);
    if (e == cudaErrorInvalidConfiguration) return YG_ERR_UNSUPPORTED;
    if (e != cudaSuccess) return YG_ERR_CUDA;
    if (ev1 && pass == npass - 1) cudaEventRecord(ev1, st);
    if (once && pass < npass - 1) continue;
    h.pol0 = once ? 0 : g.pol0;
    rc = halo_sum(h, s.npa, (unsigned)pl.ntiles_total, st);
    if (rc) return rc;
  }
  return YG_OK;
}

}  // namespace yg
