// brkga_decoder.cu — B200 (sm_100a) BRKGA chromosome decoder behind the C ABI
// of include/brkga_b200.h.
//
// Semantics: the reference's sequential decoder (paulonasc7/BRKGA_FFT2
// placement.py:94-165, binClassNew.py:45-174, numba_utils.py:50-188,
// collision_backend.py:109-213).  The reference finds collision-free
// positions with a float FFT correlation; here the correlation is evaluated
// exactly on bit-packed rows, which yields the same feasible set.
//
// A problem holds K >= 1 independent instances (own parts, machines, plate
// sizes).  Their tables are merged into one set of device arrays: part types,
// rotations, mask rows and machines get absolute indices, and each instance
// records its bases (InstDev).  A launch decodes P_k chromosomes of every
// instance k; the per-launch row/item offsets travel in the kernel
// parameters (InstRun), so one launch of each kernel serves all instances.
//
// Pipeline per launch (three kernels on one stream, no host sync):
//   1. assign_sort_kernel  one CTA per chromosome: machine of every gene from
//      the machine keys, then a bitonic sort of (machine, sequencing key,
//      gene) 64-bit keys in shared memory -> per-(chromosome, machine) part
//      order (placement.py:118-135).  order_items_kernel then sorts the
//      (chromosome, machine) items of all instances by part count.
//   2. decode_kernel       persistent CTAs of 1, 2, 4 or 8 warps (the launch
//      shape), one (chromosome, machine) item at a time, longest first, from
//      a device counter.  A plate is a grid of L rows of ceil(W/32)+2 32-bit
//      words (bit x of a row = cell x) and the coarse data derived from it
//      (erosion planes and longest free runs of blocks of rows, or the longest
//      free runs of the rows alone: coarse_ok(), coarse_blocks()); each CTA has a few plates of its own, further ones come from a global
//      pool and stay with the CTA for its later items.  For each part:
//      first-fit over plates (area filter, then the collision search), else a
//      new plate with the best rotation at (0, L-1).  The collision search
//      splits (rotation, 32 candidate rows) chunks over the warps, skipping
//      chunks that cannot beat the best position found so far; a lane runs the
//      vacancy filter of one candidate top row, then the (surviving candidate,
//      64 columns) pairs are dealt to the lanes, bottom rows first: each lane
//      tests its pair against the planes, groups of lanes test the first
//      pieces of the runs of what is left open, and the pairs still open are
//      finished in order by the whole warp, mask rows coarse to fine from the
//      bottom; the first pair with a free column gives the bottom-most
//      candidate and its leftmost x.  Results are merged with a 64-bit
//      lexicographic key (newLen, -y, x, rotation) by atomicMin in shared
//      memory, which is the reference's rotation rule
//      (binClassNew.py:101-117) — see key_of().
//   3. reduce_kernel       max over machines, 1e16 for infeasible chromosomes.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/brkga_b200.h"
#include "corr_i8.cuh"

namespace {

constexpr int kMaxMachines = 255;
constexpr int kMaxGenes = 8192;     // bitonic sort buffer: 8192 x 8 B = 64 KB shared memory
constexpr int kMaxSide = 8191;      // 13-bit fields of the selection key
constexpr int kGreedyThreads = 256;
constexpr int kGreedyCtas = 8;  // CTAs of the greedy's cluster (the portable limit)
constexpr int kResidentWarps = 32;  // automatic shape: 32 warps per SM (the register limit at 64 per thread)
constexpr int kMaxInst = BRKGA_MAX_INSTANCES;
constexpr int kMaxCtasPerSm = 32;
constexpr int kMaxSmemPlates = 8;
constexpr int kDefaultTaskMax = 8192;
// Latency launches (the 4-warp shape: few waves of items) end with their
// longest items, each sharing its SM with seven other CTAs until the queue
// drains.  The CTA that takes one of the first kCritItems items of the
// longest-first queue marks its SM, and the other CTAs there take no new
// item while the mark stands, so that SM empties and the long item gets its
// issue slots; the other SMs absorb the queue.  Measured at P100M4
// population 500: 2-4 % faster with 8 or 16 items; on throughput launches
// (2- and 1-warp shapes) draining SMs costs 2-7 %, so it is off there.
constexpr int kCritItems = 16;
constexpr int kCritSlots = 1024;  // per-SM marks, indexed by %smid
// The coarse test's erosion planes: runs of 4, 8, 16 and 32 columns (see coarse_ok()).
constexpr int kPlaneMin = 2;
constexpr int kPlaneMax = 5;
constexpr int kMaxTaskMax = 32 * 256;  // twice the pairs there can be: 32 candidates x 128 words of 64 columns
constexpr unsigned long long kKeyNone = ~0ull;
constexpr unsigned kFull = 0xFFFFFFFFu;

struct RotDev {
  int h, w;          // rows, columns
  short mw;          // 32-bit words per mask row
  short gseg;        // pieces that groups of lanes test first (0: none, see group_segs())
  int trun, ntrun;   // runs of ones of all rows in test order: truns[trun .. trun + ntrun)
  int tseg, ntseg;   // the same in pieces of at most 32 columns: truns[tseg .. tseg + ntseg), often the same list
  int mask_base;     // first word in maskbits[] (h * mw words)
};
static_assert(sizeof(RotDev) == 32, "RotDev layout");

// The coarse test of one rotation at one alignment (its entries in centry[]
// and cfilter[]); see coarse_ok() and coarse_and().
struct CoarseIdx {
  int e, ne;  // centry[e .. e + ne): cores as reads of two erosion-plane windows, ne even (the last one repeated)
  int f, nf;  // cfilter[f .. f + nf): (block row << 16 | core length), nf a multiple of kVacIlp (padded with 0)
};

// The rotations of one part type that fit one machine's plate
// (numba_utils.py:82-84), fixed per (type, machine) and so built once at
// problem creation: by height, the smallest height, and the words one
// read of the plate and of each rotated mask takes (the scan-bytes counter).
struct RotList {
  unsigned char nr;
  unsigned char rs[4];  // by height, ties in rotation order
  unsigned char pad[3];
  int hmin;
  unsigned int scan_words;
};
static_assert(sizeof(RotList) == 16, "RotList layout");

struct MachDev {
  int L, W, NW, RS;  // plate rows, columns, words per row, row stride (NW + 2 zero pad words)
  int NB;            // whole blocks of rows (the rows after them are in no core)
  double area;       // MachineData.bin_area
  double setup;      // MachineData.setup_time
};

struct BinScal {     // per-plate scalars of binClassNew.BuildingPlate
  double area, pt, pth;
  int minrow, maxrow, enc, pool;
};

// Where instance k's entries start in the merged tables.
struct InstDev {
  int N, M, T, mode;
  int gbase;    // gene_type[gbase + j]: absolute part type of gene j
  int tbase;    // first absolute part type
  int mbase;    // mach[mbase + m]
  int thrbase;  // thr[thrbase + m], M - 1 entries
  int tmbase;   // pt/pth[tmbase + m*T + t], newbin_ok/fits[tmbase + t*M + m] (t local)
};

// Merged device tables of all instances of a problem.
struct Tables {
  const InstDev* inst;
  const int32_t* gene_type;
  const double* thr;
  const MachDev* mach;
  const double* pt;
  const double* pth;
  const double* part_area;  // [absolute type]
  const int32_t* nrot;
  const int32_t* best_rot;
  const RotDev* rot;        // [absolute type * 4 + rotation]
  const CoarseIdx* cidx;    // [rotation, indexed like rot][offset of the top row in a block]
  const uint2* centry;      // (first window's column | second one's << 16, plane row from the top row's block on)
  const uint32_t* cfilter;
  const uint2* truns;       // (start | length << 16, row) per run of ones, and per piece of one
  const uint32_t* maskbits;
  const uint8_t* newbin_ok;
  const uint8_t* fits;
  const RotList* rl;        // [(type, machine)], indexed like fits
  int bsh;                  // a block of the coarse test has 2^bsh rows (0: the test is by rows, see coarse_blocks())
  int n_planes;             // erosion plane i holds the starts of free runs of 2^(kPlaneMin + i) columns; by rows none
};

// One instance's slice of a launch.
struct InstRun {
  int P;               // chromosomes of this instance in the launch
  int crow0;           // first row in chrom / makespan / infeas
  int item0;           // first (chromosome, machine) item
  int S2;              // bitonic sort width (power of two >= N)
  long long chrom_off; // first float of its chromosomes
  long long out_off;   // first makespan
  long long seq0;      // first entry of its part orders (and log entries), N per item
};

// Everything a launch needs besides the tables.
struct Run {
  int K, n_rows, n_items, Nmax;
  const float* chrom;
  double* out;
  uint16_t* seq;
  int32_t* cnt;
  int32_t* infeas;
  int32_t* order;
  double* mk;
  BrkgaPlacement* log;
  int32_t* status;
  unsigned int* item_ctr;
  unsigned int* pool_ctr;
  int* crit;           // kCritSlots marks: CTAs busy with a critical item, per SM
  int crit_items;      // items at the head of the queue that mark their SM (0 = off)
  unsigned long long* counters;
  BinScal* binscal;  // Nmax per resident CTA
  uint32_t* pool;    // grids of the plates beyond the CTAs' own, grid_words each
  uint32_t* cpool;   // their erosion planes and block vacancies, coarse_words each
  long long pool_bins;
  uint32_t* own;     // S plates per resident CTA, grid and planes
  int S, smem_grids; // plates per item that are the CTA's own; whether their grids are in shared memory instead
  int grid_words, coarse_words, vac_off;
  int task_max;  // most (survivor, word) pairs of a chunk dealt across lanes
  InstRun r[kMaxInst];
};
static_assert(sizeof(Tables) + sizeof(Run) <= 4096, "kernel parameters must stay within 4 KB");

// ---------------------------------------------------------------- device helpers

__device__ __forceinline__ unsigned ordered_bits(float v) {
  unsigned u = __float_as_uint(v);
  if (v == 0.0f) u = 0u;               // -0 and +0 compare equal in the reference's sort
  if (v != v) u = 0x7FC00000u;         // NaN sorts after every number (np.argsort)
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// placement.py:122-127 for ascending thresholds: the first machine whose
// upper threshold is >= the key, else the last; a NaN key matches no mask.
__device__ __forceinline__ int machine_of(float mv, const double* thr, int M, int mode) {
  if (M <= 1) return 0;
  if (mv != mv) return M;
  int m = 0;
  if (mode == BRKGA_THRESH_F32) {
    while (m < M - 1 && !(mv <= (float)thr[m])) ++m;
  } else {
    const double v = (double)mv;
    while (m < M - 1 && !(v <= thr[m])) ++m;
  }
  return m;
}

// Selection key, smaller is better.  Within one plate the reference keeps the
// rotation of largest packing density (area + a) / (newLen * W); numerator and
// W are shared and newLen * W are distinct integers <= 2^26, so the float64
// quotients are strictly ordered by newLen: max density == min newLen.  Ties
// go to the larger bottom row y, then the smaller x, then the first rotation.
// The row's part (newLen, y) fills the upper word, so rows compare as 32-bit values.
__device__ __forceinline__ unsigned row_key(int newlen, int y) {
  return ((unsigned)newlen << 13) | (unsigned)(kMaxSide - y);
}

__device__ __forceinline__ unsigned long long key_of(unsigned row, int x, int r) {
  return ((unsigned long long)row << 32) | ((unsigned)x << 2) | (unsigned)r;
}

// bits [p, p + 32) of a row (p >= 0; reads words p>>5 and p>>5 + 1)
__device__ __forceinline__ uint32_t bits32(const uint32_t* row, int p) {
  const int wi = p >> 5;
  return __funnelshift_r(row[wi], row[wi + 1], p & 31);
}

__device__ __forceinline__ bool range_any(const uint32_t* row, int lo, int hi) {
  const int wl = lo >> 5, wh = (hi - 1) >> 5;
  const uint32_t ml = 0xFFFFFFFFu << (lo & 31);
  const uint32_t mh = 0xFFFFFFFFu >> (31 - ((hi - 1) & 31));
  if (wl == wh) return (row[wl] & ml & mh) != 0u;
  if (row[wl] & ml) return true;
  for (int w = wl + 1; w < wh; ++w)
    if (row[w]) return true;
  return (row[wh] & mh) != 0u;
}

// For the 32 placements x' = 0..31 (absolute x = p0 - a + x'), bit x' is set
// when a run of d mask cells starting at plate column p0 + x' covers an
// occupied cell: OR of row bits [p0 + x', p0 + x' + d).
__device__ __forceinline__ uint32_t blocked(const uint32_t* row, int p0, int d) {
  if (d <= 32) {
    uint32_t lo = bits32(row, p0), hi = bits32(row, p0 + 32);
    int s = 1;
    while (2 * s <= d) {  // doubling: after a step lo bit j = OR of 2s bits from j
      lo |= __funnelshift_r(lo, hi, s);
      hi |= hi >> s;
      s <<= 1;
    }
    if (d > s) lo |= __funnelshift_r(lo, hi, d - s);
    return lo;
  }
  // d > 32: every window contains [p0 + 31, p0 + d)
  if (range_any(row, p0 + 31, p0 + d)) return 0xFFFFFFFFu;
  uint32_t res = 0u;
  const uint32_t left = bits32(row, p0) & 0x7FFFFFFFu;       // cell p0+j blocks x' <= j
  if (left) res |= (2u << (31 - __clz(left))) - 1u;
  const uint32_t right = bits32(row, p0 + d) & 0x7FFFFFFFu;  // cell p0+d+j blocks x' > j
  if (right) res |= ~((2u << (__ffs(right) - 1)) - 1u);
  return res;
}

// blocked() for a run of at most 32 cells and the 64 placements from p0, in
// straight-line code (lanes with runs of different lengths stay together).
// Reads words p0>>5 .. p0>>5 + 3, the last one only inside the row of RS words.
__device__ __forceinline__ uint2 blocked64(const uint32_t* row, int p0, int d, int RS) {
  const int wi = p0 >> 5;
  const uint32_t w0 = row[wi], w1 = row[wi + 1], w2 = row[wi + 2], w3 = wi + 3 < RS ? row[wi + 3] : 0u;
  uint32_t a = __funnelshift_r(w0, w1, p0), b = __funnelshift_r(w1, w2, p0), c = __funnelshift_r(w2, w3, p0);
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    if (d >= 2 * s) {  // after a step bit j = OR of 2s bits from j
      a |= __funnelshift_r(a, b, s);
      b |= __funnelshift_r(b, c, s);
      c |= c >> s;
    }
  }
  const int rest = d - (1 << (31 - __clz(d)));  // 0 .. 15
  return make_uint2(a | __funnelshift_r(a, b, rest), b | __funnelshift_r(b, c, rest));
}

constexpr int kTestIlp = 2;   // independent run dilations per step of the exact test
constexpr int kVacIlp = 2;    // block vacancies compared per step of the filter
constexpr int kGroupOpen = 3;  // pairs open after the coarse test from which groups of lanes first test
constexpr int kGroupSegs = 4;  // this many pieces of each (where the test is by rows: see group_segs())

// Where one open plate lives.
struct PlateRef {
  uint32_t* grid;    // L rows of RS words
  uint32_t* planes;  // NB x n_planes rows of RS words
  uint16_t* vac;     // NB longest free runs
};

// Plate b of this CTA's item: the first S in places of the CTA's own (their
// grids in shared memory if asked for), the others in the pools.
__device__ __forceinline__ PlateRef plate_ref(const Run& run, uint32_t* smem, int b, int pool) {
  PlateRef pr;
  if (b < run.S) {
    uint32_t* own = run.own + ((size_t)blockIdx.x * run.S + b) * (run.grid_words + run.coarse_words);
    pr.grid = run.smem_grids ? smem + (size_t)b * run.grid_words : own;
    pr.planes = own + run.grid_words;
  } else {
    pr.grid = run.pool + (size_t)pool * run.grid_words;
    pr.planes = run.cpool + (size_t)pool * run.coarse_words;
  }
  pr.vac = reinterpret_cast<uint16_t*>(pr.planes + run.vac_off);
  return pr;
}

// Coarse test.  The plate also keeps, for every block of 2^bsh rows, which
// columns are free in all of them, as erosion planes (plane i: columns at
// which 2^(kPlaneMin + i) such columns start), and the longest run of them.
// A rotation whose top row sits at a given offset in its block covers whole
// blocks with 2^bsh of its rows each; the columns that all of them occupy
// (the block's core) must be free in the plate's block.  That is a necessary
// condition, cheap to test (a block stands for all its rows, a core for one
// window of two plane reads instead of a dilation per row), and it rejects
// most blocked positions before the exact test: of the (row, 32-column word)
// pairs that pass the filter at P100M4, one in ten stays open.  What bounds the
// kernel is integer issue on chip, so the instructions of a rejected position
// are what counts: before, lanes walked the runs of its rows, some fifty
// instructions for each run and 32 columns.  One launch
// before / now: P100M4 1.54 / 1.04 ms (500 rows) and 8.25 / 5.47 ms (4,000),
// P200M6 3.94 / 2.45 ms (1,000), P400M8 35.9 / 18.65 ms (1,024), P50M2 0.404 /
// 0.252 ms (1 row) and 0.523 / 0.355 ms (100), 64 uneven instances x 256
// 29.5 / 19.8 ms.
//
// The filter: every block has a free run as long as the core it must take.
__device__ __forceinline__ bool coarse_ok(const Tables& tb, const uint16_t* vac, int ty, int rot) {
  const CoarseIdx ci = tb.cidx[(rot << tb.bsh) + (ty & ((1 << tb.bsh) - 1))];
  const uint32_t* f = tb.cfilter + ci.f;
  const uint16_t* v = vac + (ty >> tb.bsh);
  for (int i = 0; i < ci.nf; i += kVacIlp) {
    bool bad = false;
#pragma unroll
    for (int u = 0; u < kVacIlp; ++u) {
      const uint32_t e = __ldg(f + i + u);
      bad |= v[e >> 16] < (e & 0xFFFFu);
    }
    if (bad) return false;
  }
  return true;
}

// The 64 columns from pl's word on at which one core is free: its run is the
// union of two windows of the plane's length (the entry's plane is the longest
// that fits; longer cores are several entries).  The planes of a block lie row
// after row and the entry holds both windows' columns, so an address is one
// multiplication and no sum (with the planes one after another and the second
// window as an offset, six instructions more a core): P100M4 4,000 rows 5.67 ->
// 5.47 ms, P200M6 1,000 2.53 -> 2.45, P400M8 1,024 19.7 -> 18.65, P50M2 1 row
// 0.257 -> 0.252.
__device__ __forceinline__ uint2 coarse_window(const uint32_t* pl, unsigned RS, uint2 e) {
  const uint32_t *u = pl + e.y * RS + ((e.x & 0xFFFFu) >> 5), *v = pl + e.y * RS + (e.x >> 21);
  const uint32_t p = e.x, q = e.x >> 16;  // the shifts take their low five bits
  const uint32_t u1 = u[1], v1 = v[1];
  return make_uint2(__funnelshift_r(u[0], u1, p) & __funnelshift_r(v[0], v1, q),
                    __funnelshift_r(u1, u[2], p) & __funnelshift_r(v1, v[2], q));
}

// The bits of F at which every core of rotation rot (index into tb.rot) is free, two cores per step.
__device__ __forceinline__ uint2 coarse_and(const Tables& tb, const uint32_t* planes, const MachDev& md, int ty, int base,
                                            uint2 F, int rot) {
  const CoarseIdx ci = tb.cidx[(rot << tb.bsh) + (ty & ((1 << tb.bsh) - 1))];
  const uint4* c = reinterpret_cast<const uint4*>(tb.centry + ci.e);  // e and ne are even
  const uint32_t* pl = planes + (ty >> tb.bsh) * tb.n_planes * md.RS + (base >> 5);
  for (int q = 0; 2 * q < ci.ne && (F.x | F.y); ++q) {
    const uint4 e = __ldg(c + q);
    const uint2 a = coarse_window(pl, md.RS, make_uint2(e.x, e.y)), b = coarse_window(pl, md.RS, make_uint2(e.z, e.w));
    F.x &= a.x & b.x;
    F.y &= a.y & b.y;
  }
  return F;
}

// The valid candidate columns among base .. base + 63, for nx candidates in all.
__device__ __forceinline__ uint2 first_open(int nx, int base) {
  const int n = nx - base;
  return make_uint2(n >= 32 ? kFull : n > 0 ? (1u << n) - 1u : 0u,
                    n >= 64 ? kFull : n > 32 ? (1u << (n - 32)) - 1u : 0u);
}

// The bits of F (candidate columns base .. base + 31) at which the rotation
// fits with its top row at plate row g0: every run of ones of the mask, in
// collision-test order (widest row, then the rows coarse to fine from the
// bottom), clears the columns it would overlap; kTestIlp independent
// runs per step, stop when F is empty.
__device__ __forceinline__ uint32_t word_free(const uint32_t* g0, int RS, int base, uint32_t F, const RotDev& rd,
                                              const uint2* truns) {
  const uint2* e = truns + rd.trun;
  const int n = rd.ntrun;
  int q = 0;
  for (; q + kTestIlp <= n && F; q += kTestIlp) {
    uint32_t bl = 0u;
#pragma unroll
    for (int u = 0; u < kTestIlp; ++u) {
      const uint2 r = __ldg(e + q + u);
      bl |= blocked(g0 + (int)r.y * RS, base + (int)(r.x & 0xFFFFu), (int)(r.x >> 16));
    }
    F &= ~bl;
  }
  for (; q < n && F; ++q) {
    const uint2 r = __ldg(e + q);
    F &= ~blocked(g0 + (int)r.y * RS, base + (int)(r.x & 0xFFFFu), (int)(r.x >> 16));
  }
  return F;
}

// Leftmost x at which the rotation fits with its top row at ty, or -1
// (output words of 32 candidate columns tried left to right).
__device__ __forceinline__ int first_free_x(const Tables& tb, const PlateRef& pr, const MachDev& md, int ty, int rot,
                                            const RotDev& rd) {
  const int nx = md.W - rd.w + 1;
  const uint32_t* g0 = pr.grid + (size_t)ty * md.RS;
  for (int base = 0; base < nx; base += 64) {
    const uint2 F = coarse_and(tb, pr.planes, md, ty, base, first_open(nx, base), rot);
    const uint32_t lo = F.x ? word_free(g0, md.RS, base, F.x, rd, tb.truns) : 0u;
    if (lo) return base + __ffs(lo) - 1;
    const uint32_t hi = F.y ? word_free(g0, md.RS, base + 32, F.y, rd, tb.truns) : 0u;
    if (hi) return base + 32 + __ffs(hi) - 1;
  }
  return -1;
}

// Longest run of ones in x, branch-free: p_s marks the starts of runs of at
// least s ones (s = 1, 2, 4, 8, 16); descending, cur marks the starts of runs
// of at least n + s ones when cur & (p_s >> n) is not empty.
__device__ __forceinline__ int longest_ones(uint32_t x) {
  if (x == 0xFFFFFFFFu) return 32;
  const uint32_t p1 = x, p2 = p1 & (p1 >> 1), p4 = p2 & (p2 >> 2), p8 = p4 & (p4 >> 4), p16 = p8 & (p8 >> 8);
  const uint32_t p[5] = {p16, p8, p4, p2, p1};
  uint32_t cur = 0xFFFFFFFFu;
  int n = 0;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const uint32_t c = cur & (p[i] >> n);
    if (c) {
      cur = c;
      n += 16 >> i;
    }
  }
  return n;
}

// free columns of a block of plate rows in word w: bit set = no row occupies it (columns past W count as occupied)
__device__ __forceinline__ uint32_t block_free(const uint32_t* row, int RS, int W, int rows, int w) {
  uint32_t v = 0u;
  for (int i = 0; i < rows; ++i) v |= row[(size_t)i * RS + w];
  const int valid = W - 32 * w;
  if (valid < 32) v |= 0xFFFFFFFFu << valid;
  return ~v;
}

// longest run of free columns of one plate row (one thread)
__device__ __forceinline__ int row_free_run(const uint32_t* row, const MachDev& md) {
  int run = 0, best = 0;
  for (int w = 0; w < md.NW; ++w) {
    const uint32_t v = ~block_free(row, md.RS, md.W, 1, w);
    if (v == 0u) {
      run += 32;
      continue;
    }
    const int tz = __ffs(v) - 1;
    run += tz;
    best = max(best, run);
    const int hb = 31 - __clz(v);
    if (hb > tz + 1) best = max(best, longest_ones(~v & ((1u << hb) - 1u) & ~((2u << tz) - 1u)));
    run = __clz(v);
  }
  return max(best, run);
}

// longest run of free columns of a block of plate rows (plates wider than
// 1024 columns): a warp takes 32 words of the row at a time, a lane one of them,
// and carries the run at their end on.  One lane over the whole row took longer
// than the search: 60 parts on plates of 200 x 1500 and 300 x 1100, 4,000 rows,
// 13.8 ms and 3.7 this way; on plates 4,000 columns wide, 300 rows, 4.3 and 0.86.
// All lanes of the warp.
__device__ __forceinline__ int max_free_run(const uint32_t* row, int RS, int W, int NW, int rows) {
  const int lane = threadIdx.x & 31;
  int best = 0, carry = 0;  // carry: free columns up to these words' first one
  for (int w0 = 0; w0 < NW; w0 += 32) {
    const int w = w0 + lane;
    const uint32_t e = w < NW ? block_free(row, RS, W, rows, w) : 0u;
    const unsigned full = __ballot_sync(kFull, e == kFull);
    const int low = e == kFull ? 32 : __ffs(~e) - 1, high = e == kFull ? 32 : __clz(~e);
    // free columns up to this word: the last word below that is not full gives its upper ones
    const unsigned below = ~full & ((1u << lane) - 1u);
    const int from = below ? 31 - __clz(below) : 0;
    const int upper = __shfl_sync(kFull, high, from);
    const int before = below ? upper + 32 * (lane - 1 - from) : carry + 32 * lane;
    best = max(best, max(longest_ones(e), before + low));
    carry = __shfl_sync(kFull, e == kFull ? before + 32 : high, 31);
  }
  return __reduce_max_sync(kFull, best);
}

__device__ __forceinline__ void raise_status(int32_t* status, int code) {
  atomicCAS(status, 0, code);
}

// The window that a (candidate, 64-column word) pair of the tests reads: plate
// rows row0 .. row0 + h - 1 and, in each, at most word ((base + w - 1) >> 5) + 2
// (a run starts at s >= 0 with s + d <= w, a table invariant; the exact test
// checks the word after that one itself).  Checked once per pair, so the
// cores and runs inside need no check of their own.
__device__ __forceinline__ bool pair_in_plate(int row0, int base, int h, int w, const MachDev& md) {
  return row0 >= 0 && row0 + h <= md.L && base >= 0 && base + w <= md.W;
}

// Instance of a launch row / item: the last instance starting at or before v
// (instances with no rows share their start with the next one, which wins).
__device__ __forceinline__ int inst_of_row(const Run& run, int v) {
  int lo = 0, hi = run.K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (run.r[mid].crow0 <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int inst_of_item(const Run& run, int v) {
  int lo = 0, hi = run.K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (run.r[mid].item0 <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------- kernels

__global__ void assign_sort_kernel(const __grid_constant__ Tables tb, const __grid_constant__ Run run) {
  extern __shared__ unsigned long long keys[];
  __shared__ int s_cnt[kMaxMachines + 1];
  __shared__ int s_start[kMaxMachines + 1];
  __shared__ int s_inf;
  const int row = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int k = inst_of_row(run, row);
  const InstRun& ir = run.r[k];
  const InstDev id = tb.inst[k];
  const int N = id.N, M = id.M, S2 = ir.S2, c = row - ir.crow0;
  if (row == 0)
    for (int i = tid; i < kCritSlots; i += nt) run.crit[i] = 0;
  if (row == 0 && tid == 0) {
    *run.item_ctr = 0u;
    *run.pool_ctr = 0u;
    run.counters[0] = run.counters[1] = run.counters[2] = run.counters[3] = 0ull;
    *run.status = 0;
  }
  for (int i = tid; i <= M; i += nt) s_cnt[i] = 0;
  if (tid == 0) s_inf = 0;
  __syncthreads();
  const float* ch = run.chrom + ir.chrom_off + (long long)c * 2 * N;
  const double* thr = tb.thr + id.thrbase;
  for (int i = tid; i < S2; i += nt) {
    unsigned long long key = ~0ull;
    if (i < N) {
      const int m = machine_of(ch[N + i], thr, M, id.mode);
      atomicAdd(&s_cnt[m], 1);
      const int t = tb.gene_type[id.gbase + i] - id.tbase;
      if (m < M && !tb.fits[id.tmbase + t * M + m]) s_inf = 1;  // placement.py:47-53
      key = ((unsigned long long)m << 48) | ((unsigned long long)ordered_bits(ch[i]) << 16) |
            (unsigned long long)i;
    }
    keys[i] = key;
  }
  __syncthreads();
  for (int kk = 2; kk <= S2; kk <<= 1) {
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < S2; i += nt) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = keys[i], b = keys[ixj];
          const bool up = (i & kk) == 0;
          if ((a > b) == up) {
            keys[i] = b;
            keys[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0) {
    int acc = 0;
    for (int m = 0; m < M; ++m) {
      s_start[m] = acc;
      acc += s_cnt[m];
    }
  }
  __syncthreads();
  uint16_t* seq = run.seq + ir.seq0 + (long long)c * M * N;
  for (int i = tid; i < N; i += nt) {
    const unsigned long long key = keys[i];
    const int m = (int)(key >> 48);
    if (m < M) seq[(long long)m * N + (i - s_start[m])] = (uint16_t)(key & 0xFFFFu);
  }
  for (int m = tid; m < M; m += nt) run.cnt[ir.item0 + c * M + m] = s_cnt[m];
  if (tid == 0) run.infeas[row] = s_inf;
}

// Weight of an item for the longest-first order: its part count, 0 when the
// chromosome is infeasible (nothing to decode).
__device__ __forceinline__ int item_weight(const Tables& tb, const Run& run, int item) {
  const int k = inst_of_item(run, item);
  const int row = run.r[k].crow0 + (item - run.r[k].item0) / tb.inst[k].M;
  return run.infeas[row] ? 0 : run.cnt[item];
}

// Items of all instances in decreasing part count: the persistent CTAs pull
// them in this order, so the longest decodes start first.
__global__ void order_items_kernel(const __grid_constant__ Tables tb, const __grid_constant__ Run run) {
  extern __shared__ int start[];  // Nmax + 1 weights
  const int tid = threadIdx.x, nt = blockDim.x, Nw = run.Nmax;
  for (int i = tid; i <= Nw; i += nt) start[i] = 0;
  __syncthreads();
  for (int i = tid; i < run.n_items; i += nt) atomicAdd(&start[item_weight(tb, run, i)], 1);
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int w = Nw; w >= 0; --w) {
      const int h = start[w];
      start[w] = acc;
      acc += h;
    }
  }
  __syncthreads();
  for (int i = tid; i < run.n_items; i += nt) run.order[atomicAdd(&start[item_weight(tb, run, i)], 1)] = i;
}

// Shared state of one plate search by a CTA of kWarps warps.
template <int kWarps>
struct SearchShared {
  unsigned long long best;
  int chunk, total, nr;
  int rlist[4];
  RotDev rd[4];      // their descriptors, read by every chunk
  int nw[4];         // 64-column words of their candidates in a row
  unsigned inv[4];   // ceil(2^32 / nw)
  unsigned char surv[kWarps][32];  // per warp: lanes whose candidate passed the vacancy filter
};

// Best placement key of part type t (absolute) on one plate (kKeyNone if it
// does not fit): the CTA's warps pull (rotation, 32 candidate top rows)
// chunks from a shared counter (rotations interleaved, bottom rows first),
// skip chunks that cannot beat the best key found so far, stop once no
// rotation can at the current level, and merge with atomicMin.  Called by
// all threads of the CTA; contains __syncthreads.
template <bool kPlain, int kWarps>
__device__ __forceinline__ unsigned long long search_plate(const Tables& tb, const MachDev& md,
                                                           const PlateRef& pr, int enc,
                                                           int t, const RotList* rlp, int task_max, int32_t* status,
                                                           SearchShared<kWarps>& sh,
                                                           unsigned long long& c_tests,
                                                           unsigned long long& c_chunks,
                                                           unsigned long long& c_bytes) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 4) {  // one thread per rotation: the list was built at problem creation
    const int nr0 = rlp->nr;
    // The shortest rotation first has the smallest best-case key and prunes
    // the others sooner (measured 2-4 % off in every launch shape).
    if (tid < nr0) {
      const int r = rlp->rs[tid];
      const RotDev rd = tb.rot[t * 4 + r];
      const int nw = (md.W - rd.w + 64) >> 6;
      sh.rlist[tid] = r;
      sh.rd[tid] = rd;
      sh.nw[tid] = nw;
      sh.inv[tid] = nw > 1 ? 0xFFFFFFFFu / (unsigned)nw + 1u : 0u;
    }
    if (tid == 0) {
      sh.nr = nr0;
      sh.total = nr0 ? nr0 * ((md.L - rlp->hmin + 1 + 31) >> 5) : 0;
      sh.best = kKeyNone;
      sh.chunk = 0;
      c_tests += nr0;
      c_bytes += 4ull * rlp->scan_words;
    }
  }
  __syncthreads();
  const int nr = sh.nr, total = sh.total;
  unsigned char* surv = sh.surv[tid >> 5];
  for (int guard = 0; guard < total; ++guard) {
    int ci = 0;
    unsigned long long best = 0;
    if (lane == 0) {
      ci = atomicAdd(&sh.chunk, 1);
      best = *(volatile unsigned long long*)&sh.best;
    }
    ci = __shfl_sync(kFull, ci, 0);
    if (ci >= total) break;
    best = __shfl_sync(kFull, best, 0);
    const int level = nr == 4 ? ci >> 2 : nr == 2 ? ci >> 1 : nr == 1 ? ci : ci / 3;
    const int slot = ci - level * nr;
    const int h = sh.rd[slot].h, r = sh.rlist[slot];
    const int ty_hi = md.L - h - 32 * level;
    if (ty_hi < 0) continue;
    if (key_of(row_key(max(enc, md.L - ty_hi), ty_hi + h - 1), 0, r) >= best) {
      // The best key a chunk can give only grows with its level, and the best
      // found only shrinks: when no rotation can beat it at this level, no
      // later chunk (same level or higher) can, and the warp is done.
      bool beat = false;
      for (int j = 0; j < nr; ++j) {
        const int hj = sh.rd[j].h, tyj = md.L - hj - 32 * level;
        beat |= tyj >= 0 && key_of(row_key(max(enc, md.L - tyj), tyj + hj - 1), 0, sh.rlist[j]) < best;
      }
      if (!beat) break;
      continue;
    }
    if (lane == 0) ++c_chunks;
    // Vacancy filter, one candidate row per lane.  Then, when there are few
    // enough (surviving row, 64 candidate columns) pairs, they are dealt to the
    // lanes in rounds of 32, bottom-most row and leftmost columns first:
    //   1. each lane tests its pair's cores against the erosion planes;
    //   2. where that leaves several pairs open, groups of lanes test the first
    //      pieces of their runs;
    //   3. the pairs still open are finished in order by the whole warp: every
    //      lane walks every 32nd piece of the mask's runs, the lanes' blocked
    //      columns are ORed after each step.  The first pair that stays free is
    //      the bottom-most candidate's leftmost x, and the chunk is done.
    // Otherwise each lane tests its own candidate's words left to right.
    const int ty = ty_hi - lane, rot = t * 4 + r, nx = md.W - sh.rd[slot].w + 1;
    const bool pass = ty >= 0 && coarse_ok(tb, pr.vac, ty, rot);
    const unsigned S = __ballot_sync(kFull, pass);
    if (!S) continue;
    const int nw = sh.nw[slot], ntask = __popc(S) * nw;
    if (ntask > task_max) {
      const int x = pass ? first_free_x(tb, pr, md, ty, rot, sh.rd[slot]) : -1;
      const unsigned fm = __ballot_sync(kFull, x >= 0);
      if (fm) {
        const int l = __ffs(fm) - 1;
        const int xb = __shfl_sync(kFull, x, l);
        if (lane == 0)
          atomicMin(&sh.best, key_of(row_key(max(enc, md.L - (ty_hi - l)), ty_hi - l + h - 1), xb, r));
      }
      continue;
    }
    __syncwarp();  // the last chunk's list is read
    if (pass) surv[__popc(S & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const unsigned inv = sh.inv[slot];
    const uint2* segs = tb.truns + sh.rd[slot].tseg;
    // More than sixteen open pairs: every lane tests its own, if it is open, which
    // saves finding the lanes' pairs (P50M2 100 rows 0.323 -> 0.318 ms, 200 parts of
    // 5-15 cells 1.89 -> 1.75); not in the plain one-warp form, which is slower for
    // it (64 uneven instances x 256 19.5 -> 19.9 ms).
    constexpr bool kOwnPairs = !kPlain || kWarps > 1;
    const int nseg = sh.rd[slot].ntseg, gseg = kPlain ? kGroupSegs : sh.rd[slot].gseg;
    bool won = false;
    for (int t0 = 0; t0 < ntask && !won; t0 += 32) {
      // ---- the round's first pair has the smallest key left in the chunk: stop when it cannot win
      if (lane == 0) best = *(volatile unsigned long long*)&sh.best;
      best = __shfl_sync(kFull, best, 0);
      const int ti = t0 + lane, si = nw > 1 ? (int)__umulhi((unsigned)ti, inv) : ti;
      const int base = (ti - si * nw) << 6, row0 = ti < ntask ? ty_hi - surv[si] : 0;
      const unsigned long long low = key_of(row_key(max(enc, md.L - row0), row0 + h - 1), base, r);
      if (__shfl_sync(kFull, low, 0) >= best) break;
      // ---- coarse test of one pair per lane
      uint2 F = make_uint2(0u, 0u);
      if (ti < ntask) {
        if (pair_in_plate(row0, base, h, md.W - nx + 1, md)) {
          F = coarse_and(tb, pr.planes, md, row0, base, first_open(nx, base), rot);
        } else {  // never on consistent tables: skip the pair, flag the launch
          raise_status(status, BRKGA_ERR_INTERNAL);
        }
      }
      unsigned open = __ballot_sync(kFull, (F.x | F.y) != 0u);
      const int n_open = __popc(open), pk = row0 << 13 | base;
      int q0 = 0;
      // ---- several pairs open: 32 / 2^lg of them at once, 2^lg lanes each
      if (n_open >= kGroupOpen && gseg) {
        const int lg = n_open <= 4 ? 3 : n_open <= 8 ? 2 : n_open <= 16 ? 1 : 0;
        unsigned m = open;
        if (!kOwnPairs || lg) {
          for (int k = 0; k < (32 >> lg) - 1; ++k)
            if (k < lane >> lg) m &= m - 1u;  // drop the pairs of the groups below
        } else {
          m &= 1u << lane;  // a lane each: its own
        }
        const int src = m ? __ffs(m) - 1 : 0;
        const int pl = __shfl_sync(kFull, pk, src);
        uint32_t lo = __shfl_sync(kFull, F.x, src), hi = __shfl_sync(kFull, F.y, src);
        if (!m) lo = hi = 0u;
        const int basel = pl & 0x1FFF, n = min(max(gseg, 1 << lg), nseg);
        const uint32_t* g0 = pr.grid + (size_t)(pl >> 13) * md.RS;
        for (int q = lane & ((1 << lg) - 1); q < n && (lo | hi); q += 1 << lg) {
          const uint2 e = __ldg(segs + q);
          const uint2 b = blocked64(g0 + (size_t)e.y * md.RS, basel + (int)(e.x & 0xFFFFu), (int)(e.x >> 16), md.RS);
          lo &= ~b.x;
          hi &= ~b.y;
        }
        __syncwarp();
        for (int o = 1; o < 1 << lg; o <<= 1) {
          lo &= __shfl_xor_sync(kFull, lo, o);
          hi &= __shfl_xor_sync(kFull, hi, o);
        }
        // this lane's pair was the group's at `from`
        const int from = !kOwnPairs || lg ? __popc(open & ((1u << lane) - 1u)) << lg : lane;
        F.x &= __shfl_sync(kFull, lo, from & 31);
        F.y &= __shfl_sync(kFull, hi, from & 31);
        open &= __ballot_sync(kFull, (F.x | F.y) != 0u);
        q0 = max(gseg, 1 << lg);
      }
      // ---- exact test of the open pairs in order
      while (open) {
        const int l = __ffs(open) - 1;
        open &= open - 1u;
        const int pl = __shfl_sync(kFull, pk, l);
        uint32_t lo = __shfl_sync(kFull, F.x, l), hi = __shfl_sync(kFull, F.y, l);
        const int basel = pl & 0x1FFF, rowl = pl >> 13;
        const unsigned rk = row_key(max(enc, md.L - rowl), rowl + h - 1);
        if (key_of(rk, basel, r) >= best) break;
        const uint32_t* g0 = pr.grid + (size_t)rowl * md.RS;
        for (int q = q0; q < nseg && (lo | hi); q += 32) {
          uint32_t bx = 0u, by = 0u;
          if (q + lane < nseg) {
            const uint2 e = __ldg(segs + q + lane);
            const uint2 b = blocked64(g0 + (size_t)e.y * md.RS, basel + (int)(e.x & 0xFFFFu), (int)(e.x >> 16), md.RS);
            bx = b.x;
            by = b.y;
          }
          lo &= ~__reduce_or_sync(kFull, bx);
          hi &= ~__reduce_or_sync(kFull, by);
        }
        if (lo | hi) {
          if (lane == 0) atomicMin(&sh.best, key_of(rk, basel + (lo ? __ffs(lo) - 1 : 31 + __ffs(hi)), r));
          won = true;
          break;
        }
      }
    }
  }
  __syncthreads();
  return sh.best;
}

// The erosion planes and vacancies of whole blocks b0 .. b1 of a plate, from its
// rows.  A group of 8, 16 or 32 lanes takes a block, a lane one word of it (on
// plates wider than 1024 columns a warp walks the row in steps that overlap by
// the words an erosion reaches).  All threads of the CTA; no barrier.
template <bool kPlain>
__device__ __forceinline__ void update_blocks(const Tables& tb, const MachDev& md, const PlateRef& pr, int b0, int b1) {
  const int lane = threadIdx.x & 31;
  const int G = md.NW <= 8 ? 8 : md.NW <= 16 ? 16 : 32, gl = lane & (G - 1);
  const int groups = blockDim.x / G;
  constexpr int kReach = (1 << kPlaneMax) / 32 + 1;  // words past its own that a plane word depends on
  const int step = kPlain || md.NW <= 32 ? 32 : 32 - kReach;
  for (int bb = b0; bb <= b1; bb += groups) {
    const int b = bb + (int)threadIdx.x / G;
    const bool on = b <= b1;
    const uint32_t* row = pr.grid + (size_t)(b << tb.bsh) * md.RS;
    const int rows = min(1 << tb.bsh, md.L - (b << tb.bsh));  // 1 << bsh; written so it compiles 1 % faster
    for (int w0 = 0; w0 < md.NW; w0 += step) {
      const int w = w0 + gl;
      const uint32_t e0 = on && w < md.NW ? block_free(row, md.RS, md.W, rows, w) : 0u;
      uint32_t* dst = pr.planes + (size_t)b * tb.n_planes * md.RS + w;
      const bool put = on && w < md.NW && gl < step;
      uint32_t e = e0;
#pragma unroll
      for (int k = 1; k <= kPlaneMax; ++k) {
        if (k >= kPlaneMin + tb.n_planes) break;
        uint32_t nx = __shfl_down_sync(kFull, e, 1, G);
        if (gl + 1 >= G) nx = 0u;
        e &= __funnelshift_r(e, nx, 1 << (k - 1));
        if (k >= kPlaneMin && put) dst[(k - kPlaneMin) * md.RS] = e;
      }
      if (kPlain || md.NW <= 32) {
        // longest run of set bits over the group's words: inside a word, or
        // from a word's top bits through full words into the next one's low bits
        const unsigned fm = __ballot_sync(kFull, e0 == kFull) >> (lane - gl);
        const unsigned rest = ~(fm >> gl >> 1);  // bit i: lane gl + 1 + i is not full
        const int hop = min(__ffs(rest) - 1, G - 1 - gl);  // full lanes that follow
        const int low = e0 == kFull ? 32 : __ffs(~e0) - 1;
        int end = __shfl_sync(kFull, low, lane - gl + min(gl + 1 + hop, G - 1));
        if (gl + 1 + hop >= G) end = 0;
        int run = longest_ones(e0);
        if (e0 != kFull || gl == 0) run = max(run, (e0 == kFull ? 32 : __clz(~e0)) + 32 * hop + end);
        for (int o = G >> 1; o; o >>= 1) run = max(run, __shfl_xor_sync(kFull, run, o, G));
        if (on && gl == 0) pr.vac[b] = (uint16_t)run;
      }
    }
    if (!kPlain && md.NW > 32 && on) {  // the group is the warp
      const int run = max_free_run(row, md.RS, md.W, md.NW, rows);
      if (gl == 0) pr.vac[b] = (uint16_t)run;
    }
  }
}

// OR a mask row of mw <= kWords words into a plate row, sx bits into its first
// word: all loads first, so their latencies overlap.  Unrolled to the bound, the
// row costs kWords words' instructions whatever it holds, so rows of up to four
// words (masks to 128 columns) have their own: one launch 2 % off against eight
// for all (P100M4 500 rows 1.10 -> 1.08 ms, 4,000 5.79 -> 5.68, P400M8 1,024
// 19.95 -> 19.6), 7 % off where items hold four parts.
template <int kWords>
__device__ __forceinline__ void or_row(uint32_t* dst, const uint32_t* m, int mw, int sx) {
  uint32_t w[kWords];
#pragma unroll
  for (int j = 0; j < kWords; ++j) w[j] = j < mw ? __ldg(m + j) : 0u;
  uint32_t prev = 0u;
#pragma unroll
  for (int j = 0; j < kWords; ++j) {
    if (j < mw) {
      const uint32_t v = __funnelshift_l(prev, w[j], sx);
      if (v) dst[j] |= v;
      prev = w[j];
    }
  }
  const uint32_t v = __funnelshift_l(prev, 0u, sx);
  if (v) dst[mw] |= v;
}

// Insert rotation r of part type t (absolute) with its top row at ty and left
// column x (binClassNew.py:155-174): OR the mask rows into the plate words,
// then recompute the touched blocks' planes and vacancies (where the test is by
// rows, the row's vacancy with the row); thread 0 updates the plate scalars with the part's area and times on this machine.  Without
// `cells` (no search of the item follows) only the scalars.
// All threads of the CTA; ends with __syncthreads.
template <bool kPlain>
__device__ __forceinline__ void place_part(const Tables& tb, const MachDev& md, const PlateRef& pr, BinScal* scal, int t,
                                           int r, int x, int ty, double a, double ptv, double pthv, bool cells) {
  const int tid = threadIdx.x;
  const RotDev rd = tb.rot[t * 4 + r];
  const int sx = x & 31, wx = x >> 5, mw = rd.mw;
  const uint32_t* mb = tb.maskbits + rd.mask_base;
  const bool by_rows = !kPlain && tb.bsh == 0;
  for (int i = tid; i < rd.h && cells; i += blockDim.x) {
    uint32_t* row = pr.grid + (size_t)(ty + i) * md.RS;
    const uint32_t* m = mb + (size_t)i * mw;
    uint32_t* dst = row + wx;
    if (mw <= 4) {
      or_row<4>(dst, m, mw, sx);
    } else if (mw <= 8) {
      or_row<8>(dst, m, mw, sx);
    } else {
      uint32_t prev = 0u;
      for (int j = 0; j < mw; ++j) {
        const uint32_t cur = __ldg(m + j);
        const uint32_t v = __funnelshift_l(prev, cur, sx);
        if (v) dst[j] |= v;
        prev = cur;
      }
      const uint32_t v = __funnelshift_l(prev, 0u, sx);
      if (v) dst[mw] |= v;
    }
    if (by_rows) pr.vac[ty + i] = (uint16_t)row_free_run(row, md);
  }
  if (tid == 0) {
    BinScal s = *scal;
    s.area += a;
    s.minrow = min(s.minrow, ty);
    s.maxrow = max(s.maxrow, ty + rd.h - 1);
    s.enc = (s.minrow > s.maxrow) ? 0 : md.L - s.minrow;  // binClassNew.py:147-152
    s.pt += ptv;
    if (pthv > s.pth) s.pth = pthv;
    *scal = s;
  }
  __syncthreads();
  if (!cells || by_rows) return;
  update_blocks<kPlain>(tb, md, pr, ty >> tb.bsh, min((ty + rd.h - 1) >> tb.bsh, md.NB - 1));
  __syncthreads();
}

// Empty plate: zero words, every run of columns free (binClassNew.py:18-20),
// fresh scalars.  Without `cells` only the scalars.
template <bool kPlain>
__device__ __forceinline__ void open_plate(const Tables& tb, const MachDev& md, const PlateRef& pr, BinScal* scal,
                                           int pool_index, bool cells) {
  const int tid = threadIdx.x;
  if (cells) {
    for (int i = tid; i < md.L * md.RS; i += blockDim.x) pr.grid[i] = 0u;
    const int dw = (int)blockDim.x % md.RS, db = (int)blockDim.x / md.RS;
    for (int b = tid / md.RS, w = tid % md.RS; b < md.NB && (kPlain || tb.n_planes);) {  // w: the word's place in its row
      uint32_t* dst = pr.planes + (size_t)b * tb.n_planes * md.RS + w;
      for (int p = 0; p < tb.n_planes; ++p) {
        const int n = md.W - (1 << (kPlaneMin + p)) + 1 - 32 * w;  // run starts from this word on
        dst[p * md.RS] = n <= 0 ? 0u : n >= 32 ? kFull : (1u << n) - 1u;
      }
      b += db;
      w += dw;
      if (w >= md.RS) {
        w -= md.RS;
        ++b;
      }
    }
    for (int i = tid; i < md.NB; i += blockDim.x) pr.vac[i] = (uint16_t)md.W;
  }
  if (tid == 0) {
    BinScal z;
    z.area = 0.0;
    z.pt = 0.0;
    z.pth = 0.0;
    z.minrow = md.L;
    z.maxrow = -1;
    z.enc = 0;
    z.pool = pool_index;
    *scal = z;
  }
  __syncthreads();
}

__device__ __forceinline__ void decode_key(unsigned long long key, int* r, int* x, int* y) {
  *r = (int)(key & 3ull);
  *x = (int)((key >> 2) & 0x1FFFull);
  *y = kMaxSide - (int)((key >> 32) & 0x1FFFull);
}

// The item a CTA is decoding, set up by thread 0.
struct ItemCtx {
  int item;      // global item index, -1 when the queue is empty
  int row;       // chromosome row of the launch
  int m, M, T;   // machine (local), machines and part types of the instance
  int n;         // parts on this machine
  int N;         // genes of the instance (log entries per item)
  int gbase, tbase, tmbase;
  int infeas;
  long long seq; // first entry of its part order / log
  MachDev md;
};

// The tables go by value (every access has a fixed parameter offset); only
// the per-launch instance array, which is searched, is a grid constant.
// kThreads = 32, 64, 128 or 256 (1, 2, 4 or 8 warps per item); 32 resident warps
// per SM cap the kernel at 64 registers, which it fits without spilling.
// Launches that leave the GPU's SMs with a few items each are bound by one
// item's chain of instructions instead: kRoomyCtas CTAs of 128 threads per SM
// may use 128 registers, which saves reloads, and where every item has an SM to
// itself eight warps finish it sooner than four.  Measured (64 registers / 128 /
// eight warps): P50M2 1 row 0.31 / 0.287 / 0.262 ms, P100M4 20 rows 0.58 / 0.52 /
// 0.436 ms, 100 rows 0.71 / 0.64 / -, P200M6 20 rows 0.61 / 0.55 / 0.49 ms,
// 80 rows 0.77 / 0.66 / -; with 200 items on 148 SMs eight warps gain 2 % (P50M2)
// or lose 5 % (246 small parts).
constexpr int kRoomyCtas = 4;
// kPlain: the test is by blocks and no plate is wider than 1024 columns, as in
// most problems; without what the others need the kernel is 1 to 1.5 % faster
// (P100M4 4,000 rows 5.49 -> 5.42 ms, 500 rows 1.02 -> 0.99).
template <bool kPlain, int kThreads, int kMinCtas = kResidentWarps * 32 / kThreads>
__global__ void __launch_bounds__(kThreads, kMinCtas)
    decode_kernel(const Tables tb, const __grid_constant__ Run run) {
  extern __shared__ __align__(16) uint32_t smem[];
  // Two search states, used by alternate searches: the state a search returns
  // from is not written again until the search after next, by which time every
  // thread has passed the next search's barriers — so a search needs no
  // barrier after reading its result.
  __shared__ SearchShared<kThreads / 32> sh2[2];
  __shared__ ItemCtx ctx;
  int sh_par = 0;
  int owned = 0;  // pool plates this CTA holds, in bs[S .. S + owned)
  __shared__ int s_fail, s_pool;
  const int tid = threadIdx.x, lane = tid & 31;
  BinScal* bs = run.binscal + (size_t)blockIdx.x * run.Nmax;
  unsigned long long c_tests = 0, c_chunks = 0, c_bins = 0, c_bytes = 0;
  unsigned my_sm = 0;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(my_sm));
  my_sm &= (unsigned)(kCritSlots - 1);
  bool crit = false;  // thread 0: this CTA holds a critical item and marked its SM

  for (;;) {
    if (tid == 0) {
      if (crit) {
        atomicSub(&run.crit[my_sm], 1);
        crit = false;
      }
      ctx.item = -1;
      // While another CTA of this SM decodes a critical item, take none: the
      // CTA that holds the mark keeps pulling, so every item is still taken.
      const bool leave = run.crit_items > 0 && *(volatile int*)&run.crit[my_sm] > 0;
      const int q = leave ? run.n_items : (int)atomicAdd(run.item_ctr, 1u);
      if (q < run.crit_items && q < run.n_items) {
        crit = true;
        atomicAdd(&run.crit[my_sm], 1);
      }
      if (q < run.n_items) {
        const int item = run.order[q];
        const int k = inst_of_item(run, item);
        const InstDev id = tb.inst[k];
        const int li = item - run.r[k].item0, c = li / id.M;
        ctx.item = item;
        ctx.row = run.r[k].crow0 + c;
        ctx.m = li - c * id.M;
        ctx.M = id.M;
        ctx.T = id.T;
        ctx.n = run.cnt[item];
        ctx.N = id.N;
        ctx.gbase = id.gbase;
        ctx.tbase = id.tbase;
        ctx.tmbase = id.tmbase;
        ctx.infeas = run.infeas[ctx.row];
        ctx.seq = run.r[k].seq0 + (long long)li * id.N;
        ctx.md = tb.mach[id.mbase + ctx.m];
      }
    }
    __syncthreads();
    const int item = ctx.item;
    if (item < 0) break;
    const MachDev md = ctx.md;
    const int n = ctx.n;
    BrkgaPlacement* lg = run.log ? run.log + ctx.seq : nullptr;
    const uint16_t* seq = run.seq + ctx.seq;
    const int N = ctx.N;
    if (ctx.infeas) {  // any part too large for its machine: the whole chromosome scores 1e16
      if (lg)
        for (int k = tid; k < N; k += kThreads) lg[k] = BrkgaPlacement{-1, -1, -1, -1, -1};
      if (tid == 0) run.mk[item] = 0.0;
      __syncthreads();
      continue;
    }
    if (lg)
      for (int k = n + tid; k < N; k += kThreads) lg[k] = BrkgaPlacement{-1, -1, -1, -1, -1};

    int nb = 0;
    bool failed = false;
    for (int k = 0; k < n && !failed; ++k) {
      const int gene = seq[k];
      const int t = tb.gene_type[ctx.gbase + gene];
      const double a = tb.part_area[t];
      int pb = -1;
      unsigned long long key = kKeyNone;

      // ---- first fit over the open plates (placement.py:56-64)
      for (int b = 0; b < nb; ++b) {
        if (bs[b].area + a > md.area) continue;  // placement.py:57-59
        const PlateRef pr = plate_ref(run, smem, b, bs[b].pool);
        key = search_plate<kPlain>(tb, md, pr, bs[b].enc, t,
                           tb.rl + ctx.tmbase + (size_t)(t - ctx.tbase) * ctx.M + ctx.m, run.task_max, run.status,
                           sh2[sh_par], c_tests, c_chunks, c_bytes);
        sh_par ^= 1;
        if (key != kKeyNone) {
          pb = b;
          break;
        }
      }

      const bool last = k + 1 == n;  // no search follows: the plate's cells are not needed
      int r, x, ty;
      if (pb < 0) {
        // ---- new plate, best rotation at column 0, bottom row L-1 (placement.py:66-83)
        r = tb.best_rot[t];
        if (tid == 0) {
          s_fail = 0;
          s_pool = -1;
          if (!tb.newbin_ok[ctx.tmbase + (t - ctx.tbase) * ctx.M + ctx.m]) {
            s_fail = BRKGA_ERR_NEW_BIN_UNFIT;
          } else if (nb >= run.S) {
            // a pool plate taken for an earlier item stays this CTA's
            const unsigned idx = nb - run.S < owned ? (unsigned)bs[nb].pool : atomicAdd(run.pool_ctr, 1u);
            if ((long long)idx >= run.pool_bins) s_fail = BRKGA_ERR_CAPACITY;
            else s_pool = (int)idx;
          }
        }
        __syncthreads();
        if (s_fail) {
          if (tid == 0) {
            raise_status(run.status, s_fail);
            run.mk[item] = nan("");
          }
          failed = true;
          break;
        }
        pb = nb++;
        owned = max(owned, nb - run.S);
        open_plate<kPlain>(tb, md, plate_ref(run, smem, pb, s_pool), &bs[pb], s_pool, !last);
        if (tid == 0) ++c_bins;
        x = 0;
        ty = md.L - tb.rot[t * 4 + r].h;
      } else {
        int y;
        decode_key(key, &r, &x, &y);
        ty = y - tb.rot[t * 4 + r].h + 1;
      }

      // ---- insert (binClassNew.py:155-174)
      const size_t tm = (size_t)ctx.tmbase + (size_t)ctx.m * ctx.T + (t - ctx.tbase);
      place_part<kPlain>(tb, md, plate_ref(run, smem, pb, bs[pb].pool), &bs[pb], t, r, x, ty, a, tb.pt[tm], tb.pth[tm], !last);
      if (tid == 0 && lg) lg[k] = BrkgaPlacement{gene, pb, x, ty + tb.rot[t * 4 + r].h - 1, r};
    }
    if (!failed && tid == 0) {  // placement.py:86-89
      double ms = 0.0;
      for (int b = 0; b < nb; ++b) ms += (bs[b].pt + bs[b].pth) + md.setup;
      run.mk[item] = ms;
    }
    __syncthreads();
  }
  if (tid == 0) {
    atomicAdd(&run.counters[0], c_tests);
    atomicAdd(&run.counters[2], c_bins);
    atomicAdd(&run.counters[3], c_bytes);
  }
  if (lane == 0) atomicAdd(&run.counters[1], c_chunks);
}

__global__ void reduce_kernel(const __grid_constant__ Tables tb, const __grid_constant__ Run run) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= run.n_rows) return;
  const int k = inst_of_row(run, row);
  double* out = run.out + run.r[k].out_off + (row - run.r[k].crow0);
  if (run.infeas[row]) {
    *out = 1e16;  // placement.py:9,151-153
    return;
  }
  const int M = tb.inst[k].M;
  const double* mk = run.mk + run.r[k].item0 + (long long)(row - run.r[k].crow0) * M;
  double worst = 0.0;
  bool bad = false;
  for (int m = 0; m < M; ++m) {
    const double v = mk[m];
    if (v != v) bad = true;
    else if (v > worst) worst = v;  // placement.py:154-156
  }
  *out = bad ? nan("") : worst;
}

// Greedy initial solution (BRKGA_alg3.py:445-603 with binClassInitialSol.py):
// the parts go in the given order, each where the system makespan after
// placing it is smallest (ties: the later option wins over an earlier one on
// another machine or a new plate, the first existing plate wins within a
// machine): a new plate on some machine (best rotation at column 0, bottom row
// L-1) or any existing plate of the machine that can take it (every plate is
// tested, no area filter).
//
// A part's plate searches are independent and are most of the work, so one
// cluster of kGreedyCtas CTAs shares them: plate b belongs to CTA
// b % kGreedyCtas, which alone reads and writes its grid and scalars (in the
// global pool) and sends every search's key to the other CTAs' shared memory.
// After one cluster barrier per part each CTA has all keys and takes the same
// decision from its own copy of the makespans and of the plates' height times;
// the chosen plate's owner inserts the part while the others go on to the next
// one (the keys of alternate parts have buffers of their own, so none is
// overwritten before every CTA has read it).  What bounds it is the latency of
// one search and one insertion per part: the call took 7.4 ms on one CTA of
// four warps with the search of runs and takes 1.70 ms here at 100 parts on four
// machines (P100M4), 17.4 and 3.2 ms at 200 parts on six (P200M6), 1.34 and 0.77
// ms at 50 parts on two (P50M2).  Before the erosion planes, with four / eight /
// sixteen warps per CTA: 2.9 / 2.4 / 2.35 ms, 5.5 / 4.9 / 4.9 and 1.05 / 0.94 /
// 0.93 ms.
// Single-instance problems only, so every table base is 0.
struct GreedyArgs {
  int N, M, T;
  int32_t* status;
  BinScal* binscal;
  uint32_t* pool;
  uint32_t* cpool;
  int grid_words, coarse_words, vac_off;
  const int32_t* order;
  int n;
  int32_t* out_machine;  // [n]
  BrkgaPlacement* out;   // [n]: gene, plate index within its machine, x, bottom row y, rotation
  int32_t* plate_index;  // [n]: index of the plate within its machine
  double* machine_makespan;  // [M]
  unsigned char* state;      // the CTAs' state in global memory, state_bytes each, or NULL: in shared memory
  size_t state_bytes;
};

// A CTA's state: per plate the keys of two parts, its largest height time and
// its machine's next plate; per machine its makespan, its first and last plate
// and their number.  In shared memory as long as it fits (up to some 8,000 parts).
size_t greedy_state_bytes(int n, int M) { return (size_t)n * 28 + (size_t)M * 20; }
constexpr size_t kGreedyMaxSmem = 229 * 1024;
// Device memory of a call that stays with the problem: a grid and planes a part
// (P100M4 2 MB, P400M8 30 MB).  More, at thousands of parts or plates of thousands
// of cells, is given back by the call: beside so long a call an allocation is nothing.
constexpr size_t kGreedyKeep = (size_t)64 << 20;

__device__ __forceinline__ PlateRef greedy_plate(const GreedyArgs& g, int b) {
  uint32_t* planes = g.cpool + (size_t)b * g.coarse_words;
  return PlateRef{g.pool + (size_t)b * g.grid_words, planes, reinterpret_cast<uint16_t*>(planes + g.vac_off)};
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// All threads of all CTAs of the cluster; shared-memory writes before it, remote ones too, are seen after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Store to the same shared variable of CTA `rank` of the cluster.
__device__ __forceinline__ void cluster_store(unsigned long long* p, unsigned rank, unsigned long long v) {
  const unsigned local = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.u64 [a], %2;\n\t}" ::"r"(local),
               "r"(rank), "l"(v)
               : "memory");
}

__global__ void __launch_bounds__(kGreedyThreads, 1) greedy_kernel(const __grid_constant__ Tables tb,
                                                                const __grid_constant__ GreedyArgs g) {
  extern __shared__ __align__(16) unsigned char gsm[];
  const unsigned rank = cluster_rank();
  unsigned char* state = g.state ? g.state + rank * g.state_bytes : gsm;
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(state);  // [2][n]
  double* pth = reinterpret_cast<double*>(keys + 2 * (size_t)g.n);
  double* makespan = pth + g.n;
  int* next = reinterpret_cast<int*>(makespan + g.M);
  int* first = next + g.n;
  int* last = first + g.M;
  int* count = last + g.M;
  __shared__ SearchShared<kGreedyThreads / 32> sh2[2];  // alternate searches, as in decode_kernel
  struct Choice {
    int machine, plate;  // plate -1: a new one, machine -1: the part fits nowhere
    unsigned long long key;
    double cand;
  };
  __shared__ Choice choice;
  int sh_par = 0;
  const int tid = threadIdx.x;
  BinScal* bs = g.binscal;
  unsigned long long c_tests = 0, c_chunks = 0, c_bytes = 0;  // of search_plate, not reported here
  int nplates = 0;
  double cw = 0.0;  // current_worst_makespan
  for (int m = tid; m < g.M; m += kGreedyThreads) {
    makespan[m] = 0.0;
    first[m] = last[m] = -1;
    count[m] = 0;
  }
  // Plate b lives in pool slot b, so bs[b].pool is free to hold its machine.
  cluster_sync();
  for (int k = 0; k < g.n; ++k) {
    const int gene = g.order[k];
    const int t = tb.gene_type[gene];
    const double a = tb.part_area[t];
    unsigned long long* kk = keys + (size_t)(k & 1) * g.n;
    for (int b = (int)rank; b < nplates; b += kGreedyCtas) {
      const int m = bs[b].pool;
      const MachDev md = tb.mach[m];
      unsigned long long key = kKeyNone;
      if (tb.fits[t * g.M + m]) {  // BRKGA_alg3.py:465-470
        const PlateRef pr = greedy_plate(g, b);
        key = search_plate<false>(tb, md, pr, bs[b].enc, t,
                           tb.rl + (size_t)t * g.M + m, kDefaultTaskMax, g.status, sh2[sh_par], c_tests, c_chunks,
                           c_bytes);
        sh_par ^= 1;
      }
      if (tid < kGreedyCtas) {
        if (g.state) reinterpret_cast<unsigned long long*>(g.state + tid * g.state_bytes)[(size_t)(k & 1) * g.n + b] = key;
        else cluster_store(&kk[b], (unsigned)tid, key);
      }
    }
    cluster_sync();
    if (tid == 0) {
      Choice best{-1, -1, kKeyNone, 0.0};
      double bv = INFINITY;
      for (int m = 0; m < g.M; ++m) {
        if (!tb.fits[t * g.M + m]) continue;
        bool placed_in_exist = false;
        const double mm = makespan[m];
        const double ptm = tb.pt[(size_t)m * g.T + t], pthm = tb.pth[(size_t)m * g.T + t];
        const double cand = ((mm + tb.mach[m].setup) + ptm) + pthm;  // :472
        const double nm = cw > cand ? cw : cand;
        if (nm <= bv) {
          bv = nm;
          best = Choice{m, -1, kKeyNone, cand};
        }
        for (int b = first[m]; b >= 0; b = next[b]) {
          if (kk[b] == kKeyNone) continue;
          const double cand2 = pth[b] < pthm ? ((mm - pth[b]) + pthm) + ptm : mm + ptm;  // :486-489
          const double nm2 = cw > cand2 ? cw : cand2;
          if (nm2 <= bv) {
            if (placed_in_exist && nm2 == bv) continue;
            placed_in_exist = true;
            bv = nm2;
            best = Choice{m, b, kk[b], cand2};
          }
        }
      }
      choice = best;
      if (best.machine >= 0) {
        const int m = best.machine;
        const double pthm = tb.pth[(size_t)m * g.T + t];
        makespan[m] = best.cand;  // :541, :565
        if (best.plate < 0 && nplates < g.n) {
          const int b = nplates;
          next[b] = -1;
          if (last[m] < 0) first[m] = b;
          else next[last[m]] = b;
          last[m] = b;
          if (b % kGreedyCtas == (int)rank) g.plate_index[b] = count[m];
          ++count[m];
          pth[b] = pthm > 0.0 ? pthm : 0.0;
        } else if (best.plate >= 0 && pthm > pth[best.plate]) {
          pth[best.plate] = pthm;
        }
      }
    }
    __syncthreads();
    const Choice c = choice;
    // The same decision in every CTA, so all of them leave here together.
    if (c.machine < 0) {  // fits no machine: the reference crashes here (bestBatch == [])
      if (tid == 0 && rank == 0) raise_status(g.status, BRKGA_ERR_BAD_INSTANCE);
      return;
    }
    const MachDev md = tb.mach[c.machine];
    int r, x, ty, b = c.plate;
    const bool fresh = b < 0;
    if (fresh) {
      if (!tb.newbin_ok[t * g.M + c.machine] || nplates >= g.n) {
        if (tid == 0 && rank == 0) raise_status(g.status, BRKGA_ERR_NEW_BIN_UNFIT);
        return;
      }
      r = tb.best_rot[t];
      b = nplates++;
      x = 0;
      ty = md.L - tb.rot[t * 4 + r].h;
    } else {
      int y;
      decode_key(c.key, &r, &x, &y);
      ty = y - tb.rot[t * 4 + r].h + 1;
    }
    cw = cw > c.cand ? cw : c.cand;
    if ((unsigned)b % kGreedyCtas == rank) {
      const PlateRef pr = greedy_plate(g, b);
      if (fresh) open_plate<false>(tb, md, pr, &bs[b], c.machine, true);
      place_part<false>(tb, md, pr, &bs[b], t, r, x, ty, a, tb.pt[(size_t)c.machine * g.T + t],
                 tb.pth[(size_t)c.machine * g.T + t], true);
      if (tid == 0) {
        g.out_machine[k] = c.machine;
        g.out[k] = BrkgaPlacement{gene, g.plate_index[b], x, ty + tb.rot[t * 4 + r].h - 1, r};
      }
    }
    __syncthreads();  // `choice` is read
  }
  if (rank == 0)
    for (int m = tid; m < g.M; m += kGreedyThreads) g.machine_makespan[m] = makespan[m];
  cluster_sync();  // no CTA leaves while another may still store into its shared memory
}

// ---------------------------------------------------------------- chunk tests
// The collision test of one 32-row candidate chunk by either path, for the
// measurement that decides between them (brkga_chunk_free): the bit-packed
// run-dilation search the decode kernel uses (word_free, every word tested
// to the end, no early stop) and the INT8 tensor-core correlation
// (corr_i8.cuh).  Both write the same words: row n = candidate top row
// ty_hi - n, bit b of word k = placement at x = 32k + b is collision-free.

// The item's plate geometry and rotation, checked against the tables; false
// (and BRKGA_ERR_INVALID_ARGUMENT raised) when the item is malformed.
__device__ __forceinline__ bool chunk_item(const Tables& tb, const BrkgaChunkTest& it, int M, int T, int max_side,
                                           corr::ChunkArgs* a, RotDev* rdo, int32_t* status) {
  bool ok = it.plate && it.out && it.machine >= 0 && it.machine < M && it.part_type >= 0 && it.part_type < T &&
            it.rot >= 0 && it.rot < tb.nrot[it.part_type];
  if (ok) {
    const MachDev md = tb.mach[it.machine];
    const RotDev rd = tb.rot[it.part_type * 4 + it.rot];
    ok = rd.h <= md.L && rd.w <= md.W && rd.h <= max_side && rd.w <= max_side && it.ty_hi >= 0 &&
         it.ty_hi <= md.L - rd.h;
    a->plate = it.plate;
    a->L = md.L;
    a->W = md.W;
    a->RS = md.RS;
    a->mask = tb.maskbits + rd.mask_base;
    a->h = rd.h;
    a->w = rd.w;
    a->mw = rd.mw;
    a->ty_hi = it.ty_hi;
    a->out = it.out;
    *rdo = rd;
  }
  if (!ok && threadIdx.x == 0 && blockIdx.y == 0) raise_status(status, BRKGA_ERR_INVALID_ARGUMENT);
  return ok;
}

__global__ void __launch_bounds__(128, 8) chunk_free_bitset_kernel(const Tables tb, const BrkgaChunkTest* items, int M,
                                                                int T, int32_t* status) {
  const BrkgaChunkTest it = items[blockIdx.x];
  corr::ChunkArgs a;
  RotDev rd;
  if (!chunk_item(tb, it, M, T, kMaxSide, &a, &rd, status)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nx = a.W - a.w + 1, nwo = (nx + 31) >> 5;
  for (int n = warp; n < corr::kN; n += 4) {
    const int ty = a.ty_hi - n;
    for (int k = lane; k < nwo; k += 32) {
      uint32_t F = 0u;
      if (ty >= 0) {
        const uint32_t F0 = (k == nwo - 1 && (nx & 31)) ? ((1u << (nx & 31)) - 1u) : kFull;
        F = word_free(a.plate + (size_t)ty * a.RS, a.RS, k << 5, F0, rd, tb.truns);
      }
      a.out[(size_t)n * nwo + k] = F;
    }
  }
}

// grid (items, candidate-column tiles of 128); one CTA per SM (its shared memory)
__global__ void __launch_bounds__(corr::kThreads, 1) chunk_free_i8_kernel(const Tables tb,
                                                                          const BrkgaChunkTest* items, int M, int T,
                                                                          int32_t* status) {
  extern __shared__ __align__(1024) unsigned char csmem[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int fail;
  const BrkgaChunkTest it = items[blockIdx.x];
  corr::ChunkArgs a;
  RotDev rd;
  if (!chunk_item(tb, it, M, T, corr::kMaxSide, &a, &rd, status)) return;
  if ((int)blockIdx.y * corr::kTileM > a.W - a.w) return;  // no candidate column in this tile
  corr::chunk_tile(a, (int)blockIdx.y, csmem, bar, &tmem_slot, &fail, status);
}

// ---------------------------------------------------------------- host side

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Layout {
  size_t off_ctr, off_crit, off_seq, off_cnt, off_inf, off_ord, off_mk, off_bins, off_pool, end_pool, off_cpool, total;
};

// Sizes of one launch: chromosome rows, (chromosome, machine) items, part-order entries.
struct LaunchCounts {
  int64_t rows = 0, items = 0, seq = 0;
};

// One launch shape of the decode kernel.
struct Shape {
  int warps = 4;     // per CTA (one item per CTA)
  int ctas = 0;      // resident CTAs per SM
  int S = 0;         // plates per item that are the CTA's own
  size_t smem = 0;   // dynamic shared memory per CTA (their grids, when asked for)
  int n_slots = 0;   // resident CTAs on the GPU (the persistent grid)
};

}  // namespace

// Fixed device scratch for brkga_decode_noalloc: every GPU that loads this
// library reserves it until the process exits.  Host code must not use the
// symbol as an address; brkga_problem_create looks up its device address.
// The tables and the pool plates' grids go into the first array, their erosion
// planes and the CTAs' own plates into the second; the pool has as many plates
// as both have room for.  The second does not limit it before the start of
// another plate in the first: a plate's planes are at most as large as its grid
// (four rows for a whole block of four or eight), so the CTAs' own plates take
// at most twice the 31.5 MB of grids that shared memory would hold.  (With planes
// for a block that is only begun, plates of 13 rows had room for 8,900 plates
// instead of 10,600.)
static __device__ __align__(256) unsigned char g_noalloc_scratch[BRKGA_NOALLOC_SCRATCH_BYTES];
constexpr size_t kNoallocPlaneBytes = (size_t)2 * BRKGA_NOALLOC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_noalloc_planes[kNoallocPlaneBytes];

struct BrkgaProblem {
  int device = 0;
  void* noalloc_scratch = nullptr;  // device addresses of g_noalloc_scratch and g_noalloc_planes on `device`
  void* noalloc_planes = nullptr;
  int K = 0;                        // instances
  std::vector<InstDev> inst;
  std::vector<int> s2;              // bitonic sort width per instance
  int S2max = 1, Nmax = 0;
  int N = 0, M = 0, T = 0, mode = 0;  // instance 0 (the single-instance entry points)
  int sm_count = 0;
  int req_warps = 0, req_ctas = 0, req_plates = -1;  // requested launch shape (0 / 0 / -1 = automatic)
  int task_max = kDefaultTaskMax;
  bool plain = false;  // the kernels' plain forms serve (see decode_kernel)
  Shape shape[3];      // 4, 2 and 1 warps per item
  int64_t pool_per_cta = 0;  // plates an item may open (default_pool_bins())
  int min_S = 0;       // fewest own plates per CTA of the three shapes (pool sizing)
  int grid_words = 0, coarse_words = 0, vac_off = 0;  // words of a plate's grid, of its planes and vacancies, of the planes
  std::vector<MachDev> mach;
  std::vector<void*> allocations;
  Tables tb{};
  InstDev* d_inst = nullptr;
  int32_t* d_gene_type = nullptr;
  double* d_thr = nullptr;
  MachDev* d_mach = nullptr;
  double* d_pt = nullptr;
  double* d_pth = nullptr;
  double* d_area = nullptr;
  int32_t* d_nrot = nullptr;
  int32_t* d_best = nullptr;
  RotDev* d_rot = nullptr;
  CoarseIdx* d_cidx = nullptr;
  uint2* d_centry = nullptr;
  uint32_t* d_cfilter = nullptr;
  uint2* d_truns = nullptr;
  uint32_t* d_maskbits = nullptr;
  uint8_t* d_fits = nullptr;
  uint8_t* d_newbin_ok = nullptr;
  RotList* d_rl = nullptr;
  double* d_bin_area = nullptr;
  // brkga_evaluate_host state
  std::mutex mu;
  cudaStream_t stream = nullptr;
  float* e_chrom = nullptr;
  double* e_out = nullptr;
  int32_t* e_status = nullptr;
  BrkgaPlacement* e_log = nullptr;
  // page-locked staging of a call's results: status at 0, counters at 8,
  // makespans from 64, so the three copies back are queued without a
  // staging round trip each and waited for once
  unsigned char* e_host = nullptr;
  void* e_ws = nullptr;
  size_t e_ws_bytes = 0;
  int e_cap_P = 0;
  bool e_cap_log = false;
  int64_t e_pool_bins = 0;
  // brkga_initial_solution_host state
  void* greedy_ws = nullptr;
  size_t greedy_bytes = 0;
  int64_t last_counters[4] = {0, 0, 0, 0};
};

namespace {

int counts_of(const BrkgaProblem* pb, const int32_t* pops, LaunchCounts* lc) {
  LaunchCounts c;
  for (int k = 0; k < pb->K; ++k) {
    if (pops[k] < 0) return BRKGA_ERR_INVALID_ARGUMENT;
    c.rows += pops[k];
    c.items += (int64_t)pops[k] * pb->inst[k].M;
    c.seq += (int64_t)pops[k] * pb->inst[k].M * pb->inst[k].N;
  }
  if (c.rows >= ((int64_t)1 << 31) || c.items >= ((int64_t)1 << 31)) return BRKGA_ERR_INVALID_ARGUMENT;
  *lc = c;
  return BRKGA_OK;
}

// The shape a launch of `items` items uses: the requested CTA size, else
// 4 warps per item while the items fill at most three waves of resident
// 4-warp CTAs (per-item latency dominates), 2 warps up to sixteen waves of
// 2-warp CTAs, 1 warp beyond (throughput dominates; no CTA barriers).
const Shape& pick_shape(const BrkgaProblem* pb, int64_t items) {
  if (pb->req_warps == 4) return pb->shape[0];
  if (pb->req_warps == 2) return pb->shape[1];
  if (pb->req_warps == 1) return pb->shape[2];
  if (items <= 3 * (int64_t)pb->shape[0].n_slots) return pb->shape[0];
  if (items <= 16 * (int64_t)pb->shape[1].n_slots) return pb->shape[1];
  return pb->shape[2];
}

// CTAs whose plate scalars the workspace of a launch of `items` items holds:
// the most resident CTAs of any shape a launch of at most `items` items can
// use, so that a workspace sized for the largest population serves every
// smaller launch too.
int scratch_slots(const BrkgaProblem* pb, int64_t items) {
  if (pb->req_warps) return pick_shape(pb, items).n_slots;
  int n = pb->shape[0].n_slots;
  if (items > 3 * (int64_t)pb->shape[0].n_slots) n = std::max(n, pb->shape[1].n_slots);
  if (items > 16 * (int64_t)pb->shape[1].n_slots) n = std::max(n, pb->shape[2].n_slots);
  return n;
}

// Plates of their own of a launch's CTAs: the most of any shape that a launch
// of at most `items` items can use.
int64_t own_plates(const BrkgaProblem* pb, int64_t items) {
  auto of = [&](const Shape& s) { return std::min<int64_t>(items, s.n_slots) * s.S; };
  if (pb->req_warps) return of(pick_shape(pb, items));
  int64_t n = of(pb->shape[0]);
  if (items > 3 * (int64_t)pb->shape[0].n_slots) n = std::max(n, of(pb->shape[1]));
  if (items > 16 * (int64_t)pb->shape[1].n_slots) n = std::max(n, of(pb->shape[2]));
  return n;
}

Layout layout_of(const BrkgaProblem* pb, const LaunchCounts& lc, int64_t pool_bins) {
  Layout l;
  size_t o = 0;
  l.off_ctr = o;
  o += 64;
  l.off_crit = o = align_up(o, 256);
  o += (size_t)kCritSlots * sizeof(int);
  l.off_seq = o = align_up(o, 256);
  o += (size_t)lc.seq * sizeof(uint16_t);
  l.off_cnt = o = align_up(o, 256);
  o += (size_t)lc.items * sizeof(int32_t);
  l.off_inf = o = align_up(o, 256);
  o += (size_t)lc.rows * sizeof(int32_t);
  l.off_ord = o = align_up(o, 256);
  o += (size_t)lc.items * sizeof(int32_t);
  l.off_mk = o = align_up(o, 256);
  o += (size_t)lc.items * sizeof(double);
  l.off_bins = o = align_up(o, 256);
  o += (size_t)scratch_slots(pb, lc.items) * std::max(pb->Nmax, 1) * sizeof(BinScal);
  l.off_pool = o = align_up(o, 256);
  o += (size_t)pool_bins * pb->grid_words * sizeof(uint32_t);
  l.end_pool = l.off_cpool = o = align_up(o, 256);
  o += (size_t)pool_bins * pb->coarse_words * sizeof(uint32_t);
  o += (size_t)own_plates(pb, lc.items) * (pb->grid_words + pb->coarse_words) * sizeof(uint32_t);
  l.total = align_up(o, 256);
  return l;
}

// Pool plates of a launch whose caller names no number: two an item, four where
// some shape's CTAs have none of their own, as long as that is at most
// pool_per_cta for every CTA that is resident.  A CTA keeps its pool plates for
// its later items, so a launch of several waves needs as many as its resident
// CTAs hold at most: there the pool and the CTAs' own plates take no more memory
// than the grids alone of those two or four would, planes included.  (With planes
// for all of them P100M4 4,000 rows took 1.43 GB, now 0.93; P400M8 4,096 rows 10.0
// and 6.7; before the planes 0.97 and 6.8.)  A workspace sized for a population
// serves every smaller one: the bytes never fall as the items grow.
int64_t default_pool_bins(const BrkgaProblem* pb, int64_t items) {
  const int64_t most = std::max<int64_t>(256, items * (pb->min_S > 0 ? 2 : 4));
  const int64_t plate = pb->grid_words + pb->coarse_words;
  const int64_t fit = (most * pb->grid_words - own_plates(pb, items) * plate) / plate;
  return std::min(most, std::max(pb->pool_per_cta * scratch_slots(pb, items), fit));
}

// Plates an item may open, whatever its chromosome: all parts on the machine
// that needs most for them, plates filled to kLeastFill at least, a plate for
// each part that no second one like it fits beside; kPoolPerCta or more.
constexpr double kLeastFill = 0.4;
constexpr int kPoolPerCta = 16;
int pool_per_cta(const BrkgaProblemDesc* descs, int K) {
  double most = kPoolPerCta;
  for (int k = 0; k < K; ++k) {
    const BrkgaProblemDesc& d = descs[k];
    for (int m = 0; m < d.n_machines; ++m) {
      const double L = d.bin_length[m], W = d.bin_width[m];
      double plates = 0.0;
      for (int j = 0; j < d.n_genes; ++j) {
        const int t = d.gene_type[j], r = t * 4 + d.part_best_rot[t];
        const bool alone = 2 * std::min(d.rot_h[r], d.rot_w[r]) > std::max(L, W);
        plates += alone ? 1.0 : std::min(1.0, d.part_area[t] / (kLeastFill * L * W));
      }
      most = std::max(most, plates);
    }
  }
  return (int)std::ceil(std::min(most, (double)kMaxGenes));
}

template <typename T>
int upload(BrkgaProblem* pb, T** dst, const std::vector<T>& src) {
  const size_t bytes = std::max<size_t>(1, src.size()) * sizeof(T);
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) return BRKGA_ERR_CUDA;
  pb->allocations.push_back(p);
  if (!src.empty() && cudaMemcpy(p, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  *dst = static_cast<T*>(p);
  return BRKGA_OK;
}

class DeviceGuard {
 public:
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev_);
    if (prev_ != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() { cudaSetDevice(prev_); }

 private:
  int prev_ = 0;
};

// The forms of the decode kernel: warps per item, and with 128 registers for
// launches of few items (kRoomyCtas).
enum Form { kForm1, kForm2, kForm4, kForm4Roomy, kForm8, kForms };
using DecodeKernel = void (*)(const Tables, const Run);
template <bool kPlain>
DecodeKernel decode_form(Form f) {
  return f == kForm1        ? decode_kernel<kPlain, 32>
         : f == kForm2      ? decode_kernel<kPlain, 64>
         : f == kForm4      ? decode_kernel<kPlain, 128>
         : f == kForm4Roomy ? decode_kernel<kPlain, 128, kRoomyCtas>
                            : decode_kernel<kPlain, 256, 2>;
}

DecodeKernel decode_form(const BrkgaProblem* pb, Form f) {
  return pb->plain ? decode_form<true>(f) : decode_form<false>(f);
}

int prepare_kernel(const BrkgaProblem* pb, Form f, size_t dyn_max) {
  return cudaFuncSetAttribute(decode_form(pb, f), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_max) == cudaSuccess
             ? BRKGA_OK
             : BRKGA_ERR_CUDA;
}

int occupancy(const BrkgaProblem* pb, int warps, size_t smem, int* occ) {
  const Form f = warps == 1 ? kForm1 : warps == 2 ? kForm2 : kForm4;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, decode_form(pb, f), 32 * warps, smem) == cudaSuccess
             ? BRKGA_OK
             : BRKGA_ERR_CUDA;
}

// Launch shapes of the decode kernel, one per CTA size (4, 2 and 1 warps per
// item): resident CTAs per SM and plates per item kept in shared memory.
// For the requested CTA size (warps_req), ctas_req = 0 picks the CTAs
// automatically (32 resident warps per SM, the register limit) and
// plates_req = -1 keeps no grid in shared memory, but gives each CTA as many
// plates of its own in the workspace as would fit in its share (at most 4);
// the other CTA size, or both when warps_req = 0, gets the automatic shape.
// A requested shape that cannot be resident is refused.
int configure(BrkgaProblem* pb, int warps_req, int ctas_req, int plates_req) {
  if (warps_req == 0 && (ctas_req != 0 || plates_req != -1)) return BRKGA_ERR_INVALID_ARGUMENT;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, pb->device) != cudaSuccess) return BRKGA_ERR_CUDA;
  pb->sm_count = prop.multiProcessorCount;
  // A plate of machine m uses its own L x RS words, n_planes x NB x RS plane
  // words and NB vacancies: a slot holds the largest of each of any machine
  // (not Lmax x RSmax, which for a tall plate beside a wide one is far more
  // than either needs).
  int NBmax = 0, Lmax = 0, grid = 0, planes = 0;
  for (const MachDev& m : pb->mach) {
    NBmax = std::max(NBmax, m.NB);
    Lmax = std::max(Lmax, m.L);
    grid = std::max(grid, m.L * m.RS);
    planes = std::max(planes, pb->tb.n_planes * m.NB * m.RS);
  }
  const int grid_words = (int)align_up((size_t)grid, 4);
  const int coarse_words = (int)std::max<size_t>(4, align_up((size_t)planes + (size_t)(NBmax + 1) / 2, 4));
  const size_t grid_bytes = (size_t)grid_words * 4;
  // room of a plate in shared memory: its grid and two bytes a row
  const size_t slot_bytes = align_up((size_t)grid + (size_t)(Lmax + 1) / 2, 4) * 4;
  // Every kernel of a decode is looked up here, which loads it: a kernel first
  // used by a launch is loaded inside that call.
  cudaFuncAttributes fa[kForms], other;
  for (int f = 0; f < kForms; ++f)
    if (cudaFuncGetAttributes(&fa[f], decode_form(pb, (Form)f)) != cudaSuccess) return BRKGA_ERR_CUDA;
  if (cudaFuncGetAttributes(&other, assign_sort_kernel) != cudaSuccess ||
      cudaFuncGetAttributes(&other, order_items_kernel) != cudaSuccess ||
      cudaFuncGetAttributes(&other, reduce_kernel) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  // the forms that may have plates in shared memory
  const size_t static_smem =
      std::max({fa[kForm4].sharedSizeBytes, fa[kForm2].sharedSizeBytes, fa[kForm1].sharedSizeBytes});
  const size_t per_sm = prop.sharedMemPerMultiprocessor;
  const size_t per_block_max = prop.sharedMemPerBlockOptin - static_smem;  // dynamic part
  const size_t reserve = 1024 + static_smem;  // per-block system reservation + static shared variables
  const int max_fit = (int)std::min<size_t>(kMaxSmemPlates, per_block_max / slot_bytes);
  int st;
  for (const Form f : {kForm4, kForm2, kForm1, kForm4Roomy})
    if ((st = prepare_kernel(pb, f, per_block_max))) return st;
  if (cudaFuncSetAttribute(assign_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxGenes * 8) !=
      cudaSuccess)
    return BRKGA_ERR_CUDA;
  if (cudaFuncSetAttribute(order_items_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (kMaxGenes + 1) * (int)sizeof(int)) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  if (cudaFuncSetAttribute(chunk_free_i8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           corr::smem_bytes(corr::kMaxSide, corr::kMaxSide)) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  auto fit_for = [&](int ctas) {  // plates per item that fit when `ctas` CTAs share an SM
    const size_t share = per_sm / ctas;
    if (share <= reserve) return 0;
    return (int)std::min<size_t>((share - reserve) / slot_bytes, (size_t)max_fit);
  };
  Shape shapes[3];
  for (int v = 0; v < 3; ++v) {
    const int warps = 4 >> v;
    const int auto_ctas = kResidentWarps / warps;
    const bool req = warps_req == warps;
    const int creq = req ? ctas_req : 0, preq = req ? plates_req : -1;
    int S, ctas;
    if (creq == 0) {
      ctas = auto_ctas;
      if (preq >= 0) {
        S = preq;
        while (ctas > 1 && fit_for(ctas) < S) --ctas;
        if (fit_for(ctas) < S) return BRKGA_ERR_INVALID_ARGUMENT;
      } else {
        // Resident warps matter far more than where the plates live: in L1,
        // which all of the SM's shared memory then is, the searches' tables
        // have room beside them (measured with one to four grids, planes or
        // both per item in shared memory: P200M6, 100 rows, 0.83-0.90 ms
        // against 0.78, P50M2 0.39-0.42 against 0.39, P100M4 1.09-1.15
        // against 1.10).  Each CTA has as many plates of its own as grids
        // would fit in its share, the others come from the pool.
        S = std::min(fit_for(ctas), 4);
      }
    } else {
      ctas = creq;
      S = preq >= 0 ? preq : std::min(fit_for(ctas), 4);
    }
    if (S > max_fit) return BRKGA_ERR_INVALID_ARGUMENT;
    const size_t smem = preq > 0 ? (size_t)S * grid_bytes : 0;
    int occ = 0;
    if ((st = occupancy(pb, warps, smem, &occ))) return st;
    if (occ < 1 || (creq > 0 && occ < creq)) return BRKGA_ERR_INVALID_ARGUMENT;
    shapes[v].warps = warps;
    shapes[v].S = S;
    shapes[v].smem = smem;
    shapes[v].ctas = std::max(1, std::min(occ, ctas));
    shapes[v].n_slots = pb->sm_count * shapes[v].ctas;
  }
  pb->grid_words = grid_words;
  pb->coarse_words = coarse_words;
  pb->vac_off = planes;
  pb->min_S = shapes[0].S;
  for (int v = 0; v < 3; ++v) {
    pb->shape[v] = shapes[v];
    pb->min_S = std::min(pb->min_S, shapes[v].S);
  }
  pb->req_warps = warps_req;
  pb->req_ctas = ctas_req;
  pb->req_plates = plates_req;
  return BRKGA_OK;
}

int validate(const BrkgaProblemDesc* d) {
  if (!d) return BRKGA_ERR_INVALID_ARGUMENT;
  if (d->n_genes < 1 || d->n_genes > kMaxGenes || d->n_machines < 1 || d->n_machines > kMaxMachines ||
      d->n_types < 1 || (d->threshold_mode != BRKGA_THRESH_F32 && d->threshold_mode != BRKGA_THRESH_F64))
    return BRKGA_ERR_INVALID_ARGUMENT;
  if (!d->gene_type || (!d->thresholds && d->n_machines > 1) || !d->bin_length || !d->bin_width ||
      !d->bin_area || !d->setup_time || !d->proc_time || !d->proc_time_height || !d->part_area ||
      !d->part_nrot || !d->part_best_rot || !d->rot_h || !d->rot_w || !d->rot_mask_offset || !d->masks)
    return BRKGA_ERR_INVALID_ARGUMENT;
  for (int j = 0; j < d->n_genes; ++j)
    if (d->gene_type[j] < 0 || d->gene_type[j] >= d->n_types) return BRKGA_ERR_BAD_INSTANCE;
  for (int m = 0; m + 1 < d->n_machines; ++m) {
    if (!std::isfinite(d->thresholds[m])) return BRKGA_ERR_BAD_INSTANCE;
    if (m > 0 && d->thresholds[m] < d->thresholds[m - 1]) return BRKGA_ERR_BAD_INSTANCE;
  }
  for (int m = 0; m < d->n_machines; ++m) {
    if (d->bin_length[m] < 1 || d->bin_length[m] > kMaxSide || d->bin_width[m] < 1 ||
        d->bin_width[m] > kMaxSide || !std::isfinite(d->bin_area[m]) || !std::isfinite(d->setup_time[m]))
      return BRKGA_ERR_BAD_INSTANCE;
  }
  for (int t = 0; t < d->n_types; ++t) {
    if (!(d->part_area[t] > 0.0) || !std::isfinite(d->part_area[t])) return BRKGA_ERR_BAD_INSTANCE;
    const int nrot = d->part_nrot[t];
    if (nrot != 2 && nrot != 4) return BRKGA_ERR_BAD_INSTANCE;
    if (d->part_best_rot[t] < 0 || d->part_best_rot[t] >= nrot) return BRKGA_ERR_BAD_INSTANCE;
    for (int r = 0; r < nrot; ++r) {
      const int k = t * 4 + r;
      const int h = d->rot_h[k], w = d->rot_w[k];
      if (h < 1 || w < 1 || h > kMaxSide || w > kMaxSide) return BRKGA_ERR_BAD_INSTANCE;
      const int64_t off = d->rot_mask_offset[k];
      if (off < 0 || off + (int64_t)h * w > d->masks_bytes) return BRKGA_ERR_BAD_INSTANCE;
      for (int64_t i = 0; i < (int64_t)h * w; ++i)
        if (d->masks[off + i] > 1) return BRKGA_ERR_BAD_INSTANCE;
    }
    for (int m = 0; m < d->n_machines; ++m) {
      const size_t i = (size_t)m * d->n_types + t;
      if (!std::isfinite(d->proc_time[i]) || !std::isfinite(d->proc_time_height[i])) return BRKGA_ERR_BAD_INSTANCE;
    }
  }
  return BRKGA_OK;
}

// Host copies of the merged tables while a problem is built.
struct Merged {
  std::vector<InstDev> inst;
  std::vector<int32_t> gene_type, nrot, best;
  std::vector<double> thr, pt, pth, area, bin_area;
  std::vector<RotDev> rot;
  std::vector<CoarseIdx> cidx;
  std::vector<uint2> centry;
  std::vector<uint32_t> cfilter;
  int bsh = 0, n_planes = 0;  // rows of a block (2^bsh, 0: by rows), erosion planes that some core reads
  std::vector<std::pair<int, int>> longest;  // per mask row, rotation after rotation: [first, last + 1) of its longest run
  std::vector<int> n_runs;                   // per rotation: runs of ones of all rows
  std::vector<uint2> truns;
  std::vector<uint32_t> maskbits;
  std::vector<uint8_t> fits, newbin_ok;
  std::vector<RotList> rl;
  std::vector<MachDev> mach;
};

// Rows of the coarse test's blocks (2^shift).  Blocks of eight rows make the
// planes small and a core count for eight rows; blocks of four leave fewer rows
// of a small mask outside whole blocks, whose pairs all go to the exact test.
// Measured (eight / four rows): 14-25 cell masks 0.73 / 0.64 ms, 10-80 cell
// masks on plates filled more than once 24.5 / 21.5 ms (64 uneven instances)
// and 4.4 / 4.0 ms (231 parts on three 444 x 244 plates), on plates a quarter
// full 2.6 / 2.8 ms (P200M6); 10-120 cell masks 5.8 / 6.5 ms (P100M4), 20-240
// cell masks 20 / 26 ms (P400M8, 1,024 rows).  So four rows for small masks
// and, up to medium ones, where the parts fill most of the plates.
constexpr double kMostlyFull = 0.6;
struct MaskStats {
  double height, fill;  // over the genes: mean mask height, mean fill of their instance's plates
};
MaskStats mask_stats(const BrkgaProblemDesc* descs, int K) {
  double parts = 0.0, height = 0.0, fill = 0.0;
  for (int k = 0; k < K; ++k) {
    const BrkgaProblemDesc& d = descs[k];
    double area = 0.0, plates = 0.0;
    for (int j = 0; j < d.n_genes; ++j) {
      const int t = d.gene_type[j], nrot = d.part_nrot[t];
      area += d.part_area[t];
      for (int r = 0; r < nrot; ++r) height += (double)d.rot_h[t * 4 + r] / nrot;
    }
    for (int m = 0; m < d.n_machines; ++m) plates += d.bin_area[m];
    parts += d.n_genes;
    fill += plates > 0.0 ? d.n_genes * area / plates : 0.0;
  }
  return {height / parts, fill / parts};
}

int block_shift(const MaskStats& s) { return s.height < 28.0 || (s.height < 50.0 && s.fill >= kMostlyFull) ? 2 : 3; }

// Where the test is by rows, a rotation's filter holds this many of its rows:
// a tall, thin mask that passes 24 of them often fails at another one (200
// masks of 1-3 x 20-120 cells, 2,000 rows: 24 rows 2.19 ms, 64 1.85, all 1.97).
constexpr int kFilterRows = 64;

// Pieces of a mask that groups of lanes test before the whole warp takes the
// open pairs one by one, where the test is by rows: as many as hold kGroupCells
// cells (4 of long runs decide as much as 20 of single cells), and none for a
// mask of so few that one step of the warp tests them all and its few pairs are
// soon through.  Measured (cells 20 / 32 / 48): masks of noise 1.87 / 1.64 / 1.55
// ms, parts of 5-15 cells 1.66 / 1.80 / 1.90.  (None for up to 4 / 6 / 8 / 12
// pieces: 1-6 cell parts 2.43 / 2.09 / 2.09 / 2.09 ms, of 5-15 cells 1.59 / 1.66
// / 1.73 / 2.03, of 5-10 cells 1.36 / 1.35 / 1.27 / 1.19.)
constexpr int kGroupCells = 20, kGroupFewSegs = 6, kGroupMostSegs = 20;
int group_segs(const RotDev& rd, const Merged& g) {
  if (g.bsh) return kGroupSegs;
  if (rd.ntseg <= kGroupFewSegs) return 0;
  int cells = 0, q = 0;
  for (; q < rd.ntseg && q < kGroupMostSegs && (q < kGroupSegs || cells < kGroupCells); ++q)
    cells += (int)(g.truns[rd.tseg + q].x >> 16);
  return q;
}

// The coarse test's entries of one rotation (see coarse_ok()): for every
// offset of its top row in a block of plate rows, the blocks it covers
// whole and the core of each, widest first, then coarse to fine from the
// bottom (as the rows of the exact test).  Cores shorter than the first plane's
// runs are left to the exact test.  By rows every row is a block and its longest
// run the core, for the filter only.  Returns how many of the rotation's rows are
// part of a core, summed over the offsets.
int coarse_tables(const std::pair<int, int>* longest, const RotDev& rd, Merged& g) {
  struct Core {
    int block, lo, len;
  };
  const bool by_rows = g.bsh == 0;
  const int rows = 1 << g.bsh;
  int covered = 0;
  std::vector<Core> cores;
  std::vector<int> order;
  std::vector<char> used;
  for (int off = 0; off < rows; ++off) {
    cores.clear();
    order.clear();
    for (int i = (rows - off) % rows; i + rows <= rd.h; i += rows) {
      int lo = 0, hi = rd.w;
      for (int k = 0; k < rows; ++k) {
        lo = std::max(lo, longest[i + k].first);
        hi = std::min(hi, longest[i + k].second);
      }
      if (hi - lo >= (by_rows ? 1 : 1 << kPlaneMin)) cores.push_back({(i + off) >> g.bsh, lo, hi - lo});
    }
    const int n = (int)cores.size();
    covered += n * rows;
    used.assign(n, 0);
    if (n) {
      int widest = 0;
      for (int c = 1; c < n; ++c)
        if (cores[c].len > cores[widest].len) widest = c;
      order.push_back(widest);
      used[widest] = 1;
      for (int st = by_rows ? 16 : 4; st >= 1; st >>= 1)
        for (int c = n - 1; c >= 0; c -= st)
          if (!used[c]) {
            order.push_back(c);
            used[c] = 1;
          }
    }
    if (by_rows && n > kFilterRows) order.resize(kFilterRows);
    CoarseIdx ci;
    ci.e = (int)g.centry.size();
    ci.f = (int)g.cfilter.size();
    for (int c : order) {
      const Core& k = cores[c];
      g.cfilter.push_back(((uint32_t)k.block << 16) | (uint32_t)k.len);
      for (int at = 0; at < k.len && !by_rows;) {  // pieces of at most two windows of the longest plane
        int len = std::min(k.len - at, 2 << kPlaneMax), p = kPlaneMin;
        if (len < (1 << kPlaneMin)) {  // a short last piece: the first plane's window up to the core's end
          at = k.len - (1 << kPlaneMin);
          len = 1 << kPlaneMin;
        }
        while (p < kPlaneMax && (2 << p) <= len) ++p;
        g.centry.push_back(make_uint2((uint32_t)(k.lo + at) | ((uint32_t)(k.lo + at + len - (1 << p)) << 16),
                                      (uint32_t)k.block | ((uint32_t)(p - kPlaneMin) << 16)));
        g.n_planes = std::max(g.n_planes, p - kPlaneMin + 1);
        at += len;
      }
    }
    if ((g.centry.size() - ci.e) & 1) g.centry.push_back(g.centry.back());
    ci.ne = (int)g.centry.size() - ci.e;
    while ((g.cfilter.size() - ci.f) % kVacIlp) g.cfilter.push_back(0u);
    ci.nf = (int)g.cfilter.size() - ci.f;
    g.cidx.push_back(ci);
  }
  return covered;
}

// Rotation r of type t fits the plates of some machine of its instance (the others are never tested).
bool fits_some(const BrkgaProblemDesc& d, int t, int r) {
  for (int m = 0; m < d.n_machines; ++m)
    if (d.rot_h[t * 4 + r] <= d.bin_length[m] && d.rot_w[t * 4 + r] <= d.bin_width[m]) return true;
  return false;
}

// The coarse test's tables of every rotation for blocks of 2^g.bsh rows.
// Returns the share of the masks' rows that are part of a core, over the genes.
double coarse_tables(const BrkgaProblemDesc* descs, int K, Merged& g) {
  g.cidx.clear();
  g.centry.clear();
  g.cfilter.clear();
  g.n_planes = 0;
  double covered = 0.0, rows = 0.0;
  std::vector<std::pair<double, double>> of_type;  // rows in cores, rows
  size_t rot = 0;
  const std::pair<int, int>* longest = g.longest.data();
  for (int k = 0; k < K; ++k) {
    const BrkgaProblemDesc& d = descs[k];
    of_type.assign(d.n_types, {0.0, 0.0});
    for (int t = 0; t < d.n_types; ++t)
      for (int r = 0; r < 4; ++r, ++rot) {
        if (r >= d.part_nrot[t]) {
          g.cidx.resize(g.cidx.size() + ((size_t)1 << g.bsh), CoarseIdx{0, 0, 0, 0});
          continue;
        }
        RotDev& rd = g.rot[rot];
        const double in_cores = (double)coarse_tables(longest, rd, g) / (1 << g.bsh);
        if (fits_some(d, t, r)) {
          of_type[t].first += in_cores;
          of_type[t].second += rd.h;
        }
        rd.gseg = (short)group_segs(rd, g);
        longest += rd.h;
      }
    for (int j = 0; j < d.n_genes; ++j) {
      covered += of_type[d.gene_type[j]].first;
      rows += of_type[d.gene_type[j]].second;
    }
  }
  for (MachDev& m : g.mach) m.NB = m.L >> g.bsh;
  return covered / rows;
}

// The share of the masks' rows that belong to parts with more than kMostRuns
// runs of ones a row, over the genes.
constexpr double kMostRuns = 2.1;
double many_runs(const BrkgaProblemDesc* descs, int K, const Merged& g) {
  double many = 0.0, rows = 0.0;
  std::vector<std::pair<double, double>> of_type;  // runs, rows
  size_t rot = 0;
  for (int k = 0; k < K; ++k) {
    const BrkgaProblemDesc& d = descs[k];
    of_type.assign(d.n_types, {0.0, 0.0});
    for (int t = 0; t < d.n_types; ++t)
      for (int r = 0; r < 4; ++r, ++rot)
        if (r < d.part_nrot[t] && fits_some(d, t, r)) {
          of_type[t].first += g.n_runs[rot];
          of_type[t].second += g.rot[rot].h;
        }
    for (int j = 0; j < d.n_genes; ++j) {
      const std::pair<double, double>& p = of_type[d.gene_type[j]];
      many += p.first > kMostRuns * p.second ? p.second : 0.0;
      rows += p.second;
    }
  }
  return many / rows;
}

// Block height and tables of the coarse test.  A block's core is one run of
// columns, so it says little of masks whose rows have several runs (lattices,
// plates with holes, combs) and parts of few rows have next to none; their
// positions then went to the exact test without a filter.  Such problems are
// tested by rows: the plate keeps the longest free run of every row instead of
// planes, and a rotation's rows need one as long as their own longest run
// (numba_utils.py:50-94).  By rows from a fifth of the mask rows in parts of many
// runs on (frames, rings, H and U shapes have two runs at most), below ten rows a
// mask, and where less than half of the rows lie in cores at four rows a block
// (0.6 where the parts fill most of the plates; nearly empty plates let every row
// through anyway).  One launch, by blocks as before / by rows:
//   parts of 30-90 cells on three 300 x 300 plates, 500 rows: lattices 2.64 /
//     0.85 ms, rectangles with holes 1.24 / 0.67, bars of 5 every 12-20 cells
//     1.74 / 0.68; of solid parts and lattices 10 % lattices 0.79 / 0.86, 20 %
//     1.02 / 0.89, 33 % 1.33 / 0.90; U shapes 1.18 / 1.73, frames of 4 cells
//     0.81 / 1.27, solid parts (P100M4) 1.01 / 1.50;
//   200 parts on three plates, 1,000 rows: of 4-8 cells on 50 x 50 1.53 / 1.20 ms,
//     5-15 on 90 x 90 1.92 / 1.66, on 200 x 200 1.81 / 1.77, 5-20 on 120 x 120
//     1.98 / 1.83, on 220 x 220 1.91 / 1.99, on 400 x 400 1.90 / 2.13, 6-24 on 150
//     x 150 2.02 / 2.02, on 600 x 600 2.01 / 2.30; rectangles of 4-12 cells on 90 x
//     90 1.58 / 1.20; 1-3 x 20-120 on 200 x 200, 2,000 rows, 2.72 / 1.82, 150 on
//     600 x 600, 500 rows, 0.84 / 0.91.
constexpr double kManyRunsShare = 0.2, kLeastHeight = 10.0, kNearlyEmpty = 0.03;
void coarse_blocks(const BrkgaProblemDesc* descs, int K, Merged& g) {
  const MaskStats s = mask_stats(descs, K);
  g.bsh = many_runs(descs, K, g) > kManyRunsShare || s.height < kLeastHeight ? 0 : block_shift(s);
  const double least = s.fill < kNearlyEmpty ? 0.0 : s.fill < kMostlyFull ? 0.5 : 0.6;
  while (coarse_tables(descs, K, g) < least && g.bsh) g.bsh = g.bsh == 3 ? 2 : 0;
}

// A row's cells as bits, n <= 32 of them: eight bytes at a time, as (nonzero)
// lowest bits gathered into one byte by a multiplication.  Problem creation is
// bound by this scan of the masks: 400 parts x 8 machines 88 -> 31 ms against byte by byte.
uint32_t pack_cells(const uint8_t* cells, int n) {
  uint32_t v = 0;
  for (int at = 0; at < n; at += 8) {
    uint64_t x = 0;
    std::memcpy(&x, cells + at, std::min(8, n - at));
    x |= x >> 4;
    x |= x >> 2;
    x |= x >> 1;
    x &= 0x0101010101010101ull;
    v |= (uint32_t)((x * 0x0102040810204080ull) >> 56) << at;
  }
  return v;
}

// Append one instance: derived part tables (runs of ones, block cores,
// bit-packed rows) with absolute indices, machines, times, flags.
void merge_instance(const BrkgaProblemDesc* d, Merged& g) {
  const int N = d->n_genes, M = d->n_machines, T = d->n_types;
  InstDev id;
  id.N = N;
  id.M = M;
  id.T = T;
  id.mode = d->threshold_mode;
  id.gbase = (int)g.gene_type.size();
  id.tbase = (int)g.area.size();
  id.mbase = (int)g.mach.size();
  id.thrbase = (int)g.thr.size();
  id.tmbase = (int)g.pt.size();
  std::vector<uint32_t> runs;                // one rotation's runs of ones, row after row
  std::vector<int> row_at, order;            // where each row's runs begin; the rows in test order
  std::vector<char> used;
  for (int t = 0; t < T; ++t) {
    for (int r = 0; r < 4; ++r) {
      RotDev rd{};
      if (r < d->part_nrot[t]) {
        const int k = t * 4 + r, h = d->rot_h[k], w = d->rot_w[k];
        const uint8_t* mk = d->masks + d->rot_mask_offset[k];
        rd.h = h;
        rd.w = w;
        rd.mw = (short)((w + 31) / 32);
        rd.mask_base = (int)g.maskbits.size();
        int imax = 0, dmax = 0;  // row with the longest run of ones and that length
        runs.clear();
        row_at.assign(1, 0);
        for (int i = 0; i < h; ++i) {
          const uint8_t* cells = mk + (size_t)i * w;
          for (int j = 0; j < w; j += 32) g.maskbits.push_back(pack_cells(cells + j, std::min(32, w - j)));
          const uint32_t* row = g.maskbits.data() + g.maskbits.size() - rd.mw;
          int best = 0, from = -1;  // from: first column of the run that is open
          g.longest.push_back({0, 0});
          auto close = [&](int end) {
            runs.push_back((uint32_t)from | ((uint32_t)(end - from) << 16));
            if (end - from > best) {
              best = end - from;
              g.longest.back() = {from, end};
            }
            from = -1;
          };
          uint32_t top = 0;  // the last word's highest cell
          for (int wd = 0; wd < rd.mw; ++wd) {
            // the columns at which a run begins or has ended, in turn
            for (uint32_t edges = row[wd] ^ (row[wd] << 1 | top); edges; edges &= edges - 1) {
              const int at = 32 * wd + __builtin_ctz(edges);
              if (from < 0) from = at;
              else close(at);
            }
            top = row[wd] >> 31;
          }
          if (from >= 0) close(w);
          row_at.push_back((int)runs.size());
          if (best > dmax) {
            dmax = best;
            imax = i;
          }
        }
        // collision-test order: the widest row, then the rows coarse to fine
        // from the bottom (every 16th, then every 8th, 4th, 2nd, the rest).
        // Plates fill from the bottom, so low rows reject a blocked candidate
        // soonest; spreading the first tests over the part's height catches
        // a collision higher up without walking every row below it.
        rd.tseg = (int)g.truns.size();
        {
          order.clear();
          used.assign(h, 0);
          order.push_back(imax);
          used[imax] = 1;
          for (int st = 16; st >= 1; st >>= 1)
            for (int i = h - 1; i >= 0; i -= st)
              if (!used[i]) {
                order.push_back(i);
                used[i] = 1;
              }
          for (int i : order)
            for (int k = row_at[i]; k < row_at[i + 1]; ++k) {
              const uint32_t s = runs[k] & 0xFFFFu, d = runs[k] >> 16;
              for (uint32_t at = 0; at < d; at += 32)
                g.truns.push_back(make_uint2((s + at) | (std::min(32u, d - at) << 16), (unsigned)i));
            }
          rd.ntseg = (int)g.truns.size() - rd.tseg;
          // Pieces are runs too, so one list serves where at most an eighth of it
          // only continues a run; with two for every rotation, masks of many short
          // runs took twice the memory (lattices of 200-800 cells 145 MB, now 80).
          rd.trun = rd.tseg;
          rd.ntrun = rd.ntseg;
          if (rd.ntseg - (int)runs.size() > rd.ntseg / 8) {
            rd.trun = (int)g.truns.size();
            rd.ntrun = (int)runs.size();
            for (int i : order)
              for (int k = row_at[i]; k < row_at[i + 1]; ++k) g.truns.push_back(make_uint2(runs[k], (unsigned)i));
          }
        }
      }
      g.rot.push_back(rd);
      g.n_runs.push_back(rd.h ? (int)runs.size() : 0);
    }
    g.area.push_back(d->part_area[t]);
    g.nrot.push_back(d->part_nrot[t]);
    g.best.push_back(d->part_best_rot[t]);
  }
  std::vector<uint8_t> fits((size_t)T * M), newbin_ok((size_t)T * M);
  for (int m = 0; m < M; ++m) {
    MachDev md;
    md.L = d->bin_length[m];
    md.W = d->bin_width[m];
    md.NW = (md.W + 31) / 32;
    md.RS = md.NW + 2;
    md.NB = 0;  // coarse_tables()
    md.area = d->bin_area[m];
    md.setup = d->setup_time[m];
    g.mach.push_back(md);
    g.bin_area.push_back(d->bin_area[m]);
    for (int t = 0; t < T; ++t) {
      const int h0 = d->rot_h[t * 4], w0 = d->rot_w[t * 4];
      fits[(size_t)t * M + m] = !((h0 > md.L || w0 > md.W) && (w0 > md.L || h0 > md.W));
      const int rb = d->part_best_rot[t];
      newbin_ok[(size_t)t * M + m] = d->rot_h[t * 4 + rb] <= md.L && d->rot_w[t * 4 + rb] <= md.W;
    }
  }
  g.fits.insert(g.fits.end(), fits.begin(), fits.end());
  g.newbin_ok.insert(g.newbin_ok.end(), newbin_ok.begin(), newbin_ok.end());
  for (int t = 0; t < T; ++t)
    for (int m = 0; m < M; ++m) {
      const MachDev& md = g.mach[id.mbase + m];
      RotList l{};
      int rh[4];
      l.hmin = kMaxSide + 1;
      for (int r = 0; r < d->part_nrot[t]; ++r) {
        const int h = d->rot_h[t * 4 + r], w = d->rot_w[t * 4 + r];
        if (h <= md.L && w <= md.W) {  // numba_utils.py:82-84
          rh[l.nr] = h;
          l.rs[l.nr] = (unsigned char)r;
          ++l.nr;
          l.hmin = std::min(l.hmin, h);
          l.scan_words += (unsigned)(md.L * md.NW + h * ((w + 31) / 32));
        }
      }
      for (int i = 1; i < l.nr; ++i)  // stable insertion sort by height
        for (int j = i; j > 0 && rh[j] < rh[j - 1]; --j) {
          std::swap(rh[j], rh[j - 1]);
          std::swap(l.rs[j], l.rs[j - 1]);
        }
      g.rl.push_back(l);
    }
  for (int m = 0; m + 1 < M; ++m)
    g.thr.push_back(d->threshold_mode == BRKGA_THRESH_F32 ? (double)(float)d->thresholds[m] : d->thresholds[m]);
  for (int j = 0; j < N; ++j) g.gene_type.push_back(id.tbase + d->gene_type[j]);
  g.pt.insert(g.pt.end(), d->proc_time, d->proc_time + (size_t)M * T);
  g.pth.insert(g.pth.end(), d->proc_time_height, d->proc_time_height + (size_t)M * T);
  g.inst.push_back(id);
}

// chrom_offs / out_offs (host [K], may be NULL): where each instance's
// chromosomes (in floats) and makespans start; NULL = packed one after another.
// cpool: the pool plates' planes, NULL = in the workspace.
int fill_run(const BrkgaProblem* pb, const int32_t* pops, const int64_t* chrom_offs, const int64_t* out_offs,
             const LaunchCounts& lc, const Layout& l, char* ws, const float* d_chrom, double* d_out,
             BrkgaPlacement* d_log, int32_t* d_status, int64_t pool_bins, char* cpool, Run* run) {
  std::memset(run, 0, sizeof(Run));
  run->K = pb->K;
  run->n_rows = (int)lc.rows;
  run->n_items = (int)lc.items;
  run->Nmax = pb->Nmax;
  run->chrom = d_chrom;
  run->out = d_out;
  run->seq = reinterpret_cast<uint16_t*>(ws + l.off_seq);
  run->cnt = reinterpret_cast<int32_t*>(ws + l.off_cnt);
  run->infeas = reinterpret_cast<int32_t*>(ws + l.off_inf);
  run->order = reinterpret_cast<int32_t*>(ws + l.off_ord);
  run->mk = reinterpret_cast<double*>(ws + l.off_mk);
  run->log = d_log;
  run->status = d_status;
  unsigned int* ctr = reinterpret_cast<unsigned int*>(ws + l.off_ctr);
  run->item_ctr = ctr;
  run->pool_ctr = ctr + 1;
  run->counters = reinterpret_cast<unsigned long long*>(ws + l.off_ctr + 8);
  run->crit = reinterpret_cast<int*>(ws + l.off_crit);
  run->crit_items = pick_shape(pb, lc.items).warps == 4 ? kCritItems : 0;
  run->binscal = reinterpret_cast<BinScal*>(ws + l.off_bins);
  run->pool = reinterpret_cast<uint32_t*>(ws + l.off_pool);
  run->cpool = reinterpret_cast<uint32_t*>(cpool ? cpool : ws + l.off_cpool);
  run->pool_bins = pool_bins;
  run->S = pick_shape(pb, lc.items).S;
  run->smem_grids = pick_shape(pb, lc.items).smem > 0;
  run->own = run->cpool + (size_t)pool_bins * pb->coarse_words;
  run->grid_words = pb->grid_words;
  run->coarse_words = pb->coarse_words;
  run->vac_off = pb->vac_off;
  run->task_max = pb->task_max;
  int64_t row = 0, item = 0, seq = 0, chrom = 0;
  for (int k = 0; k < pb->K; ++k) {
    const InstDev& id = pb->inst[k];
    InstRun& r = run->r[k];
    r.P = pops[k];
    r.crow0 = (int)row;
    r.item0 = (int)item;
    r.S2 = pb->s2[k];
    r.chrom_off = chrom_offs ? chrom_offs[k] : chrom;
    r.out_off = out_offs ? out_offs[k] : row;
    r.seq0 = seq;
    row += pops[k];
    item += (int64_t)pops[k] * id.M;
    seq += (int64_t)pops[k] * id.M * id.N;
    chrom += (int64_t)pops[k] * 2 * id.N;
  }
  return BRKGA_OK;
}

int launch(const BrkgaProblem* pb, int stage, const Run& run, cudaStream_t s) {
  if (run.n_rows == 0) return BRKGA_OK;
  if (stage == 0 || stage == 1) {
    const int at = std::min(1024, std::max(64, pb->S2max / 2));
    assign_sort_kernel<<<run.n_rows, at, (size_t)pb->S2max * 8, s>>>(pb->tb, run);
    order_items_kernel<<<1, 1024, (size_t)(pb->Nmax + 1) * sizeof(int), s>>>(pb->tb, run);
  }
  if (stage == 0 || stage == 2) {
    const Shape& sh = pick_shape(pb, run.n_items);
    const int grid = (int)std::min<int64_t>(sh.n_slots, run.n_items);
    const bool alone = sh.warps == 4 && !pb->req_warps && grid <= pb->sm_count;  // every item has an SM to itself
    const Form f = sh.warps == 1                       ? kForm1
                   : sh.warps == 2                     ? kForm2
                   : alone                             ? kForm8
                   : grid <= kRoomyCtas * pb->sm_count ? kForm4Roomy
                                                       : kForm4;
    decode_form(pb, f)<<<grid, f == kForm8 ? 256 : 32 * sh.warps, sh.smem, s>>>(pb->tb, run);
  }
  if (stage == 0 || stage == 3) reduce_kernel<<<(run.n_rows + 255) / 256, 256, 0, s>>>(pb->tb, run);
  return cudaGetLastError() == cudaSuccess ? BRKGA_OK : BRKGA_ERR_CUDA;
}

// brkga_decode_multi_at with the pool plates' planes at d_planes (NULL: in the workspace).
int decode_at(int32_t stage, const BrkgaProblem* pb, const float* d_chrom, const int64_t* chrom_offsets,
              const int32_t* pops, double* d_makespan, const int64_t* makespan_offsets, BrkgaPlacement* d_log,
              int32_t* d_status, void* d_ws, size_t ws_bytes, int64_t pool_bins, void* d_planes, void* stream) {
  if (!pb || !pops || pool_bins < 0 || stage < 0 || stage > 3) return BRKGA_ERR_INVALID_ARGUMENT;
  LaunchCounts lc;
  int st = counts_of(pb, pops, &lc);
  if (st) return st;
  for (int k = 0; k < pb->K; ++k)
    if ((chrom_offsets && chrom_offsets[k] < 0) || (makespan_offsets && makespan_offsets[k] < 0))
      return BRKGA_ERR_INVALID_ARGUMENT;
  if (lc.rows == 0) return BRKGA_OK;
  if (!d_chrom || !d_makespan || !d_status || !d_ws) return BRKGA_ERR_INVALID_ARGUMENT;
  if (pool_bins == 0) pool_bins = default_pool_bins(pb, lc.items);
  const Layout l = layout_of(pb, lc, pool_bins);
  if (ws_bytes < (d_planes ? l.end_pool : l.total)) return BRKGA_ERR_WORKSPACE;
  DeviceGuard g(pb->device);
  Run run;
  fill_run(pb, pops, chrom_offsets, makespan_offsets, lc, l, static_cast<char*>(d_ws), d_chrom, d_makespan, d_log,
           d_status, pool_bins, static_cast<char*>(d_planes), &run);
  return launch(pb, stage, run, static_cast<cudaStream_t>(stream));
}

}  // namespace

extern "C" {

int brkga_abi_version(void) { return BRKGA_ABI_VERSION; }

#ifndef BRKGA_BUILD_ID
#define BRKGA_BUILD_ID "unstamped"
#endif
const char* brkga_build_id(void) { return BRKGA_BUILD_ID; }

// Device tables for the surrogate (same library, not part of the public ABI;
// single-instance problems, whose table bases are all 0).
__attribute__((visibility("hidden"))) int brkga_internal_problem_tables(
    const BrkgaProblem* pb, int* N, int* M, int* T, int* mode, const double** thr, const int32_t** gene_type,
    const double** part_area, const double** pt, const double** pth, const double** bin_area) {
  if (!pb || pb->K != 1) return BRKGA_ERR_INVALID_ARGUMENT;
  *N = pb->N;
  *M = pb->M;
  *T = pb->T;
  *mode = pb->mode;
  *thr = pb->d_thr;
  *gene_type = pb->d_gene_type;
  *part_area = pb->d_area;
  *pt = pb->d_pt;
  *pth = pb->d_pth;
  *bin_area = pb->d_bin_area;
  return BRKGA_OK;
}

const char* brkga_status_string(int status) {
  switch (status) {
    case BRKGA_OK: return "ok";
    case BRKGA_ERR_INVALID_ARGUMENT: return "invalid argument";
    case BRKGA_ERR_BAD_INSTANCE: return "bad instance";
    case BRKGA_ERR_CUDA: return "CUDA error";
    case BRKGA_ERR_WORKSPACE: return "workspace too small";
    case BRKGA_ERR_CAPACITY: return "bin pool exhausted";
    case BRKGA_ERR_NEW_BIN_UNFIT: return "new plate received a rotation that does not fit";
    case BRKGA_ERR_NO_DEVICE: return "no CUDA device";
    case BRKGA_ERR_INTERNAL: return "device consistency check failed";
    default: return "unknown status";
  }
}

void brkga_problem_destroy(BrkgaProblem* pb) {
  if (!pb) return;
  {
    DeviceGuard g(pb->device);
    for (void* p : pb->allocations) cudaFree(p);
    if (pb->e_chrom) cudaFree(pb->e_chrom);
    if (pb->e_out) cudaFree(pb->e_out);
    if (pb->e_status) cudaFree(pb->e_status);
    if (pb->e_log) cudaFree(pb->e_log);
    if (pb->e_ws) cudaFree(pb->e_ws);
    if (pb->greedy_ws) cudaFree(pb->greedy_ws);
    if (pb->e_host) cudaFreeHost(pb->e_host);
    if (pb->stream) cudaStreamDestroy(pb->stream);
  }
  delete pb;
}

int brkga_problem_create_multi(const BrkgaProblemDesc* descs, int32_t K, BrkgaProblem** out) {
  if (!out) return BRKGA_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (!descs || K < 1 || K > kMaxInst) return BRKGA_ERR_INVALID_ARGUMENT;
  for (int k = 0; k < K; ++k) {
    const int st = validate(&descs[k]);
    if (st) return st;
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return BRKGA_ERR_NO_DEVICE;
  }
  Merged g;
  for (int k = 0; k < K; ++k) merge_instance(&descs[k], g);
  coarse_blocks(descs, K, g);
  for (uint2& e : g.centry) e.y = (e.y & 0xFFFFu) * (uint32_t)g.n_planes + (e.y >> 16);  // the number of planes is known now
  if (g.maskbits.size() >= ((size_t)1 << 31) || g.truns.size() >= ((size_t)1 << 31) ||
      g.centry.size() >= ((size_t)1 << 31))
    return BRKGA_ERR_BAD_INSTANCE;
  BrkgaProblem* pb = new BrkgaProblem();
  cudaGetDevice(&pb->device);
  pb->K = K;
  pb->inst = g.inst;
  pb->mach = g.mach;
  pb->tb.bsh = g.bsh;
  pb->tb.n_planes = g.n_planes;
  pb->pool_per_cta = pool_per_cta(descs, K);
  pb->plain = g.bsh > 0;
  for (const MachDev& m : g.mach) pb->plain = pb->plain && m.NW <= 32;
  for (const InstDev& id : g.inst) {
    int s2 = 1;
    while (s2 < id.N) s2 <<= 1;
    pb->s2.push_back(s2);
    pb->S2max = std::max(pb->S2max, s2);
    pb->Nmax = std::max(pb->Nmax, id.N);
  }
  pb->N = g.inst[0].N;
  pb->M = g.inst[0].M;
  pb->T = g.inst[0].T;
  pb->mode = g.inst[0].mode;

  int st;
  if ((st = upload(pb, &pb->d_inst, g.inst)) || (st = upload(pb, &pb->d_gene_type, g.gene_type)) ||
      (st = upload(pb, &pb->d_thr, g.thr)) || (st = upload(pb, &pb->d_mach, g.mach)) ||
      (st = upload(pb, &pb->d_pt, g.pt)) || (st = upload(pb, &pb->d_pth, g.pth)) ||
      (st = upload(pb, &pb->d_area, g.area)) || (st = upload(pb, &pb->d_nrot, g.nrot)) ||
      (st = upload(pb, &pb->d_best, g.best)) || (st = upload(pb, &pb->d_rot, g.rot)) ||
      (st = upload(pb, &pb->d_cidx, g.cidx)) ||
      (st = upload(pb, &pb->d_centry, g.centry)) || (st = upload(pb, &pb->d_cfilter, g.cfilter)) || (st = upload(pb, &pb->d_truns, g.truns)) ||
      (st = upload(pb, &pb->d_maskbits, g.maskbits)) ||
      (st = upload(pb, &pb->d_fits, g.fits)) || (st = upload(pb, &pb->d_newbin_ok, g.newbin_ok)) ||
      (st = upload(pb, &pb->d_rl, g.rl)) ||
      (st = upload(pb, &pb->d_bin_area, g.bin_area)) || (st = configure(pb, 0, 0, -1))) {
    brkga_problem_destroy(pb);
    return st;
  }
  Tables& tb = pb->tb;
  tb.inst = pb->d_inst;
  tb.gene_type = pb->d_gene_type;
  tb.thr = pb->d_thr;
  tb.mach = pb->d_mach;
  tb.pt = pb->d_pt;
  tb.pth = pb->d_pth;
  tb.part_area = pb->d_area;
  tb.nrot = pb->d_nrot;
  tb.best_rot = pb->d_best;
  tb.rot = pb->d_rot;
  tb.cidx = pb->d_cidx;
  tb.centry = pb->d_centry;
  tb.cfilter = pb->d_cfilter;
  tb.truns = pb->d_truns;
  tb.maskbits = pb->d_maskbits;
  tb.newbin_ok = pb->d_newbin_ok;
  tb.fits = pb->d_fits;
  tb.rl = pb->d_rl;
  if (cudaGetSymbolAddress(&pb->noalloc_scratch, g_noalloc_scratch) != cudaSuccess ||
      cudaGetSymbolAddress(&pb->noalloc_planes, g_noalloc_planes) != cudaSuccess) {
    brkga_problem_destroy(pb);
    return BRKGA_ERR_CUDA;
  }
  *out = pb;
  return BRKGA_OK;
}

int brkga_problem_create(const BrkgaProblemDesc* d, BrkgaProblem** out) {
  if (!out) return BRKGA_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (!d) return BRKGA_ERR_INVALID_ARGUMENT;
  return brkga_problem_create_multi(d, 1, out);
}

int brkga_problem_instances(const BrkgaProblem* pb, int32_t* K) {
  if (!pb || !K) return BRKGA_ERR_INVALID_ARGUMENT;
  *K = pb->K;
  return BRKGA_OK;
}

int brkga_set_launch_config(BrkgaProblem* pb, int32_t warps_per_item, int32_t ctas_per_sm, int32_t smem_plates,
                            int32_t task_max) {
  if (!pb || (warps_per_item != 0 && warps_per_item != 1 && warps_per_item != 2 && warps_per_item != 4) ||
      ctas_per_sm < 0 ||
      ctas_per_sm > kMaxCtasPerSm || smem_plates < -1 || smem_plates > kMaxSmemPlates || task_max < -1 ||
      task_max > kMaxTaskMax)
    return BRKGA_ERR_INVALID_ARGUMENT;
  DeviceGuard g(pb->device);
  const int old_warps = pb->req_warps, old_ctas = pb->req_ctas, old_plates = pb->req_plates;
  const int st = configure(pb, warps_per_item, ctas_per_sm, smem_plates);
  if (st) {
    configure(pb, old_warps, old_ctas, old_plates);
    return st;
  }
  pb->task_max = task_max < 0 ? kDefaultTaskMax : task_max;
  return BRKGA_OK;
}

int brkga_get_launch_config(const BrkgaProblem* pb, int64_t items, int32_t* warps_per_item, int32_t* ctas_per_sm,
                            int32_t* smem_plates, int32_t* resident_ctas, int32_t* task_max) {
  if (!pb || items < 0) return BRKGA_ERR_INVALID_ARGUMENT;
  const Shape& sh = pick_shape(pb, items);
  if (warps_per_item) *warps_per_item = sh.warps;
  if (ctas_per_sm) *ctas_per_sm = sh.ctas;
  if (smem_plates) *smem_plates = sh.smem ? sh.S : 0;
  if (resident_ctas) *resident_ctas = sh.n_slots;
  if (task_max) *task_max = pb->task_max;
  return BRKGA_OK;
}

int brkga_workspace_bytes_multi(const BrkgaProblem* pb, const int32_t* pops, int64_t pool_bins, size_t* bytes) {
  if (!pb || !pops || !bytes || pool_bins < 0) return BRKGA_ERR_INVALID_ARGUMENT;
  LaunchCounts lc;
  const int st = counts_of(pb, pops, &lc);
  if (st) return st;
  if (pool_bins == 0) pool_bins = default_pool_bins(pb, lc.items);
  *bytes = layout_of(pb, lc, pool_bins).total;
  return BRKGA_OK;
}

int brkga_workspace_bytes(const BrkgaProblem* pb, int32_t P, int64_t pool_bins, size_t* bytes) {
  if (!pb || pb->K != 1) return BRKGA_ERR_INVALID_ARGUMENT;
  return brkga_workspace_bytes_multi(pb, &P, pool_bins, bytes);
}

int brkga_decode_multi_at(int32_t stage, const BrkgaProblem* pb, const float* d_chrom, const int64_t* chrom_offsets,
                          const int32_t* pops, double* d_makespan, const int64_t* makespan_offsets,
                          BrkgaPlacement* d_log, int32_t* d_status, void* d_ws, size_t ws_bytes, int64_t pool_bins,
                          void* stream) {
  return decode_at(stage, pb, d_chrom, chrom_offsets, pops, d_makespan, makespan_offsets, d_log, d_status, d_ws,
                   ws_bytes, pool_bins, nullptr, stream);
}

int brkga_decode_multi_stage(int32_t stage, const BrkgaProblem* pb, const float* d_chrom, const int32_t* pops,
                             double* d_makespan, BrkgaPlacement* d_log, int32_t* d_status, void* d_ws,
                             size_t ws_bytes, int64_t pool_bins, void* stream) {
  return brkga_decode_multi_at(stage, pb, d_chrom, nullptr, pops, d_makespan, nullptr, d_log, d_status, d_ws,
                               ws_bytes, pool_bins, stream);
}

int brkga_decode_multi(const BrkgaProblem* pb, const float* d_chrom, const int32_t* pops, double* d_makespan,
                       BrkgaPlacement* d_log, int32_t* d_status, void* d_ws, size_t ws_bytes, int64_t pool_bins,
                       void* stream) {
  return brkga_decode_multi_stage(0, pb, d_chrom, pops, d_makespan, d_log, d_status, d_ws, ws_bytes, pool_bins,
                                  stream);
}

int brkga_decode_stage(int32_t stage, const BrkgaProblem* pb, const float* d_chrom, int32_t P,
                       double* d_makespan, BrkgaPlacement* d_log, int32_t* d_status, void* d_ws,
                       size_t ws_bytes, int64_t pool_bins, void* stream) {
  if (!pb || pb->K != 1 || P < 0) return BRKGA_ERR_INVALID_ARGUMENT;
  return brkga_decode_multi_stage(stage, pb, d_chrom, &P, d_makespan, d_log, d_status, d_ws, ws_bytes, pool_bins,
                                  stream);
}

int brkga_decode(const BrkgaProblem* pb, const float* d_chrom, int32_t P, double* d_makespan,
                 BrkgaPlacement* d_log, int32_t* d_status, void* d_ws, size_t ws_bytes, int64_t pool_bins,
                 void* stream) {
  return brkga_decode_stage(0, pb, d_chrom, P, d_makespan, d_log, d_status, d_ws, ws_bytes, pool_bins, stream);
}

// Decode without allocating: the workspace is the library's fixed device
// array (address resolved when the problem was created), the bin pool takes
// whatever that array has left after the per-population tables.
int brkga_decode_noalloc(const BrkgaProblem* pb, const float* d_chrom, int32_t P, double* d_makespan,
                         BrkgaPlacement* d_log, int32_t* d_status, void* stream) {
  if (!pb || pb->K != 1 || P < 0) return BRKGA_ERR_INVALID_ARGUMENT;
  if (P == 0) return BRKGA_OK;
  if (!pb->noalloc_scratch) return BRKGA_ERR_INVALID_ARGUMENT;
  const size_t cap = (size_t)BRKGA_NOALLOC_SCRATCH_BYTES;
  LaunchCounts lc;
  if (counts_of(pb, &P, &lc)) return BRKGA_ERR_INVALID_ARGUMENT;
  const Layout fixed = layout_of(pb, lc, 0);  // offsets up to the pool do not depend on the pool size
  if (fixed.off_pool >= cap) return BRKGA_ERR_WORKSPACE;
  const size_t own = (size_t)own_plates(pb, lc.items) * (pb->grid_words + pb->coarse_words) * 4;
  if (own >= kNoallocPlaneBytes) return BRKGA_ERR_WORKSPACE;
  const int64_t planes = (int64_t)((kNoallocPlaneBytes - own) / ((size_t)pb->coarse_words * 4));
  int64_t pool_bins = std::min((int64_t)((cap - fixed.off_pool) / ((size_t)pb->grid_words * 4)), planes);
  while (pool_bins > 0 && layout_of(pb, lc, pool_bins).end_pool > cap) --pool_bins;  // 256-byte rounding
  if (pool_bins < 1) return BRKGA_ERR_WORKSPACE;
  return decode_at(0, pb, d_chrom, nullptr, &P, d_makespan, nullptr, d_log, d_status, pb->noalloc_scratch, cap,
                   pool_bins, pb->noalloc_planes, stream);
}

int brkga_evaluate_host(BrkgaProblem* pb, const float* h_chrom, int32_t P, double* h_makespan,
                        BrkgaPlacement* h_log) {
  if (!pb || pb->K != 1 || P < 0 || (P > 0 && (!h_chrom || !h_makespan))) return BRKGA_ERR_INVALID_ARGUMENT;
  if (P == 0) return BRKGA_OK;
  std::lock_guard<std::mutex> lock(pb->mu);
  DeviceGuard g(pb->device);
  if (!pb->stream && cudaStreamCreateWithFlags(&pb->stream, cudaStreamNonBlocking) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  const bool want_log = h_log != nullptr;
  if (P > pb->e_cap_P || (want_log && !pb->e_cap_log)) {
    const int cap = std::max(P, pb->e_cap_P);
    cudaFree(pb->e_chrom);
    cudaFree(pb->e_out);
    cudaFree(pb->e_status);
    cudaFree(pb->e_log);
    if (pb->e_host) cudaFreeHost(pb->e_host);
    pb->e_host = nullptr;
    pb->e_chrom = nullptr;
    pb->e_out = nullptr;
    pb->e_status = nullptr;
    pb->e_log = nullptr;
    pb->e_cap_P = 0;
    if (cudaMalloc(&pb->e_chrom, (size_t)cap * 2 * pb->N * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&pb->e_out, (size_t)cap * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&pb->e_status, sizeof(int32_t)) != cudaSuccess ||
        cudaHostAlloc(&pb->e_host, 64 + (size_t)cap * sizeof(double), cudaHostAllocDefault) != cudaSuccess)
      return BRKGA_ERR_CUDA;
    if ((want_log || pb->e_cap_log) &&
        cudaMalloc(&pb->e_log, (size_t)cap * pb->M * pb->N * sizeof(BrkgaPlacement)) != cudaSuccess)
      return BRKGA_ERR_CUDA;
    pb->e_cap_log = want_log || pb->e_cap_log;
    pb->e_cap_P = cap;
  }
  LaunchCounts lc;
  if (counts_of(pb, &P, &lc)) return BRKGA_ERR_INVALID_ARGUMENT;
  if (pb->e_pool_bins < default_pool_bins(pb, lc.items)) pb->e_pool_bins = default_pool_bins(pb, lc.items);
  if (cudaMemcpyAsync(pb->e_chrom, h_chrom, (size_t)P * 2 * pb->N * sizeof(float), cudaMemcpyHostToDevice,
                      pb->stream) != cudaSuccess)
    return BRKGA_ERR_CUDA;
  for (int attempt = 0; attempt < 12; ++attempt) {
    const Layout l = layout_of(pb, lc, pb->e_pool_bins);
    if (l.total > pb->e_ws_bytes) {
      if (cudaStreamSynchronize(pb->stream) != cudaSuccess) return BRKGA_ERR_CUDA;
      cudaFree(pb->e_ws);
      pb->e_ws = nullptr;
      pb->e_ws_bytes = 0;
      if (cudaMalloc(&pb->e_ws, l.total) != cudaSuccess) return BRKGA_ERR_CUDA;
      pb->e_ws_bytes = l.total;
    }
    int st = brkga_decode(pb, pb->e_chrom, P, pb->e_out, want_log ? pb->e_log : nullptr, pb->e_status, pb->e_ws,
                          pb->e_ws_bytes, pb->e_pool_bins, pb->stream);
    if (st) return st;
    unsigned char* hs = pb->e_host;
    if (cudaMemcpyAsync(hs, pb->e_status, sizeof(int32_t), cudaMemcpyDeviceToHost, pb->stream) != cudaSuccess ||
        cudaMemcpyAsync(hs + 8, static_cast<char*>(pb->e_ws) + l.off_ctr + 8, 4 * sizeof(unsigned long long),
                        cudaMemcpyDeviceToHost, pb->stream) != cudaSuccess ||
        cudaMemcpyAsync(hs + 64, pb->e_out, (size_t)P * sizeof(double), cudaMemcpyDeviceToHost, pb->stream) !=
            cudaSuccess)
      return BRKGA_ERR_CUDA;
    if (cudaStreamSynchronize(pb->stream) != cudaSuccess) return BRKGA_ERR_CUDA;
    int32_t status = 0;
    unsigned long long counters[4];
    std::memcpy(&status, hs, sizeof(status));
    std::memcpy(counters, hs + 8, sizeof(counters));
    std::memcpy(h_makespan, hs + 64, (size_t)P * sizeof(double));
    for (int i = 0; i < 4; ++i) pb->last_counters[i] = (int64_t)counters[i];
    if (status == BRKGA_ERR_CAPACITY) {
      pb->e_pool_bins *= 2;
      continue;
    }
    if (status) return status;
    if (want_log &&
        cudaMemcpy(h_log, pb->e_log, (size_t)P * pb->M * pb->N * sizeof(BrkgaPlacement), cudaMemcpyDeviceToHost) !=
            cudaSuccess)
      return BRKGA_ERR_CUDA;
    return BRKGA_OK;
  }
  return BRKGA_ERR_CAPACITY;
}

int brkga_initial_solution_host(BrkgaProblem* pb, const int32_t* h_order, int32_t n, int32_t* h_machine,
                                BrkgaPlacement* h_place, double* h_machine_makespan) {
  if (!pb || pb->K != 1 || n < 0 || (n > 0 && (!h_order || !h_machine || !h_place)) || !h_machine_makespan)
    return BRKGA_ERR_INVALID_ARGUMENT;
  for (int k = 0; k < n; ++k)
    if (h_order[k] < 0 || h_order[k] >= pb->N) return BRKGA_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(pb->mu);
  DeviceGuard guard(pb->device);
  const int nn = std::max(n, 1);
  // one allocation: order, outputs, plate indices, scalars, status, pool (one plate per part at most), CTA state
  size_t o = 0;
  const size_t off_order = o;
  o = align_up(o + (size_t)nn * 4, 256);
  const size_t off_mach = o;
  o = align_up(o + (size_t)nn * 4, 256);
  const size_t off_out = o;
  o = align_up(o + (size_t)nn * sizeof(BrkgaPlacement), 256);
  const size_t off_pi = o;
  o = align_up(o + (size_t)nn * 4, 256);
  const size_t off_mk = o;
  o = align_up(o + (size_t)pb->M * 8, 256);
  const size_t off_bs = o;
  o = align_up(o + (size_t)nn * sizeof(BinScal), 256);
  const size_t off_ctr = o;
  o = align_up(o + 64, 256);
  const size_t off_pool = o;
  o = align_up(o + (size_t)nn * pb->grid_words * 4, 256);
  const size_t off_cpool = o;
  o = align_up(o + (size_t)nn * pb->coarse_words * 4, 256);
  const size_t state_bytes = align_up(greedy_state_bytes(nn, pb->M), 256);
  const bool in_smem = state_bytes <= kGreedyMaxSmem - 4096;
  const size_t off_state = o;
  if (!in_smem) o += kGreedyCtas * state_bytes;
  if (o > pb->greedy_bytes) {  // up to kGreedyKeep it is kept for the next call on this problem
    cudaFree(pb->greedy_ws);
    pb->greedy_ws = nullptr;
    pb->greedy_bytes = 0;
    if (cudaMalloc(&pb->greedy_ws, o) != cudaSuccess) return BRKGA_ERR_CUDA;
    pb->greedy_bytes = o;
  }
  char* d = static_cast<char*>(pb->greedy_ws);
  int st = BRKGA_OK;
  do {
    if (cudaMemset(d, 0, off_pool) != cudaSuccess ||
        (n > 0 && cudaMemcpy(d + off_order, h_order, (size_t)n * 4, cudaMemcpyHostToDevice) != cudaSuccess)) {
      st = BRKGA_ERR_CUDA;
      break;
    }
    GreedyArgs g;
    std::memset(&g, 0, sizeof(g));
    g.N = pb->N;
    g.M = pb->M;
    g.T = pb->T;
    g.status = reinterpret_cast<int32_t*>(d + off_ctr + 40);
    g.binscal = reinterpret_cast<BinScal*>(d + off_bs);
    g.pool = reinterpret_cast<uint32_t*>(d + off_pool);
    g.cpool = reinterpret_cast<uint32_t*>(d + off_cpool);
    g.grid_words = pb->grid_words;
    g.coarse_words = pb->coarse_words;
    g.vac_off = pb->vac_off;
    g.order = reinterpret_cast<const int32_t*>(d + off_order);
    g.n = n;
    g.out_machine = reinterpret_cast<int32_t*>(d + off_mach);
    g.out = reinterpret_cast<BrkgaPlacement*>(d + off_out);
    g.plate_index = reinterpret_cast<int32_t*>(d + off_pi);
    g.machine_makespan = reinterpret_cast<double*>(d + off_mk);
    g.state = in_smem ? nullptr : reinterpret_cast<unsigned char*>(d + off_state);
    g.state_bytes = state_bytes;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = kGreedyCtas;
    cfg.blockDim = kGreedyThreads;
    cfg.dynamicSmemBytes = in_smem ? state_bytes : 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kGreedyCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int32_t status = 0;
    if (cudaFuncSetAttribute(greedy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kGreedyMaxSmem - 4096) != cudaSuccess ||
        cudaLaunchKernelEx(&cfg, greedy_kernel, pb->tb, g) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(&status, g.status, 4, cudaMemcpyDeviceToHost) != cudaSuccess) {
      st = BRKGA_ERR_CUDA;
      break;
    }
    if (status) {
      st = status;
      break;
    }
    if ((n > 0 && (cudaMemcpy(h_machine, g.out_machine, (size_t)n * 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
                   cudaMemcpy(h_place, g.out, (size_t)n * sizeof(BrkgaPlacement), cudaMemcpyDeviceToHost) !=
                       cudaSuccess)) ||
        cudaMemcpy(h_machine_makespan, g.machine_makespan, (size_t)pb->M * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
      st = BRKGA_ERR_CUDA;
  } while (false);
  if (pb->greedy_bytes > kGreedyKeep) {
    cudaFree(pb->greedy_ws);
    pb->greedy_ws = nullptr;
    pb->greedy_bytes = 0;
  }
  return st;
}

int brkga_chunk_free(const BrkgaProblem* pb, int32_t path, const BrkgaChunkTest* d_items, int32_t n_items,
                     int32_t* d_status, void* stream) {
  if (!pb || pb->K != 1 || n_items < 0 || (path != BRKGA_COLLISION_BITSET && path != BRKGA_COLLISION_INT8_TC))
    return BRKGA_ERR_INVALID_ARGUMENT;
  if (n_items == 0) return BRKGA_OK;
  if (!d_items || !d_status) return BRKGA_ERR_INVALID_ARGUMENT;
  DeviceGuard g(pb->device);
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (path == BRKGA_COLLISION_BITSET) {
    chunk_free_bitset_kernel<<<n_items, 128, 0, s>>>(pb->tb, d_items, pb->M, pb->T, d_status);
  } else {
    int wmax = 1;
    for (const MachDev& m : pb->mach) wmax = std::max(wmax, m.W);
    const dim3 grid((unsigned)n_items, (unsigned)((wmax + corr::kTileM - 1) / corr::kTileM));
    chunk_free_i8_kernel<<<grid, corr::kThreads, corr::smem_bytes(corr::kMaxSide, corr::kMaxSide), s>>>(
        pb->tb, d_items, pb->M, pb->T, d_status);
  }
  return cudaGetLastError() == cudaSuccess ? BRKGA_OK : BRKGA_ERR_CUDA;
}

int brkga_last_counters(const BrkgaProblem* pb, int64_t* tests, int64_t* chunks, int64_t* bins,
                        int64_t* scan_bytes) {
  if (!pb) return BRKGA_ERR_INVALID_ARGUMENT;
  if (tests) *tests = pb->last_counters[0];
  if (chunks) *chunks = pb->last_counters[1];
  if (bins) *bins = pb->last_counters[2];
  if (scan_bytes) *scan_bytes = pb->last_counters[3];
  return BRKGA_OK;
}

}  // extern "C"
