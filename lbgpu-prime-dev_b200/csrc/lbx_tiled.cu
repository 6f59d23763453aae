// lbx_tiled.cu -- temporal blocking of small 2D lattices.
//
// A 256 x 256 D2Q9 lattice holds 65k nodes: one step is ~0.3 us of work
// spread over 148 SMs, and a step launch (or a graph node) costs more than
// that.  Here one cooperative launch advances the lattice by many steps.
// The lattice is cut into tiles, one block (an SM) each; per round a block
// loads a halo of up to K nodes around its tile into shared memory, advances
// the tile K steps there (the region still valid shrinks by one node per
// side per step), and stores the tile's nodes.  Rounds alternate between the
// population array and a scratch copy of it, so a round never reads what a
// slower block of the same round writes.  The rounds of one launch are even
// in number (the state ends in the population array), of even length each
// (a round ends after an even step), K steps or fewer (none in the first
// round where K is 2 and the pairs are odd in number): any number of AA pairs
// from two on is one launch.
//
// Between rounds a block waits only for the tiles its halo reads (their
// round counters, polled by one lane each; the wait is bounded and records a
// timeout in a status word the host reads at lbx_sync); a counter at r + 1
// also means that tile has finished reading the buffer round r + 1 writes.
// A block keeps its tile's nodes in shared memory from round to round (they
// are valid after every round), reloads only the halo, and stores only the
// strip other halos read (every node it owns in the last round).
//
// In shared memory a step is the AA step itself, in place: the odd step
// pulls d_a from slot a of the upstream node n - c_a (the node's own slot
// opp(a) behind a solid) and pushes to the slots it pulled from, the even
// step swaps its own slots.  Every node touches its own slot set only, and
// the per-node arithmetic is the step kernels' own (collide, face_north,
// face_south): FP64 results are bit-identical to the per-step path.  A step
// in place needs one population buffer where pulling from one buffer into
// another needs two, which is what lets two substances (the flow, then the
// solute from the flow's slots with u in registers) or larger tiles fit.
// The last step can write the macro variables (a frame's step).
//
// Tile plan (host).  Columns of about equal width, each cut into heights of
// about equal work per round (fluid node updates, halo included): the
// slowest tile sets the pace, and the fluid fraction of fixed tiles of a
// porous lattice spreads from below 0.3 to near 1.  Width, rows per column
// and K come from a small cost model (see best_shapes), for all SMs or, beside
// other domains' runs, for a share of them (choose_level).  The tiles' node
// tables are made once, on the device (tile_tables), and read by every
// launch: made anew in each launch they cost 15-20 us, more than the 20
// steps between two frames of a small lattice.
//
// Eligible: 2D, no Walsh run, no plane record, faces absent or fused, a run
// of AA pairs whose launch arguments do not change (what the graph replay
// needs too).
#include "lbx.h"
#include "lbx_internal.h"
#include "lbx_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

using namespace lbx;

namespace {

constexpr int kTiledThreads = 512;
constexpr int kMaxNb = 64;             // tiles one halo may read (one warp polls them)
constexpr int kMaxK = 12;              // steps per round, at most
constexpr long long kWaitLimit = 1LL << 20;   // polls of one counter (about a second)

// Region nodes (tile and halo) a block holds in its 227 KB: Q populations
// per substance, a slot index, two list entries and a flags word per node.
template <typename T, int NS>
__host__ __device__ constexpr int tiled_cap()
{
  return (227 * 1024 - 1024) / (NS * 9 * (int)sizeof(T) + 10) / 32 * 32;
}

template <typename T, int NS>
constexpr size_t tiled_smem()
{
  return (size_t)tiled_cap<T, NS>() * (NS * 9 * sizeof(T) + 10);
}

// Row pitch of a tile's region: odd, so that the nodes of a column (the
// halo's sides in list order) lie in different banks (256^2 FP64, K = 8: 2.4
// us per step; at the even pitch of 48 3.3).
__host__ __device__ constexpr int tiled_pitch(int w, int K) { return (w + 2 * K) | 1; }

// One tile: its lattice rectangle and the bounds of its node list.  The list
// holds the region's fluid nodes (region-local indices, tiled_pitch) in
// the order: interior (at least 2K from the region's edge), strip (the
// tile's other nodes, which other halos read), then the halo's rings from
// the innermost out, each part in row order; step j of a round of k steps
// updates the nodes at least K - k + j from the edge, a prefix of the list.
// A second list holds the halo's nodes in row order, for loading it: by
// rings, the halo's sides put every lane of a load in a line of its own
// (256^2 FP64, K = 6: 2.1 us against 1.2).
struct Tile {
  int x, y, w, h;
  int at;                     // where its tables begin
  int interior, own;          // nodes in the interior; in the tile
  int ring[kMaxK + 1];        // ring[j]: nodes through the j innermost rings (ring[0] = own)
};

// A region node's flags word: bit a (a < 9) the node upstream in direction
// a (n - c_a) is solid; kWSolid the node itself is solid; kWNorth / kWSouth
// its class bits.
constexpr unsigned kWSolid = 1u << 15, kWNorth = 1u << 9, kWSouth = 1u << 10;

template <typename T>
struct TiledArgs {
  T* f0;                        // the population array [nsubs][9][P] (dense: P = N)
  T* f1;                        // scratch of the same shape
  long long P;
  const Tile* tiles;
  // per tile from Tile::at on, an entry per region node:
  const int* gidx;              // population slot
  const unsigned short* list;
  const unsigned short* wrd;    // flags words
  const unsigned short* halo;   // the halo's nodes by rows
  const int* nbrs;              // [ntiles][kMaxNb]: the tiles a halo reads, -1 after the last
  int* flags;                   // per-tile round counters
  int* status;
  int base;                     // counter value this launch starts from
  int K;
  int pairs, rounds;            // AA pairs spread over the (even) number of rounds
  int write_mv;                 // the last step writes the macro variables
};

// Rounds of a stretch of `pairs` AA pairs at K steps a round at most: an even
// number, two at least.  At K = 2 that is one more than the pairs where these
// are odd, so one round has no step.
__host__ __device__ constexpr int round_count(int pairs, int K)
{
  const int per = K / 2, least = ((pairs + per - 1) / per + 1) / 2 * 2;
  return least < 2 ? 2 : least;
}

// Steps of round r: the pairs spread evenly, the last rounds one longer, so
// that the last one always has the step that writes the macro variables.
__host__ __device__ constexpr int round_steps(int pairs, int rounds, int r)
{
  return 2 * (pairs / rounds + (r >= rounds - pairs % rounds ? 1 : 0));
}

constexpr bool rounds_end_in_steps()
{
  for (int K = 2; K <= kMaxK; K += 2)
    for (int pairs = 2; pairs <= 60; ++pairs) {
      const int rounds = round_count(pairs, K);
      int steps = 0;
      for (int r = 0; r < rounds; ++r) {
        if (round_steps(pairs, rounds, r) > K) return false;
        steps += round_steps(pairs, rounds, r);
      }
      if (steps != 2 * pairs || round_steps(pairs, rounds, rounds - 1) < 2) return false;
    }
  return true;
}
static_assert(rounds_end_in_steps(), "every stretch's steps, the last round with some");

// Round counters: tile t has stored the strips of round r when
// flags[t] >= base + r + 1 (base grows from launch to launch).
__device__ __forceinline__ void publish(int* flag, int value)
{
  __threadfence();
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}

__device__ __forceinline__ int observe(const int* flag)
{
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
  return v;
}

// One node's update in shared memory (b: [NS][9][cap]) at parity ODD.
template <typename T, int NS, int MODEL, bool ODD>
__device__ __forceinline__ void tiled_node(const StepArgs<T>& A, T* b, int node, unsigned w,
                                           int pitch, bool write_mv, int n)
{
  constexpr int cap = tiled_cap<T, NS>();
  int slot[9];                  // where d_a is read; d_opp(a) is written there
#pragma unroll
  for (int a = 0; a < 9; ++a) {
    if (ODD) {
      const int up = node - (cy(a) < 0 ? -pitch : (cy(a) > 0 ? pitch : 0)) - cx(a);
      slot[a] = ((w >> a) & 1u) ? opp(a) * cap + node : a * cap + up;
    } else {
      slot[a] = opp(a) * cap + node;
    }
  }
  T u[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    if (s == 1 && !A.solute_on) break;
    T* const fs = b + s * 9 * cap;
    T d[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) d[a] = fs[slot[a]];
    if (w & (kWNorth | kWSouth)) {
      const bool shifted = MODEL != PLAIN_COMP && s == 0;
      if (w & kWNorth)
        face_north<T>(A.face_n[s], A.rho_n[s], A.sc[s].rhoA, A.drho_n[s], shifted, d);
      if (w & kWSouth)
        face_south<T>(A.face_s[s], A.rho_s[s], A.sc[s].rhoA, A.drho_s[s], shifted, d);
    }
    collide<T, 9, MODEL>(A, s, s == 1, ODD ? 1 : 2, d, u, n, write_mv);
#pragma unroll
    for (int a = 0; a < 9; ++a) fs[slot[opp(a)]] = d[a];
  }
}

// Block t advances tile t by all rounds.  Lists keep a warp's shared-memory
// accesses runs of neighbouring nodes with no lane on a solid node.
template <typename T, int NS, int MODEL>
__global__ void __launch_bounds__(kTiledThreads, 1)
aa_tiled(StepArgs<T> A, TiledArgs<T> R)
{
  constexpr int cap = tiled_cap<T, NS>();
  extern __shared__ __align__(16) unsigned char smem[];
  T* const b = reinterpret_cast<T*>(smem);                                  // [NS][9][cap]
  int* const gidx = reinterpret_cast<int*>(b + NS * 9 * cap);               // [cap]
  unsigned short* const list = reinterpret_cast<unsigned short*>(gidx + cap);
  unsigned short* const wrd = list + cap;
  unsigned short* const halo = wrd + cap;
  __shared__ Tile tile;
  __shared__ int gave_up;
  const int K = R.K;
  if (threadIdx.x < sizeof(Tile) / 4)
    reinterpret_cast<int*>(&tile)[threadIdx.x] =
        reinterpret_cast<const int*>(R.tiles + blockIdx.x)[threadIdx.x];
  __syncthreads();
  const int pitch = tiled_pitch(tile.w, K), region = pitch * (tile.h + 2 * K);
  const size_t at = (size_t)tile.at;
  for (int i = threadIdx.x; i < region; i += kTiledThreads) {
    gidx[i] = R.gidx[at + i];
    list[i] = R.list[at + i];
    wrd[i] = R.wrd[at + i];
    halo[i] = R.halo[at + i];
  }
  __syncthreads();
  const int subs = (NS == 2 && A.solute_on) ? 2 : 1;

  for (int r = 0; r < R.rounds; ++r) {
    const T* const src = (r & 1) ? R.f1 : R.f0;
    T* const dst = (r & 1) ? R.f0 : R.f1;
    const int k = round_steps(R.pairs, R.rounds, r);
    if (r > 0) {
      // lane q of warp 0 waits for the q-th (and the 32 + q-th) tile the halo
      // reads to finish round r - 1
      if (threadIdx.x < 32) {
        int late = 0;
#pragma unroll 1
        for (int q = threadIdx.x; q < kMaxNb && !late; q += 32) {
          const int nb = R.nbrs[blockIdx.x * kMaxNb + q];
          if (nb < 0) break;
          long long polls = 0;
          // every poll is an L2 round trip: no sleep between polls, and the
          // status word, a second one, only now and then
          while (observe(R.flags + nb) < R.base + r) {
            if (++polls >= kWaitLimit || (polls % 64 == 0 && *(volatile int*)R.status != 0)) {
              late = 1;
              break;
            }
          }
        }
        late = __any_sync(0xffffffffu, late);
        if (threadIdx.x == 0) {
          if (late) atomicExch(R.status, 1);
          gave_up = late;
        }
      }
      __syncthreads();
      if (gave_up) return;          // every thread of the block leaves together
    }
    // the tile's own nodes once, the halo every round, all of a node's loads
    // in flight together (two nodes a thread at a time spilled and lost)
    auto load = [&](const unsigned short* nodes, int count) {
      for (int q = threadIdx.x; q < count; q += kTiledThreads) {
        const int i = nodes[q];
        const T* const g = src + gidx[i];
        T v[NS][9];
#pragma unroll
        for (int s = 0; s < NS; ++s)
          if (s < subs) {
#pragma unroll
            for (int a = 0; a < 9; ++a) v[s][a] = __ldcg(g + (s * 9 + a) * R.P);
          }
#pragma unroll
        for (int s = 0; s < NS; ++s)
          if (s < subs) {
#pragma unroll
            for (int a = 0; a < 9; ++a) b[(s * 9 + a) * cap + i] = v[s][a];
          }
      }
    };
    if (r == 0) load(list, tile.own);
    load(halo, tile.ring[K] - tile.own);
    __syncthreads();
    const bool last = r + 1 == R.rounds;
#pragma unroll 1
    for (int j = 1; j <= k; j += 2) {
      const int n_odd = tile.ring[k - j], n_even = tile.ring[k - j - 1];
      for (int q = threadIdx.x; q < n_odd; q += kTiledThreads) {
        const int node = list[q];
        tiled_node<T, NS, MODEL, true>(A, b, node, wrd[node], pitch, false, 0);
      }
      __syncthreads();
      const bool mv = last && j + 1 == k && R.write_mv;
      for (int q = threadIdx.x; q < n_even; q += kTiledThreads) {
        const int node = list[q];
        int n = 0;
        if (mv) {                   // an own node: inside the lattice
          const int ly = node / pitch, lx = node - ly * pitch;
          n = (tile.x + lx - K) + A.LX * (tile.y + ly - K);
        }
        tiled_node<T, NS, MODEL, false>(A, b, node, wrd[node], pitch, mv, n);
      }
      __syncthreads();
    }
    for (int q = (last ? 0 : tile.interior) + threadIdx.x; q < tile.own; q += kTiledThreads) {
      const int i = list[q];
      const int m = gidx[i];
      for (int s = 0; s < subs; ++s) {
        T* const g = dst + (size_t)s * 9 * R.P + m;
#pragma unroll
        for (int a = 0; a < 9; ++a) g[a * R.P] = b[(s * 9 + a) * cap + i];
      }
    }
    if (!last) {
      __syncthreads();              // the block's stores are issued
      if (threadIdx.x == 0) publish(R.flags + blockIdx.x, R.base + r + 1);
    }
  }
}

// The node tables of tile blockIdx.x (Tile's list bounds included).  Warp c
// gathers list part c: interior, strip, ring K-1, ..., ring 0; warp K+2 the
// halo by rows.
__global__ void __launch_bounds__(kTiledThreads)
tile_tables(const uint8_t* cls, const int* fidx, int LX, int LY, int K, Tile* tiles, int* gidx,
            unsigned short* list, unsigned short* wrd, unsigned short* halo)
{
  extern __shared__ unsigned short w[];             // [cap] flags words
  __shared__ int count[kTiledThreads / 32];
  Tile& t = tiles[blockIdx.x];
  const int width = t.w + 2 * K, pitch = tiled_pitch(t.w, K), rows = t.h + 2 * K;
  const int region = pitch * rows;
  const int x0 = t.x - K, y0 = t.y - K;
  const size_t at = (size_t)t.at;
  for (int i = threadIdx.x; i < region; i += kTiledThreads) {
    if (i % pitch >= width) {                       // the pitch's padding
      w[i] = (unsigned short)kWSolid;
      gidx[at + i] = -1;
      continue;
    }
    int gx = (x0 + i % pitch) % LX, gy = (y0 + i / pitch) % LY;
    if (gx < 0) gx += LX;
    if (gy < 0) gy += LY;
    const int n = gx + LX * gy;
    const uint8_t c = cls[n];
    w[i] = (unsigned short)(((c & CLS_SOLID) ? kWSolid : 0u) | ((c & CLS_NORTH) ? kWNorth : 0u) |
                            ((c & CLS_SOUTH) ? kWSouth : 0u));
    gidx[at + i] = (c & CLS_SOLID) ? -1 : (fidx ? fidx[n] : n);
  }
  __syncthreads();
  // upstream solid bits of the nodes a step can update (off the region's edge)
  for (int i = threadIdx.x; i < region; i += kTiledThreads) {
    const int lx = i % pitch, ly = i / pitch;
    unsigned bits = w[i];
    if (lx >= 1 && lx <= width - 2 && ly >= 1 && ly <= rows - 2 && !(bits & kWSolid)) {
#pragma unroll
      for (int a = 1; a < 9; ++a)
        if (w[i - (cx(a) + pitch * cy(a))] & kWSolid) bits |= 1u << a;
    }
    wrd[at + i] = (unsigned short)bits;
  }
  const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto in_part = [&](int i) -> bool {
    if (i >= region || (w[i] & kWSolid)) return false;
    const int lx = i % pitch, ly = i / pitch;
    const int e = min(min(lx, width - 1 - lx), min(ly, rows - 1 - ly));
    if (part == K + 2) return e < K;
    return part == 0 ? e >= 2 * K : (part == 1 ? e >= K && e < 2 * K : e == K + 1 - part);
  };
  int mine = 0;
  if (part < K + 2)
    for (int i = lane; i - lane < region; i += 32)
      mine += __popc(__ballot_sync(0xffffffffu, in_part(i)));
  if (lane == 0) count[part] = mine;
  __syncthreads();
  int pos = 0;
  for (int c = 0; c < part; ++c) pos += count[c];
  if (part < K + 2 && lane == 0) {
    if (part == 0) t.interior = pos + mine;
    else if (part == 1) t.own = t.ring[0] = pos + mine;
    else t.ring[part - 1] = pos + mine;
  }
  if (part == K + 2) pos = 0;
  unsigned short* const out = part == K + 2 ? halo : list;
  if (part < K + 3)
    for (int i = lane; i - lane < region; i += 32) {
      const bool f = in_part(i);
      const unsigned ball = __ballot_sync(0xffffffffu, f);
      if (f) out[at + pos + __popc(ball & ((1u << lane) - 1u))] = (unsigned short)i;
      pos += __popc(ball);
    }
}
static_assert(kMaxK + 3 <= kTiledThreads / 32, "a warp per list part");

// ---- the tile plan (host) ---------------------------------------------------

// Fluid counts over rectangles of the periodic lattice, halos included.
struct FluidSums {
  int LX, LY, ext, W;
  std::vector<int> s;   // prefix sums over [-ext, LY + ext) x [-ext, LX + ext)

  FluidSums(const std::vector<uint8_t>& solids, int lx, int ly, int e)
      : LX(lx), LY(ly), ext(e), W(lx + 2 * e + 1), s((size_t)(ly + 2 * e + 1) * W, 0)
  {
    std::vector<int> gx(LX + 2 * ext);
    for (int x = 0; x < LX + 2 * ext; ++x) gx[x] = ((x - ext) % LX + LX) % LX;
    for (int y = 0; y < LY + 2 * ext; ++y) {
      const uint8_t* row = solids.data() + (size_t)LX * (((y - ext) % LY + LY) % LY);
      const int* above = &s[(size_t)y * W];
      int* here = &s[(size_t)(y + 1) * W];
      int sum = 0;
      for (int x = 0; x < LX + 2 * ext; ++x) {
        sum += row[gx[x]] != 1;
        here[x + 1] = above[x + 1] + sum;
      }
    }
  }
};

// One column of tiles: fluid nodes in the rows below y (from -ext on) of the
// column widened by j on both sides, for the three j that work() asks for.
struct Band {
  int K, ext;
  std::vector<int> s[3];

  Band(const FluidSums& fs, int x, int w, int k) : K(k), ext(fs.ext)
  {
    for (int q = 0; q < 3; ++q) {
      const int j = ring(q), rows = fs.LY + 2 * ext + 1;
      s[q].resize(rows);
      const int* p = fs.s.data() + x - j + ext;
      for (int y = 0; y < rows; ++y, p += fs.W) s[q][y] = p[w + 2 * j] - p[0];
    }
  }
  int ring(int q) const { return q == 0 ? 0 : q == 1 ? (K - 1) / 2 : K - 1; }
  // fluid nodes within ring(q) of the tile of rows [y, y + h)
  long long around(int q, int y, int h) const
  {
    return s[q][y + h + ring(q) + ext] - s[q][y - ring(q) + ext];
  }
  // node updates of one round of the tile, about: the sum of the fluid nodes
  // within j over j = 0 .. K - 1 by Simpson's rule (exact where the fluid is
  // uniform)
  long long work(int y, int h) const
  {
    return K * (around(0, y, h) + 4 * around(1, y, h) + around(2, y, h)) / 6;
  }
};

struct Shape {
  int cols, rows, K;
  int tiles;            // at most this many; denser columns get more of them
  double us;            // modelled time per step
};

// Modelled microseconds per step.  A step costs a latency and its node
// updates; a round adds its boundary, a latency (counters, fence, store) and
// the halo's load.  Steps fitted to clock spans: 256^2 FP64 (tiles 32 x 9) a
// step of 261 nodes 0.75 us, of 690 1.3; FP32 of 256 nodes 0.34, of 950
// 0.93; 300 x 220 FP64 with a solute of 346 nodes 1.1, of 700 1.9.  The
// boundary to whole runs (modelled / measured, us per step): 256^2 FP64
// K = 8 1.9 / 1.8, 400^2 FP64 K = 6 3.1 / 3.1, 560^2 FP64 K = 2 5.3 / 5.6,
// 512^2 FP32 K = 6 2.8 / 2.6, 48 x 67 FP64 K = 8 1.2 / 1.2.
template <typename T, int NS>
double shape_us(double fluid, int w, int h, int K)
{
  const double lat = sizeof(T) == 8 ? 0.37 : 0.13;
  const double node = (sizeof(T) == 8 ? 1.4e-3 : 0.8e-3) * (NS == 2 ? 1.65 : 1.0);
  // the round's node updates: (w + 2 j)(h + 2 j) over j = 0 .. K - 1
  const double k = K, area = (double)w * h;
  const double nodes = k * area + (w + h) * k * (k - 1) + 2. / 3. * k * (k - 1) * (2 * k - 1);
  return (4.0 + 6.2e-3 * NS * fluid * ((w + 2 * k) * (h + 2 * k) - area) + node * fluid * nodes) / k +
         lat;
}

// The launch-per-step path's: a latency, larger for two substances (two
// launches or a joint one), and the populations, from the L2.  Fitted to
// whole runs of dependent launches, 40 % / 2 % solid nodes (modelled /
// measured, us per step): FP64 256^2 2.4, 2.8 / 2.2, 2.5, 400^2 3.2, 4.2 /
// 3.1, 4.3, 560^2 4.6, 6.4 / 4.9, 6.3; FP32 512^2 3.5, 4.6 / 3.7, 3.8; FP64
// with a solute 200^2 2.9, 3.3 / 2.9, 3.4, 380^2 4.5, 6.0 / 4.7, 6.2.  With
// the latency of launches that waited for one another (2.3 us, one
// substance) the tiled run was taken where it lost: 560^2 FP64 5.5 against
// 4.9, 380^2 with a solute 6.2 against 4.7.
double steps_us(double nodes, size_t real, int nsubs)
{
  const double per = real != 8 ? 1.1e-5 : nsubs == 2 ? 1.3e-5 : 1.5e-5;
  return (nsubs == 2 ? 2.3 : 1.8) + nodes * nsubs * per;
}

// The shapes whose regions fit a block and whose tiles fit the SMs: the best
// few, best first.
constexpr int kShapes = 8;

template <typename T, int NS>
int best_shapes(int LX, int LY, double fluid, int blocks, Shape (&best)[kShapes])
{
  int n = 0;
  for (int cols = 1; cols <= std::min(LX, blocks); ++cols) {
    const int w = (LX + cols - 1) / cols;
    for (int rows = 1, last = 0; rows <= std::min(LY, blocks / cols); ++rows) {
      const int h = (LY + rows - 1) / rows;
      if (h == last && rows != blocks / cols) continue;     // the same tiles
      last = h;
      for (int K = 2; K <= kMaxK; K += 2) {
        if (tiled_pitch(w, K) * (h + 2 * K) > tiled_cap<T, NS>()) break;
        // tiles a halo reads, about: their heights vary
        const int nx = std::min(cols, 2 * ((K + w - 1) / w) + 1);
        const int ny = std::min(rows, 2 * ((K + h - 1) / h) + 1);
        if (nx * ny > kMaxNb / 2) continue;
        const int tiles = rows == blocks / cols ? blocks : cols * rows;
        const Shape sh = {cols, rows, K, tiles, shape_us<T, NS>(fluid, w, h, K)};
        int at = n;
        while (at > 0 && sh.us < best[at - 1].us) --at;
        if (at == kShapes) continue;
        if (n < kShapes) ++n;
        for (int i = n - 1; i > at; --i) best[i] = best[i - 1];
        best[at] = sh;
      }
    }
  }
  return n;
}

// Tiles of about equal work for a shape, column by column from the first row
// up; false when a halo reads too many.
bool make_tiles(const FluidSums& fs, int LX, int LY, const Shape& sh, int cap,
                std::vector<Tile>& tiles, std::vector<int>& nbrs)
{
  const int K = sh.K;
  auto edge = [&](int c) { return (int)((long long)LX * c / sh.cols); };
  std::vector<Band> bands;
  bands.reserve(sh.cols);
  for (int c = 0; c < sh.cols; ++c) bands.emplace_back(fs, edge(c), edge(c + 1) - edge(c), K);
  std::vector<int> first(sh.cols + 1);                // a column's first tile
  auto cut = [&](long long W, std::vector<Tile>* to) -> bool {
    int n = 0;
    for (int c = 0; c < sh.cols && n <= sh.tiles; ++c) {
      const int x = edge(c), w = edge(c + 1) - x;
      const int hmax = cap / tiled_pitch(w, K) - 2 * K;
      first[c] = n;
      for (int y = 0; y < LY && n <= sh.tiles; ++n) {
        int h = 1, most = std::min(hmax, LY - y);     // the work grows with h
        while (h < most) {
          const int mid = (h + most + 1) / 2;
          if (bands[c].work(y, mid) <= W) h = mid; else most = mid - 1;
        }
        if (to) {
          Tile t;
          std::memset(&t, 0, sizeof t);
          t.x = x; t.y = y; t.w = w; t.h = h;
          to->push_back(t);
        }
        y += h;
      }
    }
    first[sh.cols] = n;
    return n <= sh.tiles;
  };
  // about the least work bound that needs no more tiles (to 2 %)
  long long hi = 0;
  for (int c = 0; c < sh.cols; ++c) hi += bands[c].work(0, (LY + sh.rows - 1) / sh.rows);
  hi = hi / sh.cols + 1;
  long long lo = 0;
  while (!cut(hi, nullptr)) {
    if (hi > (1LL << 40)) return false;
    lo = hi;
    hi *= 2;
  }
  while (hi - lo > 1 + hi / 50) {
    const long long mid = (lo + hi) / 2;
    if (cut(mid, nullptr)) hi = mid; else lo = mid;
  }
  tiles.clear();
  cut(hi, &tiles);
  // the tiles each halo reads: the columns around the tile's, in each the
  // tiles around its rows, from the one that holds the halo's first row up;
  // a halo that goes round the lattice meets a tile again
  std::vector<int> owner((size_t)sh.cols * LY);
  for (int c = 0; c < sh.cols; ++c)
    for (int t = first[c]; t < first[c + 1]; ++t)
      std::fill_n(owner.begin() + (size_t)c * LY + tiles[t].y, tiles[t].h, t);
  nbrs.assign(tiles.size() * kMaxNb, -1);
  std::vector<int> met(tiles.size(), -1);
  for (int c = 0, t = 0; c < sh.cols; ++c) {
    int c0 = c, left = K;                             // the column of the halo's first node
    for (int n = 1; left > 0 && n < sh.cols; ++n) {
      c0 = c0 == 0 ? sh.cols - 1 : c0 - 1;
      left -= edge(c0 + 1) - edge(c0);
    }
    int across = 0;                                   // columns from there on
    for (int w = left > 0 ? LX : K - left + edge(c + 1) - edge(c) + K, q = c0;
         w > 0 && across < sh.cols; ++across, q = q + 1 == sh.cols ? 0 : q + 1)
      w -= edge(q + 1) - edge(q);
    for (; t < first[c + 1]; ++t) {
      const Tile& g = tiles[t];
      int y0 = (g.y - K) % LY;
      if (y0 < 0) y0 += LY;
      int k = 0;
      int* const row = &nbrs[(size_t)t * kMaxNb];
      for (int i = 0, q = c0; i < across; ++i, q = q + 1 == sh.cols ? 0 : q + 1) {
        int o = owner[(size_t)q * LY + y0];
        for (int rows = y0 - tiles[o].y + g.h + 2 * K; rows > 0 && met[o] != t;) {
          met[o] = t;
          if (k == kMaxNb) return false;
          row[k++] = o;
          rows -= tiles[o].h;
          if (++o == first[q + 1]) o = first[q];
        }
      }
    }
  }
  return true;
}

// Region nodes of a shape's tiles, at most (heights sum to LY per column).
size_t region_nodes(const Shape& sh, int LX, int LY)
{
  return (size_t)tiled_pitch((LX + sh.cols - 1) / sh.cols, sh.K) *
         ((size_t)sh.cols * LY + (size_t)sh.tiles * 2 * sh.K);
}

// Bytes of the scratch array with the status word behind it, and of a plan's
// tables: tiles, neighbours, counters, then per region node a slot and three
// list entries.
size_t scratch_bytes(const lbx_domain* d)
{
  const long long P = d->layout == LBX_LAYOUT_COMPACT ? d->P : d->N;
  return ((size_t)d->p.nsubs * 9 * P * d->real_size + 255) / 256 * 256 + 256;
}

size_t tables_bytes(int tiles, size_t nodes)
{
  return (size_t)tiles * (sizeof(Tile) + (kMaxNb + 1) * sizeof(int)) +
         nodes * (sizeof(int) + 3 * sizeof(unsigned short));
}

int multiprocessors(const lbx_domain* d)
{
  int sms = 0, coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, d->p.device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d->p.device);
  if (coop && sms > 0) return sms;
  cudaGetLastError();
  return 0;
}

// The best shapes for level l, and their modelled time in the plan; state -1
// where none fits.
template <typename T, int NS>
int shapes_of(lbx_domain* d, int l, Shape (&shapes)[kShapes])
{
  const double fluid = (double)d->fluid / (double)d->N;
  const int n = best_shapes<T, NS>(d->p.LX, d->p.LY, fluid, multiprocessors(d) >> l, shapes);
  if (n == 0) d->tiled[l].state = -1;
  d->tiled[l].us = n == 0 ? 1e30 : shapes[0].us;
  return n;
}

// Whether the tiled run with the GPU to itself is modelled faster than a
// launch per step.
bool better(const lbx_domain* d)
{
  const double us = d->tiled[0].us;
  return us > 0.0 && us < steps_us((double)d->fluid, d->real_size, d->p.nsubs);
}

template <typename T, int NS>
size_t room(lbx_domain* d)
{
  Shape shapes[kShapes];
  const int n = shapes_of<T, NS>(d, 0, shapes);
  if (!better(d)) return 0;
  size_t most = 0;
  for (int i = 0; i < n; ++i)
    most = std::max(most, tables_bytes(shapes[i].tiles, region_nodes(shapes[i], d->p.LX, d->p.LY)));
  return scratch_bytes(d) + most;
}

// Plans the lattice's tiles for level l and makes their tables: state 1, or
// -1 where no shape fits or there is no memory for it.
template <typename T, int NS>
lbx_status make_plan(lbx_domain* d, int l)
{
  const lbx_params& p = d->p;
  TiledPlan& plan = d->tiled[l];
  Shape shapes[kShapes];
  const int ns = d->fluid == 0 ? 0 : shapes_of<T, NS>(d, l, shapes);
  plan.state = -1;
  if (ns == 0) return LBX_OK;
  const FluidSums fs(d->host_solids, p.LX, p.LY, kMaxK);
  constexpr int cap = tiled_cap<T, NS>();
  std::vector<Tile> tiles;
  std::vector<int> nbrs;
  int i = 0;
  while (i < ns && !make_tiles(fs, p.LX, p.LY, shapes[i], cap, tiles, nbrs)) ++i;
  if (i == ns) return LBX_OK;
  const int nt = (int)tiles.size();
  plan.K = shapes[i].K;
  plan.us = shapes[i].us;
  plan.ntiles = nt;
  plan.base = 0;
  size_t nodes = 0;
  for (Tile& t : tiles) {
    t.at = (int)nodes;
    nodes += (size_t)tiled_pitch(t.w, plan.K) * (t.h + 2 * plan.K);
  }
  plan.nodes = nodes;
  const size_t b_tiles = (size_t)nt * sizeof(Tile), b_nbrs = nbrs.size() * sizeof(int);
  const size_t b_flags = (size_t)nt * sizeof(int), b_gidx = nodes * sizeof(int);
  std::vector<char> head(b_tiles + b_nbrs + b_flags, 0);   // counters start at 0
  std::memcpy(head.data(), tiles.data(), b_tiles);
  std::memcpy(head.data() + b_tiles, nbrs.data(), b_nbrs);
  // the scratch array, once, and the tables of level 0: behind the population
  // array where lbx_create left room (a call here costs 0.4 ms), else on
  // their own; other levels' tables on their own
  const size_t scratch = scratch_bytes(d);
  cudaError_t e = cudaSuccess;
  if (!d->tiled_scratch) {
    char* at = (char*)d->tiled_room;
    if (at) {
      d->tiled_tables = at + scratch;
    } else {
      e = cudaMalloc(&d->tiled_own, scratch);
      at = (char*)d->tiled_own;
    }
    if (e == cudaSuccess) {
      d->tiled_scratch = at;
      d->tiled_status = (int*)(at + scratch - 256);
      e = cudaMemsetAsync(d->tiled_status, 0, sizeof(int), d->stream);
    }
  }
  char* at = nullptr;
  if (l == 0 && d->tiled_tables) {
    at = (char*)d->tiled_tables;
  } else if (e == cudaSuccess) {
    e = cudaMalloc(&plan.own, tables_bytes(nt, nodes));
    at = (char*)plan.own;
  }
  if (e == cudaSuccess) {
    plan.tiles = at;
    plan.nbrs = (int*)(at + b_tiles);
    plan.flags = (int*)(at + b_tiles + b_nbrs);
    plan.gidx = (int*)(at + b_tiles + b_nbrs + b_flags);
    plan.list = (unsigned short*)(at + b_tiles + b_nbrs + b_flags + b_gidx);
    e = cudaMemcpyAsync(at, head.data(), head.size(), cudaMemcpyHostToDevice, d->stream);
  }
  if (e == cudaSuccess) {
    tile_tables<<<nt, kTiledThreads, (size_t)cap * sizeof(unsigned short), d->stream>>>(
        d->cls, d->layout == LBX_LAYOUT_COMPACT ? d->fidx : nullptr, p.LX, p.LY, plan.K,
        (Tile*)plan.tiles, plan.gidx, plan.list, plan.list + nodes, plan.list + 2 * nodes);
    d->launches++;
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    if (e == cudaErrorMemoryAllocation && (l > 0 || d->run_mode != LBX_RUN_TILED)) {
      cudaGetLastError();             // another level, or a launch per step
      return LBX_OK;
    }
    return lbx_internal_fail(e == cudaErrorMemoryAllocation ? LBX_ERR_NOMEM : LBX_ERR_CUDA,
                             cudaGetErrorString(e));
  }
  plan.state = 1;
  return LBX_OK;
}

lbx_status plan_level(lbx_domain* d, int l)
{
  if (d->tiled[l].state != 0) return LBX_OK;
  try {
    if (d->real_size == 8)
      return d->p.nsubs == 2 ? make_plan<double, 2>(d, l) : make_plan<double, 1>(d, l);
    return d->p.nsubs == 2 ? make_plan<float, 2>(d, l) : make_plan<float, 1>(d, l);
  } catch (const std::bad_alloc&) {
    d->tiled[l].state = -1;           // no host memory for it
    return LBX_OK;
  }
}

// ---- domains side by side ---------------------------------------------------

// A tiled launch holds every SM that it has a block on.  With the GPU to
// itself a domain's tiles spread over all SMs, where a small lattice spends
// most of its time in halos and waits; launches of several domains, on
// streams of their own, would then run one after another (twelve of 48 x 67,
// 2000 steps each: FP64 26 ms, FP32 21; on a sixteenth of the GPU each, side
// by side, 4.3 and 3.4; one alone 2.2 and 2.0).  So a launch looks whether
// other domains' tiled runs are under way and takes tiles for its share.  The
// results do not depend on the tiles: every node's update is the same code on
// the same values.
//
// The listed domains are those that have taken, or might have taken, a tiled
// run.  A stretch's launch records its domain's event if another stream's
// domain is listed; one that comes later asks whether the event has passed.
// A domain that launched after this one's last launch counts as busy if the
// newest of those still is, which saves asking for each (a round of many
// domains would ask for all the others in each launch).  A launch that others
// were seen beside leaves their number for its domain's next one, which is
// the first of a new round in a program that waits for all domains between
// rounds.  The event and the question cost 2 us of a 32 us run: while nothing
// was seen beside one another in 64 launches, only every eighth is recorded.
std::mutex g_mu;                        // guards what follows, and the listed domains' fields
std::vector<lbx_domain*> g_listed;      // tiled_stream, _turn, _busy and _company
unsigned long long g_turn = 0;
unsigned g_quiet = 0;                   // launches since one saw another's run

bool under_way(lbx_domain* o)
{
  if (!o->tiled_busy) return false;
  const cudaError_t e = cudaEventQuery(o->tiled_done);
  if (e != cudaErrorNotReady) o->tiled_busy = false;
  if (e != cudaSuccess) cudaGetLastError();
  return o->tiled_busy;
}

// Other domains' tiled runs under way on d's device; *record: whether this
// one is to be seen by theirs.
int busy_beside(lbx_domain* d, bool* record)
{
  // a caller's capture elsewhere is none of these calls' business
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };
  std::lock_guard<std::mutex> lock(g_mu);
  if (!d->tiled_listed) try {
    g_listed.push_back(d);
    d->tiled_listed = true;
  } catch (const std::bad_alloc&) {}    // unseen by the others
  d->tiled_stream = d->stream;
  lbx_domain* newest = nullptr;
  bool beside = false;
  for (lbx_domain* o : g_listed) {
    if (o == d || o->p.device != d->p.device || o->tiled_stream == d->stream) continue;
    beside = true;
    if (o->tiled_busy && (!newest || o->tiled_turn > newest->tiled_turn)) newest = o;
  }
  int n = 0;
  if (newest) {
    Relaxed relaxed;
    const bool assume = under_way(newest);
    auto counts = [&](const lbx_domain* o) {
      return o != d && o->p.device == d->p.device && o->tiled_stream != d->stream && o->tiled_busy;
    };
    for (lbx_domain* o : g_listed)
      if (counts(o) && ((assume && o->tiled_turn > d->tiled_turn) || under_way(o))) ++n;
    for (lbx_domain* o : g_listed)
      if (counts(o)) o->tiled_company = std::max(o->tiled_company, n);
  }
  n = std::max(n, d->tiled_company);
  d->tiled_company = 0;
  g_quiet = n > 0 ? 0 : g_quiet + 1;
  *record = beside && (g_quiet < 64 || g_quiet % 8 == 0);
  return n;
}

}  // namespace

// After the stretch's launches: the domain's event, if others are listed.
void lbx_internal_tiled_launched(lbx_domain* d)
{
  if (!d->tiled_listed) return;
  bool busy = false;
  if (d->tiled_record) {
    cudaError_t e = d->tiled_done ? cudaSuccess
                                  : cudaEventCreateWithFlags(&d->tiled_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(d->tiled_done, d->stream);
    if (e != cudaSuccess) cudaGetLastError();
    busy = e == cudaSuccess;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  d->tiled_turn = ++g_turn;
  d->tiled_busy = busy;
}

namespace {

template <typename T, int NS>
void model_level(lbx_domain* d, int l)
{
  Shape shapes[kShapes];
  if (d->tiled[l].us == 0.0) shapes_of<T, NS>(d, l, shapes);
}

// The level whose plan a launch beside n others takes, with which all of them
// are modelled done soonest; -1: a launch per step.
// Step launches run beside one another without holding SMs, so they win
// where the lattice is large for a share of the GPU (three 300 x 300 FP64,
// 800 steps: tiled 4.9 ms, step launches 3.8).  FP32 does not take them here:
// its results would depend on the others in their last bits.
lbx_status choose_level(lbx_domain* d, int n, int* level)
{
  *level = 0;
  double best = d->tiled[0].us * (n + 1);
  for (int l = 1; l < TiledPlan::kLevels && (1 << (l - 1)) < n + 1; ++l) {
    if (d->real_size == 8)
      d->p.nsubs == 2 ? model_level<double, 2>(d, l) : model_level<double, 1>(d, l);
    else
      d->p.nsubs == 2 ? model_level<float, 2>(d, l) : model_level<float, 1>(d, l);
    const double us = d->tiled[l].us * ((n >> l) + 1);    // n + 1 runs, 2^l at a time
    if (us >= best) continue;
    if (lbx_status st = plan_level(d, l)) return st;
    if (d->tiled[l].state <= 0) continue;
    best = us;
    *level = l;
  }
  // (its launches cost the host more: by some margin)
  if (n > 0 && d->real_size == 8 && d->run_mode == LBX_RUN_AUTO &&
      1.15 * steps_us((double)d->fluid * (n + 1), d->real_size, d->p.nsubs) < best)
    *level = -1;
  return LBX_OK;
}

template <typename T, int NS, int MODEL>
lbx_status launch(lbx_domain* d, const StepArgs<T>& A, int pairs, bool write_mv)
{
  constexpr size_t smem = tiled_smem<T, NS>();
  const void* fn = (const void*)aa_tiled<T, NS, MODEL>;
  cudaError_t e = cudaSuccess;
  if (!d->tiled_attr) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return lbx_internal_fail(LBX_ERR_CUDA, cudaGetErrorString(e));
    d->tiled_attr = true;
  }
  TiledPlan& plan = d->tiled[d->tiled_level];
  const int rounds = round_count(pairs, plan.K);
  if (plan.base + rounds + 1 >= (1 << 30)) {
    // restart the counters before they could wrap
    e = cudaMemsetAsync(plan.flags, 0, (size_t)plan.ntiles * sizeof(int), d->stream);
    if (e != cudaSuccess) return lbx_internal_fail(LBX_ERR_CUDA, cudaGetErrorString(e));
    plan.base = 0;
  }
  const bool compact = d->layout == LBX_LAYOUT_COMPACT;
  StepArgs<T> a = A;
  TiledArgs<T> r;
  r.f0 = (T*)(compact ? d->fc : d->f);
  r.f1 = (T*)d->tiled_scratch;
  r.P = compact ? d->P : d->N;
  r.tiles = (const Tile*)plan.tiles;
  r.gidx = plan.gidx;
  r.list = plan.list;
  r.wrd = r.list + plan.nodes;
  r.halo = r.wrd + plan.nodes;
  r.nbrs = plan.nbrs;
  r.flags = plan.flags;
  r.status = d->tiled_status;
  r.base = plan.base;
  r.K = plan.K;
  r.pairs = pairs;
  r.rounds = rounds;
  r.write_mv = write_mv ? 1 : 0;
  void* args[] = {&a, &r};
  e = cudaLaunchCooperativeKernel(fn, plan.ntiles, kTiledThreads, args, smem, d->stream);
  if (e != cudaSuccess) return lbx_internal_fail(LBX_ERR_CUDA, cudaGetErrorString(e));
  plan.base += rounds;
  d->launches++;
  return LBX_OK;
}

template <typename T, int NS>
lbx_status run_ns(lbx_domain* d, const StepArgs<T>& A, int pairs, bool write_mv)
{
  if (d->p.accurate == 0) return launch<T, NS, PLAIN_COMP>(d, A, pairs, write_mv);
  if (d->p.compressible) return launch<T, NS, SHIFTED_COMP>(d, A, pairs, write_mv);
  return launch<T, NS, SHIFTED_INC>(d, A, pairs, write_mv);
}

}  // namespace

size_t lbx_internal_tiled_room(lbx_domain* d)
{
  if (d->fluid == 0 || d->host_solids.empty() || multiprocessors(d) == 0) return 0;
  if (d->real_size == 8) return d->p.nsubs == 2 ? room<double, 2>(d) : room<double, 1>(d);
  return d->p.nsubs == 2 ? room<float, 2>(d) : room<float, 1>(d);
}

lbx_status lbx_internal_tiled_plan(lbx_domain* d, bool* yes)
{
  *yes = false;
  if (d->host_solids.empty() || (d->run_mode != LBX_RUN_TILED && !better(d))) return LBX_OK;
  if (lbx_status st = plan_level(d, 0)) return st;
  if (d->tiled[0].state <= 0) return LBX_OK;
  const int n = busy_beside(d, &d->tiled_record);
  if (lbx_status st = choose_level(d, n, &d->tiled_level)) return st;
  *yes = d->tiled_level >= 0;
  return LBX_OK;
}

template <typename T>
lbx_status lbx_internal_tiled_run(lbx_domain* d, const StepArgs<T>& A, int pairs, bool write_mv)
{
  if (pairs < 2 || d->tiled_level < 0 || d->tiled[d->tiled_level].state <= 0)
    return lbx_internal_fail(LBX_ERR_INVALID, "tiled run without a plan or two pairs");
  return d->p.nsubs == 2 ? run_ns<T, 2>(d, A, pairs, write_mv) : run_ns<T, 1>(d, A, pairs, write_mv);
}

template lbx_status lbx_internal_tiled_run<float>(lbx_domain*, const StepArgs<float>&, int, bool);
template lbx_status lbx_internal_tiled_run<double>(lbx_domain*, const StepArgs<double>&, int, bool);

void lbx_internal_tiled_free(lbx_domain* d)
{
  if (d->tiled_listed) {
    std::lock_guard<std::mutex> lock(g_mu);
    g_listed.erase(std::find(g_listed.begin(), g_listed.end(), d));
    d->tiled_listed = false;
  }
  if (d->tiled_done) cudaEventDestroy(d->tiled_done);
  d->tiled_done = nullptr;
  for (TiledPlan& plan : d->tiled) {
    cudaFree(plan.own);
    plan = TiledPlan();
  }
  cudaFree(d->tiled_own);
  d->tiled_own = d->tiled_scratch = d->tiled_tables = nullptr;
  d->tiled_status = nullptr;
}

lbx_status lbx_internal_tiled_status(lbx_domain* d)
{
  if (!d->tiled_status) return LBX_OK;
  int st = 0;
  cudaError_t e = cudaMemcpy(&st, d->tiled_status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return lbx_internal_fail(LBX_ERR_CUDA, cudaGetErrorString(e));
  if (st == 0) return LBX_OK;
  cudaMemset(d->tiled_status, 0, sizeof(int));
  for (TiledPlan& plan : d->tiled) {
    if (plan.state <= 0) continue;
    cudaMemset(plan.flags, 0, (size_t)plan.ntiles * sizeof(int));
    plan.base = 0;
  }
  return lbx_internal_fail(LBX_ERR_CUDA, "tiled run: a block's wait for its neighbours ran out");
}
