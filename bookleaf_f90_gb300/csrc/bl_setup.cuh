// bl_setup.cuh -- the device half of bl_init: the connectivity's range
// checks and its conversion to 0-based indices, and the node -> corner
// tables of the nodal gathers.
//
// The host uploads the connectivity as the caller holds it (1-based,
// four entries per element); k_check_pack checks every range and converts
// in place, raising error bits that the host reads before anything indexes
// with the tables.  The node -> corner tables are a counting sort by node
// of a corner sequence: counts (atomics), an exclusive scan of the counts
// (the node offsets), a fill through per-node cursors (atomics, so the
// order within a node is arbitrary), then per node a sort of its corners
// by their position in the sequence, which makes the tables those of a
// stable sort: every node's corners in sequence order, the summation order
// of the reference's gathers.  Integer work only: the result does not
// depend on the order in which the atomics land.
#pragma once
#include <cuda_runtime.h>

namespace bl {
namespace setup {

// error bits, reported by bl_init in this order of precedence
enum : int { kBadConn = 1, kBadRegSort = 2, kBadPerm = 4, kBadMat = 8 };

constexpr int kThreads = 256;                     // every set-up kernel
constexpr int kScanV = 16;                        // scan values per thread
constexpr int kScanTile = kThreads * kScanV;      // scan values per block

inline int blocks_for(long n, int per) { return (int)((n + per - 1) / per); }

__device__ __forceinline__ bool in1(int v, int hi) { return (unsigned)(v - 1) < (unsigned)hi; }

// Element i: nodes nd and neighbours ee (1-based on entry, in place),
// neighbour faces fc4 (1-based, packed one byte per side into fc), region
// rg (in place), sort position srt (in place; seen[] counts each position
// to check that ielsort1 is a permutation), material mt (checked only:
// <= 0 marks a mixed cell).
__global__ void __launch_bounds__(kThreads)
    k_check_pack(int4* __restrict__ nd, int4* __restrict__ ee, const int4* __restrict__ fc4,
                 int* __restrict__ fc, int* __restrict__ rg, int* __restrict__ srt,
                 const int* __restrict__ mt, int* __restrict__ seen, int nel, int nnd,
                 int nreg, int nmat, int* __restrict__ bad) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  int b = 0;
  if (i < nel) {
    const int4 n = nd[i], e = ee[i], f = fc4[i];
    if (!(in1(n.x, nnd) && in1(n.y, nnd) && in1(n.z, nnd) && in1(n.w, nnd) && in1(e.x, nel) &&
          in1(e.y, nel) && in1(e.z, nel) && in1(e.w, nel) && in1(f.x, 4) && in1(f.y, 4) &&
          in1(f.z, 4) && in1(f.w, 4)))
      b |= kBadConn;
    const int r = rg[i], s = srt[i];
    if (!in1(r, nreg)) b |= kBadRegSort;
    if (!in1(s, nel)) {
      b |= kBadRegSort;
    } else if (atomicAdd(seen + (s - 1), 1) != 0) {
      b |= kBadPerm;
    }
    if (mt[i] > nmat) b |= kBadMat;
    nd[i] = make_int4(n.x - 1, n.y - 1, n.z - 1, n.w - 1);
    ee[i] = make_int4(e.x - 1, e.y - 1, e.z - 1, e.w - 1);
    fc[i] = (f.x - 1) | ((f.y - 1) << 8) | ((f.z - 1) << 16) | ((f.w - 1) << 24);
    rg[i] = r - 1;
    srt[i] = s - 1;
  }
  b = __reduce_or_sync(0xffffffffu, b);
  if (b && (threadIdx.x & 31) == 0) atomicOr(bad, b);
}

// corners per node (the same for every corner sequence of one mesh)
__global__ void __launch_bounds__(kThreads)
    k_count(const int4* __restrict__ nd, int nel, int nnd, int* __restrict__ cnt) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= nel) return;
  const int4 n = nd[i];
  const int c[4] = {n.x, n.y, n.z, n.w};
  for (int j = 0; j < 4; j++)
    if ((unsigned)c[j] < (unsigned)nnd) atomicAdd(cnt + c[j], 1);
}

// exclusive prefix of one value per thread over the block; *total = the
// block's sum
__device__ __forceinline__ int block_exclusive(int v, int* total) {
  __shared__ int ws[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = lane < kThreads / 32 ? ws[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < kThreads / 32) ws[lane] = s;
  }
  __syncthreads();
  const int before = (w ? ws[w - 1] : 0) + x - v;
  *total = ws[kThreads / 32 - 1];
  __syncthreads();
  return before;
}

// scan, pass 1: each block's sum of its tile of kScanTile values
__global__ void __launch_bounds__(kThreads)
    k_scan_tiles(const int* __restrict__ in, int n, int* __restrict__ bsum) {
  const long base = (long)blockIdx.x * kScanTile + (long)threadIdx.x * kScanV;
  int s = 0;
  for (int k = 0; k < kScanV; k++)
    if (base + k < n) s += in[base + k];
  int total;
  block_exclusive(s, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// scan, pass 2 (one block): the tiles' sums to their exclusive prefixes
__global__ void __launch_bounds__(kThreads) k_scan_sums(int* __restrict__ bsum, int nb) {
  int carry = 0;
  for (int c0 = 0; c0 < nb; c0 += kThreads) {
    const int i = c0 + threadIdx.x;
    const int v = i < nb ? bsum[i] : 0;
    int total;
    const int before = block_exclusive(v, &total);
    if (i < nb) bsum[i] = carry + before;
    carry += total;
  }
}

// scan, pass 3: off[i] = sum of cnt[0..i), off[n] = the total; cnt[i]
// becomes off[i] (the fill's cursor)
__global__ void __launch_bounds__(kThreads)
    k_scan_apply(int* __restrict__ cnt, int n, const int* __restrict__ bsum,
                 int* __restrict__ off) {
  const long base = (long)blockIdx.x * kScanTile + (long)threadIdx.x * kScanV;
  int v[kScanV];
  int s = 0;
  for (int k = 0; k < kScanV; k++) {
    v[k] = base + k < n ? cnt[base + k] : 0;
    s += v[k];
  }
  int total;
  int p = bsum[blockIdx.x] + block_exclusive(s, &total);
  for (int k = 0; k < kScanV; k++) {
    if (base + k < n) {
      off[base + k] = p;
      cnt[base + k] = p;
    }
    p += v[k];
  }
  if (base <= n - 1 && n - 1 < base + kScanV) off[n] = p;
}

// the cursor reset for a second corner sequence over the same offsets
__global__ void __launch_bounds__(kThreads)
    k_copy(const int* __restrict__ off, int n, int* __restrict__ cur) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i < n) cur[i] = off[i];
}

// Fill, corner-major sequence: corner j of the elements in ielsort1 order
// (position k of the sort holds element srt[k]), sequence number
// j*nel + k.  Element-major sequence (srt null): corner j of element i in
// natural order, sequence number 4*i + j.
__global__ void __launch_bounds__(kThreads)
    k_fill(const int4* __restrict__ nd, const int* __restrict__ srt, int nel, int nnd,
           int* __restrict__ cur, int* __restrict__ key) {
  const int k = blockIdx.x * kThreads + threadIdx.x;
  if (k >= nel) return;
  const int i = srt ? srt[k] : k;
  if ((unsigned)i >= (unsigned)nel) return;
  const int4 n = nd[i];
  const int c[4] = {n.x, n.y, n.z, n.w};
  for (int j = 0; j < 4; j++) {
    if ((unsigned)c[j] >= (unsigned)nnd) continue;
    const int pos = atomicAdd(cur + c[j], 1);
    key[pos] = srt ? j * nel + k : 4 * k + j;
  }
}

// Per node: its corners sorted by sequence number (insertion sort: a
// node has a handful of corners), then each sequence number replaced by
// its corner's entry 4*element + corner.
__global__ void __launch_bounds__(kThreads)
    k_sort(const int* __restrict__ off, const int* __restrict__ srt, int nel, int nnd,
           int* __restrict__ key) {
  const int n = blockIdx.x * kThreads + threadIdx.x;
  if (n >= nnd) return;
  const int b = off[n], e = off[n + 1];
  for (int a = b + 1; a < e; a++) {
    const int v = key[a];
    int c = a - 1;
    while (c >= b && key[c] > v) {
      key[c + 1] = key[c];
      c--;
    }
    key[c + 1] = v;
  }
  if (srt)
    for (int a = b; a < e; a++) {
      const int q = key[a];
      key[a] = 4 * srt[q % nel] + q / nel;
    }
}

// ---------------------------------------------------------------- edges
//
// The edge viscosity's limiter of a face compares the face with the two
// faces that continue it across the element's neighbouring sides
// (hydro_kn_edgeviscosity.f90:117-183).  On most meshes the two elements
// that share a face see the same continuing faces, so its limiter, edge
// coefficient and lengths are the same from both sides; they are then
// computed once, in a slot of that edge.  A face 0 or 3 always has a slot
// of its own (nel + nel); a face 1 or 2 uses the slot of the face across it
// when that is a face 0 or 3 with the same nodes, the same two elements and
// the same two continuing faces, whichever way round, and otherwise gets an
// extra slot.  Any mesh the range checks accept is covered: a face whose
// two sides disagree simply has two slots.
//
// The slots of the faces 0 run along the direction that crosses faces 1 and
// 3 where the mesh's numbering has a constant stride S that way (the first
// element's neighbour across face 1, if S divides the mesh): slot
// j * (n / S) + i for element i * S + j.  The faces 3 run along the
// element numbers.  In both, an edge and the one that continues it then
// take adjacent slots on meshes numbered along mesh lines, which k_edge
// shares between adjacent threads; where they do not, the table holds the
// continuing face's nodes instead.
enum : int { kEndWall = -1, kEndMirror = -2, kEndAdjacent = -3 };

__device__ __forceinline__ int at4(const int4& v, int j) {
  return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
}
__device__ __forceinline__ int face_byte(int packed, int j) { return (packed >> (8 * j)) & 3; }

// Marks (bit 0x80 << 8 f) the faces f = 1, 2 whose nodes the element across
// holds as its face 0 or 3, the other way round: the volume such a face sweeps
// is exactly the negative of the one across, whichever way the connectivity
// leads back.
__global__ void __launch_bounds__(kThreads)
    k_swept_faces(const int4* __restrict__ nd, const int4* __restrict__ ee, int* __restrict__ fc,
                  int nel) {
  const int e = blockIdx.x * kThreads + threadIdx.x;
  if (e >= nel) return;
  const int4 n = nd[e], nb = ee[e];
  int v = fc[e];
  for (int f = 1; f <= 2; f++) {
    const int g = face_byte(v, f);
    const int4 m = nd[at4(nb, f)];
    if ((g == 0 || g == 3) && at4(m, g) == at4(n, f + 1) && at4(m, (g + 1) & 3) == at4(n, f))
      v |= 0x80 << (8 * f);
  }
  fc[e] = v;
}

// the nodes of the two faces that continue face f of element e, or the
// boundary rule's ratio there (kEndWall: 0, kEndMirror: 1) in both entries
struct EdgeEnds {
  int p1, q1, p2, q2;
};
__device__ __forceinline__ EdgeEnds edge_ends(const int4* nd, const int4* ee, const int* fc,
                                              const int* it, int e, int f) {
  const int4 n = nd[e], nb = ee[e];
  const int fcp = fc[e];
  const int s = (f & 1) ? 0 : 1;            // the neighbours across sides s and s + 2
  const bool first = f == 3 || f == 0;
  const int in1 = at4(nb, s), in2 = at4(nb, s + 2);
  const int f1 = face_byte(fcp, s), f2 = face_byte(fcp, s + 2);
  EdgeEnds r;
  if (in1 == e) {
    const bool m = it[at4(n, s)] < 0 && it[at4(n, (s + 1) & 3)] < 0 && in2 != e;
    r.p1 = r.q1 = m ? kEndMirror : kEndWall;
  } else {
    const int4 m = nd[in1];
    const int k = (f1 + (first ? 1 : 3)) & 3;
    r.p1 = at4(m, k);
    r.q1 = at4(m, (k + 1) & 3);
  }
  if (in2 == e) {
    const bool m = it[at4(n, s + 2)] < 0 && it[at4(n, (s + 3) & 3)] < 0 && in1 != e;
    r.p2 = r.q2 = m ? kEndMirror : kEndWall;
  } else {
    const int4 m = nd[in2];
    const int k = (f2 + (first ? 3 : 1)) & 3;
    r.p2 = at4(m, k);
    r.q2 = at4(m, (k + 1) & 3);
  }
  return r;
}

// the mesh of element or slot i: the last one that begins at or before it
__device__ __forceinline__ int mesh_at(const int* moff, int nmesh, int i) {
  int lo = 0, hi = nmesh - 1;
  while (lo < hi) {
    const int m = (lo + hi + 1) >> 1;
    if (moff[m] <= i) lo = m;
    else hi = m - 1;
  }
  return lo;
}
// the slots of a mesh's faces 0: n elements from off, stride S (1: in order)
struct SlotMap {
  int off, n, S;
};
__device__ __forceinline__ SlotMap slot_map(const int* moff, int nmesh, const int4* ee, int i) {
  const int m = mesh_at(moff, nmesh, i);
  SlotMap r;
  r.off = moff[m];
  r.n = moff[m + 1] - r.off;
  r.S = ee[r.off].y - r.off;
  if (r.S < 2 || r.S >= r.n || r.n % r.S != 0) r.S = 1;
  return r;
}
__device__ __forceinline__ int slot_of(const SlotMap& r, int e) {
  const int l = e - r.off;
  return r.S == 1 ? e : r.off + (l % r.S) * (r.n / r.S) + l / r.S;
}
__device__ __forceinline__ int element_of(const SlotMap& r, int slot) {
  const int p = slot - r.off, R = r.n / r.S;
  return r.S == 1 ? slot : r.off + (p % R) * r.S + p / R;
}

// Each element's four slots; the faces that need an extra one go to exl
// (4 * element + face) in any order, counted in *nex.
__global__ void __launch_bounds__(kThreads)
    k_edge_refs(const int4* __restrict__ nd, const int4* __restrict__ ee,
                const int* __restrict__ fc, const int* __restrict__ it, int nel,
                const int* __restrict__ moff, int nmesh, uint4* __restrict__ er,
                int* __restrict__ exl, int* __restrict__ nex) {
  const int e = blockIdx.x * kThreads + threadIdx.x;
  if (e >= nel) return;
  const SlotMap sm = slot_map(moff, nmesh, ee, e);
  unsigned ref[4];
  ref[0] = 2u * (unsigned)slot_of(sm, e);
  ref[3] = 2u * ((unsigned)nel + (unsigned)e);
  const int4 n = nd[e], nb = ee[e];
  const int fcp = fc[e];
  for (int f = 1; f <= 2; f++) {
    const int w = at4(nb, f), g = face_byte(fcp, f);
    const int a = at4(n, f), b = at4(n, f + 1);
    bool same = false, rev = false;
    if (w != e && (g == 0 || g == 3) && at4(ee[w], g) == e && face_byte(fc[w], g) == f) {
      const int4 m = nd[w];
      const int c = at4(m, g), d = at4(m, (g + 1) & 3);
      rev = a == d && b == c;
      if (rev || (a == c && b == d)) {
        const EdgeEnds x = edge_ends(nd, ee, fc, it, e, f);
        EdgeEnds y = edge_ends(nd, ee, fc, it, w, g);
        if (rev) {
          int t = y.p1;
          y.p1 = y.q1;
          y.q1 = t;
          t = y.p2;
          y.p2 = y.q2;
          y.q2 = t;
        }
        same = (x.p1 == y.p1 && x.q1 == y.q1 && x.p2 == y.p2 && x.q2 == y.q2) ||
               (x.p1 == y.p2 && x.q1 == y.q2 && x.p2 == y.p1 && x.q2 == y.q1);
      }
    }
    if (same) {
      const unsigned slot = g == 3 ? (unsigned)nel + (unsigned)w
                                   : (unsigned)slot_of(slot_map(moff, nmesh, ee, w), w);
      ref[f] = 2u * slot + (rev ? 1u : 0u);
    } else {
      const int k = atomicAdd(nex, 1);
      exl[k] = 4 * e + f;
      ref[f] = 2u * (2u * (unsigned)nel + (unsigned)k);
    }
  }
  er[e] = make_uint4(ref[0], ref[1], ref[2], ref[3]);
}

// The slots' tables: en = (node a, node b, element, element across), eq =
// the continuing faces' nodes (p1, q1, p2, q2), with kEndAdjacent in p1
// where the first is the edge of the slot before and in p2 where the second
// is that of the slot after (the two ends change places if that makes them
// so: the limiter is symmetric in them).
__global__ void __launch_bounds__(kThreads)
    k_edge_slots(const int4* __restrict__ nd, const int4* __restrict__ ee,
                 const int* __restrict__ fc, const int* __restrict__ it, int nel,
                 const int* __restrict__ moff, int nmesh, const int* __restrict__ exl, int nslot,
                 int4* __restrict__ en, int4* __restrict__ eq) {
  const int slot = blockIdx.x * kThreads + threadIdx.x;
  if (slot >= nslot) return;
  int e, f, ep = -1, ex = -1;  // the elements of the slots before and after
  if (slot < 2 * nel) {
    f = slot < nel ? 0 : 3;
    const int k = slot < nel ? slot : slot - nel;
    const SlotMap sm = slot_map(moff, nmesh, ee, k);
    e = f == 0 ? element_of(sm, k) : k;
    if (k > sm.off) ep = f == 0 ? element_of(sm, k - 1) : k - 1;
    if (k + 1 < sm.off + sm.n) ex = f == 0 ? element_of(sm, k + 1) : k + 1;
  } else {
    const int v = exl[slot - 2 * nel];
    e = v >> 2;
    f = v & 3;
  }
  const int4 n = nd[e];
  EdgeEnds r = edge_ends(nd, ee, fc, it, e, f);
  auto is_edge = [&](int el, int p, int q) {
    if (el < 0) return false;
    const int4 m = nd[el];
    return p == at4(m, f) && q == at4(m, (f + 1) & 3);
  };
  bool before1 = is_edge(ep, r.p1, r.q1), before2 = is_edge(ep, r.p2, r.q2);
  bool after1 = is_edge(ex, r.p1, r.q1), after2 = is_edge(ex, r.p2, r.q2);
  if (!before1 && !after2 && (before2 || after1)) {
    const EdgeEnds o = r;
    r.p1 = o.p2;
    r.q1 = o.q2;
    r.p2 = o.p1;
    r.q2 = o.q1;
    before1 = before2;
    after2 = after1;
  }
  if (before1) r.p1 = kEndAdjacent;
  if (after2) r.p2 = kEndAdjacent;
  en[slot] = make_int4(at4(n, f), at4(n, (f + 1) & 3), e, at4(ee[e], f));
  eq[slot] = make_int4(r.p1, r.q1, r.p2, r.q2);
}

}  // namespace setup
}  // namespace bl
