// Tiles of the fused FP32 stage (swm_stage32.cu): the layout's cells cut into
// contiguous runs, each with the cells, edges and triangles around it that one
// block needs to step it.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <new>

#include <omp.h>

#include "swm_layout.h"

namespace imodel {
namespace {

// A set of entities by device index, emptied by a new tag.  The memory is
// mapped zeroed and touched only around the tiles that a thread works on.
class Marks {
 public:
  explicit Marks(size_t n)
      : v_(static_cast<int32_t *>(std::calloc(n ? n : 1, sizeof(int32_t)))) {}
  ~Marks() { std::free(v_); }
  Marks(const Marks &) = delete;
  bool valid() const { return v_ != nullptr; }
  void start(int tag) { tag_ = tag + 1; }
  bool has(int32_t k) const { return v_[k] == tag_; }
  // true when k was not there
  bool add(int32_t k) {
    if (has(k)) return false;
    v_[k] = tag_;
    return true;
  }

 private:
  int32_t *v_;
  int32_t tag_ = 0;
};

// cells whose flux terms a tile of the cells [c0, c1) needs: its own and the
// higher-numbered neighbours; the last c1 <= end with at most cap of them
int tile_end(const Layout &L, int c0, int end, int cap, Marks &ring) {
  const size_t NV = L.nv;
  ring.start(c0);
  int above = 0;  // ring cells >= c1
  int c1 = c0;
  for (; c1 < end; ++c1) {
    const int was = ring.has(c1) ? 1 : 0;  // moves from the ring into the tile
    int fresh[kMaxNb], n = 0;
    for (int j = 0; j < L.c_nnb[c1]; ++j) {
      const int nb = L.c_nb[j * NV + c1];
      if (nb > c1 && !ring.has(nb)) fresh[n++] = nb;
    }
    if ((c1 + 1 - c0) + above - was + n > cap) break;
    above += n - was;
    for (int k = 0; k < n; ++k) ring.add(fresh[k]);
  }
  return c1;
}

}  // namespace

// One kind of a tile's entities, in device numbering; more than a tile may have
// are counted only
struct TileList {
  int n = 0;
  int32_t v[1024];
  void add(int32_t k) {
    if (n < 1024) v[n] = k;
    ++n;
  }
};

bool build_tiles(const Layout &L, int cap, TileLayout &T) {
  const size_t NV = L.nv, NE = L.ne, NT = L.nt;
  T = TileLayout();
  T.cap = cap;
  // no exception leaves a parallel region: out of memory is thrown after it
  bool oom = false;
  // edge e belongs to the tile of its lower cell: edges are numbered by it, and
  // first[c] is the first with a lower cell of c or above
  auto lower = [&](size_t e) { return std::min(L.e_v[e], L.e_v[NE + e]); };
  bool ok = true;
#pragma omp parallel for schedule(static) reduction(&& : ok)
  for (size_t e = 1; e < NE; ++e) ok = ok && lower(e) >= lower(e - 1);
  if (!ok || NE == 0) return false;
  HVec<int32_t> first;
  first.resize(NV + 1);
#pragma omp parallel for schedule(static)
  for (size_t e = 0; e <= NE; ++e) {
    const int c1 = e < NE ? lower(e) : static_cast<int>(NV);
    for (int c = e > 0 ? lower(e - 1) + 1 : 0; c <= c1; ++c) first[c] = static_cast<int32_t>(e);
  }
  // cut: fixed segments of the curve, each cut on its own (the result does
  // not depend on the thread count)
  const int kSeg = 16384, nseg = static_cast<int>((NV + kSeg - 1) / kSeg);
  std::vector<std::vector<int32_t>> cuts(nseg);
#pragma omp parallel reduction(&& : ok) reduction(|| : oom)
  {
    Marks ring(NV);
    oom = !ring.valid();
#pragma omp for schedule(static)
    for (int s = 0; s < nseg; ++s) {
      if (oom) continue;
      try {
        const int end = static_cast<int>(std::min(NV, static_cast<size_t>(s + 1) * kSeg));
        for (int c = s * kSeg; c < end;) {
          cuts[s].push_back(c);
          const int c1 = tile_end(L, c, end, cap, ring);
          if (c1 == c) {
            ok = false;
            break;
          }
          c = c1;
        }
      } catch (const std::bad_alloc &) {
        oom = true;
      }
    }
  }
  if (oom) throw std::bad_alloc();
  if (!ok) return false;
  std::vector<int32_t> start;
  for (const auto &c : cuts) start.insert(start.end(), c.begin(), c.end());
  const int nt = static_cast<int>(start.size());
  start.push_back(L.nv);
  T.ntiles = nt;
  T.head.resize(static_cast<size_t>(nt));
  // the lists of every tile, one thread's behind one another, then their places
  std::vector<HVec<int32_t>> lists(omp_get_max_threads());
  std::vector<int32_t> owner(nt);
#pragma omp parallel reduction(&& : ok) reduction(|| : oom)
  {
    Marks cells(NV), edges(NE), tris(NT);
    oom = !cells.valid() || !edges.valid() || !tris.valid();
    TileList z, hx, ux, tri;
    HVec<int32_t> &mine = lists[omp_get_thread_num()];
#pragma omp for schedule(static)
    for (int b = 0; b < nt; ++b) {
      if (oom) continue;
      try {
        const int c0 = start[b], c1 = start[b + 1], e0 = first[c0], e1 = first[c1];
        z.n = hx.n = ux.n = tri.n = 0;
        cells.start(b);
        edges.start(b);
        tris.start(b);
        // a tile's own cells and edges are told by their range
        auto other_cell = [&](int c) { return (c < c0 || c >= c1) && cells.add(c); };
        auto other_edge = [&](int e) { return (e < e0 || e >= e1) && edges.add(e); };
        for (int e = e0; e < e1; ++e) {
          const int hi = std::max(L.e_v[e], L.e_v[NE + e]);
          if (other_cell(hi)) z.add(hi);
        }
        auto around = [&](int c) {
          for (int j = 0; j < L.c_nnb[c]; ++j) {
            const int nb = L.c_nb[j * NV + c], t = L.c_tr[j * NV + c], e = L.c_ed[j * NV + c];
            if (other_cell(nb)) hx.add(nb);
            if (tris.add(t)) tri.add(t);
            if (other_edge(e)) ux.add(e);
          }
        };
        // (the cut bounds own and ring cells by cap; checked before the lists
        // are read)
        if (c1 - c0 + z.n > cap || z.n > 1024) {
          ok = false;
          continue;
        }
        for (int c = c0; c < c1; ++c) around(c);
        for (int k = 0; k < z.n; ++k) around(z.v[k]);
        for (int k = 0; k < std::min(tri.n, 1024); ++k)
          for (int s = 0; s < 3; ++s) {
            const int e = L.t_ed[s * NT + tri.v[k]], v = L.t_v[s * NT + tri.v[k]];
            if (other_edge(e)) ux.add(e);
            if (other_cell(v)) hx.add(v);
          }
        const int nz = c1 - c0 + z.n, nh = nz + hx.n, nu = e1 - e0 + ux.n, ntr = tri.n;
        if (nh > 1024 || nu > 1024 || ntr > 1024) {
          ok = false;
          continue;
        }
        // the flux terms must fit where the triangles' records were
        if (6 * nz > 8 * ntr) ok = false;
        TileHead &H = T.head[b];
        H = TileHead{};
        H.c0 = c0;
        H.nc = c1 - c0;
        H.nz = nz;
        H.nh = nh;
        H.e0 = e0;
        H.ne = e1 - e0;
        H.nu = nu;
        H.nt = ntr;
        auto up = [](int n) { return (n + 15) & ~15; };
        H.ux = up(4 * (nh - H.nc));
        H.slot = H.ux + up(4 * (nu - H.ne));
        H.triA = H.slot + 16 * kMaxNb * nz;
        H.triB = H.triA + 16 * ntr;
        H.triC = H.triB + 16 * ntr;
        H.edge = H.triC + up(4 * ntr);
        H.meta = H.edge + up(8 * H.ne);
        H.bt = H.meta + up(4 * nz);
        H.inva = H.bt + up(4 * nz);
        H.bytes = H.inva + up(4 * H.nc);
        if (mine.size() > INT32_MAX - 4096) {
          ok = false;
          continue;
        }
        H.lists = static_cast<int32_t>(mine.size());
        owner[b] = omp_get_thread_num();
        for (const TileList *q : {&z, &hx, &ux, &tri}) mine.insert(mine.end(), q->v, q->v + q->n);
      } catch (const std::bad_alloc &) {
        oom = true;
      }
    }
  }
  if (oom) throw std::bad_alloc();
  if (!ok) return false;
  std::vector<size_t> base(lists.size() + 1, 0);
  for (size_t k = 0; k < lists.size(); ++k) base[k + 1] = base[k] + lists[k].size();
  if (base.back() > INT32_MAX) return false;
  size_t bytes = 0;
  for (int b = 0; b < nt; ++b) {
    TileHead &H = T.head[b];
    if (bytes / 16 > INT32_MAX) return false;
    H.block = static_cast<int32_t>(bytes / 16);
    H.lists += static_cast<int32_t>(base[owner[b]]);
    bytes += H.bytes;
    T.max_h = std::max(T.max_h, H.nh);
    T.max_u = std::max(T.max_u, H.nu);
    T.max_t = std::max(T.max_t, H.nt);
    T.max_bytes = std::max(T.max_bytes, H.bytes);
  }
  T.data_bytes = bytes;
  T.lists.resize(base.back());
#pragma omp parallel for schedule(static, 1)
  for (int k = 0; k < static_cast<int>(lists.size()); ++k)
    std::copy(lists[k].begin(), lists[k].end(), T.lists.begin() + base[k]);
  return true;
}

}  // namespace imodel
