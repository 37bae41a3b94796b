// Tiles of the fused FP32 stage (swm_stage32.cu): the layout's cells cut into
// contiguous runs, each with the cells, edges and triangles around it that one
// block needs to step it.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <new>

#include "swm_layout.h"

namespace imodel {
namespace {

// Local numbers of one tile's entities, by device index: a value per index,
// forgotten when the tile changes.  The memory is mapped zeroed and touched
// only around the tiles that a thread works on.
class LocalNumbers {
 public:
  explicit LocalNumbers(size_t n)
      : v_(static_cast<uint64_t *>(std::calloc(n ? n : 1, sizeof(uint64_t)))) {}
  ~LocalNumbers() { std::free(v_); }
  LocalNumbers(const LocalNumbers &) = delete;
  bool valid() const { return v_ != nullptr; }
  void start(int tile) { tag_ = static_cast<uint64_t>(tile) + 1; }
  bool has(int32_t k) const { return v_[k] >> 32 == tag_; }
  void set(int32_t k, uint32_t local) { v_[k] = tag_ << 32 | local; }
  // true when k was not there
  bool add(int32_t k) {
    if (has(k)) return false;
    set(k, 0);
    return true;
  }
  uint32_t operator[](int32_t k) const { return static_cast<uint32_t>(v_[k]); }

 private:
  uint64_t *v_;
  uint64_t tag_ = 0;
};

// cells whose flux terms a tile of the cells [c0, c1) needs: its own and the
// higher-numbered neighbours; the last c1 <= end with at most cap of them
int tile_end(const Layout &L, int c0, int end, int cap, LocalNumbers &ring) {
  const size_t NV = L.nv;
  ring.start(c0);
  int above = 0;  // ring cells >= c1
  int c1 = c0;
  for (; c1 < end; ++c1) {
    const int was = ring.has(c1) ? 1 : 0;  // moves from the ring into the tile
    int fresh = 0;
    for (int j = 0; j < L.c_nnb[c1]; ++j) {
      const int nb = L.c_nb[j * NV + c1];
      if (nb > c1 && !ring.has(nb)) ++fresh;
    }
    if ((c1 + 1 - c0) + above - was + fresh > cap) break;
    above += fresh - was;
    for (int j = 0; j < L.c_nnb[c1]; ++j) {
      const int nb = L.c_nb[j * NV + c1];
      if (nb > c1) ring.add(nb);
    }
  }
  return c1;
}

}  // namespace

// One tile's lists, in device numbering
struct TileLists {
  std::vector<int32_t> z, hx, ux, tri;  // ring cells, other depths, other edges, triangles
};

bool build_tiles(const Layout &L, int cap, TileLayout &T) {
  const size_t NV = L.nv, NE = L.ne, NT = L.nt;
  T = TileLayout();
  T.cap = cap;
  // no exception leaves a parallel region: out of memory is thrown after it
  bool oom = false;
  // edge e belongs to the tile of its lower cell: edges are numbered by it
  std::vector<int32_t> first(NV + 1, 0);
  for (size_t e = 0; e < NE; ++e) {
    const int lo = std::min(L.e_v[e], L.e_v[NE + e]);
    if (e > 0 && lo < std::min(L.e_v[e - 1], L.e_v[NE + e - 1])) return false;
    first[lo + 1] = static_cast<int32_t>(e + 1);
  }
  for (size_t i = 0; i < NV; ++i) first[i + 1] = std::max(first[i + 1], first[i]);
  // cut: fixed segments of the curve, each cut on its own (the result does
  // not depend on the thread count)
  const int kSeg = 16384, nseg = static_cast<int>((NV + kSeg - 1) / kSeg);
  std::vector<std::vector<int32_t>> cuts(nseg);
  bool ok = true;
#pragma omp parallel reduction(&& : ok) reduction(|| : oom)
  {
    LocalNumbers ring(NV);
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
  // pass 1: the lists of every tile; pass 2: their places; pass 3: the records
  std::vector<TileLists> lists(nt);
#pragma omp parallel reduction(&& : ok) reduction(|| : oom)
  {
    LocalNumbers cells(NV), edges(NE), tris(NT);
    oom = !cells.valid() || !edges.valid() || !tris.valid();
#pragma omp for schedule(static)
    for (int b = 0; b < nt; ++b) {
      if (oom) continue;
      try {
        const int c0 = start[b], c1 = start[b + 1], e0 = first[c0], e1 = first[c1];
        TileLists &Q = lists[b];
        cells.start(b);
        edges.start(b);
        tris.start(b);
        for (int c = c0; c < c1; ++c) cells.add(c);
        for (int e = e0; e < e1; ++e) {
          edges.add(e);
          const int hi = std::max(L.e_v[e], L.e_v[NE + e]);
          if (cells.add(hi)) Q.z.push_back(hi);
        }
        std::sort(Q.z.begin(), Q.z.end());
        auto around = [&](int c) {
          for (int j = 0; j < L.c_nnb[c]; ++j) {
            const int nb = L.c_nb[j * NV + c], t = L.c_tr[j * NV + c], e = L.c_ed[j * NV + c];
            if (cells.add(nb)) Q.hx.push_back(nb);
            if (tris.add(t)) Q.tri.push_back(t);
            if (edges.add(e)) Q.ux.push_back(e);
          }
        };
        for (int c = c0; c < c1; ++c) around(c);
        for (int c : Q.z) around(c);
        for (int t : Q.tri)
          for (int s = 0; s < 3; ++s) {
            const int e = L.t_ed[s * NT + t], v = L.t_v[s * NT + t];
            if (edges.add(e)) Q.ux.push_back(e);
            if (cells.add(v)) Q.hx.push_back(v);
          }
        std::sort(Q.hx.begin(), Q.hx.end());
        std::sort(Q.ux.begin(), Q.ux.end());
        std::sort(Q.tri.begin(), Q.tri.end());
        const int nz = c1 - c0 + static_cast<int>(Q.z.size());
        const int nh = nz + static_cast<int>(Q.hx.size());
        const int nu = e1 - e0 + static_cast<int>(Q.ux.size());
        const int ntr = static_cast<int>(Q.tri.size());
        if (nz > cap || nh > 1024 || nu > 1024 || ntr > 1024) ok = false;
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
      } catch (const std::bad_alloc &) {
        oom = true;
      }
    }
  }
  if (oom) throw std::bad_alloc();
  if (!ok) return false;
  size_t bytes = 0;
  for (TileHead &H : T.head) {
    if (bytes / 16 > INT32_MAX) return false;
    H.block = static_cast<int32_t>(bytes / 16);
    bytes += H.bytes;
    T.max_h = std::max(T.max_h, H.nh);
    T.max_u = std::max(T.max_u, H.nu);
    T.max_t = std::max(T.max_t, H.nt);
    T.max_bytes = std::max(T.max_bytes, H.bytes);
  }
  T.data.resize(bytes / 4);
  auto bits = [](float f) {
    uint32_t v;
    std::memcpy(&v, &f, sizeof(v));
    return v;
  };
#pragma omp parallel reduction(|| : oom)
  {
    LocalNumbers cells(NV), edges(NE), tris(NT);
    oom = !cells.valid() || !edges.valid() || !tris.valid();
#pragma omp for schedule(static)
    for (int b = 0; b < nt; ++b) {
      if (oom) continue;
      const TileHead &H = T.head[b];
      const TileLists &Q = lists[b];
      cells.start(b);
      edges.start(b);
      tris.start(b);
      uint32_t *base = T.data.data() + 4 * static_cast<size_t>(H.block);
      std::memset(base, 0, H.bytes);
      auto part = [&](int off) { return base + off / 4; };
      // local numbers: depths own, ring, others; edges own, others
      for (int k = 0; k < H.nc; ++k) cells.set(H.c0 + k, k);
      int n = H.nc;
      for (const std::vector<int32_t> *list : {&Q.z, &Q.hx})
        for (int c : *list) {
          part(0)[n - H.nc] = static_cast<uint32_t>(c);
          cells.set(c, n++);
        }
      for (int k = 0; k < H.ne; ++k) edges.set(H.e0 + k, k);
      n = H.ne;
      for (int e : Q.ux) {
        part(H.ux)[n - H.ne] = static_cast<uint32_t>(e);
        edges.set(e, n++);
      }
      n = 0;
      for (int t : Q.tri) tris.set(t, n++);
      for (int k = 0; k < H.nt; ++k) {
        const int t = Q.tri[k];
        uint32_t *A = part(H.triA) + 4 * k, *B = part(H.triB) + 4 * k;
        uint32_t ie = 0, iv = 0;
        for (int s = 0; s < 3; ++s) {
          ie |= edges[L.t_ed[s * NT + t]] << (10 * s);
          iv |= cells[L.t_v[s * NT + t]] << (10 * s);
          A[s] = bits(L.t_circ32[s * NT + t]);
          B[s] = bits(L.t_kite32[s * NT + t]);
        }
        A[3] = bits(L.t_f32[t]);
        B[3] = ie;
        part(H.triC)[k] = iv;
      }
      for (int z = 0; z < H.nz; ++z) {
        const int c = z < H.nc ? H.c0 + z : Q.z[z - H.nc];
        part(H.meta)[z] = L.c_meta[c];
        part(H.bt)[z] = bits(static_cast<float>(L.c_bt[c]));
        if (z < H.nc) part(H.inva)[z] = bits(L.c_inva32[c]);
        for (int j = 0; j < kMaxNb; ++j) {
          // c_pk: {edge, neighbour, triangle, kite fraction}; c_kd: {KE
          // weight, ttgout d}; unused slots repeat slot 0 with zero weights
          const size_t src = j * NV + c;
          uint32_t *q = part(H.slot) + 4 * (j * H.nz + z);
          q[0] = edges[L.c_pk[4 * src]] | cells[L.c_pk[4 * src + 1]] << 10 |
                 tris[L.c_pk[4 * src + 2]] << 20;
          q[1] = static_cast<uint32_t>(L.c_pk[4 * src + 3]);
          q[2] = bits(L.c_kd[2 * src]);
          q[3] = bits(L.c_kd[2 * src + 1]);
        }
      }
      for (int k = 0; k < H.ne; ++k) {
        const size_t e = H.e0 + k;
        const uint32_t w1 = L.e_vs[e], w2 = L.e_vs[NE + e];
        const uint32_t z1 = cells[static_cast<int32_t>(w1 & 0x0FFFFFFFu)];
        const uint32_t z2 = cells[static_cast<int32_t>(w2 & 0x0FFFFFFFu)];
        uint32_t *q = part(H.edge) + 2 * k;
        q[0] = z1 | (w1 >> 28) << 10 | z2 << 13 | (w2 >> 28) << 23;
        q[1] = bits(L.e_grad32[e]);
      }
    }
  }
  if (oom) throw std::bad_alloc();
  return true;
}

}  // namespace imodel
