// stage_pair.cu -- host side of the paired z-marching stage kernels: TMA
// tensor maps, launch plan (persistent grid, z-chunk length) and dispatch.
// The kernels themselves are in stage_pair_impl.cuh, instantiated by
// pair_*.cu.
#include "once_per_device.h"
#include "stage_pair_impl.cuh"

#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

namespace cgfd {
namespace pair {
namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

// 4-D map {x: nx, y: ny, z: nz, component: nc} over float arrays with the
// given pitches (elements), box {bx, by, 1, bc}
bool make_map(CUtensorMap *m, const void *base, int nx, int ny, int nz, int nc, size_t pitch_y,
              size_t pitch_z, size_t pitch_c, int bx, int by, int bc, int elem = ELEM_F32) {
  auto fn = encode_fn();
  if (!fn || !base) return false;
  const size_t es_b = elem_size(elem);
  cuuint64_t dims[4] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz, (cuuint64_t)nc};
  cuuint64_t strides[3] = {(cuuint64_t)(pitch_y * es_b), (cuuint64_t)(pitch_z * es_b),
                           (cuuint64_t)(pitch_c * es_b)};
  cuuint32_t box[4] = {(cuuint32_t)bx, (cuuint32_t)by, 1, (cuuint32_t)bc};
  cuuint32_t es[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = elem == ELEM_F16    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                 : elem == ELEM_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                     : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = fn(m, dt, 4, (void *)base, dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}
// a map over ncomp arrays of the internal field layout
bool field_map(CUtensorMap *m, const Geom &g, const void *base, int ncomp, int bx, int by,
               int bc, int elem = ELEM_F32) {
  return make_map(m, base, g.px, g.nyi, g.nzi, ncomp, g.px, g.plane, g.fstride, bx, by, bc,
                  elem);
}
// a map over one auxiliary set (9 components) of direction d
bool aux_map(CUtensorMap *m, const Geom &g, int d, const float *base, int bc) {
  if (d == 0)
    return make_map(m, base, g.nxa, g.nyi, g.nzi, g.ncaux, g.nxa, (size_t)g.nxa * g.nyi, g.astride[0],
                    CX, TY, bc);
  if (d == 1)
    return make_map(m, base, g.px, g.nya, g.nzi, g.ncaux, g.px, (size_t)g.px * g.nya, g.astride[1],
                    CX, TY, bc);
  return make_map(m, base, g.px, g.nyi, g.nza, g.ncaux, g.px, g.plane, g.astride[2], CX, TY, bc);
}

}  // namespace
}  // namespace pair

using namespace pair;

bool pair_supported(const Geom &g) {
  // tile boxes start on 16-byte boundaries (XO and i0 multiples of 4, px of 32);
  // the free surface and the two layers below it are distinct planes
  return (XO % 4) == 0 && XO >= 4 && g.px % 32 == 0 && g.nk >= 4;
}

namespace pair {
namespace {

// entry points by storage type (ELEM_*), RK stage kind and launch
const Entry &entry(int elem, int kind, int list) {
#define CGFD_ENTRIES(E)                                  \
  {{entry_##E##0v(), entry_##E##0s(), entry_##E##0l()},  \
   {entry_##E##1v(), entry_##E##1s(), entry_##E##1l()},  \
   {entry_##E##2v(), entry_##E##2s(), entry_##E##2l()}}
  static const Entry e[3][3][NLIST] = {CGFD_ENTRIES(f), CGFD_ENTRIES(h), CGFD_ENTRIES(b)};
#undef CGFD_ENTRIES
  return e[elem][kind][list];
}

// kernel attributes of one storage type on the current device (each call loads
// its kernels, so a process pays for the types and devices it uses only)
bool set_attrs_of(int elem) {
  static OncePerDevice once;
  return once.run(elem, [&] {
    cudaError_t e = cudaSuccess;
    for (int kind = 0; kind < 3; ++kind)
      for (int list = 0; list < NLIST && e == cudaSuccess; ++list)
        e = entry(elem, kind, list).attrs();
    return e;
  });
}

// tensor maps of one model's buffers
bool model_maps(ModelMaps *pl, int *has_aux, const Geom &g, int elem, void *const sets[4],
                const float *media, const float *metric, float *const aux[3]) {
  bool ok = true;
  constexpr int NCV = PartInfo<PART_VEL>::NC, NCS = PartInfo<PART_STR>::NC;
  const int hx = (elem == ELEM_F32) ? Halo<float>::HX : Halo<__half>::HX;
  for (int q = 0; q < 4; ++q) {
    ok = ok && field_map(&pl->haloV[q], g, sets[q], 9, hx, HY, NCV, elem);
    ok = ok && field_map(&pl->haloS[q], g, sets[q], 9, hx, HY, NCS, elem);
    ok = ok && field_map(&pl->ctrV[q], g, sets[q], 9, CX, TY, 3, elem);
    ok = ok && field_map(&pl->ctrT[q], g, sets[q], 9, CX, TY, 6, elem);
  }
  ok = ok && field_map(&pl->coefV, g, media, 3, CX, TY, PartInfo<PART_VEL>::NCOEF);
  ok = ok && field_map(&pl->coefS, g, media, 3, CX, TY, PartInfo<PART_STR>::NCOEF);
  ok = ok && field_map(&pl->met, g, metric, 4, CX, TY, 3);
  for (int d = 0; d < 3; ++d) {
    has_aux[d] = aux[d] != nullptr;
    if (!aux[d]) continue;
    const size_t ss = (size_t)g.ncaux * g.astride[d];
    for (int t = 0; t < 3; ++t) {  // FA, A, tA
      ok = ok && aux_map(&pl->auxV[d][t], g, d, aux[d] + t * ss, 3);
      ok = ok && aux_map(&pl->auxT[d][t], g, d, aux[d] + t * ss, 3);
    }
  }
  return ok;
}

// the maps of one stage (stage input set, RK kind, stage index) for the
// velocity (mv) and stress (ms) parts
// (rebuild: the second stage under tW elision, whose u1 is the stage input)
// (tw_delta: 16-bit storage, tW kept as tW - FW; the final stage reads FW as
// its first register set and the difference as its second)
void stage_maps(const ModelMaps &pl, int rk, int in_set, bool rebuild, bool tw_delta, Maps &mv,
                Maps &ms) {
  const int kind = rk == 0 ? 0 : (rk < 3 ? 1 : 2);
  const bool fw_first = kind != 2 || tw_delta;
  mv.halo = pl.haloV[in_set];
  mv.u0 = fw_first ? pl.ctrV[0] : pl.ctrV[3];
  mv.u1 = rebuild ? pl.ctrV[in_set] : pl.ctrV[3];
  mv.coef = pl.coefV;
  mv.met = pl.met;
  ms.halo = pl.haloS[in_set];
  ms.u0 = fw_first ? pl.ctrT[0] : pl.ctrT[3];
  ms.u1 = rebuild ? pl.ctrT[in_set] : pl.ctrT[3];
  ms.coef = pl.coefS;
  ms.met = pl.met;
  for (int d = 0; d < 3; ++d) {
    // prefetched sets: stage input (FA in the first stage, else A), FA, tA
    const int in = (rk == 0) ? 0 : 1;
    mv.aux[d][0] = pl.auxV[d][in]; mv.aux[d][1] = pl.auxV[d][0]; mv.aux[d][2] = pl.auxV[d][2];
    ms.aux[d][0] = pl.auxT[d][in]; ms.aux[d][1] = pl.auxT[d][0]; ms.aux[d][2] = pl.auxT[d][2];
  }
}

// Tile origins along one axis of n cells with layers of lo and hi cells:
// tiles of `size` cells that start at `first`, tiles inside the layers' inner
// faces marked interior.
struct Tile {
  int at;
  bool interior;
};
// x: origins at multiples of CX from 0, which keeps every tile row of the
// field, media and metric boxes on a 128-byte boundary
std::vector<Tile> x_tiles(const Geom &g) {
  std::vector<Tile> t;
  for (int i = 0; i < g.ni; i += CX)
    t.push_back({i, i >= g.nabs[0] && i + CX <= g.ni - g.nabs[1]});
  return t;
}
// y: the interior tiles start at the low layer's inner face (its own tiles
// lie before them, the first one partly left of the grid when the layer is
// no multiple of TY), so that layers of any width cost no more boundary tiles
// than they fill
std::vector<Tile> y_tiles(const Geom &g) {
  std::vector<Tile> t;
  const int lo = g.nabs[2], nin = (g.nj - lo - g.nabs[3]) / TY;
  for (int j = lo - (lo + TY - 1) / TY * TY; j < g.nj; j += TY)
    t.push_back({j, j >= lo && j < lo + nin * TY});
  return t;
}

// Work items of one or more models, in two lists: lean items (no PML cell, no
// cell outside the grid; `plain` models only) and general ones (part 0, both
// parts' launches walk them).  The bottom PML layer is a z-chunk of
// its own (in general columns when it has >= 8 planes), the rest is cut into
// pieces.  Order: the most expensive first (estimated cost: planes x sum over
// the tile's valid columns of (1 + pml_weight x number of PML directions)), so
// the cheap items fill the tail; equal costs keep the (model, z-chunk, tile)
// order, so neighbouring tiles of a class run together and share halo rows in
// L2, and the two parts of a tile follow one another.
std::vector<int4> build_items(const std::vector<Geom> &gs, const std::vector<char> &plain,
                              bool lean, int G, const WorkParams &wp, int *zchunk) {
  struct It { Item v; double cost; };
  struct Col { int i0, j0, z0, z1, mdl; double w; bool cut; };
  std::vector<Col> cols;  // columns with their z range, to be cut into pieces
  double planes = 0;
  for (size_t mdl = 0; mdl < gs.size(); ++mdl) {
    const Geom &g = gs[mdl];
    const int zlo = LFD + g.nabs[4], ztop = g.nk + LFD;
    const bool split = plain[mdl] && ztop - zlo >= 8;  // lean columns exist
    for (const Tile &ty : y_tiles(g))
      for (const Tile &tx : x_tiles(g)) {
        const bool in = split && tx.interior && ty.interior;
        if (lean && !in) continue;
        auto add = [&](int z0, int z1, bool cut) {
          if (z0 >= z1) return;
          double w = 0;
          for (int j = std::max(ty.at, 0); j < ty.at + TY && j < g.nj; ++j) {
            const bool yp = j < g.nabs[2] || j >= g.nj - g.nabs[3];
            for (int i = tx.at; i < tx.at + CX && i < g.ni; ++i) {
              const bool xp = i < g.nabs[0] || i >= g.ni - g.nabs[1];
              w += 1 + wp.pml_weight * ((xp ? 1 : 0) + (yp ? 1 : 0) + (z0 < zlo ? 1 : 0));
            }
          }
          cols.push_back({tx.at, ty.at, z0, z1, (int)mdl, w, cut});
          planes += z1 - z0;
        };
        if (lean) {
          add(zlo, ztop, true);
        } else if (in) {
          add(LFD, zlo, true);
        } else if (g.nabs[4] >= 8 && ztop - zlo >= 8) {
          add(LFD, zlo, true);
          add(zlo, ztop, true);
        } else {
          add(LFD, ztop, true);
        }
      }
  }
  if (cols.empty()) return {};
  // chunk length: about items_per_cta items per resident CTA, min_chunk planes at
  // the least; but where that leaves resident CTAs without an item, as
  // many planes as share the work out over all of them, down to one (the stage
  // then takes a few planes' latency: 28x24x20 cells 103 us per step with
  // chunks of at least 4 planes, 73 with 2, 60 with 1; 62x54x40 cells, where
  // the work fills 1.4 planes per CTA, 132, 126 and 129, hence rounded up)
  const int parts = lean ? 2 : 1;
  const double fill = parts * planes / G;
  double len = std::max(fill / wp.items_per_cta, (double)wp.min_chunk);
  if (fill < len) len = std::max(std::ceil(fill), 1.0);
  const int min_len = (int)std::min(len, 4.0);
  std::vector<It> items;
  for (const Col &c : cols) {
    const int n = c.z1 - c.z0;
    int pieces = std::max(1, (int)(n / len + 0.5));
    while (pieces > 1 && n / pieces < min_len) --pieces;
    if (zchunk && items.empty()) *zchunk = (n + pieces - 1) / pieces;
    for (int q = 0; q < pieces; ++q) {
      const int a0 = c.z0 + (int)((long)n * q / pieces);
      const int a1 = c.z0 + (int)((long)n * (q + 1) / pieces);
      items.push_back({Item{c.i0, c.j0, a0, a1, c.mdl, 0}, c.w * (a1 - a0)});
    }
  }
  // z-chunks of a class together: columns were cut one by one
  std::stable_sort(items.begin(), items.end(), [](const It &x, const It &y) {
    if (x.cost != y.cost) return x.cost > y.cost;
    if (x.v.model != y.v.model) return x.v.model < y.v.model;
    return x.v.z0 < y.v.z0;
  });
  std::vector<int4> hv;
  hv.reserve(2 * items.size());
  auto push = [&](Item v) {
    for (int part : {PART_VEL, PART_STR}) {
      v.part = part;
      if (lean || part == PART_VEL) hv.push_back(pack_item(v));
    }
  };
  // guided end: the last items (the cheapest, one per resident CTA) become
  // short chunks, ordered piece by piece (the first piece of every cut item,
  // then the second...) so that CTAs running together stay on neighbouring
  // columns
  size_t ncut = 0;
  if (wp.tail_chunk >= 4) {
    while (parts * ncut < (size_t)G && ncut < items.size()) {
      const Item &v = items[items.size() - 1 - ncut].v;
      if (v.z1 - v.z0 < 2 * wp.tail_chunk) break;
      ++ncut;
    }
  }
  const size_t keep = items.size() - ncut;
  for (size_t q = 0; q < keep; ++q) push(items[q].v);
  std::vector<std::vector<Item>> pieces(ncut);
  size_t maxp = 0;
  for (size_t q = 0; q < ncut; ++q) {
    Item v = items[keep + q].v;
    const int z0 = v.z0, n = v.z1 - z0, np = n / wp.tail_chunk;
    for (int t = 0; t < np; ++t) {
      v.z0 = z0 + (int)((long)n * t / np);
      v.z1 = z0 + (int)((long)n * (t + 1) / np);
      pieces[q].push_back(v);
    }
    maxp = std::max(maxp, pieces[q].size());
  }
  for (size_t t = 0; t < maxp; ++t)
    for (size_t q = 0; q < ncut; ++q)
      if (t < pieces[q].size()) push(pieces[q][t]);
  return hv;
}

// uploads the two work lists into the plan; the earlier ones are replaced, and
// freed, only when the new ones are complete
bool upload_items(Plan *pl, const std::vector<int4> (&hv)[2],
                  const int (&G)[NLIST]) {
  Work &wk = pl->wk;
  if (hv[0].empty() && hv[1].empty()) return false;
  int4 *d[2] = {nullptr, nullptr};
  bool ok = true;
  for (int l = 0; l < 2; ++l)
    if (ok && !hv[l].empty())
      ok = cudaMalloc(&d[l], hv[l].size() * sizeof(int4)) == cudaSuccess &&
           cudaMemcpy(d[l], hv[l].data(), hv[l].size() * sizeof(int4), cudaMemcpyHostToDevice) ==
               cudaSuccess;
  if (ok && !wk.counter) {
    int *c = nullptr;
    ok = cudaMalloc(&c, 2 * NLIST * sizeof(int)) == cudaSuccess &&
         cudaMemset(c, 0, 2 * NLIST * sizeof(int)) == cudaSuccess;
    if (ok) wk.counter = c;
    else cudaFree(c);
  }
  if (!ok) {
    for (int4 *p : d) cudaFree(p);
    return false;
  }
  for (int l = 0; l < 2; ++l) {
    cudaFree((void *)wk.items[l]);
    wk.items[l] = d[l];
    wk.nitems[l] = (int)hv[l].size();
  }
  for (int q = 0; q < NLIST; ++q) {
    const int n = wk.nitems[q == LEAN_BOTH];
    pl->grid[q] = n < G[q] ? n : G[q];
  }
  return true;
}

// builds the work lists of a shape and of the models' `plain` flags; on failure
// the plan keeps its lists, shape and flags
bool rebuild(Plan *pl, const WorkParams &wp, const std::vector<char> &plain) {
  std::vector<int4> hv[2];
  int G[NLIST], zchunk = pl->zchunk;
  for (int q = 0; q < NLIST; ++q) {
    G[q] = entry(pl->elem, 1, q).resident[pl->nmodels > 0]();
    if (G[q] < 1) return false;
  }
  for (int l = 0; l < 2; ++l)
    hv[l] = build_items(pl->geoms, plain, l != 0,
                        l ? G[LEAN_BOTH] : std::min(G[GEN_VEL], G[GEN_STR]), wp, &zchunk);
  if (!upload_items(pl, hv, G)) return false;
  pl->list_id = 14695981039346656037ull;  // FNV-1a over both lists
  for (const auto &list : hv)
    for (const int4 &v : list)
      for (int w : {v.x, v.y, v.z, v.w}) pl->list_id = (pl->list_id ^ (unsigned)w) * 1099511628211ull;
  pl->zchunk = zchunk;
  pl->params = wp;
  pl->plain = plain;
  return true;
}

}  // namespace
}  // namespace pair

void *pair_create_plan(const Geom &g, int elem, void *const sets[4], const float *media,
                       const float *metric, float *const aux[3]) {
  if (!set_attrs_of(elem)) return nullptr;
  Plan *pl = new (std::nothrow) Plan();
  if (!pl) return nullptr;
  pl->elem = elem;
  pl->sms = sm_count();
  pl->geoms.push_back(g);
  pl->plain.assign(1, 1);
  pl->mm.resize(1);
  if (!model_maps(&pl->mm[0], pl->wk.has_aux, g, elem, sets, media, metric, aux) ||
      !pair_set_work(pl, WorkParams{})) {
    pair_destroy_plan(pl);
    return nullptr;
  }
  return pl;
}

WorkParams pair_get_work(const void *plan) {
  return reinterpret_cast<const Plan *>(plan)->params;
}

unsigned long long pair_work_id(const void *plan) {
  return reinterpret_cast<const Plan *>(plan)->list_id;
}

bool pair_set_work(void *plan, const WorkParams &wp) {
  Plan *pl = reinterpret_cast<Plan *>(plan);
  return rebuild(pl, wp, std::vector<char>(pl->plain));
}

bool pair_set_plain(void *plan, const char *plain) {
  Plan *pl = reinterpret_cast<Plan *>(plan);
  const std::vector<char> v(plain, plain + pl->geoms.size());
  return v == pl->plain || rebuild(pl, pl->params, v);
}

bool pair_set_wait_test(void *plan, double wait_s, int withhold) {
  Plan *pl = reinterpret_cast<Plan *>(plan);
  if (!pl || !(wait_s > 0.0) || wait_s > 60.0) return false;
  pl->wk.wait_us = withhold >= 0 ? (unsigned)(wait_s * 1e6) : ptx::WAIT_US;
  pl->wk.withhold = withhold >= 0 ? withhold : -1;
  return true;
}

void pair_destroy_plan(void *plan) {
  Plan *pl = reinterpret_cast<Plan *>(plan);
  if (!pl) return;
  for (const int4 *p : pl->wk.items) cudaFree((void *)p);
  cudaFree(pl->wk.counter);
  cudaFree(pl->d_bargs);
  cudaFree(pl->d_bmaps);
  delete pl;
}

void launch_stage_pair(const void *plan, const StageArgs &a, int in_set, int *err, void *stream,
                       const SideStream *side) {
  const Plan &pl = *reinterpret_cast<const Plan *>(plan);
  cudaStream_t s = (cudaStream_t)stream;
  const int kind = a.rk == 0 ? 0 : (a.rk < 3 ? 1 : 2);
  Maps m[2];
  stage_maps(pl.mm[0], a.rk, in_set, a.tw_skip && a.rk == 1, pl.elem != ELEM_F32, m[0], m[1]);
  // the parts of the general items, the lean items and the traction image (the
  // top three layers' V, their tW and x/y auxiliaries) need only the stage
  // input and write disjoint values: with side streams they run beside one
  // another
  cudaStream_t ls[NLIST] = {s, s, s};
  if (side) {
    cudaEventRecord((cudaEvent_t)side->fork, s);
    for (int q = 0; q < SideStream::N; ++q)
      cudaStreamWaitEvent((cudaStream_t)side->stream[q], (cudaEvent_t)side->fork, 0);
    if (pl.grid[GEN_STR] > 0) ls[GEN_STR] = (cudaStream_t)side->stream[1];
    if (pl.grid[GEN_VEL] > 0) ls[LEAN_BOTH] = (cudaStream_t)side->stream[2];
  }
  for (int q : {GEN_STR, GEN_VEL, LEAN_BOTH})
    if (pl.grid[q] > 0) entry(pl.elem, kind, q).launch[0](pl, m, a, pl.wk, err, ls[q]);
  launch_timg(a, side ? side->stream[0] : stream, pl.sms);
  if (side)
    for (int q = 0; q < SideStream::N; ++q) {
      cudaEventRecord((cudaEvent_t)side->join[q], (cudaStream_t)side->stream[q]);
      cudaStreamWaitEvent(s, (cudaEvent_t)side->join[q], 0);
    }
}

// ---------------------------- batched models ------------------------------

void *pair_create_batch_plan(int n, const Geom *gs, void *const *sets, const float *const *media,
                             const float *const *metric, float *const *aux, int elem) {
  if (n > ITEM_MODELS || !set_attrs_of(elem)) return nullptr;
  Plan *pl = new (std::nothrow) Plan();
  if (!pl) return nullptr;
  pl->elem = elem;
  pl->nmodels = n;
  pl->geoms.assign(gs, gs + n);
  pl->plain.assign(n, 1);
  pl->wk.nmodels = n;
  pl->mm.resize(n);
  bool ok = true;
  for (int i = 0; i < n && ok; ++i) {
    int ha[3];
    ok = model_maps(&pl->mm[i], ha, gs[i], elem, sets + 4 * i, media[i], metric[i],
                    aux + 3 * i);
  }
  // per stage, part and model: the maps of that stage (input set per stage
  // as in the step schedule: FW, Wa, Wb, Wa; batched stages run with tW
  // elision)
  static const int ins[4] = {0, 1, 2, 1};
  std::vector<Maps> hm((size_t)8 * n);
  for (int rk = 0; rk < 4 && ok; ++rk)
    for (int i = 0; i < n; ++i)
      stage_maps(pl->mm[i], rk, ins[rk], rk == 1, elem != ELEM_F32, hm[(size_t)(rk * 2) * n + i],
                 hm[(size_t)(rk * 2 + 1) * n + i]);
  ok = ok && cudaMalloc(&pl->d_bmaps, hm.size() * sizeof(Maps)) == cudaSuccess &&
       cudaMemcpy(pl->d_bmaps, hm.data(), hm.size() * sizeof(Maps), cudaMemcpyHostToDevice) ==
           cudaSuccess &&
       cudaMalloc(&pl->d_bargs, (size_t)16 * n * sizeof(StageArgs)) == cudaSuccess;
  if (!ok || !pair_set_work(pl, WorkParams{})) {
    pair_destroy_plan(pl);
    return nullptr;
  }
  return pl;
}

bool pair_batch_set_args(void *plan, const StageArgs *args) {
  Plan *pl = reinterpret_cast<Plan *>(plan);
  return cudaMemcpy(pl->d_bargs, args, (size_t)16 * pl->nmodels * sizeof(StageArgs),
                    cudaMemcpyHostToDevice) == cudaSuccess;
}

void launch_stage_pair_batch(const void *plan, int pattern, const StageArgs &rep, int *err,
                             void *stream) {
  const Plan &pl = *reinterpret_cast<const Plan *>(plan);
  cudaStream_t s = (cudaStream_t)stream;
  const int rk = rep.rk, kind = rk == 0 ? 0 : (rk < 3 ? 1 : 2), n = pl.nmodels;
  Work wk = pl.wk;
  wk.bargs = pl.d_bargs + (size_t)(pattern * 4 + rk) * n;
  wk.bmaps = pl.d_bmaps + (size_t)(rk * 2) * n;
  const Maps none[2] = {};
  for (int q : {GEN_STR, GEN_VEL, LEAN_BOTH})
    if (pl.grid[q] > 0) entry(pl.elem, kind, q).launch[1](pl, none, rep, wk, err, s);
  int mi = 0, mj = 0;
  for (const Geom &g : pl.geoms) {
    mi = g.ni > mi ? g.ni : mi;
    mj = g.nj > mj ? g.nj : mj;
  }
  launch_timg_batch(wk.bargs, n, mi, mj, pl.elem, s);
}

int pair_plan_info(const void *plan, int *zchunk, int *grid_general, int *grid_lean) {
  const Plan &pl = *reinterpret_cast<const Plan *>(plan);
  if (zchunk) *zchunk = pl.zchunk;
  if (grid_general) *grid_general = pl.grid[GEN_VEL];
  if (grid_lean) *grid_lean = pl.grid[LEAN_BOTH];
  return pl.wk.nitems[0] + pl.wk.nitems[1];
}

}  // namespace cgfd
