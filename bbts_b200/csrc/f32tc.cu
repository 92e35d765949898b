// Host side of the FP32 tensor-core product (f32tc.h).
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include "bbts_b200.h"
#include "common.h"
#include "f32tc.h"
#include "gemm_f32tc.cuh"
#include "launch.h"

namespace bbx {

namespace {
thread_local bool t_fma_chain = false;
}
FmaChain::FmaChain(bool on) : before_(t_fma_chain) { t_fma_chain = before_ || on; }
FmaChain::~FmaChain() { t_fma_chain = before_; }
bool FmaChain::active() { return t_fma_chain; }

// The lesser of two measured times of a lone product (us): the SIMT kernel takes
// 0.105 us per step of K for each round of 128 x 128 tiles over the chip; the
// tensor cores 1.15 us per 64 steps, after about 10 us more of launches (two
// kernels, their prologues) and the operands' split (10 bytes moved per element at 4 TB/s):
// 128 x 128 x 64 7 against 17 us, 256^3 29 against 28, 512^3 54 against 29, 4096^3 2700 against 750.
// From K = 64 on its error is below the FMA chain's for every size measured, on normals and
// on data of one sign (normwise 0.8e-7 against 1.4e-7 at K = 64, 1.7e-7 against 11e-7 at
// K = 4096). Only short sums that one huge term dominates are summed better by the chain
// (log-normals, sigma = 2, K <= 256: 3.7e-7 against 1.9e-7).
bool f3_wanted(long long m, long long n, long long k, long long batch) {
  if (k < 64 || std::min(m, n) < 16 || batch <= 0 || batch > 65535) return false;
  const double tiles = (double)((m + 127) / 128) * ((n + 127) / 128) * batch;
  const double rounds = std::ceil(tiles / 148);
  const double simt = 6.0 + 0.105 * k * rounds;
  const double tc = 16.0 + 1.15 * ((k + 63) / 64) * rounds + 2.5e-6 * ((double)m * k + (double)k * n) * batch;
  return tc < simt;
}

bool f3_contraction_wanted(const ContractionLowering& L) {
  return !L.empty && L.nn <= 65535ll * 128 && f3_wanted(L.nm, L.nn, L.kdim, L.nb);
}

F3Mat f3_dense(const float* src, long long rows, long long cols, long long ld, long long batch, long long stride, bool mn) {
  F3Mat t;
  t.src = src;
  t.mn = mn;
  t.rows = rows;
  t.cols = cols;
  t.pitch = (cols + 7) / 8 * 8;
  t.batch = batch;
  GatherArgs& g = t.g;
  g.rank_o = 3;
  g.odims[0] = batch; g.istride[0] = stride; g.ostride[0] = rows * t.pitch;
  g.odims[1] = rows;  g.istride[1] = ld;     g.ostride[1] = t.pitch;
  g.odims[2] = cols;  g.istride[2] = 1;      g.ostride[2] = 1;
  simplify_gather(&g);
  return t;
}

void f3_contraction(const ContractionLowering& L, const float* lhs, const float* rhs, float* c, float alpha, F3Mat* lc,
                    F3Mat* rc, F3Spec* out) {
  auto mat = [&](const float* src, const GatherArgs& g, bool mn, long long mode, long long pitch_mn) {
    F3Mat t;
    t.src = src;
    t.g = g;
    simplify_gather(&t.g);
    t.mn = mn;
    t.rows = mn ? L.kdim : mode;
    t.cols = mn ? mode : L.kdim;
    t.pitch = mn ? pitch_mn : L.pk;
    t.batch = L.nb;
    return t;
  };
  *lc = mat(lhs, L.ga, L.lc_mn, L.nm, L.pm);
  *rc = mat(rhs, L.gb, L.rc_mn, L.nn, L.pn);
  F3Spec s;
  // the longer side is M, as in contraction_gemm; C holds element (m, n) of the output at m + n * nm
  const bool l_first = L.nm > L.nn;
  s.a = l_first ? 0 : 1;
  s.b = l_first ? 1 : 0;
  s.m = (int)(l_first ? L.nm : L.nn);
  s.n = (int)(l_first ? L.nn : L.nm);
  s.k = (int)L.kdim;
  s.c = c;
  s.ldc = L.nm;
  s.c_batch = L.nn * L.nm;
  s.c_col = l_first;
  s.alpha = alpha;
  *out = s;
}

namespace {

long long plane_elems(const F3Mat& m) { return m.batch * m.rows * m.pitch; }

// Chunks of a split: one CTA each, of 512 items (eight elements), two a thread:
// a 1024^2 matrix alone then has 256 CTAs (with 64 of eight items a thread, 10 us instead of 4).
// One a thread while that leaves no more than a CTA an SM: a lone 501^3 product 25.0 -> 22.8 us
// (each item of a row record waits for its own loads), 512^3 18.7 and 18.6.
// At most 1024 chunks, the words that a reader of the maximum takes.
struct Chunks { long long rows, items, per, count; };
Chunks chunks_of(const F3Mat& m) {
  const GatherArgs& g = m.g;
  Chunks c;
  c.rows = 1;
  for (int d = 0; d + 1 < g.rank_o; ++d) c.rows *= g.odims[d];
  c.items = c.rows * ((g.odims[g.rank_o - 1] + 7) / 8);
  c.per = c.items < 148 * 256 ? 256 : std::max(512ll, (c.items / 1024 + 256) / 256 * 256);
  c.count = (c.items + c.per - 1) / c.per;
  return c;
}

size_t planes_bytes(const F3Mat& m) { return ((size_t)plane_elems(m) * 6 + 255) & ~(size_t)255; }

F3Split split_record(const F3Mat& m, int chunk_start) {
  const GatherArgs& g = m.g;
  const Chunks ch = chunks_of(m);
  F3Split r;
  std::memset(&r, 0, sizeof(r));
  r.src = m.src;
  r.dst = (__nv_bfloat16*)m.ws;
  r.plane = plane_elems(m);
  const int outer = g.rank_o - 1;
  for (int d = 0; d < 3; ++d) r.odims[d] = 1;
  for (int d = 0; d < outer; ++d) {  // into the last places
    const int q = 3 - outer + d;
    r.odims[q] = g.odims[d];
    r.istride[q] = g.istride[d];
    r.ostride[q] = g.ostride[d];
  }
  r.len = g.odims[outer];
  r.inner = g.istride[outer];
  r.oinner = g.ostride[outer];
  r.items = ch.items;
  r.items_per_chunk = ch.per;
  r.amax = (uint32_t*)((char*)m.ws + planes_bytes(m));
  r.chunk_start = chunk_start;
  r.rank_s = g.rank_s;
  for (int d = 0; d < g.rank_s; ++d) {
    r.sdims[d] = g.sdims[d];
    r.sstride[d] = g.sstride[d];
  }
  return r;
}

// Tile shapes of the product kernel.
enum Shape { PAIR256 = 0, ONE128 = 1 };
struct ShapeInfo { int tile, sms; double chunk_cycles; };
// chunk_cycles: measured per chunk of K of one tile (see the head of gemm_f32tc.cuh)
constexpr ShapeInfo kShapes[2] = {{256, 2, 3700.0}, {128, 1, 2200.0}};

int operand_map(const F3Mat& m, CUtensorMap* map) {
  return make_map3(map, m.ws, m.cols, m.rows, 3 * m.batch, m.pitch, m.rows * m.pitch, 64, m.mn ? 64 : 128);
}

int build_problem(const F3Mat* mats, const F3Spec& s, Shape shape, F3Problem* out) {
  const F3Mat &a = mats[s.a], &b = mats[s.b];
  std::memset(out, 0, sizeof(*out));
  const ShapeInfo& sh = kShapes[shape];
  int rc = operand_map(a, &out->tmap_a);
  if (!rc) rc = operand_map(b, &out->tmap_b);
  if (rc) return rc;
  out->f.a = (const __nv_bfloat16*)a.ws;
  out->f.b = (const __nv_bfloat16*)b.ws;
  out->f.c = s.c;
  out->f.bias = s.bias;
  out->f.amax_a = (const uint32_t*)((const char*)a.ws + planes_bytes(a));
  out->f.amax_b = (const uint32_t*)((const char*)b.ws + planes_bytes(b));
  out->f.na = (int)chunks_of(a).count;
  out->f.nb = (int)chunks_of(b).count;
  out->f.a_plane = plane_elems(a);
  out->f.b_plane = plane_elems(b);
  out->f.a_batch = a.rows * a.pitch;
  out->f.b_batch = b.rows * b.pitch;
  out->f.a_row = a.mn ? 1 : a.pitch;
  out->f.a_k = a.mn ? a.pitch : 1;
  out->f.b_col = b.mn ? 1 : b.pitch;
  out->f.b_k = b.mn ? b.pitch : 1;
  out->f.ldc = s.ldc;
  out->f.c_batch = s.c_batch;
  out->f.m = s.m; out->f.n = s.n; out->f.k = s.k;
  out->f.batch = (int)a.batch;
  out->f.tiles_m = (s.m + sh.tile - 1) / sh.tile;
  out->f.tiles_n = (s.n + sh.tile - 1) / sh.tile;
  out->f.a_mn = a.mn ? 1 : 0;
  out->f.b_mn = b.mn ? 1 : 0;
  out->f.c_col = s.c_col ? 1 : 0;
  out->f.alpha = s.alpha;
  out->f.beta = s.beta;
  return BBX_OK;
}

// Modelled time of a group in one shape: the longest unit's share of the tile
// list (the kernel's own order), a tile costing its K chunks times the measured
// cost of a chunk.
double group_cost(const std::vector<std::pair<long long, int>>& tiles_k, int units, double per_chunk) {
  long long total = 0;
  for (auto& t : tiles_k) total += t.first;
  if (total <= units) {
    double most = 0;
    for (auto& t : tiles_k) most = std::max(most, (double)((t.second + kF3BK - 1) / kF3BK));
    return most * per_chunk;
  }
  double sum = 0, most = 0;
  for (auto& t : tiles_k) {
    const double c = (t.second + kF3BK - 1) / kF3BK;
    sum += c * t.first;
    most = std::max(most, c);
  }
  if (tiles_k.size() == 1) return (double)((total + units - 1) / units) * most * per_chunk;
  return std::max(most, sum / units + 0.5 * most) * per_chunk;
}

Shape pick_shape(const F3Mat* mats, const F3Spec* specs, const int* order, int count, int sms) {
  Shape best = PAIR256;
  double best_cost = 0;
  for (Shape sh : {PAIR256, ONE128}) {
    const ShapeInfo& si = kShapes[sh];
    std::vector<std::pair<long long, int>> t;
    for (int i = 0; i < count; ++i) {
      const F3Spec& s = specs[order ? order[i] : i];
      t.push_back({mats[s.a].batch * ((s.m + si.tile - 1) / si.tile) * ((s.n + si.tile - 1) / si.tile), s.k});
    }
    const double cost = group_cost(t, sms / si.sms, si.chunk_cycles);
    if (sh == PAIR256 || cost < best_cost) {
      best = sh;
      best_cost = cost;
    }
  }
  return best;
}

int launch(const F3Args& args, Shape shape, int sms, cudaStream_t st) {
  const int grid = kShapes[shape].sms * std::min(args.total_tiles, sms / kShapes[shape].sms);
  launch_dependent(shape == PAIR256 ? f32_gemm_pair_kernel : f32_gemm_kernel, grid, kF3Threads, kF3Smem, st, args);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? BBX_OK : set_error(BBX_ERR_CUDA, "f32_gemm: %s", cudaGetErrorString(e));
}

// The split kernel of a record.
enum SplitKind { GENERAL = 0, ROWS = 1, FLAT = 2 };
bool rows_ok(const F3Split& r) {
  if (r.rank_s != 0 || r.inner != 1 || r.oinner != 1 || r.plane % 8 != 0 || r.items >= (1ll << 30)) return false;
  // a row's last piece is written whole: the row stride has to leave it room
  const bool one_row = r.items == (r.len + 7) / 8;
  return r.odims[0] == 1 && r.odims[1] == 1 && r.ostride[2] % 8 == 0 && r.istride[2] >= 0 && r.len < (1ll << 31) &&
         (one_row ? r.plane : r.ostride[2]) >= (r.len + 7) / 8 * 8;
}
SplitKind split_kind(const F3Split& r) {
  if (!rows_ok(r)) return GENERAL;
  return r.items == r.len / 8 && r.len % 8 == 0 && (((uintptr_t)r.src) & 15) == 0 ? FLAT : ROWS;
}

int launch_split(const F3SplitArgs& args, int chunks, int kind, cudaStream_t st) {
  if (chunks == 0) return BBX_OK;
  launch_dependent(kind == FLAT ? k_f32_split_flat : kind == ROWS ? k_f32_split_rows : k_f32_split, chunks, 256, 0, st, args);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? BBX_OK : set_error(BBX_ERR_CUDA, "k_f32_split: %s", cudaGetErrorString(e));
}

long long tiles_of(const F3Problem& p) { return (long long)p.f.batch * p.f.tiles_m * p.f.tiles_n; }

}  // namespace

size_t f3_mat_bytes(const F3Mat& m) {
  return planes_bytes(m) + (((size_t)chunks_of(m).count * 4 + 255) & ~(size_t)255);
}

int f3_init() {
  cudaError_t e = cudaSuccess;
  for (auto f : {(const void*)f32_gemm_pair_kernel, (const void*)f32_gemm_kernel})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kF3Smem);
  return e == cudaSuccess ? BBX_OK : set_error(BBX_ERR_CUDA, "f32_gemm attribute: %s", cudaGetErrorString(e));
}

int f3_run(const F3Mat* mats, const F3Spec& spec, void* stream) {
  uint32_t* status = nullptr;
  int sms = 148;
  int rc = device_status_and_sms(&status, &sms);
  if (rc) return rc;
  const Shape shape = pick_shape(mats, &spec, nullptr, 1, sms);
  F3Args args;
  std::memset(&args, 0, sizeof(args));
  rc = build_problem(mats, spec, shape, &args.one);
  if (rc) return rc;
  args.num_problems = 1;
  args.status = status;
  if (tiles_of(args.one) > (1ll << 30)) return set_error(BBX_ERR_INVALID, "f32 product: too many tiles");
  args.total_tiles = (int)tiles_of(args.one);
  F3SplitArgs sp;
  std::memset(&sp, 0, sizeof(sp));
  int chunks = 0;
  int kind = FLAT;  // one launch: the most general kernel of the two (a flat record is also one of rows)
  for (int i : {spec.a, spec.b}) {
    sp.inl[sp.count] = split_record(mats[i], chunks);
    kind = std::min(kind, (int)split_kind(sp.inl[sp.count++]));
    chunks += (int)chunks_of(mats[i]).count;
    if (spec.a == spec.b) break;
  }
  rc = launch_split(sp, chunks, kind, (cudaStream_t)stream);
  return rc ? rc : launch(args, shape, sms, (cudaStream_t)stream);
}

struct F3Plan {
  struct Part { int first, count, tiles, shape; };
  F3Problem* d_problems = nullptr;
  F3Split* d_splits = nullptr;     // flat records, row records, the others
  int n_splits[3] = {0, 0, 0}, chunks[3] = {0, 0, 0};  // by SplitKind
  std::vector<Part> parts;
};

int f3_plan_create(const F3Mat* mats, int n_mats, const F3Spec* specs, int n_specs, F3Plan** out) {
  if (!mats || !specs || n_mats <= 0 || n_specs <= 0 || !out) return set_error(BBX_ERR_INVALID, "bad f32 plan arguments");
  uint32_t* status = nullptr;
  int sms = 148;
  int rc = device_status_and_sms(&status, &sms);
  if (rc) return rc;
  std::unique_ptr<F3Plan, void (*)(F3Plan*)> p(new F3Plan(), f3_plan_destroy);
  std::vector<F3Split> splits;
  for (int kind : {FLAT, ROWS, GENERAL})
    for (int i = 0; i < n_mats; ++i) {
      if (!mats[i].split) continue;
      const F3Split r = split_record(mats[i], p->chunks[kind]);
      if (split_kind(r) != kind) continue;
      splits.push_back(r);
      p->chunks[kind] += (int)chunks_of(mats[i]).count;
      p->n_splits[kind]++;
    }
  // descending K: the longest tiles first, the shortest even out the end
  std::vector<int> order(n_specs);
  for (int i = 0; i < n_specs; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return specs[x].k > specs[y].k; });
  std::vector<F3Problem> probs(n_specs);
  for (int first = 0; first < n_specs; first += kF3MaxProblems) {
    const int count = std::min(kF3MaxProblems, n_specs - first);
    const Shape shape = pick_shape(mats, specs, order.data() + first, count, sms);
    long long tiles = 0;
    for (int i = first; i < first + count; ++i) {
      rc = build_problem(mats, specs[order[i]], shape, &probs[i]);
      if (rc) return rc;
      probs[i].f.tile_start = (int)tiles;
      tiles += tiles_of(probs[i]);
      if (tiles > (1ll << 30)) return set_error(BBX_ERR_INVALID, "f32 plan: too many tiles");
    }
    p->parts.push_back({first, count, (int)tiles, (int)shape});
  }
  cudaError_t e = device_alloc((void**)&p->d_problems, sizeof(F3Problem) * n_specs);
  if (e == cudaSuccess) e = cudaMemcpy(p->d_problems, probs.data(), sizeof(F3Problem) * n_specs, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = device_alloc((void**)&p->d_splits, sizeof(F3Split) * splits.size());
  if (e == cudaSuccess) e = cudaMemcpy(p->d_splits, splits.data(), sizeof(F3Split) * splits.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return set_error(BBX_ERR_CUDA, "f32 plan upload: %s", cudaGetErrorString(e));
  *out = p.release();
  return BBX_OK;
}

int f3_plan_launch(F3Plan* p, void* stream) {
  if (!p) return set_error(BBX_ERR_INVALID, "null f32 plan");
  uint32_t* status = nullptr;
  int sms = 148;
  int rc = device_status_and_sms(&status, &sms);
  if (rc) return rc;
  int first = 0;
  for (int kind : {FLAT, ROWS, GENERAL}) {
    F3SplitArgs sp;
    std::memset(&sp, 0, sizeof(sp));
    sp.table = p->d_splits + first;
    sp.count = p->n_splits[kind];
    first += sp.count;
    rc = launch_split(sp, p->chunks[kind], kind, (cudaStream_t)stream);
    if (rc) return rc;
  }
  for (const auto& part : p->parts) {
    if (rc) return rc;
    F3Args args;
    std::memset(&args, 0, sizeof(args));
    args.table = p->d_problems + part.first;
    args.num_problems = part.count;
    args.total_tiles = part.tiles;
    args.status = status;
    rc = launch(args, (Shape)part.shape, sms, (cudaStream_t)stream);
  }
  return rc;
}

void f3_plan_destroy(F3Plan* p) {
  if (!p) return;
  if (p->d_problems) cudaFree(p->d_problems);
  if (p->d_splits) cudaFree(p->d_splits);
  delete p;
}

}  // namespace bbx
