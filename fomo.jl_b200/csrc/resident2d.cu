// resident2d.cu -- tile plan of the on-chip 2D time loops (resident2d.cuh).
#include <algorithm>
#include <numeric>

#include "resident2d.cuh"

namespace fomo {
namespace res {

namespace {
constexpr int kMaxSmem = 227 * 1024;
int align4(int n) { return (n + 3) & ~3; }
}  // namespace

Plan make_plan(const Needs& nd, int N, int nx, int nz, int ld, int nbc, int ns, int nsm,
               int extra) {
  Plan best;
  if (ns < 1 || ns > nsm) return best;
  const int per = nsm / ns, H = N + 1, L = align4(N);
  double best_cost = 0.0;
  for (int gx = 1; gx <= per; ++gx) {
    int TW = 0, narrow = nx, nq = 0;
    for (int i = 0; i < gx; ++i) {
      const int a = tile_x(nx, gx, i), b = tile_x(nx, gx, i + 1), first = a ? a - 1 : 0;
      TW = std::max(TW, b - a);
      narrow = std::min(narrow, b - a);
      nq = std::max(nq, (std::min(b, nx - 1) - first) / 4 + 1);
    }
    if (gx > 1 && narrow < H) break;
    const int gz = std::max(1, std::min(per / gx, nz / H));
    for (int z = std::max(1, gz - 2); z <= gz; ++z) {
      const int TH = (nz + z - 1) / z;
      for (int form = 0; form < nd.forms; ++form) {
        const int R = kForms[form].R, CX = kForms[form].CX, nb = 4 * nq / CX;
        const int ngr = (TH + 2 + R - 1) / R, thr = nb * ngr;
        if (thr > kForms[form].threads) continue;
        const int rows = ngr * R + 2 * N + 1;
        // columns: L + the quads + the right halo, padded so that the 16-byte reads
        // of a warp that spans row groups miss each other's banks
        const int need = L + 4 * nq + (N == 5 ? 8 : 4);
        const bool mreg = CX * R <= nd.mreg, small = CX * R <= kSmallBlock;
        for (int gmat = 0; gmat <= (mreg || small ? 0 : 1); ++gmat)
          for (int pad = 28; pad >= 0; pad -= 4) {
            const int pitch = need + pad;
            if (pad && (R * (pitch / 4) - nq) % 8 != 0) continue;
            const int ext = nd.ext + (mreg || gmat ? 0 : nd.mats);
            const int floats = (nd.hal * rows * pitch + ext * ngr * R * 4 * nq + extra + 3) & ~3;
            // words put (4 bytes of table each) and got (8 bytes) by both half steps
            const int put = (2 * N + 1 + nd.wide) * (nd.strips * TH + nd.bands * TW) +
                            2 * (nd.rows * TW + nd.cols * TH);
            const int get = put + 2 * (2 * N + 1 + nd.wide) * (nd.strips + nd.bands);
            const size_t smem = sizeof(float) * floats + sizeof(int) * (put + 2) + sizeof(Word) * get;
            if (smem > (size_t)kMaxSmem) continue;
            // the slowest tile sets the pace: its extended cells, plus the halo it reads
            const double cost = 4.0 * R * nq * ngr + form + 2.0 * (TW + TH) * (2 * N + 2) * 0.3 +
                                gmat * 1000.0;
            if (best.ok && cost >= best_cost) continue;
            best_cost = cost;
            best.ok = true;
            best.form = form;
            // idle threads of a small tile still move words
            best.threads = (std::min(kForms[form].threads, std::max(thr, get / 6)) + 31) & ~31;
            best.tiles = gx * z * ns;
            best.smem = smem;
            best.g = Geom{nx,  nz, ld,    (long long)ld * nz, N,      nbc, gx,  z,
                          nq, ngr, nb, pitch, rows, floats, put, gmat};
          }
      }
    }
  }
  return best;
}

void plan_entries(Plan& p, int ns, const CellTagHost& tags) {
  const Geom& g = p.g;
  struct Item {
    int tile, thread, cell, e;
  };
  std::vector<Item> items;
  for (int e = 0; e < (int)tags.lin.size(); ++e) {
    const int x = tags.lin[e] % g.ld, z = tags.lin[e] / g.ld;
    int tx = 0, tz = 0;
    while (tile_x(g.nx, g.gx, tx + 1) <= x) ++tx;
    while (tile_z(g.nz, g.gz, tz + 1) <= z) ++tz;
    const int x0 = tile_x(g.nx, g.gx, tx);
    const int ex = x - (x0 ? x0 - 1 : 0), ez = z - tile_z(g.nz, g.gz, tz) + 1;  // extended
    const Form f = kForms[p.form];
    const int thread = (ez / f.R) * g.nb + ex / f.CX, cell = (ez % f.R) * f.CX + ex % f.CX;
    for (int s = 0; s < ns; ++s)
      items.push_back(Item{(s * g.gz + tz) * g.gx + tx, thread, cell, e});
  }
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
    return a.tile != b.tile ? a.tile < b.tile : a.thread < b.thread;
  });
  p.off.assign(p.tiles + 1, 0);
  p.key.resize(items.size());
  p.ent.resize(items.size());
  for (const Item& it : items) ++p.off[it.tile + 1];
  std::partial_sum(p.off.begin(), p.off.end(), p.off.begin());
  for (size_t k = 0; k < items.size(); ++k) {
    p.key[k] = make_int2(items[k].thread, items[k].cell);
    p.ent[k] = items[k].e;
  }
}

Tables take_tables(Arena& ar, const Plan& p) {
  Tables t;
  if (!p.ok) return t;
  t.ll_words = (size_t)4 * p.tiles * p.g.per;
  t.ll = ar.take<uint64_t>(t.ll_words);
  t.off = ar.take<int>(p.off.size());
  t.key = ar.take<int2>(std::max<size_t>(p.key.size(), 1));
  t.ent = ar.take<int>(std::max<size_t>(p.ent.size(), 1));
  return t;
}

cudaError_t upload_tables(cudaStream_t st, char* ws, const Plan& p, const Tables& t,
                          const CellTags& tags, Run& run) {
  int* off = reinterpret_cast<int*>(ws + t.off);
  int2* key = reinterpret_cast<int2*>(ws + t.key);
  int* ent = reinterpret_cast<int*>(ws + t.ent);
  run.g = p.g;
  run.E = Entries{off, key, ent, tags};
  run.ll = reinterpret_cast<uint64_t*>(ws + t.ll);
  cudaError_t e = cudaMemcpyAsync(off, p.off.data(), sizeof(int) * p.off.size(),
                                  cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && !p.key.empty())
    e = cudaMemcpyAsync(key, p.key.data(), sizeof(int2) * p.key.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && !p.ent.empty())
    e = cudaMemcpyAsync(ent, p.ent.data(), sizeof(int) * p.ent.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(run.ll, 0, sizeof(uint64_t) * t.ll_words, st);
  return e;
}

int sm_count(int device) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace res
}  // namespace fomo
