// Hyperplane-column schedule of the sweep tasks (WaveJobs, declared in piks_internal.h).
#include <algorithm>
#include <atomic>
#include <thread>

#include "piks_internal.h"

namespace piks {

namespace {

int worker_count() {
  const unsigned hw = std::thread::hardware_concurrency();
  return (int)std::max(1u, std::min(hw ? hw : 1u, 16u));
}

// Runs fn(worker) on `n` threads.
template <typename F>
void on_workers(int n, F fn) {
  if (n <= 1) { fn(0); return; }
  std::vector<std::thread> th;
  for (int i = 0; i < n; ++i) th.emplace_back([&fn, i] { fn(i); });
  for (auto &t : th) t.join();
}

constexpr int kFw = 1 << 30;

// A row that a column holds: its code and where it stands (batch, list, index in the list).
struct Held { int32_t code, batch, idx; };   // idx | list << 28 (0 own, 1 static, 2 dependent)

// Scratch of one worker for the batches of a column.
struct ColumnScan {
  // rows by voxel (four z layers of the cross-section with its two upwind layers) and
  // variant: 0 the octant's own slot, 1 / 2 what a y / z reader finds in a wall
  std::vector<Held> cell;
  std::vector<int32_t> stat, dep;
  int32_t own[4], ns[4];          // own rows and static rows of the last four batches
  int64_t pos[4];                 // ring position of their first row
  int32_t stamp = 0;              // batches scanned so far, over all columns
};

}  // namespace

// One column: `fill` writes its rows and records, otherwise only the batch sizes.
struct WaveBuilder {
  const Geometry &g;
  WaveJobs &wj;
  int ncu, ncv;                                // columns per octant along x and y
  std::vector<int32_t> ux[2], vy[2], wz[2];    // frame coordinates by ghosted coordinate, sign + / -
  BigVec<uint64_t> xyz;
  BigVec<int32_t> order;
  std::vector<int32_t> col_of_key, key_of_col;
  std::vector<int64_t> task_begin;

  void scan(int col, ColumnScan &c, bool fill) {
    const int A = wj.A, B = wj.B;
    const int key = key_of_col[(size_t)col];
    const int o = key / (ncu * ncv), ka = key % ncu, kb = key / ncu % ncv;
    const int sx = oct_sx(o) < 0, sy = oct_sy(o) < 0, sz = oct_sz(o) < 0;
    const int64_t t0 = task_begin[(size_t)col], t1 = task_begin[(size_t)col + 1];
    int32_t *hdr = &wj.cols[(size_t)col * 8];
    const int s_first = hdr[3];
    int64_t batch = hdr[0];
    int64_t row_off = 0, p = t0, pos = 0;  // pos: rows of the column so far
    const int stride_v = A + 2, stride_w = (A + 2) * (B + 2);
    auto local = [&](int32_t node, int &lu, int &lv, int &w) {
      const uint64_t q = xyz[(size_t)node];
      lu = ux[sx][(size_t)(q & 0x1FFFFF)] - 1 - ka * A;
      lv = vy[sy][(size_t)((q >> 21) & 0x1FFFFF)] - 1 - kb * B;
      w = wz[sz][(size_t)(q >> 42)];
    };
    const int32_t first_stamp = c.stamp + 1;
    for (int s = s_first; s < s_first + hdr[1]; ++s, ++batch) {
      const int32_t k = ++c.stamp;
      int64_t e = p;
      for (; e < t1; ++e) {
        int lu, lv, w;
        const int32_t *r = &g.tasks[(size_t)order[(size_t)e] * 8];
        local(r[0], lu, lv, w);
        if (lu + lv + w - 1 != s) break;
        c.cell[(size_t)(((w & 3) * stride_w + (lv + 2) * stride_v + lu + 2) * 3)] = {r[0] * 8 + o, k, (int32_t)(e - p)};
      }
      const int32_t nt = (int32_t)(e - p);
      c.stat.clear();
      c.dep.clear();
      // the row of a read: found in the column's last batches, or added to this one
      auto find = [&](int32_t code, int axis, int back, int lu, int lv, int w) -> const Held & {
        int cu = lu, cv = lv, cw = w;
        (axis == 0 ? cu : axis == 1 ? cv : cw) -= back;
        const bool fw = code & kFw;
        const int variant = !fw && (code & 7) == o ? 0 : axis;
        Held &h = c.cell[(size_t)(((cw & 3) * stride_w + (cv + 2) * stride_v + cu + 2) * 3 + variant)];
        if (h.code == code && h.batch >= first_stamp && h.batch >= k - 2) return h;
        // swept by an upwind column: a fluid node of this octant past the inflow plane
        const bool swept = !fw && (code >> 3) < g.NF &&
                           (axis == 0 ? ka * A + cu >= 0 : axis == 1 ? kb * B + cv >= 0 : cw >= 1);
        std::vector<int32_t> &list = swept ? c.dep : c.stat;
        h = {code, k, (int32_t)list.size() | (swept ? 2 : 1) << 28};
        list.push_back(code);
        return h;
      };
      for (int64_t q = p; q < e; ++q) {
        const int32_t *r = &g.tasks[(size_t)order[(size_t)q] * 8];
        int lu, lv, w;
        local(r[0], lu, lv, w);
        for (int j = 0; j < 6; ++j)
          if (r[2 + j] >= 0) find(r[2 + j], j >> 1, 1 + (j & 1), lu, lv, w);
      }
      const int32_t ns = (int32_t)c.stat.size(), nd = (int32_t)c.dep.size(), nrows = nt + ns + nd;
      int32_t *b = &wj.batch[(size_t)batch * 4];
      if (!fill) {
        b[2] = nrows | nt << 16;
        b[3] = nt + ns;
        row_off += (nrows + 3) / 4 * 4;
        p = e;
        continue;
      }
      c.own[k & 3] = nt;
      c.ns[k & 3] = ns;
      c.pos[k & 3] = pos;
      const int R = wj.ring;
      b[3] |= (int32_t)(1 + pos % R) << 16;
      int32_t *rows = &wj.rows[(size_t)b[0] * 4];
      auto slot = [&](const Held &h) -> int32_t {
        const int list = h.idx >> 28, m = h.batch & 3;
        const int64_t at = c.pos[m] + (h.idx & 0xFFFFFFF) + (list > 0 ? c.own[m] : 0) + (list > 1 ? c.ns[m] : 0);
        return (int32_t)(1 + at % R);
      };
      for (int64_t q = p; q < e; ++q) {
        const int32_t *r = &g.tasks[(size_t)order[(size_t)q] * 8];
        rows[q - p] = r[0] * 8 + o;
        int lu, lv, w;
        local(r[0], lu, lv, w);
        int32_t sl[6];
        for (int j = 0; j < 6; ++j) sl[j] = r[2 + j] < 0 ? 0 : slot(find(r[2 + j], j >> 1, 1 + (j & 1), lu, lv, w));
        const int fl = r[1];
        int32_t *tr = &wj.tasks[(size_t)q * 4];
        tr[0] = r[0] | ((fl & 8) ? 1 << 27 : 0) | ((fl & 16) ? 1 << 28 : 0) | ((fl & 32) ? 1 << 29 : 0);
        tr[1] = sl[0] | sl[1] << 16;
        tr[2] = sl[2] | sl[3] << 16;
        tr[3] = sl[4] | sl[5] << 16;
      }
      const int32_t fw0 = (int32_t)(g.node_g.size() * 8);
      for (int32_t i = 0; i < ns; ++i) rows[nt + i] = c.stat[(size_t)i] & kFw ? fw0 + (c.stat[(size_t)i] & ~kFw) : c.stat[(size_t)i];
      std::copy(c.dep.begin(), c.dep.end(), rows + nt + ns);
      std::fill(rows + nrows, rows + (nrows + 3) / 4 * 4, 0);
      pos += nrows;
      p = e;
    }
    if (!fill) hdr[6] = (int32_t)(row_off / 4);  // row groups of the column (an offset later)
  }
};

bool build_wave_jobs(const Geometry &g, int A, int B, const std::function<int(int, int)> &ring, WaveJobs &wj) {
  wj = WaveJobs{};
  wj.A = A;
  wj.B = B;
  const int64_t ntask = (int64_t)(g.tasks.size() / 8);
  if (ntask <= 0 || ntask > INT32_MAX || A < 2 || B < 2) return false;
  WaveBuilder wb{g, wj, 0, 0, {}, {}, {}, {}, {}, {}, {}, {}};
  // frame coordinates: 0 on the inflow plane of the octant's sign, the swept planes from 1
  const int ux_pos = g.wglob ? 1 : g.xl - 1, ux_neg = g.eglob ? g.Nx : g.xu + 1;
  auto axis = [](int G, int at_pos, int at_neg, std::vector<int32_t> *out) {
    for (int s = 0; s < 2; ++s) {
      out[s].resize((size_t)G);
      for (int X = 0; X < G; ++X) out[s][(size_t)X] = s ? at_neg - (X - 1) : (X - 1) - at_pos;
    }
  };
  axis(g.GX, ux_pos, ux_neg, wb.ux);
  axis(g.GY, 1, g.Ny, wb.vy);
  axis(g.GZ, 1, g.Nz, wb.wz);
  const int umax = std::max(g.xu - ux_pos, ux_neg - g.xl), vmax = g.Ny - 1;
  const int ncu = wb.ncu = std::max(1, (umax + A - 1) / A), ncv = wb.ncv = std::max(1, (vmax + B - 1) / B);
  const int64_t nkeys = (int64_t)8 * ncu * ncv;
  const int nw = ntask < 4096 ? 1 : worker_count();
  const int64_t nnode = (int64_t)g.node_g.size(), GX = g.GX, GXY = (int64_t)g.GX * g.GY;
  wb.xyz.resize((size_t)nnode);
  on_workers(nw, [&](int t) {
    for (int64_t n = nnode * t / nw; n < nnode * (t + 1) / nw; ++n) {
      const int64_t gi = g.node_g[(size_t)n];
      wb.xyz[(size_t)n] = (uint64_t)(gi % GX) | (uint64_t)(gi / GX % g.GY) << 21 | (uint64_t)(gi / GXY) << 42;
    }
  });
  // tasks by column, keeping their order (by hyperplane): counts per worker and key over
  // contiguous parts of the task list, then each worker places its part
  auto key_of = [&](int64_t t) -> int32_t {
    const int32_t *r = &g.tasks[(size_t)t * 8];
    const int o = r[1] & 7;
    const uint64_t q = wb.xyz[(size_t)r[0]];
    const int a = (wb.ux[oct_sx(o) < 0][(size_t)(q & 0x1FFFFF)] - 1) / A;
    const int b = (wb.vy[oct_sy(o) < 0][(size_t)((q >> 21) & 0x1FFFFF)] - 1) / B;
    return (int32_t)(o * (ncu * ncv) + a + ncu * b);
  };
  BigVec<int32_t> key((size_t)ntask);
  std::vector<std::vector<int32_t>> count((size_t)nw, std::vector<int32_t>((size_t)nkeys, 0));
  on_workers(nw, [&](int t) {
    auto &c = count[(size_t)t];
    for (int64_t q = ntask * t / nw; q < ntask * (t + 1) / nw; ++q) c[(size_t)(key[(size_t)q] = key_of(q))]++;
  });
  wb.col_of_key.assign((size_t)nkeys, -1);
  wb.task_begin.assign(1, 0);
  for (int64_t k = 0; k < nkeys; ++k) {
    int64_t at = wb.task_begin.back(), n = 0;
    for (int t = 0; t < nw; ++t) {
      const int32_t c = count[(size_t)t][(size_t)k];
      count[(size_t)t][(size_t)k] = (int32_t)(at + n);
      n += c;
    }
    if (!n) continue;
    wb.col_of_key[(size_t)k] = (int32_t)wb.key_of_col.size();
    wb.key_of_col.push_back((int32_t)k);
    wb.task_begin.push_back(at + n);
  }
  const int ncol = wj.ncol = (int)wb.key_of_col.size();
  wb.order.resize((size_t)ntask);
  on_workers(nw, [&](int t) {
    auto &c = count[(size_t)t];
    for (int64_t q = ntask * t / nw; q < ntask * (t + 1) / nw; ++q) wb.order[(size_t)c[(size_t)key[(size_t)q]]++] = (int32_t)q;
  });
  key.clear();
  key.shrink_to_fit();
  // column headers: first batch, batches, octant, local step of the first batch, the columns
  // upwind in x and y, then (for now) the row groups
  wj.cols.assign((size_t)ncol * 8, 0);
  int64_t nbatch = 0;
  for (int col = 0; col < ncol; ++col) {
    const int k = wb.key_of_col[(size_t)col], o = k / (ncu * ncv), a = k % ncu, b = k / ncu % ncv;
    auto step = [&](int64_t q) {
      const int32_t *r = &g.tasks[(size_t)wb.order[(size_t)q] * 8];
      const uint64_t c = wb.xyz[(size_t)r[0]];
      return wb.ux[oct_sx(o) < 0][(size_t)(c & 0x1FFFFF)] - 1 - a * A + wb.vy[oct_sy(o) < 0][(size_t)((c >> 21) & 0x1FFFFF)] -
             1 - b * B + wb.wz[oct_sz(o) < 0][(size_t)(c >> 42)] - 1;
    };
    int32_t *h = &wj.cols[(size_t)col * 8];
    const int s0 = step(wb.task_begin[(size_t)col]), s1 = step(wb.task_begin[(size_t)col + 1] - 1);
    h[0] = (int32_t)nbatch;
    h[1] = (s1 - s0 + kWaveGroup) / kWaveGroup * kWaveGroup;  // empty batches fill the last group
    h[2] = o;
    h[3] = s0;
    h[4] = a > 0 ? wb.col_of_key[(size_t)(k - 1)] : -1;
    h[5] = b > 0 ? wb.col_of_key[(size_t)(k - ncu)] : -1;
    nbatch += h[1];
  }
  if (nbatch > INT32_MAX / 4) return false;
  wj.batch.assign((size_t)nbatch * 4, 0);
  auto each_column = [&](bool fill) {
    std::atomic<int> next{0};
    on_workers(nw, [&](int) {
      ColumnScan c;
      c.cell.assign((size_t)4 * (A + 2) * (B + 2) * 3, Held{-1, 0, 0});
      for (int col; (col = next.fetch_add(1)) < ncol;) wb.scan(col, c, fill);
    });
  };
  each_column(false);
  // windows of three batches: the rows that have to be on chip at once (a batch's rows are
  // read in the next two)
  int64_t groups = 0;
  int win_rows = 0, max_tasks = 0, max_rows = 0;
  for (int col = 0; col < ncol; ++col) {
    int32_t *h = &wj.cols[(size_t)col * 8];
    int32_t *b = &wj.batch[(size_t)h[0] * 4];
    int64_t at = groups, task = wb.task_begin[(size_t)col];
    int list = 0;
    for (int i = 0; i < h[1]; ++i) {
      int r = 0;
      for (int j = std::max(0, i - 2); j <= i; ++j) r += b[4 * j + 2] & 0xFFFF;
      win_rows = std::max(win_rows, r);
      max_tasks = std::max(max_tasks, b[4 * i + 2] >> 16);
      const int nr = b[4 * i + 2] & 0xFFFF;
      if (i % kWaveGroup == 0) list = 0;
      max_rows = std::max(max_rows, list += (nr + 3) / 4 * 4);
      b[4 * i] = (int32_t)at;
      b[4 * i + 1] = (int32_t)task;
      at += (nr + 3) / 4;
      task += b[4 * i + 2] >> 16;
    }
    groups += h[6];
    h[6] = 0;
  }
  wj.max_rows = max_rows;
  wj.win_rows = win_rows;
  wj.task_ring = 3 * kWaveGroup * max_tasks;  // three groups of the largest batches
  if (groups > INT32_MAX) return false;
  wj.ring = std::min(ring(wj.task_ring, wj.max_rows), 65000);
  if (wj.ring < win_rows) return false;
  wj.rows.resize((size_t)groups * 4);
  wj.tasks.resize((size_t)ntask * 4);
  each_column(true);
  // columns in dependency order: by the x + y column diagonal of the octant's frame
  wj.col_list.resize((size_t)ncol);
  for (int i = 0; i < ncol; ++i) wj.col_list[(size_t)i] = i;
  auto diag = [&](int32_t c) { const int k = wb.key_of_col[(size_t)c]; return k % ncu + k / ncu % ncv; };
  std::stable_sort(wj.col_list.begin(), wj.col_list.end(), [&](int32_t a, int32_t b) { return diag(a) < diag(b); });
  wj.diag.resize((size_t)ncol);
  for (int i = 0; i < ncol; ++i) wj.diag[(size_t)i] = diag(wj.col_list[(size_t)i]);
  return true;
}

}  // namespace piks
