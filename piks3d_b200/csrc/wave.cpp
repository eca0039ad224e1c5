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

constexpr int kFw = 1 << 30;

// A row that a column holds: its code and where it stands (batch, list, index in the list).
struct Held { int32_t code, batch, idx; };   // idx | list << 28 (0 own, 1 static, 2 dependent)

// Scratch of one worker for the batches of a column.
struct ColumnScan {
  // rows by voxel (four z layers of the cross-section with its two upwind layers) and
  // variant: 0 the octant's own slot, 1 / 2 what a y / z reader finds in a wall
  std::vector<Held> cell;
  std::vector<int32_t> stat, dep;
  std::vector<int32_t> refs;      // the six reads of each task of a batch: back << 30 | list << 28 | index, -1 none
  std::vector<int32_t> rows;      // the row lists of the worker's columns
  int32_t own[4], ns[4];          // own rows and static rows of the last four batches
  int64_t pos[4];                 // ring position of their first row
  int32_t stamp = 0;              // batches scanned so far, over all columns
};

}  // namespace

struct WaveBuilder {
  const Geometry &g;
  WaveJobs &wj;
  int ncu, ncv;                                // columns per octant along x and y
  std::vector<int32_t> ux[2], vy[2], wz[2];    // frame coordinates by ghosted coordinate, sign + / -
  BigVec<uint64_t> xyz;
  BigVec<int32_t> order;
  std::vector<int32_t> col_of_key, key_of_col;
  std::vector<int64_t> task_begin;
  std::vector<ColumnScan> scratch;             // by worker
  std::vector<std::pair<int32_t, int64_t>> rows_at;  // worker and offset of each column's row list

  // One column's batches, row list and records. The ring's size is not known yet: a record
  // holds the distance of a read's row from the first row two batches back, plus one.
  void scan(int col, int worker) {
    ColumnScan &c = scratch[(size_t)worker];
    const int A = wj.A, B = wj.B;
    const int key = key_of_col[(size_t)col];
    const int o = key / (ncu * ncv), ka = key % ncu, kb = key / ncu % ncv;
    const int32_t *tu = ux[oct_sx(o) < 0].data(), *tv = vy[oct_sy(o) < 0].data(), *tw = wz[oct_sz(o) < 0].data();
    const int u0 = 1 + ka * A, v0 = 1 + kb * B;
    const int64_t t1 = task_begin[(size_t)col + 1];
    int32_t *hdr = &wj.cols[(size_t)col * 8];
    const int s_first = hdr[3];
    int64_t batch = hdr[0], p = task_begin[(size_t)col], pos = 0;  // pos: rows of the column so far
    const int stride_v = A + 2, stride_w = (A + 2) * (B + 2);
    const int32_t first_stamp = c.stamp + 1;
    const int64_t row0 = (int64_t)c.rows.size();
    rows_at[(size_t)col] = {worker, row0};
    auto where = [&](int32_t node, int &lu, int &lv, int &w) {
      const uint64_t q = xyz[(size_t)node];
      lu = tu[q & 0x1FFFFF] - u0;
      lv = tv[(q >> 21) & 0x1FFFFF] - v0;
      w = tw[q >> 42];
    };
    const int32_t fw0 = (int32_t)(g.node_g.size() * 8);
    for (int s = s_first; s < s_first + hdr[1]; ++s, ++batch) {
      const int32_t k = ++c.stamp;
      int64_t e = p;
      const int64_t list0 = (int64_t)c.rows.size();
      for (; e < t1; ++e) {
        int lu, lv, w;
        const int32_t *r = &g.tasks[(size_t)order[(size_t)e] * 8];
        where(r[0], lu, lv, w);
        if (lu + lv + w - 1 != s) break;
        const int32_t code = r[0] * 8 + o;
        c.cell[(size_t)(((w & 3) * stride_w + (lv + 2) * stride_v + lu + 2) * 3)] = {code, k, (int32_t)(e - p)};
        c.rows.push_back(code);
      }
      const int32_t nt = (int32_t)(e - p);
      c.stat.clear();
      c.dep.clear();
      c.refs.resize((size_t)nt * 6);
      for (int64_t q = p; q < e; ++q) {
        const int32_t *r = &g.tasks[(size_t)order[(size_t)q] * 8];
        int32_t *ref = &c.refs[(size_t)(q - p) * 6];
        int lu, lv, w;
        where(r[0], lu, lv, w);
        for (int j = 0; j < 6; ++j) {
          const int32_t code = r[2 + j];
          if (code < 0) { ref[j] = -1; continue; }
          // the row of the read: one the column's last batches hold, or a new one of this batch
          const int axis = j >> 1, back = 1 + (j & 1);
          const int cu = axis == 0 ? lu - back : lu, cv = axis == 1 ? lv - back : lv, cw = axis == 2 ? w - back : w;
          const bool fw = code & kFw;
          const int variant = !fw && (code & 7) == o ? 0 : axis;
          Held &h = c.cell[(size_t)(((cw & 3) * stride_w + (cv + 2) * stride_v + cu + 2) * 3 + variant)];
          if (h.code != code || h.batch < first_stamp || h.batch < k - 2) {
            // swept by an upwind column: a fluid node of this octant past the inflow plane
            const bool swept = !fw && (code >> 3) < g.NF &&
                               (axis == 0 ? u0 + cu >= 1 : axis == 1 ? v0 + cv >= 1 : cw >= 1);
            std::vector<int32_t> &list = swept ? c.dep : c.stat;
            h = {code, k, (int32_t)list.size() | (swept ? 2 : 1) << 28};
            list.push_back(fw ? fw0 + (code & ~kFw) : code);
          }
          ref[j] = (int32_t)((uint32_t)(k - h.batch) << 30 | (uint32_t)h.idx);
        }
      }
      const int32_t ns = (int32_t)c.stat.size(), nd = (int32_t)c.dep.size(), nrows = nt + ns + nd;
      c.rows.insert(c.rows.end(), c.stat.begin(), c.stat.end());
      c.rows.insert(c.rows.end(), c.dep.begin(), c.dep.end());
      c.rows.resize((size_t)(list0 + (nrows + 3) / 4 * 4), 0);
      int32_t *b = &wj.batch[(size_t)batch * 4];
      b[2] = nrows | nt << 16;
      b[3] = nt + ns;
      c.own[k & 3] = nt;
      c.ns[k & 3] = ns;
      c.pos[k & 3] = pos;
      int32_t from[3][3];  // by batches back and list: 1 + the position of its first row past the base
      const int64_t base = c.pos[std::max(first_stamp, k - 2) & 3];
      for (int back = 0; back < 3 && k - back >= first_stamp; ++back) {
        const int m = (k - back) & 3;
        from[back][0] = (int32_t)(1 + c.pos[m] - base);
        from[back][1] = from[back][0] + c.own[m];
        from[back][2] = from[back][1] + c.ns[m];
      }
      for (int64_t q = p; q < e; ++q) {
        const int32_t *r = &g.tasks[(size_t)order[(size_t)q] * 8], *ref = &c.refs[(size_t)(q - p) * 6];
        uint32_t sl[6];
        for (int j = 0; j < 6; ++j) {
          const uint32_t v = (uint32_t)ref[j];
          sl[j] = ref[j] == -1 ? 0u : (uint32_t)from[v >> 30][v >> 28 & 3] + (v & 0xFFFFFFF);
        }
        const int fl = r[1];
        int32_t *tr = &wj.tasks[(size_t)q * 4];
        tr[0] = r[0] | ((fl & 8) ? 1 << 27 : 0) | ((fl & 16) ? 1 << 28 : 0) | ((fl & 32) ? 1 << 29 : 0);
        for (int j = 0; j < 3; ++j) tr[1 + j] = (int32_t)(sl[2 * j] | sl[2 * j + 1] << 16);
      }
      pos += nrows;
      p = e;
    }
    hdr[6] = (int32_t)(((int64_t)c.rows.size() - row0) / 4);  // row groups of the column (an offset later)
  }

  // The column's row list to its place, its records' distances to ring slots.
  void place(int col) {
    const int32_t *hdr = &wj.cols[(size_t)col * 8];
    int32_t *b = &wj.batch[(size_t)hdr[0] * 4];
    const auto &[worker, row0] = rows_at[(size_t)col];
    const int32_t *rows = scratch[(size_t)worker].rows.data() + row0;
    std::copy(rows, rows + (int64_t)hdr[6] * 4, &wj.rows[(size_t)b[0] * 4]);
    const uint32_t R = (uint32_t)wj.ring;
    uint32_t at = 0, start[3] = {0, 0, 0};  // positions (mod R) of the batch and the two before it
    for (int i = 0; i < hdr[1]; ++i, b += 4) {
      start[2] = i > 1 ? start[1] : 0; start[1] = i > 0 ? start[0] : 0; start[0] = at;
      b[3] |= (int32_t)(1 + at) << 16;
      int32_t *tr = &wj.tasks[(size_t)b[1] * 4];
      const uint32_t base = start[2];
      // a window of three batches is at most the ring: one wrap
      auto slot = [&](uint32_t d) { return d == 0 ? 0u : base + d > R ? base + d - R : base + d; };
      for (int32_t q = 0; q < b[2] >> 16; ++q, tr += 4)
        for (int j = 1; j < 4; ++j) {
          const uint32_t v = (uint32_t)tr[j];
          tr[j] = (int32_t)(slot(v & 0xFFFF) | slot(v >> 16) << 16);
        }
      at = (at + (uint32_t)(b[2] & 0xFFFF)) % R;
    }
  }
};

bool build_wave_jobs(const Geometry &g, int A, int B, const std::function<int(int, int)> &ring, WaveJobs &wj) {
  wj = WaveJobs{};
  wj.A = A;
  wj.B = B;
  const int64_t ntask = (int64_t)(g.tasks.size() / 8);
  // (the distances of a window of three batches have to fit 16 bits)
  if (ntask <= 0 || ntask > INT32_MAX || A < 2 || B < 2 || A * B > 2048) return false;
  WaveBuilder wb{g, wj, 0, 0, {}, {}, {}, {}, {}, {}, {}, {}, {}, {}};
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
  on_threads(nw, [&](int t) {
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
  on_threads(nw, [&](int t) {
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
  on_threads(nw, [&](int t) {
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
  wj.tasks.resize((size_t)ntask * 4);
  wb.scratch.resize((size_t)nw);
  wb.rows_at.resize((size_t)ncol);
  std::atomic<int> next{0};
  on_threads(nw, [&](int t) {
    wb.scratch[(size_t)t].cell.assign((size_t)4 * (A + 2) * (B + 2) * 3, Held{-1, 0, 0});
    for (int col; (col = next.fetch_add(1)) < ncol;) wb.scan(col, t);
  });
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
  }
  wj.max_rows = max_rows;
  wj.win_rows = win_rows;
  wj.task_ring = 3 * kWaveGroup * max_tasks;  // three groups of the largest batches
  if (groups > INT32_MAX) return false;
  wj.ring = std::min(ring(wj.task_ring, wj.max_rows), 65000);
  if (wj.ring < win_rows) return false;
  wj.rows.resize((size_t)groups * 4);
  next = 0;
  on_threads(nw, [&](int) {
    for (int col; (col = next.fetch_add(1)) < ncol;) wb.place(col);
  });
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
