// Builds the tiles of the fast forms' stage kernel (tiles.hpp) on host threads;
// tiles are independent, so every thread builds a range of them.
#include "tiles.hpp"

#include <algorithm>
#include <exception>
#include <mutex>
#include <stdexcept>
#include <system_error>
#include <thread>
#include <utility>

#include "mesh.hpp"

namespace nf {

namespace {

// Numbers of the staged cells and ghosts outside the tile, by open addressing.
class Places {
 public:
  explicit Places(size_t most) {
    size_t n = 64;
    while (n < 2 * most) n *= 2;
    key_.assign(n, kEmpty);
    val_.resize(n);
  }
  int* find(int key, bool* fresh) {
    size_t i = (uint32_t(key) * 2654435769u) & (key_.size() - 1);
    while (key_[i] != kEmpty && key_[i] != key) i = (i + 1) & (key_.size() - 1);
    *fresh = key_[i] == kEmpty;
    if (*fresh) {
      key_[i] = key;
      used_.push_back(i);
    }
    return &val_[i];
  }
  void clear() {
    for (size_t i : used_) key_[i] = kEmpty;
    used_.clear();
  }

 private:
  static constexpr int kEmpty = INT32_MIN;
  std::vector<int> key_, val_;
  std::vector<size_t> used_;
};

}  // namespace

Tiles build_tiles(int n, int stride, int tile, const std::vector<int>& nbvf, const std::vector<int>& nbsf,
                  const std::vector<int>& cnode, const std::vector<int>& gcode, const std::vector<int>& b_cell) {
  Tiles all;
  all.tile = tile;
  all.n_tiles = (n + tile - 1) / tile;
  all.head.resize(size_t(all.n_tiles));
  all.code.assign(size_t(4) * all.n_tiles * tile, kFaceNone);
  all.vert.assign(size_t(4) * all.n_tiles * tile, 0);
  const int n_threads = std::max(1, std::min(build_threads(size_t(n)), all.n_tiles / 16));
  std::vector<Tiles> part(static_cast<size_t>(n_threads));
  std::exception_ptr failed;
  std::mutex failed_mutex;

  auto build = [&](int w) {
    Tiles& p = part[size_t(w)];
    const int t0 = int(int64_t(all.n_tiles) * w / n_threads), t1 = int(int64_t(all.n_tiles) * (w + 1) / n_threads);
    Places places(size_t(16) * tile), nodes(size_t(4) * tile);
    struct Cut {
      int cell, slot, t, q;
    };
    std::vector<Cut> cuts;
    std::vector<int> far;
    for (int ti = t0; ti < t1; ti++) {
      const int c0 = ti * tile, c1 = std::min(n, c0 + tile);
      TileHead h{};
      h.b0 = int(std::lower_bound(b_cell.begin(), b_cell.end(), c0) - b_cell.begin());
      h.nb = int(std::lower_bound(b_cell.begin(), b_cell.end(), c1) - b_cell.begin()) - h.b0;
      auto present = [&](int c, int q) { return (gcode[size_t(c)] >> (3 * q) & 1) != 0; };
      // the tile's own faces
      cuts.clear();
      for (int c = c0; c < c1; c++)
        for (int q = 0; q < 4; q++) {
          uint16_t& code = all.code[size_t(4) * c + q];
          if (!present(c, q)) {
            h.open = 1;
            continue;
          }
          const int o = nbvf[size_t(q) * stride + c];
          if (o < 0) code = 1;  // numbered below, once the cut faces are known
          else if (o >= c0 && o < c1) code = uint16_t((nbsf[size_t(q) * stride + c] & 3) * tile + (o - c0));
          else cuts.push_back({o, nbsf[size_t(q) * stride + c] & 3, c - c0, q});
        }
      std::sort(cuts.begin(), cuts.end(), [](const Cut& x, const Cut& y) {
        return x.cell != y.cell ? x.cell < y.cell : x.slot < y.slot;
      });
      h.cut0 = int(p.cut_cell.size());
      h.ncut = int(cuts.size());
      places.clear();
      for (int i = 0; i < h.ncut; i++) {
        const Cut& x = cuts[size_t(i)];
        all.code[size_t(4) * (c0 + x.t) + x.q] = uint16_t(4 * tile + i);
        p.cut_cell.push_back(x.cell);
        bool fresh;
        int* at = places.find(x.cell, &fresh);
        if (fresh) *at = tile + i;
      }
      for (int c = c0; c < c1; c++)
        for (int q = 0; q < 4; q++)
          if (present(c, q) && nbvf[size_t(q) * stride + c] < 0)
            all.code[size_t(4) * c + q] = uint16_t(4 * tile + h.ncut + (-nbvf[size_t(q) * stride + c] - 1 - h.b0));
      // what the outside cells touch beyond the staged values so far
      far.clear();
      const int base = tile + h.ncut + h.nb;
      for (const Cut& x : cuts)
        for (int q = 0; q < 4; q++) {
          if (!present(x.cell, q)) {
            h.open = 1;
            continue;
          }
          const int o = nbvf[size_t(q) * stride + x.cell];
          if (o >= c0 && o < c1) continue;
          bool fresh;
          places.find(o, &fresh);
          if (fresh) far.push_back(o);
        }
      std::sort(far.begin(), far.end());
      for (size_t i = 0; i < far.size(); i++) {
        bool fresh;
        *places.find(far[i], &fresh) = base + int(i);
      }
      h.far0 = int(p.far_id.size());
      h.nfar = int(far.size());
      p.far_id.insert(p.far_id.end(), far.begin(), far.end());
      for (int i = 0; i < h.ncut; i++) {
        const Cut& x = cuts[size_t(i)];
        for (int q = 0; q < 4; q++) {
          const int o = present(x.cell, q) ? nbvf[size_t(q) * stride + x.cell] : x.cell;
          bool fresh;
          int at = !present(x.cell, q) ? tile + i : (o >= c0 && o < c1) ? o - c0 : *places.find(o, &fresh);
          if (at > kVertIndex) throw std::runtime_error("tile lists too long");
          if (q == 0) at |= x.slot << 14;
          p.cut_nb.push_back(uint16_t(at));
        }
      }
      // vertices
      nodes.clear();
      far.clear();
      for (int c = c0; c < c1; c++)
        for (int q = 0; q < 4; q++) {
          bool fresh;
          nodes.find(cnode[size_t(q) * stride + c], &fresh);
          if (fresh) far.push_back(cnode[size_t(q) * stride + c]);
        }
      std::sort(far.begin(), far.end());
      for (size_t i = 0; i < far.size(); i++) {
        bool fresh;
        *nodes.find(far[i], &fresh) = int(i);
      }
      h.node0 = int(p.node_id.size());
      h.nnode = int(far.size());
      p.node_id.insert(p.node_id.end(), far.begin(), far.end());
      for (int c = c0; c < c1; c++)
        for (int q = 0; q < 4; q++) {
          const int bits = gcode[size_t(c)] >> (3 * q);
          bool fresh;
          all.vert[size_t(4) * c + q] = uint16_t(*nodes.find(cnode[size_t(q) * stride + c], &fresh) |
                                                 ((bits & 4) ? kVertSide : 0) | ((bits & 2) ? kVertFlip : 0));
        }
      // the next tile's lists start on multiples of four entries
      while (p.cut_cell.size() % 4) {
        p.cut_cell.push_back(0);
        p.cut_nb.insert(p.cut_nb.end(), 4, 0);
      }
      while (p.far_id.size() % 4) p.far_id.push_back(0);
      while (p.node_id.size() % 4) p.node_id.push_back(0);
      p.max_staged1 = std::max(p.max_staged1, base);
      p.max_staged2 = std::max(p.max_staged2, base + h.nfar);
      p.max_nodes = std::max(p.max_nodes, h.nnode);
      p.max_states = std::max(p.max_states, 4 * tile + h.ncut + h.nb);
      all.head[size_t(ti)] = h;
    }
  };
  auto guarded = [&](int w) {
    try {
      build(w);
    } catch (...) {
      std::lock_guard<std::mutex> lock(failed_mutex);
      failed = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(size_t(n_threads));
  for (int w = 1; w < n_threads; w++) {
    try {
      pool.emplace_back(guarded, w);
    } catch (const std::system_error&) {  // no further thread: its range by this one
      guarded(w);
    }
  }
  guarded(0);
  for (auto& th : pool) th.join();
  if (failed) std::rethrow_exception(failed);

  // the threads' lists one after another; each tile's offsets moved along
  for (int w = 0; w < n_threads; w++) {
    const Tiles& p = part[size_t(w)];
    const int t0 = int(int64_t(all.n_tiles) * w / n_threads), t1 = int(int64_t(all.n_tiles) * (w + 1) / n_threads);
    for (int ti = t0; ti < t1; ti++) {
      TileHead& h = all.head[size_t(ti)];
      h.cut0 += int(all.cut_cell.size());
      h.far0 += int(all.far_id.size());
      h.node0 += int(all.node_id.size());
    }
    all.cut_cell.insert(all.cut_cell.end(), p.cut_cell.begin(), p.cut_cell.end());
    all.cut_nb.insert(all.cut_nb.end(), p.cut_nb.begin(), p.cut_nb.end());
    all.far_id.insert(all.far_id.end(), p.far_id.begin(), p.far_id.end());
    all.node_id.insert(all.node_id.end(), p.node_id.begin(), p.node_id.end());
    all.max_staged1 = std::max(all.max_staged1, p.max_staged1);
    all.max_staged2 = std::max(all.max_staged2, p.max_staged2);
    all.max_nodes = std::max(all.max_nodes, p.max_nodes);
    all.max_states = std::max(all.max_states, p.max_states);
  }
  return all;
}

}  // namespace nf
