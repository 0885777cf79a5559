// Checks nf::build_tiles (netflux_b200/csrc/tiles.cpp) on random cells: every code and list entry must
// lead back to the neighbour, boundary face or vertex that it stands for. Usage:
//   tiles_check CELLS TILE SPREAD SEED THREADS
// SPREAD is how far apart neighbouring cells lie (cells of a well-ordered mesh: a few hundred); THREADS
// is how many threads the system grants before it refuses the next (-1: all).
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../netflux_b200/csrc/tiles.hpp"

static int g_threads = -1;

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
  if (g_threads == 0) return EAGAIN;
  if (g_threads > 0) g_threads--;
  return real(t, a, f, arg);
}

#define REQUIRE(x)                                        \
  do {                                                    \
    if (!(x)) {                                           \
      std::printf("line %d: %s\n", __LINE__, #x);         \
      return 1;                                           \
    }                                                     \
  } while (0)

int main(int argc, char** argv) {
  if (argc != 6) return 2;
  const int n = std::atoi(argv[1]), tile = std::atoi(argv[2]), spread = std::atoi(argv[3]);
  std::mt19937 rng(unsigned(std::atoi(argv[4])));
  const int stride = (n + 63) / 64 * 64;
  constexpr int kNone = 1 << 30;  // a face that no marker lists
  std::vector<int> nbvf(size_t(4) * stride, 0), nbsf(size_t(4) * stride, 0), cnode(size_t(4) * stride, 0),
      gcode(size_t(stride), 0), b_cell;
  std::vector<int> other(size_t(4) * stride, kNone);  // [slot][cell]: cell << 2 | slot, -(1 + boundary face), kNone
  auto at = [&](int c, int q) { return size_t(q) * stride + c; };
  for (int c = 0; c < n; c++)
    for (int q = 0; q < 4; q++) {
      if (other[at(c, q)] != kNone || rng() % 10 == 0) continue;
      const int o = c + 1 + int(rng() % unsigned(spread)), oq = int(rng() % 4);
      if (o < n && other[at(o, oq)] == kNone) {
        other[at(c, q)] = o << 2 | oq;
        other[at(o, oq)] = c << 2 | q;
      }
    }
  for (int c = 0; c < n; c++)
    for (int q = 0; q < 4; q++) {
      if (other[at(c, q)] == kNone && rng() % 2) {  // a boundary face, numbered in the order of the cells
        other[at(c, q)] = -int(b_cell.size()) - 1;
        b_cell.push_back(c);
      }
      const int o = other[at(c, q)];
      nbvf[at(c, q)] = o == kNone ? c : o < 0 ? o : o >> 2;
      nbsf[at(c, q)] = o == kNone ? (c << 2 | q) : o;
      gcode[size_t(c)] |= int(o != kNone ? 1u | (rng() % 4) << 1 : 0u) << (3 * q);
      cnode[at(c, q)] = c / 8 + int(rng() % 60);
    }

  g_threads = std::atoi(argv[5]);
  const nf::Tiles t = nf::build_tiles(n, stride, tile, nbvf, nbsf, cnode, gcode, b_cell);
  REQUIRE(t.tile == tile && t.n_tiles == (n + tile - 1) / tile && int(t.head.size()) == t.n_tiles);
  REQUIRE(t.cut_nb.size() == 4 * t.cut_cell.size());
  int b0 = 0;
  for (int ti = 0; ti < t.n_tiles; ti++) {
    const nf::TileHead& h = t.head[size_t(ti)];
    const int c0 = ti * tile, c1 = std::min(n, c0 + tile), n_states = 4 * tile + h.ncut;
    REQUIRE(h.cut0 % 4 == 0 && h.far0 % 4 == 0 && h.node0 % 4 == 0 && h.b0 == b0);
    b0 += h.nb;
    REQUIRE(size_t(h.cut0 + (h.ncut + 3) / 4 * 4) <= t.cut_cell.size());
    REQUIRE(size_t(h.far0 + (h.nfar + 3) / 4 * 4) <= t.far_id.size());
    REQUIRE(size_t(h.node0 + (h.nnode + 3) / 4 * 4) <= t.node_id.size());
    const int staged = tile + h.ncut + h.nb + h.nfar;
    REQUIRE(staged <= t.max_staged2 && staged - h.nfar <= t.max_staged1 && h.nnode <= t.max_nodes);
    REQUIRE(n_states + h.nb <= t.max_states && staged <= 17 * tile && h.nnode <= 4 * tile);
    // the cell (or -(1 + boundary face)) behind a staged number
    auto behind = [&](int s) {
      if (s < tile) return c0 + s;
      if (s < tile + h.ncut) return t.cut_cell[size_t(h.cut0 + s - tile)];
      if (s < tile + h.ncut + h.nb) return -(1 + h.b0 + s - tile - h.ncut);
      return t.far_id[size_t(h.far0 + s - tile - h.ncut - h.nb)];
    };
    bool open = false;
    for (int c = c0; c < c1; c++)
      for (int q = 0; q < 4; q++) {
        const int o = other[at(c, q)], code = t.code[size_t(4) * c + q];
        open = open || o == kNone;
        if (o == kNone) {
          REQUIRE(code == nf::kFaceNone);
        } else {
          REQUIRE(code < n_states + h.nb);
          REQUIRE(behind(nf::staged_of(code, tile)) == (o < 0 ? o : o >> 2));
          if (code < 4 * tile) REQUIRE(code / tile == (o & 3));
          else if (code < n_states) REQUIRE(t.cut_nb[4 * size_t(h.cut0 + code - 4 * tile)] >> 14 == (o & 3));
        }
        const int v = t.vert[size_t(4) * c + q], bits = gcode[size_t(c)] >> (3 * q);
        REQUIRE((v & nf::kVertIndex) < h.nnode);
        REQUIRE(t.node_id[size_t(h.node0 + (v & nf::kVertIndex))] == cnode[at(c, q)]);
        REQUIRE(((v & nf::kVertFlip) != 0) == ((bits & 2) != 0) && ((v & nf::kVertSide) != 0) == ((bits & 4) != 0));
      }
    for (int i = 0; i < h.ncut; i++) {
      const int x = t.cut_cell[size_t(h.cut0 + i)];
      REQUIRE(x >= 0 && x < n && !(x >= c0 && x < c1));
      for (int q = 0; q < 4; q++) {
        const int o = other[at(x, q)], s = t.cut_nb[4 * size_t(h.cut0 + i) + q] & (q == 0 ? 0x3fff : 0xffff);
        open = open || o == kNone;
        REQUIRE(s < staged);
        if (o == kNone) REQUIRE(s == tile + i);
        else REQUIRE(behind(s) == (o < 0 ? o : o >> 2));
      }
    }
    REQUIRE((h.open != 0) == open);
  }
  REQUIRE(b0 == int(b_cell.size()));
  std::printf("tiles ok\n");
  return 0;
}
