// Tiles of the fast forms' stage kernel: a tile is kTile consecutive cells of
// the device order (compact, because that order is a space-filling curve) with
// the lists the kernel needs to hold everything the tile reads in shared memory.
#pragma once

#include <cstdint>
#include <vector>

namespace nf {

// One tile's slices of the lists below. The lists of a tile start on multiples of
// four entries (16 bytes or more).
struct TileHead {
  int cut0, ncut;    // faces between a cell of the tile and a cell outside it
  int far0, nfar;    // further cells and ghosts the outside cells of those faces touch
  int b0, nb;        // boundary faces of the tile's cells (consecutive in owner order)
  int node0, nnode;  // vertices of the tile's cells
  int open;          // some cell of the tile or of its cut faces has a face no marker lists
  int case_id;       // the case all its cells belong to, -1: several (filled by the caller)
  int pad[2];
};

// Face codes of a cell (16 bits, face m opposite vertex m): the number of what
// is on the face's other side. Face states are numbered q * tile + t for face q
// of the tile's cell t, then one per cut face, then one per boundary face (its
// flux); kFaceNone is a face no marker lists. The staged number of the other
// side follows from the code (staged_of).
constexpr uint16_t kFaceNone = 0xffff;
// Vertex codes of a cell: the vertex's place in the tile's vertex list, and for
// the face opposite it whether the normal of its ascending vertices points
// into the cell (kVertFlip) and whether the cell is on the neighbour's side
constexpr uint16_t kVertIndex = 0x3fff, kVertSide = 0x4000, kVertFlip = 0x8000;

// Staged values are numbered: the tile's cells, one per cut face (its outside
// cell), the tile's boundary faces (their ghosts), then the far list.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int staged_of(int code, int tile) { return code < 4 * tile ? code % tile : code - 3 * tile; }
struct Tiles {
  int tile = 0, n_tiles = 0;
  int max_staged1 = 0;  // cells, cut faces and ghosts of any tile
  int max_staged2 = 0;  // the same with the far list (second order)
  int max_nodes = 0;
  int max_states = 0;   // 4 tile + cut + boundary faces of any tile
  std::vector<TileHead> head;
  std::vector<uint16_t> code;      // [n_tiles * tile][4]
  std::vector<uint16_t> vert;      // [n_tiles * tile][4]
  std::vector<int> cut_cell;       // outside cell of each cut face
  std::vector<uint16_t> cut_nb;    // [.][4] staged numbers of its neighbours (itself: no face);
                                   // bits 14-15 of the first: which of them the cut face is
  std::vector<int> far_id;         // cell, or -(1 + boundary face)
  std::vector<int> node_id;
};

// nbvf, nbsf, cnode: [4][stride], gcode: [stride] (the node-based layout of
// nf_create); b_cell: owner cell of each boundary face, ascending.
Tiles build_tiles(int n, int stride, int tile, const std::vector<int>& nbvf, const std::vector<int>& nbsf,
                  const std::vector<int>& cnode, const std::vector<int>& gcode, const std::vector<int>& b_cell);

}  // namespace nf
