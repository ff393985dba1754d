// node_setup.cpp -- host-side structure of a vertex-level problem assembled
// over its distinct points (nb_nodes.h).
#include <algorithm>

#include "nb_nodes.h"

namespace nb {

void node_setup(const GsMaps &maps, long n, const std::vector<int> &masked, int most_nodes,
                NodeHost &H) {
  // points with one gather-scatter id are one node; points outside the maps
  // are nodes of their own
  std::vector<int> id(n, -1);
  int ids = 0;
  for (int q = 0; q < maps.nlocal; q++) {
    id[maps.gs_dof[q] - 1] = maps.dof_gs[q] - 1;
    ids = std::max(ids, maps.dof_gs[q]);
  }
  std::vector<char> zero(ids, 0);  // a masked copy masks the whole node
  std::vector<char> mine(n, 0);
  for (int q : masked) {
    mine[q] = 1;
    if (id[q] >= 0) zero[id[q]] = 1;
  }
  std::vector<int> node(ids, -1);
  H.node_of.assign(n, -1);
  H.nn = 0;
  for (long i = 0; i < n; i++) {
    if (id[i] < 0) {
      if (!mine[i]) H.node_of[i] = H.nn++;
    } else if (!zero[id[i]]) {
      if (node[id[i]] < 0) node[id[i]] = H.nn++;
      H.node_of[i] = node[id[i]];
    }
  }
  const int nn = H.nn;
  if (nn > most_nodes) return;
  H.eptr.assign(nn + 1, 0);
  for (int v : H.node_of)
    if (v >= 0) H.eptr[v + 1]++;
  for (int v = 0; v < nn; v++) H.eptr[v + 1] += H.eptr[v];
  H.ent.resize(H.eptr[nn]);
  std::vector<int> fill(H.eptr.begin(), H.eptr.end() - 1);
  for (long i = 0; i < n; i++)
    if (H.node_of[i] >= 0) H.ent[fill[H.node_of[i]]++] = (int)i;

  H.slot.assign(8 * H.ent.size(), -1);
  H.soff.assign(1, 0);
  H.col.clear();
  H.col.reserve(27 * (size_t)nn + 27 * 32);
  H.maxw = 0;
  // columns of a row in order of first appearance over its copies' corners;
  // at[v] is the position of node v in the row that stamped it last
  std::vector<int> at(nn), stamp(nn, -1), rows[32];
  for (int r0 = 0; r0 < nn; r0 += 32) {
    int width = 0;
    for (int l = 0; l < 32; l++) {
      std::vector<int> &c = rows[l];
      c.clear();
      const int r = r0 + l;
      if (r >= nn) continue;
      for (int k = H.eptr[r]; k < H.eptr[r + 1]; k++)
        for (int b = 0; b < 8; b++) {
          const int v = H.node_of[(H.ent[k] & ~7) + b];
          if (v < 0) continue;
          if (stamp[v] != r) {
            stamp[v] = r;
            at[v] = (int)c.size();
            c.push_back(v);
          }
          H.slot[8 * (size_t)k + b] = at[v];
        }
      width = std::max(width, (int)c.size());
    }
    const size_t base = H.col.size();
    H.col.resize(base + 32 * (size_t)width);
    for (int l = 0; l < 32; l++) {
      const int own = std::min(r0 + l, nn - 1);
      for (int k = 0; k < width; k++)
        H.col[base + 32 * (size_t)k + l] = k < (int)rows[l].size() ? rows[l][k] : own;
    }
    H.soff.push_back(H.soff.back() + width);
    H.maxw = std::max(H.maxw, width);
  }
}

}  // namespace nb
