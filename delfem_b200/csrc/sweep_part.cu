// Row partition of the range sweeps made from the factor's own pattern.
//
// What crosses CTAs costs about 1 us on the level path (a store to L2, a poll,
// a store to shared memory).  Once per pair of neighbouring CTAs that is a lag
// and no more, as long as the dependencies between the two go one way: both
// then run at the speed of their own rounds.  Where two CTAs read each other's
// rows, every level waits for the other one (measured on a 100x20x20 box cut
// by the coordinates of its jittered nodes, whose cuts zigzag: rounds of 1 us
// instead of 0.26).  So the parts are cut along monotone directions that the
// dependencies themselves give:
//
//   chains  a row continues the chain of the nearest row it reads that is one
//           level below it and has no continuation yet;
//   lines   the same among the chains (by their depth in the order in which
//           chains read each other): a chain has a line and a position in it.
//
// In a lexicographically numbered grid the chains are its x lines, a line is an
// xy plane of them and the position is y.  Parts are blocks of consecutive
// lines and positions: every dependency goes to the same or a later block in
// both.  In a plane grid all chains form one line, and the parts are strips.
#include <algorithm>
#include <cmath>

#include "dfm_internal.h"

namespace dfm {

constexpr unsigned kNone = 0xffffffffu;

// M->own_of: a partition into at most G parts (M->own_n of them), see above.
int sweep_own_partition(dfm_ilu M, unsigned G) {
  if (M->own_for == G && G) return DFM_OK;
  M->own_for = 0;
  const unsigned N = M->N;
  const std::vector<unsigned>& rp = M->A->h_rowptr;
  const std::vector<unsigned>& ci = M->A->h_colind;
  // chains, numbered by their first rows
  std::vector<unsigned> chain(N, kNone);
  std::vector<unsigned char> taken(N, 0);
  unsigned nc = 0;
  for (unsigned i = 0; i < N; i++) {
    unsigned from = kNone;
    for (unsigned s = M->h_diaind[i]; s-- > rp[i] && from == kNone;)
      if (M->lev_f[ci[s]] + 1 == M->lev_f[i] && !taken[ci[s]]) from = ci[s];
    if (from == kNone) {
      chain[i] = nc++;
    } else {
      taken[from] = 1;
      chain[i] = chain[from];
    }
  }
  // the earlier chains each chain reads
  std::vector<unsigned> ptr(nc + 1, 0), rows(N), mark(nc, kNone), pred, pptr(nc + 1, 0);
  for (unsigned c : chain) ptr[c + 1]++;
  for (unsigned c = 0; c < nc; c++) ptr[c + 1] += ptr[c];
  {
    std::vector<unsigned> fill(ptr.begin(), ptr.end() - 1);
    for (unsigned i = 0; i < N; i++) rows[fill[chain[i]]++] = i;
  }
  for (unsigned c = 0; c < nc; c++) {
    for (unsigned k = ptr[c]; k < ptr[c + 1]; k++)
      for (unsigned s = rp[rows[k]]; s < M->h_diaind[rows[k]]; s++) {
        const unsigned d = chain[ci[s]];
        if (d >= c || mark[d] == c) continue;
        mark[d] = c;
        pred.push_back(d);
      }
    std::sort(pred.begin() + pptr[c], pred.end());
    pptr[c + 1] = (unsigned)pred.size();
  }
  // lines, numbered by their first chains
  std::vector<unsigned> depth(nc, 0), line(nc, kNone), pos(nc, 0);
  taken.assign(nc, 0);
  unsigned nl = 0, npos = 0;
  for (unsigned c = 0; c < nc; c++) {
    for (unsigned k = pptr[c]; k < pptr[c + 1]; k++) depth[c] = std::max(depth[c], depth[pred[k]] + 1);
    unsigned from = kNone;
    for (unsigned k = pptr[c + 1]; k-- > pptr[c] && from == kNone;)
      if (depth[pred[k]] + 1 == depth[c] && !taken[pred[k]]) from = pred[k];
    if (from == kNone) {
      line[c] = nl++;
    } else {
      taken[from] = 1;
      line[c] = line[from];
      pos[c] = pos[from] + 1;
    }
    npos = std::max(npos, pos[c] + 1);
  }
  // gl bands of lines x gp ranges of positions, blocks about as many lines as positions
  G = std::max(G, 1u);
  unsigned gl = 1, gp = 1;
  const double want = nc ? std::sqrt((double)G * nl / std::max(1.0, (double)nc / nl)) : 1.0;
  for (int d = -1; d <= 1; d++) {
    const unsigned a = std::min({(unsigned)std::max(1.0, std::floor(want + 0.5) + d), std::max(nl, 1u), G});
    const unsigned b = std::min(G / a, std::max(npos, 1u));
    if (a * b > gl * gp) {
      gl = a;
      gp = b;
    }
  }
  std::vector<unsigned long long> wl(nl + 1, 0), wp(npos + 1);
  std::vector<unsigned> band(nl), cut(npos);
  for (unsigned c = 0; c < nc; c++) wl[line[c] + 1] += ptr[c + 1] - ptr[c];
  for (unsigned l = 0; l < nl; l++) wl[l + 1] += wl[l];
  for (unsigned l = 0; l < nl; l++)  // the band of a line's middle weight
    band[l] = (unsigned)std::min<unsigned long long>(gl - 1, (wl[l] + wl[l + 1]) * gl / (2 * std::max(1u, N)));
  std::vector<std::vector<unsigned>> of_band(gl);
  for (unsigned c = 0; c < nc; c++) of_band[band[line[c]]].push_back(c);
  M->own_of.assign(N, 0);
  for (unsigned b = 0; b < gl; b++) {
    std::fill(wp.begin(), wp.end(), 0);
    for (unsigned c : of_band[b]) wp[pos[c] + 1] += ptr[c + 1] - ptr[c];
    for (unsigned p = 0; p < npos; p++) wp[p + 1] += wp[p];
    for (unsigned p = 0; p < npos; p++)
      cut[p] = (unsigned)std::min<unsigned long long>(
          gp - 1, (wp[p] + wp[p + 1]) * gp / (2 * std::max<unsigned long long>(1, wp[npos])));
    for (unsigned c : of_band[b])
      for (unsigned k = ptr[c]; k < ptr[c + 1]; k++) M->own_of[rows[k]] = b * gp + cut[pos[c]];
  }
  M->own_n = gl * gp;
  M->own_for = G;
  return DFM_OK;
}

}  // namespace dfm
