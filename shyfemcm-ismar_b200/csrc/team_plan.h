// team_plan.h -- how the resident solver (k_zeta_team.cuh) deals the rows of
// one system to the CTAs of its team: compact shares by bisection of the
// plane, their ghosts, local columns and tails.  Host code alone but for the
// packing of a row's diagonal place; no CUDA header, so that it compiles with
// a plain C++ compiler.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <thread>
#include <vector>

#ifdef __CUDACC__
#define SHY_HD __host__ __device__ __forceinline__
#else
#define SHY_HD inline
#endif

namespace shy {

// what a CTA of the resident solver holds
struct TeamShape {
  int rows;      // rows at most (the first place of a ghost)
  int ghosts;    // ghost copies at most
  int entries;   // off-diagonal entries in a row's block
  int capacity;  // CTAs that fit the device at once (0 on error)
};

// the place of the diagonal among a row's CSR slots and the count of the
// other slots, 16 bits each: a row's columns are rows and ghosts of one
// share, at most 2560 (shares with more ghosts are refused before a row is
// packed)
SHY_HD int dpos_pack(int place, int count) { return place | count << 16; }
SHY_HD int dpos_place(int v) { return v & 0xffff; }
SHY_HD int dpos_count(int v) { return (int)((unsigned)v >> 16); }

// fn(i) for i = 0 .. n-1 on up to nt threads, the caller's among them; false
// when a call threw.  Threads that the system refuses are done without.
template <class F>
inline bool on_threads(int n, int nt, F fn) {
  std::atomic<int> next{0};
  std::atomic<bool> ok{true};
  auto work = [&] {
    try {
      for (int i; (i = next++) < n;) fn(i);
    } catch (...) {
      ok = false;
    }
  };
  std::vector<std::thread> pool;
  try {
    for (int q = 1; q < std::min(n, nt); q++) pool.emplace_back(work);
  } catch (...) {
  }
  work();
  for (std::thread &t : pool) t.join();
  return ok;
}

// a row with its place in the plane
struct PlaneRow { float x[2]; int i; };

// rows v[0, n) cut into T compact patches of nearly equal size by recursive
// bisection, across the longer side; patch r holds v[cut[r], cut[r+1]),
// rows in order (gathers of neighbours stay local); `at` is v's place
inline void bisect_rows(PlaneRow *v, int n, int at, int r, int T, int *cut) {
  if (T == 1) {
    cut[r] = at;
    std::sort(v, v + n, [](const PlaneRow &p, const PlaneRow &q) { return p.i < q.i; });
    return;
  }
  float a[2] = {INFINITY, INFINITY}, b[2] = {-INFINITY, -INFINITY};
  for (int i = 0; i < n; i++)
    for (int c = 0; c < 2; c++) { a[c] = std::min(a[c], v[i].x[c]); b[c] = std::max(b[c], v[i].x[c]); }
  const int c = b[1] - a[1] > b[0] - a[0] ? 1 : 0;
  const int T1 = T / 2, mid = (int)((long long)n * T1 / T);
  std::nth_element(v, v + mid, v + n, [c](const PlaneRow &p, const PlaneRow &q) {
    return p.x[c] != q.x[c] ? p.x[c] < q.x[c] : p.i < q.i;
  });
  bisect_rows(v, mid, at, r, T1, cut);
  bisect_rows(v + mid, n - mid, at + mid, r + T1, T - T1, cut);
}

// what the resident solver needs to know of one basin (rows k0 .. k0+nk-1)
struct TeamBasin {
  std::vector<int> cut;                            // first row of each share, and nk
  std::vector<int> ghost, gptr;                    // ghosts of the shares, offsets
  std::vector<int> tcount, tslot;                  // rows' tail lengths, tail slots
  std::vector<unsigned short> tcol;
  std::vector<int> rows, dpos;
  std::vector<unsigned short> lcol;                // K columns a row
  int most = 0;                                    // most ghosts of a share
};

// shares of the rows k0 .. k0+nk-1 of the CSR pattern with coordinates xy
inline void team_basin(const int *rowptr, const int *col, const float *xy, int k0, int nk, int T, const TeamShape &sh,
                       TeamBasin &B) {
  const int K = sh.entries;
  std::vector<PlaneRow> v(nk);
  for (int j = 0; j < nk; j++) {         // NaN has no place in the order that bisect_rows needs
    const float *p = xy + 2 * (size_t)(k0 + j);
    v[j] = PlaneRow{{p[0] == p[0] ? p[0] : 0.f, p[1] == p[1] ? p[1] : 0.f}, k0 + j};
  }
  B.cut.assign(T + 1, nk);
  bisect_rows(v.data(), nk, 0, 0, T, B.cut.data());
  std::vector<int> own(nk), place(nk), seen(nk, -1), gplace(nk), gl;
  std::vector<char> sent(nk, 0);
  for (int r = 0; r < T; r++)
    for (int j = B.cut[r]; j < B.cut[r + 1]; j++) { own[v[j].i - k0] = r; place[v[j].i - k0] = j - B.cut[r]; }
  B.rows.resize(nk);
  B.dpos.resize(nk);
  B.lcol.resize((size_t)K * nk);
  B.tcount.assign(nk, 0);
  B.gptr.assign(1, 0);
  for (int r = 0; r < T; r++) {
    gl.clear();
    for (int j = B.cut[r]; j < B.cut[r + 1]; j++)
      for (int s = rowptr[v[j].i]; s < rowptr[v[j].i + 1]; s++) {
        const int c = col[s] - k0;
        if (own[c] != r && seen[c] != r) { seen[c] = r; gl.push_back(c); sent[c] = 1; }
      }
    std::sort(gl.begin(), gl.end());
    B.most = std::max(B.most, (int)gl.size());
    for (size_t g = 0; g < gl.size(); g++) { gplace[gl[g]] = sh.rows + (int)g; B.ghost.push_back(k0 + gl[g]); }
    B.gptr.push_back((int)B.ghost.size());
    if (B.most > sh.ghosts) return;       // refused by the caller
    for (int j = B.cut[r]; j < B.cut[r + 1]; j++) {
      const int i = v[j].i, s0 = rowptr[i];
      unsigned short *lc = &B.lcol[(size_t)K * j];
      int n = 0, dp = 0;
      for (int s = s0; s < rowptr[i + 1]; s++) {
        const int c = col[s] - k0;
        if (c == i - k0) { dp = s - s0; continue; }
        const int l = own[c] == r ? place[c] : gplace[c];
        if (n < K) lc[n] = (unsigned short)(4 * l);
        else { B.tcol.push_back((unsigned short)l); B.tslot.push_back(s); B.tcount[j]++; }
        n++;
      }
      for (int k = n; k < K; k++) lc[k] = (unsigned short)(4 * (j - B.cut[r]));
      B.dpos[j] = dpos_pack(dp, n);
    }
  }
  for (int j = 0; j < nk; j++) B.rows[j] = v[j].i | (sent[v[j].i - k0] ? (int)0x80000000u : 0);
}

}  // namespace shy
