// Host-side check of the site indexing the kernels use (lattice.cuh): the
// functions are __host__ __device__, so the exact device code runs here on
// the CPU, over every site of each lattice given on the command line
// ("Lx,Ly,Lz,Lt/NBx,NBy,NBz,NBt ...", or "planted:..." to check that a
// planted mistake is caught).  For every site g:
//   * decode_site(g) gives in-range block and in-block coordinates, and
//     dd_index of the site's coordinates is g again (the DD order is a
//     bijection of [0, V));
//   * for each of the eight hops, the neighbour's index -- g + rot_step(...)
//     when it lies in the same block, nbr_across(...) when it crosses a block
//     face (periodic wrap included) -- equals dd_index of the neighbour's
//     coordinates and lies in [0, V), and the colour nbr_across reports is
//     the neighbour's block colour;
//   * on_block_face(g), which makes the face kernels' site lists, holds
//     exactly when some hop of g leaves its block.
// And for the even-odd kernels, for each parity:
//   * the threads on pairs of sites (eo_first) visit every site of the parity once and no other;
//   * eo_coords and eo_index are inverse to one another, in [0, V/2);
//   * a hop's neighbour on the full planes (eo_neighbour) is a site of the
//     other parity next to this one -- up to a step in x where it crosses a
//     boundary of odd extent -- and its compact index is eo_step's.
// It prints one line per lattice and exits non-zero on the first failure.
// Built and run by tests/test_geometry_host.py (nvcc, no GPU needed).
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../qws_b200/csrc/lattice.cuh"

using namespace qwsg;

static int fail(const char* what, const int L[4], const int NB[4], long g, int mu, int dir) {
  std::printf("FAIL %s: lattice %dx%dx%dx%d blocks %d,%d,%d,%d site %ld mu %d dir %d\n", what,
              L[0], L[1], L[2], L[3], NB[0], NB[1], NB[2], NB[3], g, mu, dir);
  return 1;
}

// planted: a mistake put in on purpose (two in-block strides swapped after
// the layout is made), which the checks must catch
static int check(const int L[4], const int NB[4], bool planted) {
  Geom G{};
  for (int mu = 0; mu < 4; mu++) {
    G.L[mu] = L[mu];
    G.NB[mu] = NB[mu];
    G.B[mu] = L[mu] / NB[mu];
  }
  G.tbc = -1;
  G.nr = 1;
  geom_layout(G);
  if (planted) {
    const int t = G.str[0];
    G.str[0] = G.str[1];
    G.str[1] = t;
  }
  for (long g = 0; g < G.V; g++) {
    Site s;
    decode_site(G, (int)g, s);
    int x[4];
    for (int mu = 0; mu < 4; mu++) {
      if (s.lc[mu] < 0 || s.lc[mu] >= G.B[mu] || s.bc[mu] < 0 || s.bc[mu] >= G.NB[mu])
        return fail("decoded coordinates out of range", L, NB, g, mu, 0);
      x[mu] = s.bc[mu] * G.B[mu] + s.lc[mu];
    }
    if ((s.bc[0] + s.bc[1] + s.bc[2] + s.bc[3]) % 2 != s.col)
      return fail("block colour", L, NB, g, -1, 0);
    if (dd_index(G, x) != g) return fail("dd_index(decode_site(g)) != g", L, NB, g, -1, 0);
    bool face = false;  // some hop leaves the block
    for (int mu = 0; mu < 4; mu++) face |= s.lc[mu] == 0 || s.lc[mu] == G.B[mu] - 1;
    if (on_block_face(G, (int)g) != face) return fail("face-site test", L, NB, g, -1, 0);
    for (int mu = 0; mu < 4; mu++)
      for (int dir = -1; dir <= 1; dir += 2) {
        int y[4] = {x[0], x[1], x[2], x[3]};
        y[mu] = (y[mu] + dir + G.L[mu]) % G.L[mu];
        const long want = dd_index(G, y);
        const int l = s.lc[mu] + dir;
        long got;
        if (l >= 0 && l < G.B[mu]) {
          got = g + rot_step(G, mu, s.lc[mu], dir);
        } else {
          int ncol = -1;
          got = nbr_across(G, s, mu, dir, &ncol);
          const int yb = (y[0] / G.B[0] + y[1] / G.B[1] + y[2] / G.B[2] + y[3] / G.B[3]) % 2;
          if (ncol != yb) return fail("nbr_across colour", L, NB, g, mu, dir);
        }
        if (got < 0 || got >= G.V) return fail("neighbour index out of [0, V)", L, NB, g, mu, dir);
        if (got != want) return fail("neighbour index", L, NB, g, mu, dir);
      }
  }
  std::printf("ok %dx%dx%dx%d blocks %d,%d,%d,%d (rotated direction %d, strides %d %d %d %d)\n",
              L[0], L[1], L[2], L[3], NB[0], NB[1], NB[2], NB[3], G.rot, G.str[0], G.str[1],
              G.str[2], G.str[3]);
  return 0;
}

static auto neighbour(int mu, int dir) {
  using F = void (*)(const Geom&, const int*, int, int*);
  static const F f[4][2] = {{eo_neighbour<0, -1>, eo_neighbour<0, 1>},
                            {eo_neighbour<1, -1>, eo_neighbour<1, 1>},
                            {eo_neighbour<2, -1>, eo_neighbour<2, 1>},
                            {eo_neighbour<3, -1>, eo_neighbour<3, 1>}};
  return f[mu][dir > 0];
}

// planted: the parity of the pairs' second sites is taken as the first's
static int check_eo(const int L[4], const int NB[4], bool planted) {
  Geom G{};
  for (int mu = 0; mu < 4; mu++) {
    G.L[mu] = L[mu];
    G.NB[mu] = NB[mu];
    G.B[mu] = L[mu] / NB[mu];
  }
  G.tbc = -1;
  G.nr = 1;
  geom_layout(G);
  for (int p = 0; p < 2; p++) {
    std::vector<char> seen(G.V, 0);
    for (int i = 0; 2 * i < G.V; i++) {
      int x[4], x1[4];
      site_coords(G, 2 * i, x);
      site_coords(G, 2 * i + 1, x1);
      bool second;
      int g = eo_first(x, x1, p, second);
      if (planted) second = g == 0;
      if (g < 0) continue;
      g += 2 * i;
      for (;;) {
        if (g >= G.V || seen[g]++) return fail("pair's site", L, NB, g, -1, p);
        if (dd_index(G, x) != g) return fail("pair's coordinates", L, NB, g, -1, p);
        if (((x[0] + x[1] + x[2] + x[3]) & 1) != p) return fail("pair's parity", L, NB, g, -1, p);
        const int e = eo_index(G, x);
        int xe[4];
        eo_coords(G, e, p, xe);
        if (e < 0 || e >= G.Vh || dd_index(G, xe) != g) return fail("compact index", L, NB, g, -1, p);
        for (int mu = 0; mu < 4; mu++)
          for (int dir = -1; dir <= 1; dir += 2) {
            int xn[4];
            neighbour(mu, dir)(G, x, p, xn);
            for (int k = 0; k < 4; k++)
              if (xn[k] < 0 || xn[k] >= L[k]) return fail("parity neighbour's range", L, NB, g, mu, dir);
            if (((xn[0] + xn[1] + xn[2] + xn[3]) & 1) == p)
              return fail("parity neighbour's parity", L, NB, g, mu, dir);
            int y[4] = {x[0], x[1], x[2], x[3]};
            y[mu] = (y[mu] + dir + L[mu]) % L[mu];
            const bool odd_wrap = L[mu] % 2 != 0 && (dir > 0 ? x[mu] == L[mu] - 1 : x[mu] == 0);
            for (int k = 0; k < 4; k++)
              if (k == 0 && odd_wrap ? xn[0] / 2 != y[0] / 2 : xn[k] != y[k])
                return fail("parity neighbour", L, NB, g, mu, dir);
            if (eo_step(G, e, mu, dir, x[mu], x[0] / 2, x[0] & 1) != eo_index(G, xn))
              return fail("compact neighbour", L, NB, g, mu, dir);
          }
        if (!second) break;
        second = false;
        g++;
        site_coords(G, g, x);
      }
    }
    for (int g = 0; g < G.V; g++) {
      int x[4];
      site_coords(G, g, x);
      if (seen[g] != (((x[0] + x[1] + x[2] + x[3]) & 1) == p)) return fail("sites of a parity", L, NB, g, -1, p);
    }
  }
  return 0;
}

int main(int argc, char** argv) {
  for (int i = 1; i < argc; i++) {
    int L[4], NB[4];
    const bool eo = std::strncmp(argv[i], "planted-eo:", 11) == 0;
    const bool planted = std::strncmp(argv[i], "planted:", 8) == 0;
    if (std::sscanf(argv[i] + (planted ? 8 : eo ? 11 : 0), "%d,%d,%d,%d/%d,%d,%d,%d", &L[0], &L[1], &L[2],
                    &L[3], &NB[0], &NB[1], &NB[2], &NB[3]) != 8) {
      std::printf("FAIL bad argument %s\n", argv[i]);
      return 2;
    }
    if (check_eo(L, NB, eo) || check(L, NB, planted)) return 1;
  }
  return 0;
}
