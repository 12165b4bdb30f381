// Ghost exchange of field blocks on one periodic block (the reference's
// transfer(), source_beta_to_omega/src/trans.c:1939-1996, when every
// Cartesian neighbour is the rank itself).
//
// The reference packs front/back planes, then top/bottom slabs, then
// left/right slabs, all from the block as it stood before the exchange, and
// unpack() (trans.c:154-251) writes left, right, top, bottom, front, back in
// that order.  The net effect is a fixed gather: a ghost cell takes the
// pre-exchange value of its one-axis periodic image along its highest-priority
// ghost axis (z over y over x); the other two coordinates stay as they are,
// so edge and corner ghosts copy other ghost cells' previous values.
//
// The dependences form small trees, one per ghost cell with a single ghost axis:
// its source is an owned cell, and only ghosts with that cell's other two
// coordinates follow from it.  A thread does a whole tree, in place: it reads the
// tree's previous values first and is the only one to read or write them.
#include "sclet_internal.cuh"

namespace sclet {

// Root r (0 .. 12 N^2 - 1) of a block's trees: a ghost cell with one ghost axis
// (0 z, 1 y, 2 x), its source, and the tree's other cells (offsets, -1 for none):
//   axis 1: c[0] one z ghost on; axis 2: c[0] a z ghost on, c[1] a y ghost on,
//   c[2] a z ghost on from there.
// A coordinate within two of a face is the image of exactly one ghost (N >= 4).
struct GhostTree {
  int axis;
  long long cell, source, c[3];
};
__device__ __forceinline__ GhostTree ghost_tree(int n, int r) {
  const int N = n - 4, face = 4 * N * N;
  const int axis = r / face, i = r - axis * face;
  // the ghost coordinate's layer and the two owned ones; x ghosts: layer fastest
  int p, a, b;
  if (axis < 2) {
    const int q = i / N;
    b = i - q * N;
    a = axis == 0 ? q % N : q >> 2;
    p = axis == 0 ? q / N : q & 3;
  } else {
    p = i & 3;
    a = (i >> 2) / N;
    b = (i >> 2) - a * N;
  }
  const int g = p < 2 ? p : n - 4 + p;
  const int z = axis == 0 ? g : a + 2, y = axis == 1 ? g : axis == 0 ? a + 2 : b + 2, x = axis == 2 ? g : b + 2;
  auto at = [&](int zz, int yy, int xx) { return ((long long)zz * n + yy) * n + xx; };
  // the ghost whose image v is, or -1
  auto ghost_of = [&](int v) { return v < 4 ? v + n - 4 : v >= n - 4 ? v - (n - 4) : -1; };
  GhostTree t;
  t.axis = axis;
  t.cell = at(z, y, x);
  t.source = axis == 0 ? at(wrap1(n, z), y, x) : axis == 1 ? at(z, wrap1(n, y), x) : at(z, y, wrap1(n, x));
  t.c[0] = t.c[1] = t.c[2] = -1;
  if (axis > 0) {
    const int gz = ghost_of(z);
    if (gz >= 0) t.c[0] = at(gz, y, x);
    if (axis == 2) {
      const int gy = ghost_of(y);
      if (gy >= 0) {
        t.c[1] = at(z, gy, x);
        if (gz >= 0) t.c[2] = at(gz, gy, x);
      }
    }
  }
  return t;
}

// `per` CTAs for each group of FILL blocks of u (a tree's cells are found once for
// the group; finding them is most of the work).
constexpr int FILL = 3;
template <typename T>
__global__ void ghost_fill(T *__restrict__ u, int count, int n, int per) {
  chain_wait();
  const int b = blockIdx.x / per, roots = 12 * (n - 4) * (n - 4), live = min(FILL, count - b * FILL);
  const long long n3 = (long long)n * n * n;
  u += b * FILL * n3;
  for (int r = (blockIdx.x - b * per) * blockDim.x + threadIdx.x; r < roots; r += per * blockDim.x) {
    const GhostTree t = ghost_tree(n, r);
    T v[FILL], g[FILL], h[FILL];
#pragma unroll
    for (int f = 0; f < FILL; f++)
      if (f < live) {
        v[f] = u[f * n3 + t.source];
        if (t.c[0] >= 0 || t.c[1] >= 0) g[f] = u[f * n3 + t.cell];
        if (t.c[2] >= 0) h[f] = u[f * n3 + t.c[1]];
      }
#pragma unroll
    for (int f = 0; f < FILL; f++)
      if (f < live) {
        u[f * n3 + t.cell] = v[f];
        if (t.c[0] >= 0) u[f * n3 + t.c[0]] = g[f];
        if (t.c[1] >= 0) u[f * n3 + t.c[1]] = g[f];
        if (t.c[2] >= 0) u[f * n3 + t.c[2]] = h[f];
      }
  }
}

// CTAs over a block's trees
static int tree_ctas(int n) {
  const int c = (12 * (n - 4) * (n - 4) + 255) / 256;
  return c > 152 * 16 ? 152 * 16 : c;
}

template <typename T>
cudaError_t launch_ghost_fill(T *u, int count, int n, cudaStream_t s) {
  const int per = tree_ctas(n);
  chain_launch(true, ghost_fill<T>, per * ((count + FILL - 1) / FILL), 256, 0, s, u, count, n, per);
  launch_counter()++;
  return cudaGetLastError();
}

// The elastic force is written into one shared scratch block per field p in
// order (elastic_calculate_ElasDri, elastic.c:617-687): interior = the field's
// result, ghosts = the exchange of that block, whose stale ghost cells still
// hold the previously exchanged field.  A ghost of field p whose one-axis image
// is an owned cell takes this field's value there; one whose image is itself a
// ghost takes field p - 1's value at the image, and before field 0 comes the
// last field of the previous call (zero before the first).  So a tree's cells
// two and three steps from the owned cell hold the fields one and two earlier,
// and all fields of a tree are one thread's.  (As a gather into a shell buffer
// and a scatter, and the fields above as well: two launches more a step, 98 us for
// 4 fields of 36^3, now 95.)  felas: runs x nac blocks, `per` CTAs a run.
template <typename T>
__global__ void elastic_ghosts(T *__restrict__ felas, int n, int nac, int first, int per) {
  chain_wait();
  const int run = blockIdx.x / per, roots = 12 * (n - 4) * (n - 4);
  const long long n3 = (long long)n * n * n;
  felas += run * (nac * n3);
  const T *last = felas + (nac - 1) * n3;
  for (int r = (blockIdx.x - run * per) * blockDim.x + threadIdx.x; r < roots; r += per * blockDim.x) {
    const GhostTree t = ghost_tree(n, r);
    // one step back: the previous field's root; two: its predecessor's
    T g = (T)0, h = (T)0;
    if (!first) {
      if (t.c[0] >= 0 || t.c[1] >= 0) g = last[t.cell];
      if (t.c[2] >= 0) h = last[t.c[1]];
    }
    for (int p = 0; p < nac; p++) {
      T *f = felas + p * n3;
      const T v = f[t.source];
      f[t.cell] = v;
      if (t.c[0] >= 0) f[t.c[0]] = g;
      if (t.c[1] >= 0) f[t.c[1]] = g;
      if (t.c[2] >= 0) f[t.c[2]] = h;
      h = g;
      g = v;
    }
  }
}

template <typename T>
cudaError_t launch_elastic_ghosts(T *felas, int nac, int n, cudaStream_t s, int runs, bool first) {
  const int per = tree_ctas(n);
  chain_launch(true, elastic_ghosts<T>, per * (runs > 0 ? runs : 1), 256, 0, s, felas, n, nac, first ? 1 : 0, per);
  launch_counter()++;
  return cudaGetLastError();
}

template cudaError_t launch_ghost_fill<double>(double *, int, int, cudaStream_t);
template cudaError_t launch_ghost_fill<float>(float *, int, int, cudaStream_t);
template cudaError_t launch_elastic_ghosts<double>(double *, int, int, cudaStream_t, int, bool);
template cudaError_t launch_elastic_ghosts<float>(float *, int, int, cudaStream_t, int, bool);

long long &launch_counter() {
  static long long c = 0;
  return c;
}

}  // namespace sclet
