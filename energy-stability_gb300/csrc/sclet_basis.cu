// What the eigenbasis of a run allows the transforms to save (host side).
//
// The basis read_matrices selects for a periodic single block (variant 3,
// source_beta_to_omega/src/vars.c:488-582) diagonalises the second difference
// T with zero values outside the block.  Its eigenvectors are even or odd
// about the block's centre, alternating along the spectrum, so
//   V^-1 x : the even modes see only x[j] + x[n-1-j], the odd ones x[j] - x[n-1-j]
//   V x    : the even modes give E, the odd ones O, x[i] = E[i] + O[i] and
//            x[n-1-i] = E[i] - O[i]
// and each n x n product is two of half the edge: half the multiplications.
// And V diag(d) V^-1 is T itself, so the linear operator of a step can be
// applied to the state in place, as a stencil (sclet_api.cu, increments).
#include <math.h>

#include <vector>

#include "sclet_internal.cuh"

namespace sclet {

// True when (d, v, vi) is that basis, eigenvalues ascending, to 1e-11 of each
// vector's largest entry: T v_k = d_k v_k, vi_k T = d_k vi_k and vi_k v_k = 1.
// The eigenvalues of T are simple, so this makes V V^-1 the identity and
// gives every vector its parity.  (Files hold 16 digits of sines of arguments
// up to n pi: about 1e-13.)
bool basis_is_dirichlet(int n, const double *d, const double *v, const double *vi) {
  const double tol = 1e-11;
  for (int k = 0; k < n; k++) {
    if (k > 0 && !(d[k] > d[k - 1])) return false;
    double mv = 0.0, mw = 0.0, dot = 0.0;
    for (int i = 0; i < n; i++) {
      mv = fmax(mv, fabs(v[(size_t)i * n + k]));
      mw = fmax(mw, fabs(vi[(size_t)k * n + i]));
      dot += vi[(size_t)k * n + i] * v[(size_t)i * n + k];
    }
    if (!(mv > 0.0) || !(mw > 0.0) || !(fabs(dot - 1.0) <= tol)) return false;
    for (int i = 0; i < n; i++) {
      const double a = v[(size_t)i * n + k], b = vi[(size_t)k * n + i];
      const double av = (i > 0 ? v[(size_t)(i - 1) * n + k] : 0.0) + (i < n - 1 ? v[(size_t)(i + 1) * n + k] : 0.0);
      const double bv = (i > 0 ? vi[(size_t)k * n + i - 1] : 0.0) + (i < n - 1 ? vi[(size_t)k * n + i + 1] : 0.0);
      if (!(fabs(av - (2.0 + d[k]) * a) <= tol * mv) || !(fabs(bv - (2.0 + d[k]) * b) <= tol * mw)) return false;
    }
  }
  return true;
}

// Folded halves of a matrix whose rows (fwd) or columns (inverse) are modes:
// part 0 the even modes, part 1 the odd ones, each h x h (h = fold_half(n)),
// contraction index slowest: out[part][k][o].  The odd part of an odd n has
// one row and column less (zeros).  Mode k is even when n - k is odd.
//   fwd:     k = j (block position, j < h), o = m (mode 2 m + p)
//   inverse: k = m,                         o = i (block position)
// Entries are the mean of the two mirrored ones.
std::vector<double> fold_matrix(int n, const double *m, bool inverse) {
  const int h = fold_half(n);
  std::vector<double> out((size_t)2 * h * h, 0.0);
  for (int part = 0; part < 2; part++) {
    const double s = part == 0 ? 1.0 : -1.0;
    const int live = part == 0 ? h : n / 2;
    for (int q = 0; q < live; q++) {
      const int mode = 2 * q + fold_mode0(n, part);
      for (int i = 0; i < live; i++) {
        const double a = inverse ? m[(size_t)i * n + mode] : m[(size_t)mode * n + i];
        const double b = inverse ? m[(size_t)(n - 1 - i) * n + mode] : m[(size_t)mode * n + n - 1 - i];
        const int k = inverse ? q : i, o = inverse ? i : q;
        out[((size_t)part * h + k) * h + o] = 0.5 * (a + s * b);
      }
    }
  }
  return out;
}

}  // namespace sclet
