// icf_solve.cu -- the Newton linear solve on the device.
//
// The reference copies the upper-triangular BCSR matrix and the rhs to the
// host every Newton iteration and solves them with MKL PARDISO (symmetric,
// mtype -2, BSR 3x3; LinearSystem.cs:45-64, PardisoLoader2/dllmain.cpp:30-79).
// Here the system stays where it was assembled and is solved by
// the minimal residual method (MINRES: the matrix is symmetric but, with
// softening cohesive zones, may be indefinite, as PARDISO's mtype -2 allows)
// with a block-Jacobi (3x3) preconditioner, positive definite as MINRES needs
// (a row whose diagonal block is indefinite uses |S|^-1 of the block's
// symmetric part).  The whole iteration is one cooperative kernel, k_minres:
// the product with A, the dot products, the plane rotations and the stopping
// test run on the device, two grid-wide exchanges per iteration; every sum has
// a fixed order, so a solve is identical run to run.
// The solution stays on the device for icf_apply_dx (du += dx, the
// reference's _XtoDU, ImplicitModel3.cs:247-256).
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>

#include "icf_internal.cuh"

namespace {

// ---- the solver's form of the structure -------------------------------------------
// Rows go in Morton order of their nodes' rest positions (position p holds row
// perm[p]; copies of a split node lie side by side), so that contiguous
// positions are a compact piece of the body with few columns outside it.
// Only the upper blocks are stored.  A row of the product needs its own
// (upper) blocks and, transposed, the blocks of its column above the diagonal:
// per structure, every position gets the list of both, padded to steps of
// three entries: eslot {slot << 1 | transposed, or -1}, ecol {column position}.

// bounding box of the nodes (one block): lo[3], hi[3]
__global__ void k_bounds(int n, const double4 *__restrict__ x0, double *__restrict__ box) {
  __shared__ double sh[6][32];
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double4 x = x0[i];
    const double v[3] = {x.x, x.y, x.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      lo[k] = fmin(lo[k], v[k]);
      hi[k] = fmax(hi[k], v[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
      hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
    }
    if ((threadIdx.x & 31) == 0) {
      sh[k][threadIdx.x >> 5] = lo[k];
      sh[3 + k][threadIdx.x >> 5] = hi[k];
    }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double v = sh[threadIdx.x][0];
    for (int i = 1; i < (int)(blockDim.x >> 5); i++)
      v = threadIdx.x < 3 ? fmin(v, sh[threadIdx.x][i]) : fmax(v, sh[threadIdx.x][i]);
    box[threadIdx.x] = v;
  }
}

__device__ __forceinline__ unsigned spread3(unsigned v) {  // 10 bits, two zeros between each
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  return (v | (v << 2)) & 0x09249249u;
}

// Morton code of every row (preset to all ones): the smallest of its nodes'
__global__ void k_morton(int n, int N, const double4 *__restrict__ x0, const int *__restrict__ alt,
                         const double *__restrict__ box, unsigned *__restrict__ code) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = alt[i];
  if (r < 0 || r >= N) return;
  const double ext = fmax(fmax(box[3] - box[0], box[4] - box[1]), box[5] - box[2]);
  const double sc = ext > 0 ? 1023.0 / ext : 0.0;
  const double4 x = x0[i];
  const unsigned c = spread3((unsigned)((x.x - box[0]) * sc)) | spread3((unsigned)((x.y - box[1]) * sc)) << 1 |
                     spread3((unsigned)((x.z - box[2]) * sc)) << 2;
  atomicMin(code + r, c);
}

__global__ void k_fill_iota(int n, int *__restrict__ a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = i;
}
__global__ void k_invert(int n, const int *__restrict__ perm, int *__restrict__ iperm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) iperm[perm[i]] = i;
}

// sort key of slot s: its column, N for a diagonal block (after every column) and
// for a column without a row (a contact with a node that no unit holds), which
// sets *outside
__global__ void k_lower_keys(int N, int nnz, const unsigned long long *__restrict__ mkeys, unsigned *__restrict__ key,
                             int *__restrict__ slot, int *__restrict__ outside) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nnz) return;
  const unsigned long long k = mkeys[s];
  const unsigned r = (unsigned)(k >> 32), c = (unsigned)(k & 0xffffffffull);
  key[s] = r == c || c >= (unsigned)N ? (unsigned)N : c;
  if (c >= (unsigned)N) *outside = 1;
  slot[s] = s;
}

// row r: its first block among the blocks sorted by column
__global__ void k_lower_rows(int N, int nnz, const unsigned *__restrict__ key, int *__restrict__ lrow) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > N) return;
  int lo = 0, hi = nnz;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (key[mid] < (unsigned)r) lo = mid + 1;
    else hi = mid;
  }
  lrow[r] = lo;
}

// steps of the row at position p, at least one (steps[N] = 0, for the scan)
__global__ void k_steps(int N, const int *__restrict__ perm, const int *__restrict__ rows,
                        const int *__restrict__ lrow, int *__restrict__ steps) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > N) return;
  int n = 0;
  if (p < N) {
    const int r = perm[p];
    n = max(1, (rows[r + 1] - rows[r]) + (lrow[r + 1] - lrow[r]));
  }
  steps[p] = (n + 2) / 3;
}

// one thread per stored block: its entry in its own row and, off the diagonal,
// the transposed entry in its column's row (q: its place among the blocks
// sorted by column).  Padding entries keep the preset slot -1, column 0.
__global__ void k_entries(int N, int nnz, const unsigned long long *__restrict__ mkeys,
                          const unsigned *__restrict__ key, const int *__restrict__ slot,
                          const int *__restrict__ rows, const int *__restrict__ lrow, const int *__restrict__ iperm,
                          const int *__restrict__ sstep, int *__restrict__ eslot, int *__restrict__ ecol) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nnz) return;
  {
    const unsigned long long k = mkeys[q];
    const int r = (int)(k >> 32), p = iperm[r], i = q - rows[r];
    const int e = 3 * sstep[p] + i;
    eslot[e] = (int)((unsigned)q << 1);
    ecol[e] = iperm[min((int)(k & 0xffffffffull), N - 1)];
  }
  const unsigned c = key[q];
  if (c < (unsigned)N) {
    const int s = slot[q], e = 3 * sstep[iperm[c]] + (rows[c + 1] - rows[c]) + (q - lrow[c]);
    eslot[e] = (int)((unsigned)s << 1 | 1u);
    ecol[e] = iperm[(int)(mkeys[s] >> 32)];
  }
}

// The positions of warp w of n: [part[w], part[w + 1]), the warps evenly loaded
// (a row weighs its steps and MR_ROW_WEIGHT more for its vectors).  A warp's
// steps start at a multiple of MR_BATCH: first[w], the number of batches before
// it (turned into a prefix sum by k_first).  most[0]: the largest thread block's
// rows, most[2]: the largest warp's batches.  Row weights of 0 to 6, and 16 to 48
// rows a block at least (MR_MIN_ROWS), take the same time.  They decide the order
// of the sums, though, and with it the last digits that the Newton runs of the
// tests carry through contact events: these are the values those runs were
// checked with.
constexpr int MR_ROW_WEIGHT = 5;
constexpr int MR_WARPS = 16;  // of a thread block of k_minres
constexpr int MR_BATCH = 8;   // steps a warp reads together
__device__ int first_at(const int *__restrict__ raw, int lo, int hi, long long target) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (raw[mid] + (long long)MR_ROW_WEIGHT * mid < target) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
__global__ void k_part(int N, int n, const int *__restrict__ raw, int *__restrict__ part, int *__restrict__ first,
                       int *__restrict__ most) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w > n) return;
  const long long all = raw[N] + (long long)MR_ROW_WEIGHT * N;
  auto at = [&](int i) { return i >= n ? N : first_at(raw, 0, N, all * i / n); };
  const int p = at(w), e = at(w + 1);
  part[w] = p;
  const int nb = w < n ? (raw[e] - raw[p] + MR_BATCH - 1) / MR_BATCH : 0;
  first[w] = nb;
  atomicMax(most + 2, nb);
  if (w % MR_WARPS == 0 && w < n) atomicMax(most, at(w + MR_WARPS) - p);
}
// exclusive prefix sum of first[0 .. n] in place (one thread block)
__global__ void __launch_bounds__(1024) k_first(int n, int *__restrict__ first) {
  __shared__ int ws[32];
  const int tid = threadIdx.x, per = (n + 1 + 1023) / 1024, lo = min(n + 1, tid * per), hi = min(n + 1, lo + per);
  int sum = 0;
  for (int i = lo; i < hi; i++) sum += first[i];
  int inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if ((tid & 31) >= o) inc += v;
  }
  if ((tid & 31) == 31) ws[tid >> 5] = inc;
  __syncthreads();
  int base = inc - sum;
  for (int i = 0; i < (tid >> 5); i++) base += ws[i];
  for (int i = lo; i < hi; i++) {
    const int v = first[i];
    first[i] = base;
    base += v;
  }
}
// the first step of every position, behind its warp's, and the mark of its
// last (last: preset to zero)
__global__ void k_place_steps(int N, int n, const int *__restrict__ raw, const int *__restrict__ part,
                              const int *__restrict__ first, int *__restrict__ sstep,
                              unsigned char *__restrict__ last) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  int lo = 0, hi = n;  // the last warp that starts at or before p
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (part[mid] <= p) lo = mid;
    else hi = mid;
  }
  const int st = MR_BATCH * first[lo] + (raw[p] - raw[part[lo]]);
  sstep[p] = st;
  last[st + (raw[p + 1] - raw[p]) - 1] = 1;
}

// The columns a thread block's rows use, its halo (own rows included): sorted
// positions hcol[MR_HALO b + i], their count hcount[b], and every entry's
// place in it, eidx.  One thread block each; a bit per position, then ranks.
constexpr int MR_HALO = 6144;  // most positions of a halo (most[1]: the largest found)
__global__ void __launch_bounds__(512) k_halo(int N, const int *__restrict__ first, const int *__restrict__ eslot,
                                              const int *__restrict__ ecol, int *__restrict__ hcol,
                                              int *__restrict__ hcount, unsigned short *__restrict__ eidx,
                                              int *__restrict__ most) {
  extern __shared__ unsigned bits[];
  __shared__ int wsum[16];
  const int nw = (N + 31) / 32, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, b = blockIdx.x;
  unsigned short *rank = reinterpret_cast<unsigned short *>(bits + nw);  // set bits before each word
  for (int i = tid; i < nw; i += blockDim.x) bits[i] = 0;
  __syncthreads();
  const int e0 = 3 * MR_BATCH * first[MR_WARPS * b], e1 = 3 * MR_BATCH * first[MR_WARPS * (b + 1)];
  for (int e = e0 + tid; e < e1; e += blockDim.x)
    if (eslot[e] != -1) atomicOr(bits + (ecol[e] >> 5), 1u << (ecol[e] & 31));
  __syncthreads();
  // each thread ranks a run of words
  const int per = (nw + (int)blockDim.x - 1) / (int)blockDim.x, w0 = min(nw, tid * per), w1 = min(nw, w0 + per);
  int n = 0;
  for (int i = w0; i < w1; i++) n += __popc(bits[i]);
  int inc = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  int base = inc - n, total = 0;
  for (int i = 0; i < 16; i++) {
    if (i < wid) base += wsum[i];
    total += wsum[i];
  }
  if (tid == 0) {
    hcount[b] = total;
    atomicMax(most + 1, total);
  }
  if (total > MR_HALO) return;  // too large: the solve reads y from global memory instead
  for (int i = w0; i < w1; i++) {
    rank[i] = (unsigned short)base;
    for (unsigned m = bits[i]; m; m &= m - 1) hcol[(size_t)MR_HALO * b + base++] = 32 * i + __ffs(m) - 1;
  }
  __syncthreads();
  for (int e = e0 + tid; e < e1; e += blockDim.x) {
    const int c = ecol[e];
    eidx[e] = eslot[e] == -1 ? 0 : (unsigned short)(rank[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1)));
  }
}

// The matrix of a solve, one record per batch of steps: the columns by block of
// a step, [3][MR_BATCH], three times a place in the halo (16 bits) or a position
// (32 bits); a mask of the steps that end a row; then the steps' blocks as their
// row uses them (27 doubles each).  224 bytes a step (232 with positions), which
// is 75 a block.  One thread per 64-bit word.
constexpr int rec_head(bool halo) { return halo ? 8 : 16; }
constexpr int rec_words(bool halo) { return rec_head(halo) + 27 * MR_BATCH; }
template <bool HALO>
__global__ void k_records(long long n, const int *__restrict__ eslot, const int *__restrict__ ecol,
                          const unsigned short *__restrict__ eidx, const unsigned char *__restrict__ last,
                          const double *__restrict__ vals, double *__restrict__ rec) {
  constexpr int W = rec_words(HALO), H = rec_head(HALO);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long k = t / W;
  int c = (int)(t - k * W);
  if (k >= n) return;
  const long long s0 = MR_BATCH * k;
  if (c >= H) {
    c -= H;
    const int u = c / 27, e = c - 27 * u, q = e / 9, ij = e - 9 * q;
    const int sl = __ldg(eslot + 3 * (s0 + u) + q);
    rec[t] = sl == -1 ? 0.0 : __ldg(vals + 9 * (size_t)((unsigned)sl >> 1) + ((sl & 1) ? 3 * (ij % 3) + ij / 3 : ij));
    return;
  }
  constexpr int P = H / 4;  // words of a block's columns
  const int g = c / P, j = c - P * g;
  unsigned long long v = 0;
  if (g == 3) {
    if (j == 0)
      for (int u = 0; u < MR_BATCH; u++) v |= (unsigned long long)(last[s0 + u] ? 1u : 0u) << u;
  } else if (HALO) {
    for (int u = 0; u < 4; u++) v |= (unsigned long long)(3u * eidx[3 * (s0 + 4 * j + u) + g]) << (16 * u);
  } else {
    for (int u = 0; u < 2; u++) v |= (unsigned long long)(unsigned)ecol[3 * (s0 + 2 * j + u) + g] << (32 * u);
  }
  rec[t] = __longlong_as_double((long long)v);
}

// |S|^-1 for a symmetric 3x3 block S = V diag(l) V^T: V diag(1 / |l|) V^T,
// the eigenvalues by cyclic Jacobi rotations (Golub & Van Loan, Matrix
// Computations, section 8.5), |l| floored at 1e-14 of the largest.  Returns
// false when S is zero or not finite.
__device__ bool abs_inverse_sym3(const double S[9], double *o) {
  double a[3][3], v[3][3];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      a[i][j] = S[3 * i + j];
      v[i][j] = i == j ? 1.0 : 0.0;
    }
  for (int sweep = 0; sweep < 10; sweep++) {
    const double off = fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]);
    const double dia = fabs(a[0][0]) + fabs(a[1][1]) + fabs(a[2][2]);
    if (!(off > 1e-300) || off <= 1e-18 * dia) break;
    for (int p = 0; p < 2; p++)
      for (int q = p + 1; q < 3; q++) {
        if (a[p][q] == 0.0) continue;
        const double th = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
        const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
        // A <- J^T A J, V <- V J with J the rotation in the (p, q) plane
        for (int k = 0; k < 3; k++) {
          const double akp = a[k][p], akq = a[k][q];
          a[k][p] = c * akp - sn * akq;
          a[k][q] = sn * akp + c * akq;
        }
        for (int k = 0; k < 3; k++) {
          const double apk = a[p][k], aqk = a[q][k];
          a[p][k] = c * apk - sn * aqk;
          a[q][k] = sn * apk + c * aqk;
        }
        for (int k = 0; k < 3; k++) {
          const double vkp = v[k][p], vkq = v[k][q];
          v[k][p] = c * vkp - sn * vkq;
          v[k][q] = sn * vkp + c * vkq;
        }
      }
  }
  double l[3], lmax = 0;
  for (int i = 0; i < 3; i++) {
    l[i] = fabs(a[i][i]);
    lmax = fmax(lmax, l[i]);
  }
  if (!(lmax > 0) || !isfinite(lmax)) return false;
  for (int i = 0; i < 3; i++) l[i] = 1.0 / fmax(l[i], 1e-14 * lmax);
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) o[3 * i + j] = v[i][0] * l[0] * v[j][0] + v[i][1] * l[1] * v[j][1] + v[i][2] * l[2] * v[j][2];
  return true;
}

// The preconditioner of a row with diagonal block a: its inverse when the
// block is positive definite; otherwise (softening cohesive zones can make it
// indefinite) |S|^-1 of its symmetric part S, which keeps the preconditioner
// positive definite as MINRES needs.  bad[0]: bit 0 a zero or non-finite
// block; bad[1]: blocks replaced by |S|^-1.
__device__ void precond_row(const double *__restrict__ a, double *o, int *bad) {
  const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
  const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
  const double m2 = a[0] * a[4] - 0.25 * (a[1] + a[3]) * (a[1] + a[3]);
  if (!(a[0] > 0 && m2 > 0 && det > 0) || !isfinite(det)) {
    double S[9];
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) S[3 * i + j] = 0.5 * (a[3 * i + j] + a[3 * j + i]);
    if (!abs_inverse_sym3(S, o)) {
      atomicOr(bad, 1);
      for (int k = 0; k < 9; k++) o[k] = (k % 4 == 0) ? 1.0 : 0.0;
    } else {
      atomicAdd(bad + 1, 1);
    }
    return;
  }
  const double id = 1.0 / det;
  o[0] = c00 * id;
  o[1] = (a[2] * a[7] - a[1] * a[8]) * id;
  o[2] = (a[1] * a[5] - a[2] * a[4]) * id;
  o[3] = c01 * id;
  o[4] = (a[0] * a[8] - a[2] * a[6]) * id;
  o[5] = (a[2] * a[3] - a[0] * a[5]) * id;
  o[6] = c02 * id;
  o[7] = (a[1] * a[6] - a[0] * a[7]) * id;
  o[8] = (a[0] * a[4] - a[1] * a[3]) * id;
}

// ---- preconditioned MINRES (Paige & Saunders 1975) in one kernel ------------------
// The matrix is symmetric and possibly indefinite (softening cohesive zones),
// the preconditioner M the SPD 3x3 block-Jacobi.  With y = M^-1 r2 the
// Lanczos vector is v = y / beta; per iteration
//   q    = A v - (beta / oldb) r1,             alfa = v . q
//   r1   = r2,  r2 = q - (alfa / beta) r1,     y = M^-1 r2,  beta^2 = r2 . y
//   rotation (delta, gamma, phi, ...),         w = (v - oldeps w1 - delta w2) / gamma,
//   x   += phi w.
// One thread block per SM, all co-resident (cooperative launch), owns contiguous
// positions, a warp of it some of them.  Per product a block gathers the y of its
// halo into shared memory (HALO), and each warp reads its records from L2 (a
// step is three blocks of a row, nine lanes each, one lane per entry of the
// block: one contiguous request), up to two batches of eight steps ahead of the
// one it multiplies.  At a row's last step its 27 lane sums go to shared memory;
// ten rows at a time are added up there, three lanes a row.  The block keeps its rows' vectors in shared
// memory as far as they fit (LEVEL 2: all, and M^-1; 1: r1, r2, y and q; 0:
// none), and in what is left the first batches of every warp.
//
// Why this form: seven launches an iteration spent 40 us and more on launches,
// on two sums of 296 partials by one thread (10 us each) and on a product with
// four lanes a row whose 72-byte blocks were nine scattered loads.  Reading the
// upper blocks in place, transposed ones too, streams less (72 against 150 bytes
// an off-diagonal block) but is bound by the chain entry -> block and y of every
// row (34 us an iteration at N = 56,603); records through a ring of bulk copies
// cost the shared memory's bandwidth twice (27 us); records in registers 17 us.
// What bounds it now: small systems, the two exchanges (a store to L2, its read
// by all blocks and a fence: about half of an iteration) and the product's serial
// chain; from N = 30,000 the product's instructions and L2 reads; beyond the L2
// the records' and vectors' stream from HBM.
// Measured, an iteration, before and after (B200, rtol 1e-12, resident data):
//   N =     600 (2,304-tet cantilever)             41 -> 5.6 us
//   N =   1,317 (ice blocks, 3,072 tets)           47 -> 6.2 us
//   N =   6,339 (polycrystal, 20,250 tets)         46 -> 7.7 us
//   N =  18,775 (ice blocks, 63,888 tets)          47 -> 10.2 us
//   N =  56,603 (polycrystal, 196,608 tets)        61 -> 18 us
//   N = 203,704 (polycrystal, 663,552 tets)       128 -> 88 us
//
// The exchange: every block sends its partial sum to every block and adds up
// what it got in block order (so all blocks hold the same scalars bit for bit),
// which is also the grid-wide barrier after which y is new.  (One word per block
// that all blocks poll is slower: 148 blocks reading the same 19 lines, 7,500
// clocks against 4,800 for the second exchange at N = 6,339.)  A partial travels as two 64-bit words, half a double and
// the exchange's number in each, so a word that carries the number is valid by
// itself; two sets of words alternate, and a block can only come back to a set
// after all have read it.  y alternates
// between two buffers as well: the first exchange of an iteration (alfa) then
// orders nothing in memory and needs no fence.  A wait that runs out of polls
// sets the status and every block returns.
constexpr int MR_THREADS = 32 * MR_WARPS;
constexpr int MR_MIN_ROWS = 24;          // a block is given at least so many rows (see k_part)
constexpr int MR_CAP = 10;               // rows a warp adds up together
constexpr int MR_ITERS = 2048;           // iterations per launch (a multiple of MR_CHECK)
constexpr int MR_CHECK = 4;              // the stopping test, every so many iterations
constexpr unsigned MR_POLLS = 1u << 24;  // bound of a wait (some 10 s)
// state carried between launches and read by the host
enum { SC_BETA, SC_IBETA, SC_F1, SC_DBAR, SC_EPSLN, SC_CS, SC_SN, SC_PHIBAR, SC_BETA1, SC_IT, SC_STATUS, SC_BAD, NSC = 16 };
enum { MR_RUNNING = 0, MR_DONE = 1, MR_BREAKDOWN = 2, MR_TIMEOUT = 3, MR_PAUSE = 4 };

struct mr_args {
  int N, halo_cap;  // rows; the largest halo of a block
  int res;          // batches of every warp that shared memory holds
  const int *rows, *perm, *part, *first, *hcol, *hcount;
  const double *rec;                                  // the matrix's records
  const double *vals, *rhs;
  double *y4;                                         // y, four doubles per position, two buffers
  double *r1, *r2, *w, *w2, *ya, *yb, *x, *q, *dinv;  // vectors by position
  double *sol;                                        // the solution by row
  unsigned long long *slots;                          // [2][to block][from block][2] exchange words
  double *sc;
  unsigned epoch0;  // number of the last exchange before this launch
  int max_iter, fresh;
  int iters;        // iterations of this launch (a multiple of MR_CHECK)
  double tol;
};

struct mr_shared {
  double part[MR_WARPS];
  // the scalars (in shared memory: they would cost every thread 36 registers):
  // 1 / beta of this iteration and the last, beta / oldb, alfa / beta, the
  // last rotation's oldeps, delta, 1 / gamma, phi; warp 0's recurrence
  double ibeta, vscale, f1, f2, oldeps, delta, igamma, phi;
  double beta, dbar, epsln, cs, sn, phibar, beta1, alfa;
  int status;
  double rows[MR_WARPS][MR_CAP * 27];  // lane sums of finished rows
};

// Block sum of v, sent to every block as this block's partial of exchange
// `epoch`.  RELEASE: the block's writes before the call are visible to every
// block that has collected the exchange.
template <bool RELEASE>
__device__ __forceinline__ void mr_publish(mr_shared &S, unsigned long long *slots, unsigned epoch, double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) S.part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int G = gridDim.x;
    double p = S.part[threadIdx.x % MR_WARPS];
#pragma unroll
    for (int o = MR_WARPS / 2; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
    if (RELEASE) asm volatile("fence.acq_rel.gpu;" ::: "memory");
    const unsigned long long n = (unsigned long long)epoch << 32, u = (unsigned long long)__double_as_longlong(p);
    unsigned long long *o = slots + 2 * ((epoch & 1) * (size_t)G * G + blockIdx.x);
    for (int i = threadIdx.x; i < G; i += 32)
      asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(o + 2 * (size_t)G * i),
                   "l"(n | (u & 0xffffffffull)), "l"(n | (u >> 32))
                   : "memory");
  }
}

// The sum of all partials of exchange `epoch`, in a fixed order (warp 0; every
// lane returns it).  False when the wait ran out.
template <bool ACQUIRE>
__device__ __forceinline__ bool mr_collect(const unsigned long long *slots, unsigned epoch, double &sum) {
  const int G = gridDim.x;
  const unsigned long long *base = slots + 2 * (size_t)G * ((epoch & 1) * (size_t)G + blockIdx.x);
  double acc = 0;
  bool ok = true;
  constexpr int PER = 5;  // words a lane polls side by side (148 blocks: all of them)
  for (int i0 = threadIdx.x; i0 < G; i0 += 32 * PER) {
    unsigned long long a[PER], b[PER];
    unsigned n = 0;
    for (;;) {
      bool all = true;
#pragma unroll
      for (int k = 0; k < PER; k++) {
        const int i = min(i0 + 32 * k, G - 1);
        asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a[k]), "=l"(b[k]) : "l"(base + 2 * i) : "memory");
      }
#pragma unroll
      for (int k = 0; k < PER; k++) all &= (unsigned)(a[k] >> 32) == epoch && (unsigned)(b[k] >> 32) == epoch;
      if (all) break;
      if (++n > MR_POLLS) {
        ok = false;
        break;
      }
    }
#pragma unroll
    for (int k = 0; k < PER; k++)
      if (i0 + 32 * k < G) acc += __longlong_as_double((long long)((a[k] & 0xffffffffull) | (b[k] << 32)));
  }
  if (ACQUIRE) asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  sum = acc;
  return __all_sync(0xffffffffu, ok);
}

template <bool HALO, int LEVEL, bool STREAM>
__global__ void __launch_bounds__(MR_THREADS, 1) k_minres(const mr_args A) {
  constexpr int W = rec_words(HALO), H = rec_head(HALO);
  extern __shared__ __align__(16) double smem[];
  __shared__ mr_shared S;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int b = blockIdx.x;
  const int row0 = A.part[MR_WARPS * b], nr = A.part[MR_WARPS * (b + 1)] - row0, ne = 3 * nr;  // positions, elements
  // shared memory: halo (y, then positions), vectors, the warps' first batches
  double *yh = smem;
  int *hpos = reinterpret_cast<int *>(yh + 3 * (size_t)A.halo_cap);
  double *vsm = reinterpret_cast<double *>(hpos + A.halo_cap + (A.halo_cap & 1));
  const int nh = HALO ? A.hcount[b] : 0;
  // element i of the block's rows: its vectors in shared memory or, by
  // position, in global memory
  auto vec = [&](int level, int i, double *g) -> double * {
    return LEVEL >= level ? vsm + i * ne : g + 3 * (size_t)row0;
  };
  double *r1 = vec(1, 0, A.r1), *r2 = vec(1, 1, A.r2), *y = vec(1, 2, A.ya), *yo = vec(1, 3, A.yb), *q = vec(1, 4, A.q);
  double *w = vec(2, 5, A.w), *w2 = vec(2, 6, A.w2), *x = vec(2, 7, A.x);
  double *D = LEVEL >= 2 ? vsm + 8 * ne : A.dinv + 9 * (size_t)row0;
  unsigned epoch = A.epoch0;
  int it = 0;

  // ---- the halo and the warp's rows
  for (int t = tid; t < nh; t += MR_THREADS) hpos[t] = A.hcol[(size_t)MR_HALO * b + t];
  const int wr0 = A.part[MR_WARPS * b + wid];  // its first position
  const int nb = A.first[MR_WARPS * b + wid + 1] - A.first[MR_WARPS * b + wid];  // its batches
  // the first batches, for good; the others (STREAM) come from L2, two at a time
  const int nres = STREAM ? min(A.res, nb) : nb, nstr = nb - nres;
  const double *rec = A.rec + (size_t)W * A.first[MR_WARPS * b + wid];
  const int vwords = (LEVEL >= 2 ? 11 : (LEVEL >= 1 ? 5 : 0)) * ne;
  double *kept = vsm + vwords + ((vsm - smem + vwords) & 1) + wid * (A.res * W);  // (16-byte aligned)
  for (int i = lane; i < nres * W; i += 32) kept[i] = __ldg(rec + i);
  rec += (size_t)W * nres;
  __syncwarp();
  // ---- start: M^-1, r1 = r2 = rhs, y = M^-1 rhs; or the state of the last
  // launch (what is kept in global memory is in place)
  double acc = 0;
  for (int t = tid; t < nr; t += MR_THREADS) {
    const int o = 3 * t;
    const size_t g = 3 * (size_t)(row0 + t);
    double *d = D + 3 * (size_t)o;
    if (A.fresh) {
      const int r = A.perm[row0 + t];
      double m[9];
      precond_row(A.vals + 9 * (size_t)A.rows[r], m, reinterpret_cast<int *>(A.sc + SC_BAD));
#pragma unroll
      for (int k = 0; k < 9; k++) d[k] = m[k];
      const double bv[3] = {A.rhs[3 * (size_t)r], A.rhs[3 * (size_t)r + 1], A.rhs[3 * (size_t)r + 2]};
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const double z = m[3 * k] * bv[0] + m[3 * k + 1] * bv[1] + m[3 * k + 2] * bv[2];
        r1[o + k] = r2[o + k] = bv[k];
        w[o + k] = w2[o + k] = x[o + k] = 0.0;
        y[o + k] = z;
        A.y4[4 * (size_t)(row0 + t) + k] = z;
        acc += bv[k] * z;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        if (LEVEL >= 1) {
          r1[o + k] = A.r1[g + k];
          r2[o + k] = A.r2[g + k];
          y[o + k] = A.ya[g + k];
        }
        if (LEVEL >= 2) {
          w[o + k] = A.w[g + k];
          w2[o + k] = A.w2[g + k];
          x[o + k] = A.x[g + k];
        }
      }
      if (LEVEL >= 2)
#pragma unroll
        for (int k = 0; k < 9; k++) d[k] = A.dinv[3 * g + k];
    }
  }
  if (A.fresh) {
    mr_publish<true>(S, A.slots, ++epoch, acc);
    if (wid == 0) {
      double b2;
      int st = mr_collect<true>(A.slots, epoch, b2) ? MR_RUNNING : MR_TIMEOUT;
      if (st == MR_RUNNING && (b2 < 0 || !isfinite(b2))) st = MR_BREAKDOWN;
      const double beta = b2 > 0 ? sqrt(b2) : 0.0;
      if (st == MR_RUNNING && (beta == 0 || A.tol >= 1.0)) st = MR_DONE;
      if (lane == 0) {
        S.beta = S.beta1 = S.phibar = beta;
        S.ibeta = b2 > 0 ? rsqrt(b2) : 0.0;
        S.f1 = S.dbar = S.epsln = S.sn = 0.0;
        S.cs = -1.0;
        S.status = st;
      }
    }
  } else {
    if (tid == 0) {
      S.beta = A.sc[SC_BETA]; S.ibeta = A.sc[SC_IBETA]; S.f1 = A.sc[SC_F1]; S.dbar = A.sc[SC_DBAR];
      S.epsln = A.sc[SC_EPSLN]; S.cs = A.sc[SC_CS]; S.sn = A.sc[SC_SN]; S.phibar = A.sc[SC_PHIBAR];
      S.beta1 = A.sc[SC_BETA1];
      S.status = MR_RUNNING;
    }
    it = (int)A.sc[SC_IT];
  }
  __syncthreads();
  int status = S.status;
  const int it_stop = it + A.iters;
  bool pending = false;  // the last iteration's w and x are still to be formed
  double *yin = A.y4, *yout = A.y4 + 4 * (size_t)A.N;

  // w = (v - oldeps w1 - delta w2) / gamma, x += phi w, with v = yo vscale; w
  // takes the place of w1
  auto update_x = [&]() {
    const double vscale = S.vscale, oldeps = S.oldeps, delta = S.delta, igamma = S.igamma, phi = S.phi;
    for (int o = tid; o < ne; o += MR_THREADS) {
      const double wn = (yo[o] * vscale - oldeps * w2[o] - delta * w[o]) * igamma;
      w2[o] = wn;
      x[o] += phi * wn;
    }
    double *z = w;
    w = w2;
    w2 = z;
  };

  // this lane: block g of a step and its column ck there (lanes 27 and up: the
  // mask of a batch); in the flush, row fj and component fi
  const int g = lane / 9, ck = lane % 3, word = min(lane, 26);
  const int fj = lane / 3, fi = lane - 3 * fj;
  double *lsum = S.rows[wid];
  struct batch {
    double B[MR_BATCH];
    uint4 c[HALO ? 1 : 2];
  };
  batch P0, P1;  // the next two streamed batches, P0 the even ones
  auto fetch = [&](batch &P, int k) {
    const double *r = rec + (size_t)W * k;
#pragma unroll
    for (int i = 0; i < (HALO ? 1 : 2); i++) P.c[i] = __ldg(reinterpret_cast<const uint4 *>(r + H / 4 * g) + i);
#pragma unroll
    for (int u = 0; u < MR_BATCH; u++) P.B[u] = __ldg(r + H + 27 * u + word);
  };
  if (STREAM && nstr > 0) {
    fetch(P0, 0);
    if (nstr > 1) fetch(P1, 1);
  }
  while (status == MR_RUNNING) {
    // ---- q = A v - (beta / oldb) r1, alfa = v . q
    if (HALO) {
      for (int t = tid; t < nh; t += MR_THREADS) {
        const double2 *p = reinterpret_cast<const double2 *>(yin + 4 * (size_t)hpos[t]);
        const double2 a = p[0];
        const double c = p[1].x;
        yh[3 * t] = a.x;
        yh[3 * t + 1] = a.y;
        yh[3 * t + 2] = c;
      }
      __syncthreads();
    }
    acc = 0;
    double s = 0;
    int cnt = 0, o0 = 3 * (wr0 - row0);  // rows in lsum, the first one's element
    auto flush = [&]() {
      __syncwarp();
      if (fj < cnt) {
        const double *l = lsum + 27 * fj + 3 * fi;
        double t = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) t += (l[9 * k] + l[9 * k + 1]) + l[9 * k + 2];
        const int o = o0 + lane;
        const double ibeta = S.ibeta, qi = t * ibeta - S.f1 * r1[o];
        q[o] = qi;
        acc += (y[o] * ibeta) * qi;
      }
      __syncwarp();
      o0 += 3 * cnt;
      cnt = 0;
    };
    auto multiply = [&](const batch &P, unsigned ends) {
      double yv[MR_BATCH];
#pragma unroll
      for (int u = 0; u < MR_BATCH; u++) {
        const uint4 c = P.c[HALO ? 0 : u / 4];
        const int i = HALO ? u / 2 : u % 4;
        unsigned v = i == 0 ? c.x : (i == 1 ? c.y : (i == 2 ? c.z : c.w));
        if (HALO) v = u % 2 ? v >> 16 : v & 0xffffu;
        if (g == 3) v = 0;
        yv[u] = HALO ? yh[v + ck] : yin[4 * (size_t)v + ck];
      }
#pragma unroll
      for (int u = 0; u < MR_BATCH; u++) {
        s += P.B[u] * yv[u];
        const bool end = ends >> u & 1;  // (the same for all lanes)
        if (end && lane < 27) lsum[27 * cnt + lane] = s;
        s = end ? 0.0 : s;
        cnt += end;
      }
    };
    auto ends_of = [&](const batch &P) -> unsigned { return __shfl_sync(0xffffffffu, P.c[0].x, 27); };
    for (int k = 0; k <= nres; k++) {  // (the flush after the last batch at k == nres)
      batch P;
      unsigned ends = 0;
      if (k < nres) {
        const double *r = kept + W * k;
#pragma unroll
        for (int i = 0; i < (HALO ? 1 : 2); i++) P.c[i] = *(reinterpret_cast<const uint4 *>(r + H / 4 * g) + i);
#pragma unroll
        for (int u = 0; u < MR_BATCH; u++) P.B[u] = r[H + 27 * u + word];
        ends = ends_of(P);
      }
      if (k == nres || cnt + __popc(ends) > MR_CAP) flush();
      if (k < nres) multiply(P, ends);
    }
    if (STREAM && nstr > 0) {
      for (int k = 0; k < nstr; k += 2) {
        unsigned ends = ends_of(P0);
        if (cnt + __popc(ends) > MR_CAP) flush();
        multiply(P0, ends);
        fetch(P0, k + 2 < nstr ? k + 2 : 0);
        if (k + 1 == nstr) break;
        ends = ends_of(P1);
        if (cnt + __popc(ends) > MR_CAP) flush();
        multiply(P1, ends);
        fetch(P1, k + 3 < nstr ? k + 3 : 1);
      }
      flush();
    }
    mr_publish<false>(S, A.slots, ++epoch, acc);
    if (pending) update_x();  // while the partials travel
    if (wid == 0) {
      double alfa;
      const bool ok = mr_collect<false>(A.slots, epoch, alfa);
      if (lane == 0) {
        S.alfa = alfa;
        S.f2 = alfa * S.ibeta;
        if (!ok) S.status = MR_TIMEOUT;
      }
    }
    __syncthreads();
    status = S.status;
    if (status != MR_RUNNING) break;
    // ---- r2 = q - (alfa / beta) r2, y = M^-1 r2, beta^2 = r2 . y.  The new r2
    // takes the place of r1, the new y that of the one before
    acc = 0;
    const double f2 = S.f2;
    for (int o = tid; o < ne; o += MR_THREADS) {
      const int t = o / 3, c = o - 3 * t, e = 3 * t;
      const double *d = D + 3 * (size_t)o;
      double rn[3];
#pragma unroll
      for (int m = 0; m < 3; m++) rn[m] = q[e + m] - f2 * r2[e + m];
      const double z = d[0] * rn[0] + d[1] * rn[1] + d[2] * rn[2];
      const double rc = c == 0 ? rn[0] : (c == 1 ? rn[1] : rn[2]);
      r1[o] = rc;
      yo[o] = z;
      yout[4 * (size_t)(row0 + t) + c] = z;
      acc += rc * z;
    }
    mr_publish<true>(S, A.slots, ++epoch, acc);
    {
      double *z = r1;
      r1 = r2;
      r2 = z;
      z = y;
      y = yo;
      yo = z;
      z = yin;
      yin = yout;
      yout = z;
    }
    it++;
    if (wid == 0) {
      // the plane rotation of this iteration
      double b2;
      int st = mr_collect<true>(A.slots, epoch, b2) ? MR_RUNNING : MR_TIMEOUT;
      if (st == MR_RUNNING && (b2 < 0 || !isfinite(b2))) st = MR_BREAKDOWN;
      const double ioldb = S.ibeta, cs = S.cs, sn = S.sn, alfa = S.alfa, dbar = S.dbar, phibar = S.phibar;
      const double ib = b2 > 0 ? rsqrt(b2) : 0.0;  // beta = 0: converged exactly, nothing left to add
      const double beta = b2 * ib, gbar = sn * dbar - cs * alfa, g2 = gbar * gbar + b2;
      const double igamma = g2 > 0 ? rsqrt(g2) : 1e300;
      const double cs2 = gbar * igamma, sn2 = beta * igamma, phibar2 = sn2 * phibar;
      if (st == MR_RUNNING && (it % MR_CHECK == 0 || it >= A.max_iter)) {
        if (!(phibar2 > A.tol * S.beta1) || it >= A.max_iter) st = MR_DONE;
        else if (it >= it_stop) st = MR_PAUSE;
      }
      __syncwarp();
      if (lane == 0) {
        S.beta = beta;
        S.ibeta = ib;
        S.vscale = ioldb;
        S.f1 = beta * ioldb;
        S.oldeps = S.epsln;
        S.epsln = sn * beta;
        S.delta = cs * dbar + sn * alfa;
        S.dbar = -cs * beta;
        S.igamma = igamma;
        S.cs = cs2;
        S.sn = sn2;
        S.phi = cs2 * phibar;
        S.phibar = phibar2;
        S.status = st;
      }
    }
    __syncthreads();
    status = S.status;
    pending = true;
  }

  if (pending && (status == MR_DONE || status == MR_PAUSE)) update_x();
  // any block's time-out is the launch's (a word of its own)
  if (tid == 0 && status == MR_TIMEOUT) reinterpret_cast<volatile int *>(A.sc + SC_BAD + 1)[0] = 1;
  if (b == 0 && tid == 0) {
    A.sc[SC_BETA] = S.beta; A.sc[SC_IBETA] = S.ibeta; A.sc[SC_F1] = S.f1; A.sc[SC_DBAR] = S.dbar;
    A.sc[SC_EPSLN] = S.epsln; A.sc[SC_CS] = S.cs; A.sc[SC_SN] = S.sn; A.sc[SC_PHIBAR] = S.phibar;
    A.sc[SC_BETA1] = S.beta1;
    A.sc[SC_IT] = it;
    A.sc[SC_STATUS] = status;
  }
  // the solution by row, and on a pause the rest of the state (vectors in global
  // memory are in place: a pause comes at an even iteration, when the pairs
  // that swap are back in theirs)
  __syncthreads();
  const size_t g0 = 3 * (size_t)row0;
  for (int o = tid; o < ne; o += MR_THREADS) {
    const int t = o / 3;
    A.sol[3 * (size_t)A.perm[row0 + t] + (o - 3 * t)] = x[o];
    if (status != MR_PAUSE) continue;
    if (LEVEL >= 1) {
      A.r1[g0 + o] = r1[o];
      A.r2[g0 + o] = r2[o];
      A.ya[g0 + o] = y[o];
    }
    if (LEVEL >= 2) {
      A.w[g0 + o] = w[o];
      A.w2[g0 + o] = w2[o];
      A.x[g0 + o] = x[o];
#pragma unroll
      for (int k = 0; k < 3; k++) A.dinv[3 * (g0 + o) + k] = D[3 * (size_t)o + k];
    }
  }
}

template <typename T>
int grow(icf_ctx *ctx, T **p, long long *cap, long long n) {
  return n <= *cap ? ICF_OK : icf_grow(ctx, cap, n + n / 4 + 16, p);
}
// a function's temporaries on the context's stream
#define SOLVE_TMP(p, n)                                                                    \
  do {                                                                                     \
    if (!tmp.alloc(&(p), n)) return icf_fail(ctx, ICF_ERR_CUDA, "linear solve: out of memory"); \
  } while (0)

}  // namespace

void icf_free_solver(icf_ctx *ctx) {
  icf_solver &S = ctx->solver;
  void *ptrs[] = {S.perm, S.iperm, S.sstep, S.eslot, S.ecol, S.eidx, S.last, S.part, S.hcol, S.rec, S.x, S.vec,
                  S.sc, S.slots};
  for (void *p : ptrs) cudaFree(p);
  if (S.h_sc) cudaFreeHost(S.h_sc);
  S = icf_solver();
}

// The row order, once per static pattern.
static int build_order(icf_ctx *ctx) {
  icf_solver &S = ctx->solver;
  cudaStream_t s = ctx->stream;
  const int N = ctx->N, n = ctx->n_nodes;
  ICF_TRY_RC(grow(ctx, &S.perm, &S.perm_cap, N));
  ICF_TRY_RC(grow(ctx, &S.iperm, &S.iperm_cap, N));
  unsigned *k0, *k1;
  int *i0;
  double *box;
  icf_stream_mem mem{s};
  icf_temps<icf_stream_mem> tmp(mem);
  SOLVE_TMP(k0, N);
  SOLVE_TMP(k1, N);
  SOLVE_TMP(i0, N);
  SOLVE_TMP(box, 6);
  k_bounds<<<1, 1024, 0, s>>>(n, ctx->d_x0, box);
  ICF_CUDA(ctx, cudaMemsetAsync(k0, 0xff, sizeof(unsigned) * (size_t)N, s));
  k_morton<<<icf_blocks(n, 256), 256, 0, s>>>(n, N, ctx->d_x0, ctx->d_alt, box, k0);
  k_fill_iota<<<icf_blocks(N, 256), 256, 0, s>>>(N, i0);
  size_t tb = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tb, k0, k1, i0, S.perm, N, 0, 32, s);
  if (icf_scratch(ctx, tb)) return ICF_ERR_CUDA;
  ICF_CUDA(ctx, cub::DeviceRadixSort::SortPairs(ctx->d_tmp, tb, k0, k1, i0, S.perm, N, 0, 32, s));
  k_invert<<<icf_blocks(N, 256), 256, 0, s>>>(N, S.perm, S.iperm);
  ICF_CUDA(ctx, cudaGetLastError());
  S.order_rows = N;
  return ICF_OK;
}

// The solver's form of the current structure (rebuilt when that changes): the
// blocks sorted by column (a stable sort over the bits of the row count, so
// each column's rows ascend), every position's entries, the thread blocks'
// positions and halos.  One synchronisation.
static int build_steps(icf_ctx *ctx) {
  icf_solver &S = ctx->solver;
  cudaStream_t s = ctx->stream;
  const int N = ctx->N, nnz = ctx->nnz;
  if (S.order_rows != N) ICF_TRY_RC(build_order(ctx));
  // at most: a row's padding to steps, a warp's to batches
  const int G = std::min(ctx->n_sm, (N + MR_MIN_ROWS - 1) / MR_MIN_ROWS), nw = MR_WARPS * G;
  const long long scap = 2LL * nnz / 3 + N + (long long)MR_BATCH * nw;
  ICF_TRY_RC(grow(ctx, &S.sstep, &S.sstep_cap, N));
  ICF_TRY_RC(grow(ctx, &S.eslot, &S.eslot_cap, 3 * scap));
  ICF_TRY_RC(grow(ctx, &S.ecol, &S.ecol_cap, 3 * scap));
  ICF_TRY_RC(grow(ctx, &S.eidx, &S.eidx_cap, 3 * scap));
  ICF_TRY_RC(grow(ctx, &S.last, &S.last_cap, scap));
  // the warps' first positions and batches, the halo counts, the maxima and a flag
  ICF_TRY_RC(grow(ctx, &S.part, &S.part_cap, (2 * MR_WARPS + 1) * (long long)ctx->n_sm + 8));
  ICF_TRY_RC(grow(ctx, &S.hcol, &S.hcol_cap, (long long)MR_HALO * ctx->n_sm));
  S.first = S.part + MR_WARPS * ctx->n_sm + 1;
  S.hcount = S.first + MR_WARPS * ctx->n_sm + 1;
  int *d_most = S.hcount + ctx->n_sm;
  unsigned *k0, *k1;
  int *s0, *s1, *lrow, *steps, *raw;
  icf_stream_mem mem{s};
  icf_temps<icf_stream_mem> tmp(mem);
  SOLVE_TMP(k0, nnz);
  SOLVE_TMP(k1, nnz);
  SOLVE_TMP(s0, nnz);
  SOLVE_TMP(s1, nnz);
  SOLVE_TMP(lrow, 3 * (N + 1LL));
  steps = lrow + N + 1;
  raw = steps + N + 1;
  ICF_CUDA(ctx, cudaMemsetAsync(d_most, 0, 4 * sizeof(int), s));
  k_lower_keys<<<icf_blocks(nnz, 256), 256, 0, s>>>(N, nnz, ctx->d_mkeys, k0, s0, d_most + 3);
  int bits = 1;
  while ((1LL << bits) <= (long long)N) bits++;
  size_t tb = 0, tb2 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tb, k0, k1, s0, s1, nnz, 0, bits, s);
  cub::DeviceScan::ExclusiveSum(nullptr, tb2, steps, raw, N + 1, s);
  if (icf_scratch(ctx, std::max(tb, tb2))) return ICF_ERR_CUDA;
  ICF_CUDA(ctx, cub::DeviceRadixSort::SortPairs(ctx->d_tmp, tb, k0, k1, s0, s1, nnz, 0, bits, s));
  k_lower_rows<<<icf_blocks(N + 1LL, 256), 256, 0, s>>>(N, nnz, k1, lrow);
  k_steps<<<icf_blocks(N + 1LL, 256), 256, 0, s>>>(N, S.perm, ctx->d_rows, lrow, steps);
  ICF_CUDA(ctx, cub::DeviceScan::ExclusiveSum(ctx->d_tmp, tb2, steps, raw, N + 1, s));
  k_part<<<icf_blocks(nw + 1LL, 128), 128, 0, s>>>(N, nw, raw, S.part, S.first, d_most);
  k_first<<<1, 1024, 0, s>>>(nw, S.first);
  ICF_CUDA(ctx, cudaMemsetAsync(S.eslot, 0xff, sizeof(int) * 3 * (size_t)scap, s));
  ICF_CUDA(ctx, cudaMemsetAsync(S.ecol, 0, sizeof(int) * 3 * (size_t)scap, s));
  ICF_CUDA(ctx, cudaMemsetAsync(S.last, 0, (size_t)scap, s));
  k_place_steps<<<icf_blocks(N, 256), 256, 0, s>>>(N, nw, raw, S.part, S.first, S.sstep, S.last);
  k_entries<<<icf_blocks(nnz, 256), 256, 0, s>>>(N, nnz, ctx->d_mkeys, k1, s1, ctx->d_rows, lrow, S.iperm, S.sstep,
                                                 S.eslot, S.ecol);
  // six bytes of shared memory per 32 positions
  const size_t hsm = 6 * (((size_t)N + 31) / 32);
  const bool try_halo = hsm <= 200 * 1024;
  if (try_halo) {
    ICF_CUDA(ctx, cudaFuncSetAttribute(k_halo, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    k_halo<<<G, 512, hsm, s>>>(N, S.first, S.eslot, S.ecol, S.hcol, S.hcount, S.eidx, d_most);
  }
  ICF_CUDA(ctx, cudaGetLastError());
  int h[5] = {0, 0, 0, 0, 0};
  ICF_CUDA(ctx, cudaMemcpyAsync(h, d_most, 4 * sizeof(int), cudaMemcpyDeviceToHost, s));
  ICF_CUDA(ctx, cudaMemcpyAsync(h + 4, S.first + nw, sizeof(int), cudaMemcpyDeviceToHost, s));
  ICF_CUDA(ctx, cudaStreamSynchronize(s));
  if (h[3]) return icf_fail(ctx, ICF_ERR_STATE, "linear solve: a contact joins a row to a node outside the system");
  std::copy(h, h + 3, S.most);
  S.n_steps = MR_BATCH * (long long)h[4];
  S.blocks = G;
  S.halo = try_halo && h[1] <= MR_HALO;
  S.gen = ctx->struct_gen;
  return ICF_OK;
}

// Iterations per launch of this context's solves until its next static data: a
// multiple of MR_CHECK up to 65,536, or 0 for MR_ITERS.  Not part of the
// interface; for the tests of a solve that spans launches.
extern "C" int icf_solver_slice(icf_ctx *ctx, int iters) {
  if (!ctx || iters < 0 || iters > 65536 || iters % MR_CHECK != 0) return ICF_ERR_ARG;
  ctx->solver.slice = iters;
  return ICF_OK;
}

int icf_solve_impl(icf_ctx *ctx, double rel_tol, int max_iter, int *iters, double *relres) {
  icf_solver &S = ctx->solver;
  cudaStream_t s = ctx->stream;
  const int N = ctx->N;
  const long long n3 = 3LL * N;
  if (S.gen != ctx->struct_gen) ICF_TRY_RC(build_steps(ctx));
  // shared memory: the halo, then as many vectors as fit; without room for the
  // halo y comes from global memory
  const int G = S.blocks;
  int smem_max = 0;
  ICF_CUDA(ctx, cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const size_t room = (size_t)smem_max - sizeof(mr_shared) - 1024, el = sizeof(double) * 3 * (size_t)S.most[0];
  const bool halo = S.halo && 28 * (size_t)(S.most[1] + 1) <= room;
  const int halo_cap = halo ? S.most[1] : 0;
  const size_t fixed = 28 * (size_t)(halo_cap + 1) + 8, vbytes[3] = {0, 5 * el, 11 * el};
  int level = halo ? 2 : 0;
  while (level > 0 && fixed + vbytes[level] > room) level--;
  const size_t batch = sizeof(double) * MR_WARPS * rec_words(halo);  // a batch of every warp
  const int res = (int)std::min<size_t>((room - fixed - vbytes[level]) / batch, S.most[2]);
  const size_t smem = fixed + vbytes[level] + res * batch;
  ICF_TRY_RC(grow(ctx, &S.x, &S.x_cap, n3));
  // y4 (twice), then r1, r2, w, w2, ya, yb, x, q, M^-1
  ICF_TRY_RC(grow(ctx, &S.vec, &S.vec_cap, 8LL * N + 11 * n3));
  if (!S.sc) ICF_CUDA(ctx, cudaMalloc(&S.sc, sizeof(double) * NSC));
  if (!S.h_sc) ICF_CUDA(ctx, cudaMallocHost(&S.h_sc, sizeof(double) * NSC));
  if (!S.slots || S.epoch > 0xf0000000u) {
    const size_t bytes = sizeof(unsigned long long) * 4 * (size_t)ctx->n_sm * ctx->n_sm;
    if (!S.slots) ICF_CUDA(ctx, cudaMalloc(&S.slots, bytes));
    ICF_CUDA(ctx, cudaMemsetAsync(S.slots, 0, bytes, s));
    S.epoch = 0;
  }
  ICF_CUDA(ctx, cudaMemsetAsync(S.sc, 0, sizeof(double) * NSC, s));
  // the matrix's records
  const long long nbat = S.n_steps / MR_BATCH, words = rec_words(halo) * nbat;
  ICF_TRY_RC(grow(ctx, &S.rec, &S.rec_cap, words));
  (halo ? k_records<true> : k_records<false>)<<<icf_blocks(words, 256), 256, 0, s>>>(
      nbat, S.eslot, S.ecol, S.eidx, S.last, ctx->d_vals, S.rec);
  ICF_CUDA(ctx, cudaGetLastError());
  mr_args A;
  A.N = N;
  A.res = res;
  A.halo_cap = halo_cap;
  A.rows = ctx->d_rows;
  A.perm = S.perm;
  A.part = S.part;
  A.first = S.first;
  A.hcol = S.hcol;
  A.hcount = S.hcount;
  A.rec = S.rec;
  A.vals = ctx->d_vals;
  A.rhs = ctx->d_rhs;
  A.y4 = S.vec;
  double *v0 = S.vec + 8 * (size_t)N;
  double **vecs[] = {&A.r1, &A.r2, &A.w, &A.w2, &A.ya, &A.yb, &A.x, &A.q, &A.dinv};
  for (int i = 0; i < 9; i++) *vecs[i] = v0 + i * (size_t)n3;
  A.sol = S.x;
  A.slots = S.slots;
  A.sc = S.sc;
  A.max_iter = max_iter;
  A.iters = S.slice > 0 ? S.slice : MR_ITERS;
  A.tol = rel_tol;
  A.fresh = 1;
  const void *fn = !halo                              ? (const void *)k_minres<false, 0, true>
                   : level == 2 && res == S.most[2] ? (const void *)k_minres<true, 2, false>
                   : level == 2                       ? (const void *)k_minres<true, 2, true>
                   : level == 1                       ? (const void *)k_minres<true, 1, true>
                                                      : (const void *)k_minres<true, 0, true>;
  ICF_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int it = 0, status = MR_RUNNING;
  double rel = 0;
  const int *flags = reinterpret_cast<const int *>(S.h_sc + SC_BAD);
  do {
    A.epoch0 = S.epoch;
    S.epoch += 2 * A.iters + 2;
    void *args[] = {&A};
    ICF_CUDA(ctx, cudaLaunchCooperativeKernel(fn, dim3(G), dim3(MR_THREADS), args, smem, s));
    ICF_CUDA(ctx, cudaMemcpyAsync(S.h_sc, S.sc, sizeof(double) * NSC, cudaMemcpyDeviceToHost, s));
    ICF_CUDA(ctx, cudaStreamSynchronize(s));
    A.fresh = 0;
    status = (int)S.h_sc[SC_STATUS];
    it = (int)S.h_sc[SC_IT];
    const double phibar = S.h_sc[SC_PHIBAR], beta1 = S.h_sc[SC_BETA1];
    if (flags[2] || status == MR_TIMEOUT) return icf_fail(ctx, ICF_ERR_CUDA, "linear solve: a grid-wide wait ran out");
    if (status == MR_BREAKDOWN)
      return icf_fail(ctx, ICF_ERR_NUMERIC, "linear solve: breakdown (preconditioned residual norm negative or not finite)");
    rel = beta1 > 0 ? phibar / beta1 : 0.0;
    if (!std::isfinite(rel)) return icf_fail(ctx, ICF_ERR_NUMERIC, "linear solve: non-finite residual");
  } while (status == MR_PAUSE);
  if (flags[0]) return icf_fail(ctx, ICF_ERR_NUMERIC, "linear solve: zero or non-finite diagonal block");
  S.n_indefinite = flags[1];
  if (iters) *iters = it;
  if (relres) *relres = rel;
  if (rel > rel_tol && it >= max_iter)
  {
    char buf[64];
    snprintf(buf, sizeof(buf), "%.3e", rel);
    return icf_fail(ctx, ICF_ERR_NUMERIC, "linear solve: no convergence in " + std::to_string(max_iter) +
                                              " iterations (relative residual " + buf + ")");
  }
  return ICF_OK;
}
