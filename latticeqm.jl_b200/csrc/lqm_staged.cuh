// Staged eigensolver for orders whose lower triangle fits the registers of one CTA
// (n <= kStMaxN): the per-k dense Hermitian eigenproblem of a whole list of k-points
// as a few kernels, each with the work split and the occupancy its own stage wants.
//
//   st_hetrd_kernel   H(k) and its Householder reduction to a real tridiagonal, one
//                     warp or one CTA per k-point, the lower triangle in registers;
//                     reflectors, tau, d, e to HBM
//   st_dc_kernel      eigenpairs of the tridiagonal: implicit QL on leaves of at most 16
//                     rows, divide-and-conquer merges above; the eigenvector columns that
//                     are needed, in ascending order
//   st_tfac_kernel    compact-WY factors of the reflectors, eight at a time
//   st_back_kernel    U = H_0 ... H_{n-2} Z on the FP64 tensor path, eight columns of U
//                     per warp held in accumulator fragments throughout
//   st_rho_kernel     rho_k = U g U^H (+ I) on the FP64 tensor path, lower blocks mirrored
//
// The stages pass 30 to 40 n^2 bytes per k-point through HBM, a few per cent of their
// time.  Every sum has a fixed order.  Measured on B200 (rho passes; milliseconds of
// hetrd, dc, tfac, back, rho; then the one-CTA kernel that ran them before):
//   n = 24, 16384 k-points: 0.42, 0.85, 0.16, 0.19, 0.10; 9.3
//   n = 96,  4096 k-points: 3.24, 3.56, 0.19, 0.96, 0.43; 26.8
//   n = 144, 2304 k-points: 7.45, 6.48, 0.19, 1.87, 0.81; 40.0
// (dc before the branch-free quotients and the first guess of the secular roots, which took
// the whole n = 96 pass on 8100 k-points from 17.5 to 16.3 ms).  The reference's counterpart is LAPACK's zheevr on
// Hermitian(M) (src/modules/Eigen/Eigen.jl:22-23); the steps are zhetd2, Cuppen's divide and
// conquer over implicit QL (EISPACK's imtql2), and zlarft / zlarfb.
#pragma once
#include "lqm_kernels.cuh"

namespace lqm {

constexpr int kStMaxN = 144;    // the lower triangle in four warps' registers and, above 64, shared memory
constexpr int kStNB = 8;        // reflectors per compact-WY block

__host__ __device__ inline int st_chunks(int n) { return (n + 31) / 32; }

// ---------------------------------------------------------------------------
// 1. H(k) and the Householder reduction.
// ---------------------------------------------------------------------------
struct StHetrdArgs {
  int n, nR, dim;
  const double2* blocks;
  const int64_t* keys;
  int64_t nk;
  const double* ks;
  double2* V;    // nk x (n x n): reflector j in column j, rows j+1.., leading 1
  double2* tau;  // nk x n
  double* d;     // nk x n
  double* e;     // nk x n
  unsigned long long* phase_cycles;
};

// Thread grid of one k-point: WR x WC warps of 4 x 8 lanes; thread (tr, tc) holds the
// elements (TR a + tr, TC b + tc) of the block lower triangle: the NA x NB blocks without
// those above the diagonal squares.  The diagonal squares (TC x TC) are held whole, so no
// element needs a mask.  The first KEPT blocks (by columns) are kept in shared memory, one
// element per thread and block and so without conflicts: they are finished first, and the
// registers they would take are worth more as a further CTA per SM.
template <int WR_, int WC_, int NB_, int KEPT_>
struct StGrid {
  static constexpr int WR = WR_, WC = WC_, W = WR * WC, TR = 4 * WR, TC = 8 * WC, KEPT = KEPT_;
  static constexpr int NB = NB_, NP = TC * NB, NA = NP / TR;
  static_assert(TC % TR == 0, "a diagonal square is a whole number of row blocks");
  // block (a, b) is below or in a diagonal square / in one
  static __host__ __device__ constexpr bool has(int a, int b) { return a < NA && TR * (a + 1) > TC * b; }
  static __host__ __device__ constexpr bool diag(int a, int b) { return has(a, b) && TR * a < TC * (b + 1); }
  // number of a block, column by column
  static __host__ __device__ constexpr int index(int a, int b) {
    int i = 0;
    for (int q = 0; q < b; ++q)
      for (int p = 0; p < NA; ++p) i += has(p, q) ? 1 : 0;
    for (int p = 0; p < a; ++p) i += has(p, b) ? 1 : 0;
    return i;
  }
  static __host__ __device__ constexpr bool kept(int a, int b) { return index(a, b) < KEPT; }
  static __host__ __device__ constexpr int at(int a, int b) { return 32 * W * index(a, b); }
  // complex per k-point: the kept blocks, x, v, w, the next column, row sums (WC parts),
  // column sums (WR parts), three scalars
  static constexpr int vec = 32 * W * KEPT + (4 + WC + WR) * NP + 3;
};
template <class G>
__host__ __device__ inline size_t st_hetrd_complex(int nR) {
  return (size_t)G::vec + nR + 2;  // .. | phases | k
}

// Sum over the warp in two tensor steps: ones times the lanes' values as a 4 x 8 operand
// gives the eight column sums, two per lane; the same again adds those.  Every lane gets
// the result.  Half the latency of five shuffle levels.
__device__ __forceinline__ double st_warp_sum(double v) {
  double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
  dmma_884(a0, a1, 1.0, v);
  dmma_884(b0, b1, 1.0, a0 + a1);
  return b0;
}

// Barrier of warps 0 and 1 of a CTA.
__device__ __forceinline__ void st_pair_sync() { asm volatile("bar.sync 1, 64;\n" ::: "memory"); }

// One pass over the trailing block of step j (columns and rows below j are finished: x, v
// and w are zero there): the rank-2 update by (v, w), then the Hermitian product with x in
// two halves: row sums of A(r, c) x_c (over the lanes of a row and WC warps) and, for the
// blocks below the diagonal squares, column sums of conj(A(r, c)) x_r (over the lanes of a
// column and WR warps).  Four row blocks at a time, so that a block column's 64
// multiply-adds come in independent chains; every exchange of a reduction halves what a
// lane keeps.  sA: the thread's elements of the blocks in shared memory.
template <class G>
__device__ __forceinline__ void st_pass(double2 (&A)[G::NA][G::NB], double2* sA, int j, const double2* x,
                                        const double2* v, const double2* w, double2* qr, double2* qc, int tr, int tc,
                                        int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int RG = 4;
  const int b0 = j / G::TC;
  double2 ca[G::NB];
#pragma unroll
  for (int b = 0; b < G::NB; ++b) ca[b] = cmk(0.0, 0.0);
#pragma unroll
  for (int a = 0; a < G::NA; a += RG) {
    if (G::TR * (a + RG) <= j) continue;  // these row blocks are finished (uniform)
    double2 rs[RG];
#pragma unroll
    for (int i = 0; i < RG; ++i) rs[i] = cmk(0.0, 0.0);
#pragma unroll
    for (int b = 0; b < G::NB; ++b) {
      if (!G::has(a, b) && !G::has(a + 1, b) && !G::has(a + 2, b) && !G::has(a + 3, b)) continue;
      if (b < b0) continue;  // finished columns (uniform)
      const int c = G::TC * b + tc;
      const double2 cv = cconj(v[c]), cw = cconj(w[c]), xc = x[c];
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        if (!G::has(a + i, b)) continue;
        const int r = G::TR * (a + i) + tr;
        const double2 t = cfms(cfms(G::kept(a + i, b) ? sA[G::at(a + i, b)] : A[a + i][b], v[r], cw), w[r], cv);
        if (G::kept(a + i, b)) sA[G::at(a + i, b)] = t;
        else A[a + i][b] = t;
        rs[i] = cfma(rs[i], t, xc);
        if (!G::diag(a + i, b)) ca[b] = cfma_conj(ca[b], t, x[r]);
      }
    }
    const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
    double2 k0 = h4 ? rs[2] : rs[0], k1 = h4 ? rs[3] : rs[1];
    const double2 s0 = h4 ? rs[0] : rs[2], s1 = h4 ? rs[1] : rs[3];
    k0.x += __shfl_xor_sync(FULL, s0.x, 4);
    k0.y += __shfl_xor_sync(FULL, s0.y, 4);
    k1.x += __shfl_xor_sync(FULL, s1.x, 4);
    k1.y += __shfl_xor_sync(FULL, s1.y, 4);
    double2 m = h2 ? k1 : k0;
    const double2 z = h2 ? k0 : k1;
    m.x += __shfl_xor_sync(FULL, z.x, 2);
    m.y += __shfl_xor_sync(FULL, z.y, 2);
    double u = h1 ? m.y : m.x;
    u += __shfl_xor_sync(FULL, h1 ? m.x : m.y, 1);
    const int ra = a + (h4 ? 2 : 0) + (h2 ? 1 : 0);
    if (ra < G::NA) ((double*)(qr + G::TR * ra + tr))[h1 ? 1 : 0] = u;
  }
#pragma unroll
  for (int b = 0; b < G::NB; ++b) {
    if (b < b0) continue;
    const bool h8 = lane & 8;
    double u = h8 ? ca[b].y : ca[b].x;
    u += __shfl_xor_sync(FULL, h8 ? ca[b].x : ca[b].y, 8);
    u += __shfl_xor_sync(FULL, u, 16);
    if (!(lane & 16)) ((double*)(qc + G::TC * b + tc))[h8 ? 1 : 0] = u;
  }
}

// Householder reduction of H(k) with the lower triangle in registers (LAPACK zhetd2 /
// zlarfg conventions: reflector j is zero above row j + 1 and one there, e real).  Only
// vectors pass through shared memory; 16 multiply-adds per element and step.
// Reflectors are kept unscaled: x = A(j+1:, j) with x_o = alpha - beta at o = j + 1, H = I -
// tau' x x^H with tau' = tau / |alpha - beta|^2.  H(k) is first scaled by a power of two to
// entries below one, so that their squares and cubes stay in range; a column whose squares
// fall below 1e-290 counts as zero.  The pass runs with x_o = 0, t = A x, so that it does
// not wait for the column's norm; with a the column o of the updated block,
//   q = t + (alpha - beta) a,   gamma = x^H q = x^H t + 2 Re((alpha - beta) conj(t_o)) +
//   |alpha - beta|^2 a_o        (a^H x = t_o, A being Hermitian),
//   w = tau' q - 1/2 |tau'|^2 gamma x,   next column = a - x conj(w_o) - w conj(x_o).
// Per step: the pass, a barrier, then warp 1 takes beta and tau while warp 0 sums t and
// x^H t, and warp 0 the rest; a barrier.  Bound by instruction issue and the latency of a
// step's serial part (n = 96: 1.55 instructions per cycle and SM with three CTAs, a third of
// them FP64; the FP64 pipe is 27% busy).  With the triangle in shared memory it took 6.37 ms
// at n = 96 and 4096 k-points, with eight warps per k-point 3.95, without the blocks in
// shared memory (two CTAs per SM) 3.93.
template <class G>
__device__ __forceinline__ void st_hetrd_body(const StHetrdArgs& p, int64_t k, double2* sm, int warp, int lane) {
  constexpr int NP = G::NP, NQ = (NP + 31) / 32, WC = G::WC, WR = G::WR;
  const int n = p.n;
  double2* xb = sm + 32 * G::W * G::KEPT;
  double2* vb = xb + NP;
  double2* wb = vb + NP;
  double2* cb = wb + NP;
  double2* qr = cb + NP;       // WC x NP
  double2* qc = qr + WC * NP;  // WR x NP
  double2* sc = qc + WR * NP;  // alpha, alpha - beta, tau'
  double2* ph = sc + 3;
  double* kpt = (double*)(ph + p.nR);
  const int tid = warp * 32 + lane;
  const int wr = warp % WR, wc = warp / WR;
  const int tr = 4 * wr + (lane >> 3), tc = 8 * wc + (lane & 7);
  auto sync = [&] {
    if (G::W == 1) __syncwarp();
    else __syncthreads();
  };
  const bool prof = p.phase_cycles != nullptr && tid == 0;
  long long t0 = prof ? clock64() : 0;
  if (tid < p.dim) kpt[tid] = p.ks[k * p.dim + tid];
  for (int r = tid; r < 3 * NP; r += 32 * G::W) xb[r] = cmk(0.0, 0.0);  // x, v, w
  sync();
  for (int r = tid; r < p.nR; r += 32 * G::W) {
    double dot = 0.0;
    for (int c = 0; c < p.dim; ++c) dot += kpt[c] * (double)p.keys[(int64_t)r * p.dim + c];
    double s, co;
    lqm_sincospi(2.0 * dot, &s, &co);
    ph[r] = cmk(co, s);
  }
  sync();
  // the upper triangle is the source: (r, c) below the diagonal = conj of the sum at (c, r)
  const int64_t nn = (int64_t)n * n;
  double2 A[G::NA][G::NB];
  double mx = 0.0;
#pragma unroll
  for (int b = 0; b < G::NB; ++b) {
    const int c = G::TC * b + tc;
    double2 s[G::NA];
#pragma unroll
    for (int a = 0; a < G::NA; ++a) s[a] = cmk(0.0, 0.0);
    for (int R = 0; R < p.nR; ++R) {
      const double2 f = ph[R];
      const double2* blk = p.blocks + R * nn;
#pragma unroll
      for (int a = 0; a < G::NA; ++a) {
        if (!G::has(a, b)) continue;
        const int r = G::TR * a + tr;
        const int u = G::diag(a, b) ? min(r, c) : c, l = G::diag(a, b) ? max(r, c) : r;
        if (l < n) s[a] = cadd(s[a], cmul(__ldg(blk + u + l * n), f));
      }
    }
#pragma unroll
    for (int a = 0; a < G::NA; ++a) {
      if (!G::has(a, b)) continue;
      const int r = G::TR * a + tr;
      if (G::diag(a, b) && c == r) s[a].y = 0.0;
      if (!G::diag(a, b) || c < r) s[a].y = -s[a].y;
      mx = fmax(mx, fmax(fabs(s[a].x), fabs(s[a].y)));
      if (b == 0 && c == 0 && r < n) cb[r] = s[a];  // column 0
      if (G::kept(a, b)) sm[G::at(a, b) + tid] = s[a];
      else A[a][b] = s[a];
    }
  }
  // entries below one: a power of two, exact both ways
  mx = warp_max(mx);
  if (G::W > 1) {
    if (lane == 0) qr[warp].x = mx;
    sync();
    mx = qr[0].x;
    for (int u = 1; u < G::W; ++u) mx = fmax(mx, qr[u].x);
  }
  double unit = 1.0;
  if (mx > 0.0 && mx <= 1.7976931348623157e308) { int ex; frexp(mx, &ex); unit = ldexp(1.0, ex); }
  const double inv = 1.0 / unit;
#pragma unroll
  for (int b = 0; b < G::NB; ++b)
#pragma unroll
    for (int a = 0; a < G::NA; ++a) {
      if (!G::has(a, b)) continue;
      if (G::kept(a, b)) sm[G::at(a, b) + tid] = cscale(inv, sm[G::at(a, b) + tid]);
      else A[a][b] = cscale(inv, A[a][b]);
    }
  sync();
  if (prof) {
    const long long t1 = clock64();
    atomicAdd(&p.phase_cycles[PH_BLOCH], (unsigned long long)(t1 - t0));
    t0 = t1;
  }
  double2* Vk = p.V + k * nn;
  double2* tauk = p.tau + k * n;
  double* dk = p.d + k * n;
  double* ek = p.e + k * n;
  if (warp == 0) {  // x_0, its alpha and d_0
    for (int r = 2 + lane; r < n; r += 32) xb[r] = cscale(inv, cb[r]);
    if (lane == 0) {
      dk[0] = cb[0].x;
      if (n > 1) sc[0] = cscale(inv, cb[1]);
    }
  }
  double2* x = xb;
  double2* v = vb;
  constexpr int WB = G::W > 1 ? 1 : 0;  // the warp of the norm, beta and tau
  for (int j = 0; j <= n - 2; ++j) {
    const int o = j + 1;
    sync();
    double2 alpha = cmk(0.0, 0.0);
    double nrm = 0.0;
    if (warp == WB) {
      alpha = sc[0];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int r = 32 * q + lane;
        if (r < NP) { const double2 t = x[r]; nrm = fma(t.x, t.x, fma(t.y, t.y, nrm)); }
      }
      nrm = st_warp_sum(nrm);
    }
    st_pass<G>(A, sm + tid, j, x, v, wb, qr + wc * NP, qc + wr * NP, tr, tc, lane);
    {  // column j + 1 of the updated block, for warp 0
      const int bo = o / G::TC, oc = o % G::TC;
#pragma unroll
      for (int b = 0; b < G::NB; ++b) {
        if (b != bo) continue;
        if (tc == oc)
#pragma unroll
          for (int a = 0; a < G::NA; ++a)
            if (G::has(a, b)) cb[G::TR * a + tr] = G::kept(a, b) ? sm[G::at(a, b) + tid] : A[a][b];
      }
    }
    sync();
    double2 amb = cmk(0.0, 0.0), tp = amb, scal = amb;
    if (warp == WB) {
      double2 tau = cmk(0.0, 0.0);
      double beta = alpha.x;
      if (fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, nrm)) >= 1e-290)
        zlarfg_scalars(alpha, nrm, &tau, &beta, &scal);  // scal = 1 / (alpha - beta); zero reflector: tau = scal = 0
      if (!(tau.x == 0.0 && tau.y == 0.0)) amb = cmk(alpha.x - beta, alpha.y);
      tp = cscale(scal.x * scal.x + scal.y * scal.y, tau);
      if (lane == 0) {
        sc[1] = amb;
        sc[2] = tp;
        tauk[j] = tau;
        ek[j] = beta * unit;
      }
    }
    if (warp == 0) {
      double2 tv[NQ], xv[NQ], ac[NQ];
      auto total = [&](int r) {
        double2 t = qr[r];
#pragma unroll
        for (int u = 1; u < WC; ++u) t = cadd(t, qr[u * NP + r]);
#pragma unroll
        for (int u = 0; u < WR; ++u) t = cadd(t, qc[u * NP + r]);
        return t;
      };
      double gam = 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int r = 32 * q + lane;
        tv[q] = xv[q] = ac[q] = cmk(0.0, 0.0);
        if (r >= o && r < n) {
          tv[q] = total(r);
          ac[q] = cb[r];
          xv[q] = x[r];
          gam = fma(xv[q].x, tv[q].x, fma(xv[q].y, tv[q].y, gam));
        }
      }
      const double2 to = total(o), ao = cb[o];
      gam = st_warp_sum(gam);
      if (G::W > 1) {
        st_pair_sync();
        amb = sc[1];
        tp = sc[2];
      }
      gam += 2.0 * (amb.x * to.x + amb.y * to.y) + (amb.x * amb.x + amb.y * amb.y) * ao.x;
      const double h = 0.5 * (tp.x * (tp.x * gam) + tp.y * (tp.y * gam));  // |tau'|^2 alone may overflow
      const double2 wo = csub(cmul(tp, cfma(to, amb, cmk(ao.x, 0.0))), cscale(h, amb));
      const double2 cw = cconj(wo), cx = cconj(amb);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int r = 32 * q + lane;
        if (r < NP) {
          const double2 xx = (r == o) ? amb : xv[q];
          const double2 wv = (r == o) ? wo : csub(cmul(tp, cfma(tv[q], amb, ac[q])), cscale(h, xx));
          wb[r] = wv;  // zero outside o .. n - 1
          const double2 t = cfms(cfms(ac[q], xx, cw), wv, cx);
          if (r == o) {
            x[o] = amb;
            dk[o] = t.x * unit;
          }
          if (r == o + 1) sc[0] = t;
          v[r] = (r > o + 1) ? t : cmk(0.0, 0.0);  // becomes x of the next step
        }
      }
    } else if (warp == WB) {
      st_pair_sync();
    }
    if (warp == WB) {  // the reflector, scaled (x_o is not read)
      if (lane == 0) Vk[o + (int64_t)j * n] = cmk(1.0, 0.0);
      for (int r = o + 1 + lane; r < n; r += 32) Vk[r + (int64_t)j * n] = cmul(scal, x[r]);
    }
    double2* t = x;
    x = v;
    v = t;
  }
  if (prof) atomicAdd(&p.phase_cycles[PH_HETRD], (unsigned long long)(clock64() - t0));
}

// One warp per k-point, WPC of them per CTA.
template <int NB, int WPC, int MINB>
__global__ void __launch_bounds__(32 * WPC, MINB) st_hetrd_warp_kernel(StHetrdArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  using G = StGrid<1, 1, NB, 0>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t k = (int64_t)blockIdx.x * WPC + warp;
  if (k >= a.nk) return;
  st_hetrd_body<G>(a, k, (double2*)smem + warp * st_hetrd_complex<G>(a.nR), 0, lane);
}

// One CTA of WR x WC warps per k-point.
template <int WR, int WC, int NB, int KEPT, int MINB>
__global__ void __launch_bounds__(32 * WR * WC, MINB) st_hetrd_kernel(StHetrdArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  st_hetrd_body<StGrid<WR, WC, NB, KEPT>>(a, blockIdx.x, (double2*)smem, threadIdx.x >> 5, threadIdx.x & 31);
}

// ---------------------------------------------------------------------------
// 2. Eigenpairs of the tridiagonal: QL leaves, divide-and-conquer merges.
// ---------------------------------------------------------------------------
constexpr int kStLeaf = 16;      // rows of a leaf at most (a half-warp solves one)
constexpr int kStMaxLeaves = 16;

struct StDcArgs {
  int n, depth;  // 2^depth leaves
  int64_t nk;
  const double* d;  // nk x n
  const double* e;  // nk x n
  double* bands;    // nk x n, ascending
  double* Z;        // nk x (n x n): the needed columns in ascending order, packed; null: eigenvalues only
  // occupation (rho_k wanted alone); eband_k null: every column
  double mu, T;
  const double* w;
  double* eband_k;  // nk
  double* occ;      // nk x n: the weight of each packed column in rho_k
  int* ncol;        // nk: packed columns
  int* comp;        // nk: 1 where rho_k = I + sum of the (negative) weights
  int* redo;        // nk flags: 1 where a leaf did not converge; then their count (zeroed before)
  int sweeps;       // QL sweeps of a leaf at most
  unsigned long long* phase_cycles;
};

__host__ __device__ inline int st_depth(int n) {
  int D = 0;
  while (((n - 1) >> D) + 1 > kStLeaf) ++D;
  return D;
}
// doubles of shared memory per k-point: Q (n x n) or the leaves' Z (16 n) and the boundary
// rows (4 n), then 12 n + 80 doubles and 12 n + 160 ints
__host__ __device__ inline size_t st_dc_doubles(int n, bool vec) {
  return (vec ? (size_t)n * n : (size_t)20 * n) + 12 * (size_t)n + 80 + (12 * (size_t)n + 160 + 1) / 2;
}

// Implicit QL (EISPACK imtql2's recurrences, the plane rotation from one reciprocal square
// root) of the leaf rows lo .. lo + s - 1 by a half-warp: lane i of it keeps d_i and e_i
// in registers and row i of Z in shared memory (Zl: (row, column) at row + ld column);
// every lane computes the rotation's scalars, on values passed by shuffles, and rotates
// its own row.  The two halves of a warp take their sweeps together: every loop's trip
// count comes from a vote or is a constant, so that the warp stays together and only
// assignments are conditional.  An off-diagonal entry is dropped below eps (|d_i| +
// |d_{i+1}|) + eps / 16 (of a matrix scaled to a largest entry below one).  Returns false
// where `sweeps` were not enough (about 2 s are needed).
constexpr int kStLeafSweeps = 30 * kStLeaf;
__device__ __forceinline__ bool st_leaf_ql(int s, double& d, double& e, double* Zl, int ld, int lane, int sweeps) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr double EPS = 2.0 * LQM_DEPS;
  const int i0 = lane & 15, half = lane & 16;
  const bool row = i0 < s;
  int l = 0;
  unsigned rem = 1;
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    const double dn = __shfl_down_sync(FULL, d, 1);
    const bool tiny = i0 >= s - 1 || fabs(e) <= EPS * (fabs(d) + fabs(dn)) + EPS / 16.0;
    const unsigned mask = (__ballot_sync(FULL, tiny) >> half) & 0xffffu;  // bit i: no coupling of i and i + 1
    // the first block [l, m] that is not diagonal yet (bits from s - 1 on are set)
    rem = ~mask & (0xffffu << l) & 0xffffu;
    if (!__any_sync(FULL, rem != 0u)) break;
    const bool live = rem != 0u;
    if (live) l = __ffs(rem) - 1;
    const int m = live ? l + __ffs(mask >> l) - 1 : l;
    // Wilkinson shift from its top 2 x 2
    const double dl = __shfl_sync(FULL, d, half + l), el = __shfl_sync(FULL, e, half + l);
    const double d1 = __shfl_sync(FULL, d, half + (l < 15 ? l + 1 : 15)), dm = __shfl_sync(FULL, d, half + m);
    const double gg = (d1 - dl) / (live ? 2.0 * el : 1.0);
    const double rr0 = sqrt(fma(gg, gg, 1.0));
    double g = dm - dl + (fabs(gg) > 1e150 ? 0.0 : el / (gg + (gg >= 0.0 ? rr0 : -rr0)));
    double sn = 1.0, c = 1.0, p = 0.0, di = dm;
    bool run = live;
    double h = (live && row) ? Zl[i0 + m * ld] : 0.0;
    int last = m;  // column that the carried entry of Z belongs to
    const int len = max(m - l, __shfl_xor_sync(FULL, m - l, 16));
    for (int u = 1; u <= len; ++u) {
      const int i = m - u;
      const bool act = run && i >= l;
      const int src = half + (act ? i : 0);
      const double ei = __shfl_sync(FULL, e, src), dd = __shfl_sync(FULL, d, src);
      const double zi = (act && row) ? Zl[i0 + i * ld] : 0.0;
      const double f = sn * ei, b = c * ei;
      const double t = fma(f, f, g * g);
      const bool split = act && t < 1e-290;  // nothing left of the bulge: the block splits at i + 1
      const bool rot = act && !split;
      const double ri = rsqrt(rot ? t : 1.0);
      const double r = t * ri, s1 = f * ri, c1 = g * ri, g1 = di - p;
      const double rr = fma(dd - g1, s1, 2.0 * c1 * b), p1 = s1 * rr;
      if (act && i0 == i + 1) {
        d = split ? g1 : g1 + p1;
        e = split ? 0.0 : i + 1 < m ? r : e;
      }
      if (split && i0 == m) e = 0.0;
      if (rot && row) Zl[i0 + (i + 1) * ld] = fma(s1, zi, c1 * h);
      if (rot) {
        h = fma(c1, zi, -(s1 * h));
        sn = s1;
        c = c1;
        p = p1;
        g = fma(c1, rr, -b);
        di = dd;
        last = i;
      }
      run = run && !split;
    }
    if (live && row) Zl[i0 + last * ld] = h;
    if (run && i0 == l) { d = di - p; e = g; }
    if (run && i0 == m) e = 0.0;
  }
  return rem == 0u;
}

// One CTA of NT threads per k-point.  The tridiagonal is torn into 2^depth leaves of at
// most 16 rows (Cuppen), a half-warp each; then the merges, depth by depth, as dc_solve
// makes them (same deflation, secular solver and Gu-Eisenstat z), with two differences:
//   * eigenvectors stay in their physical column (pc: the column of each sorted value);
//     a merge overwrites the columns of its non-deflated values only;
//   * the update Q <- Q U runs on the FP64 tensor path.  A warp takes eight new columns
//     and all rows of the node; the secular vectors are formed in the B fragments, one
//     division per lane and step, and never stored.  The columns of the upper and the lower
//     half are zero in the other half's rows: with the values ordered upper, mixed (by a
//     deflation rotation), lower, each half sums over its own range only.  Below the root
//     the new columns are held in registers (at most two sets of eight per warp, RT row
//     tiles) until every warp has read the old ones; at the root (RR row tiles) they go to
//     HBM in ascending order, and for rho_k alone only those that carry it.
template <int NT, int RT, int RR, int MINB>
__global__ void __launch_bounds__(NT, MINB) st_dc_kernel(StDcArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int NW = NT / 32, SETS = 2;
  const int n = a.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t k = blockIdx.x;
  const bool vec = a.Z != nullptr;
  const long long t0 = a.phase_cycles ? clock64() : 0;
  auto sync = [&] {
    if (NT == 32) __syncwarp();
    else __syncthreads();
  };
  double* Q = (double*)smem;
  double* QF = Q + 16 * n;  // eigenvalues only: first and last row of each node's Q, by sorted value
  double* QL = QF + n;
  double* FT = QL + n;
  double* LT = FT + n;
  double* ev = vec ? Q + (size_t)n * n : LT + n;
  double* ee = ev + n;
  double* zs = ee + n;
  double* ds = zs + n;
  EighVec S;
  S.dl = ds + n;
  S.zl = S.dl + n;
  S.troot = S.zl + n;
  S.zhat = S.troot + n;
  S.vals = S.zhat + n;
  S.dval = S.vals + n;
  S.rc = S.dval + n;
  S.rs = S.rc + n;
  double* red = S.rs + n;       // 48
  S.nrho = red + 48;            // 16
  double* sgn = S.nrho + 16;    // 16: the torn entry's sign times its modulus
  int* ib = (int*)(sgn + 16);
  int* pc = ib;                 // physical column of the sorted value
  int* own = pc + n;
  S.perm = own + n;
  S.colnd = S.perm + n;
  S.org = S.colnd + n;
  S.dcol = S.org + n;
  S.newpos = S.dcol + n;
  S.ri = S.newpos + n;
  S.rj = S.ri + n;
  int* pl = S.rj + n;           // the non-deflated values by half: upper, mixed, lower
  int* pq = pl + n;             // their physical columns
  int* typ = pq + n;            // 1: the value's column mixes both halves
  int* bnd = typ + n;           // 17
  int* nlo = bnd + 20;
  int* nmid = nlo + 16;
  int* nhi = nmid + 16;
  S.nk = nhi + 16;
  S.nrot = S.nk + 16;
  S.ndef = S.nrot + 16;
  int* k1 = S.ndef + 16;        // upper
  int* k12 = k1 + 16;           // upper and mixed
  if (vec)  // a column is zero outside its node's rows
    for (int i = tid; i < n * n; i += NT) Q[i] = 0.0;
  const int D = a.depth, nleaf = 1 << D;
  // leaf boundaries by repeated halving
  for (int i = tid; i <= nleaf; i += NT) {
    int lo = 0, hi = n;
    if (i == nleaf) lo = n;
    else
      for (int q = D - 1; q >= 0; --q) {
        const int mid = lo + (hi - lo) / 2;
        if ((i >> q) & 1) lo = mid;
        else hi = mid;
      }
    bnd[i] = lo;
  }
  // scale by a power of two to a largest entry in [1/2, 1)
  double mx = 0.0;
  for (int i = tid; i < n; i += NT) {
    ev[i] = a.d[k * n + i];
    ee[i] = i < n - 1 ? a.e[k * n + i] : 0.0;
    mx = fmax(mx, fmax(fabs(ev[i]), fabs(ee[i])));
  }
  mx = warp_max(mx);
  if (lane == 0) red[wid] = mx;
  sync();
  mx = red[0];
  for (int q = 1; q < NW; ++q) mx = fmax(mx, red[q]);
  double scale = 1.0;
  if (mx > 0.0 && mx <= 1.7976931348623157e308) { int ex; frexp(mx, &ex); scale = ldexp(1.0, ex); }
  const double inv = 1.0 / scale;
  if (tid == 0) {
    for (int i = 1; i < nleaf; ++i) {
      const double b = fabs(ee[bnd[i] - 1]);
      ev[bnd[i] - 1] -= b;
      ev[bnd[i]] -= b;
    }
  }
  sync();
  bool ok = true;
  for (int f0 = 2 * wid; f0 < nleaf; f0 += 2 * NW) {
    const int f = f0 + (lane >> 4), i0 = lane & 15;
    const bool have = f < nleaf;
    const int lo = have ? bnd[f] : 0, s = have ? bnd[f + 1] - lo : 0;
    double d = i0 < s ? ev[lo + i0] * inv : 0.0, e = i0 < s - 1 ? ee[lo + i0] * inv : 0.0;
    double* Zl = vec ? Q + lo + (size_t)lo * n : Q + 16 * lo;
    const int ld = vec ? n : 16;
    if (i0 < s)
      for (int c = 0; c < s; ++c) Zl[i0 + c * ld] = i0 == c ? 1.0 : 0.0;
    __syncwarp();
    ok = st_leaf_ql(s, d, e, Zl, ld, lane, a.sweeps) && ok;
    __syncwarp();
    int pos = 0;
    const long long b = __double_as_longlong(d);
    const long long key = d == d ? b ^ ((b >> 63) & 0x7fffffffffffffffLL) : 0x7fffffffffffffffLL;  // NaN last (dc_less)
    for (int j = 0; j < 16; ++j) {
      const long long o = __shfl_sync(FULL, key, (lane & 16) + j);
      pos += j < s && (o < key || (o == key && j < i0));
    }
    if (i0 < s) {
      ev[lo + pos] = d;
      pc[lo + pos] = lo + i0;
      if (!vec) {
        QF[lo + pos] = Zl[i0 * ld];
        QL[lo + pos] = Zl[s - 1 + i0 * ld];
      }
    }
  }
  if (!ok && (lane & 15) == 0) {
    if (atomicExch(a.redo + k, 1) == 0) atomicAdd(a.redo + a.nk, 1);
  }
  sync();
  int cbeg = 0, cend = n;
  // the packed columns that rho_k needs (values ascending, final in ev): see StDcArgs
  auto occupation = [&] {
    if (!a.eband_k) return;
    int* redi = (int*)(red + 16);
    double eb = 0.0;
    int cnt[4] = {0, 0, n, -1};  // exactly full, exactly empty, first not full, last not empty
    for (int c = tid; c < n; c += NT) {
      const double ej = ev[c] * scale, f = fermi(ej - a.mu, a.T);
      eb += ej * f;
      cnt[0] += f == 1.0;
      cnt[1] += f == 0.0;
      if (f != 1.0) cnt[2] = min(cnt[2], c);
      if (f != 0.0) cnt[3] = max(cnt[3], c);
    }
    eb = warp_sum(eb);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      cnt[0] += __shfl_xor_sync(FULL, cnt[0], s);
      cnt[1] += __shfl_xor_sync(FULL, cnt[1], s);
      cnt[2] = min(cnt[2], __shfl_xor_sync(FULL, cnt[2], s));
      cnt[3] = max(cnt[3], __shfl_xor_sync(FULL, cnt[3], s));
    }
    if (lane == 0) {
      red[wid] = eb;
#pragma unroll
      for (int q = 0; q < 4; ++q) redi[4 * wid + q] = cnt[q];
    }
    sync();
    eb = 0.0;
    cnt[0] = cnt[1] = 0;
    cnt[2] = n;
    cnt[3] = -1;
    for (int q = 0; q < NW; ++q) {
      eb += red[q];
      cnt[0] += redi[4 * q];
      cnt[1] += redi[4 * q + 1];
      cnt[2] = min(cnt[2], redi[4 * q + 2]);
      cnt[3] = max(cnt[3], redi[4 * q + 3]);
    }
    // rho_k = sum f u u^H over the states that are not exactly empty or, when more states
    // are exactly full than exactly empty, I - sum (1 - f) u u^H over those not exactly full
    const bool comp = cnt[0] > cnt[1];
    if (comp) cbeg = cnt[2];
    else cend = cnt[3] + 1;
    for (int c = cbeg + tid; c < cend; c += NT) {
      const double f = fermi(ev[c] * scale - a.mu, a.T);
      a.occ[k * n + (c - cbeg)] = comp ? f - 1.0 : f;
    }
    if (tid == 0) {
      a.eband_k[k] = a.w[k] * eb;
      a.comp[k] = comp ? 1 : 0;
    }
  };
  double* Zk = vec ? a.Z + k * (int64_t)n * n : nullptr;
  if (D == 0 && vec) {
    occupation();
    for (int c = cbeg + wid; c < cend; c += NW)
      for (int r = lane; r < n; r += 32) Zk[(c - cbeg) * n + r] = Q[r + pc[c] * n];
  }
  for (int dep = D - 1; dep >= 0; --dep) {
    const int nn = 1 << dep, sh = D - dep;
    const bool root = dep == 0;
    for (int q = tid; q < nn; q += NT) {
      const int lo = bnd[q << sh], m = bnd[(2 * q + 1) << (sh - 1)];
      nlo[q] = lo;
      nmid[q] = m;
      nhi[q] = bnd[(q + 1) << sh];
      sgn[q] = ee[m - 1] * inv;
    }
    sync();
    // A: node of each value, z (scaled by 1 / sqrt 2), the merged order
    for (int i = tid; i < n; i += NT) {
      int q = 0;
      while (nhi[q] <= i) ++q;
      own[i] = q;
      const int lo = nlo[q], m = nmid[q], hi = nhi[q];
      const bool up = i < m;
      const double sg = sgn[q] < 0.0 ? -1.0 : 1.0;
      double z;
      if (vec) {
        z = up ? Q[m - 1 + pc[i] * n] : sg * Q[m + pc[i] * n];
      } else {
        z = up ? QL[i] : sg * QF[i];
        FT[i] = up ? QF[i] : 0.0;
        LT[i] = up ? 0.0 : QL[i];
      }
      const double di = ev[i];
      int p, b, c;
      if (up) {  // first value of the lower half that is >= di
        for (p = m, b = hi; p < b;) { c = (p + b) >> 1; if (dc_less(ev[c], di)) p = c + 1; else b = c; }
        p = i + (p - m);
      } else {   // first value of the upper half that is > di
        for (p = lo, b = m; p < b;) { c = (p + b) >> 1; if (!dc_less(di, ev[c])) p = c + 1; else b = c; }
        p = p + (i - m);
      }
      zs[p] = z * 0.70710678118654752440;
      ds[p] = di;
      S.perm[p] = i;
      typ[i] = 0;
    }
    sync();
    // B: deflation, a warp per node.  Values with a tiny z drop out; when no neighbours
    // among the others are close enough to be rotated, that is all, else one lane
    // goes through them in order (deflate_node).
    DCPlan P;
    P.lo = nlo;
    P.mid = nmid;
    P.hi = nhi;
    for (int q = wid; q < nn; q += NW) {
      const int lo = nlo[q], hi = nhi[q];
      const double beta = fabs(sgn[q]), rho = 2.0 * beta;
      double zm = 0.0, dm = 0.0;
      for (int p = lo + lane; p < hi; p += 32) { zm = fmax(zm, fabs(zs[p])); dm = fmax(dm, fabs(ds[p])); }
      zm = __shfl_sync(FULL, warp_max(zm), 0);
      dm = __shfl_sync(FULL, warp_max(dm), 0);
      const double tol = 8.0 * LQM_DEPS * fmax(dm, zm);
      int kk = 0, nd = 0;
      if (rho * zm > tol)
        for (int p0 = lo; p0 < hi; p0 += 32) {
          const int p = p0 + lane;
          const bool in = p < hi;
          const double z = in ? zs[p] : 0.0, dv = in ? ds[p] : 0.0;
          const bool tiny = in && rho * fabs(z) <= tol, live = in && !tiny;
          const unsigned ml = __ballot_sync(FULL, live), mt = __ballot_sync(FULL, tiny);
          const unsigned below = (1u << lane) - 1u;
          if (live) {
            const int x = lo + kk + __popc(ml & below);
            S.dl[x] = dv;
            S.zl[x] = z;
            S.colnd[x] = S.perm[p];
          }
          if (tiny) {
            const int x = lo + nd + __popc(mt & below);
            S.dval[x] = dv;
            S.dcol[x] = S.perm[p];
          }
          kk += __popc(ml);
          nd += __popc(mt);
        }
      __syncwarp();
      bool close = !(rho * zm > tol);
      for (int p = lane; p < kk - 1; p += 32) {
        const double za = S.zl[lo + p], zb = S.zl[lo + p + 1];
        close = close || fabs((S.dl[lo + p + 1] - S.dl[lo + p]) * zb * za) <= tol * (zb * zb + za * za);
      }
      if (__any_sync(FULL, close)) {
        if (lane == 0) {
          deflate_node(q, P, S, beta, zs, ds);
          for (int r = 0; r < S.nrot[q]; ++r) {  // survivors of a rotation across the halves are mixed
            const int i = S.ri[lo + r], j = S.rj[lo + r];
            if (typ[i] || (i < nmid[q]) != (j < nmid[q])) typ[i] = typ[j] = 1;
          }
        }
      } else if (lane == 0) {
        S.nk[q] = kk;
        S.ndef[q] = nd;
        S.nrot[q] = 0;
        S.nrho[q] = rho;
      }
      __syncwarp();
      if (vec) {  // the non-deflated values by half
        const int nk = S.nk[q], mid = nmid[q];
        int c0 = 0, c1 = 0, c2 = 0;
        for (int pass = 0; pass < 2; ++pass) {
          int x0 = lo, x1 = lo + c0, x2 = lo + c0 + c1;
          if (pass == 1 && lane == 0) { k1[q] = c0; k12[q] = c0 + c1; }
          for (int p0 = 0; p0 < nk; p0 += 32) {
            const int p = p0 + lane;
            const int i = p < nk ? S.colnd[lo + p] : -1;
            const bool mi = i >= 0 && typ[i], up = i >= 0 && !mi && i < mid, dn = i >= 0 && !mi && i >= mid;
            const unsigned mu_ = __ballot_sync(FULL, up), mm = __ballot_sync(FULL, mi), md = __ballot_sync(FULL, dn);
            const unsigned below = (1u << lane) - 1u;
            if (pass == 0) {
              c0 += __popc(mu_);
              c1 += __popc(mm);
              c2 += __popc(md);
            } else {
              const int x = up ? x0 + __popc(mu_ & below) : mi ? x1 + __popc(mm & below) : x2 + __popc(md & below);
              if (i >= 0) { pl[x] = p; pq[x] = pc[i]; }
              x0 += __popc(mu_);
              x1 += __popc(mm);
              x2 += __popc(md);
            }
          }
        }
      }
    }
    sync();
    // C: secular roots
    {
      int kmax = 1;
      for (int q = 0; q < nn; ++q) kmax = max(kmax, S.nk[q]);
      const int gw = secular_width(kmax, 32), gpw = 32 / gw, gl = lane % gw;
      for (int base = wid * gpw; base < n; base += NW * gpw) {
        const int i = base + lane / gw;
        int lo = 0, q = 0, kk = 0;
        bool active = false;
        if (i < n) {
          q = own[i];
          lo = nlo[q];
          kk = S.nk[q];
          active = i - lo < kk;
        }
        int org = 0;
        double tr = 0.0;
        secular_root_group(active, gw, gl, active ? kk : 1, S.dl + lo, S.zl + lo, active ? S.nrho[q] : 1.0, i - lo,
                           &org, &tr);
        if (active && gl == 0) { S.org[i] = org; S.troot[i] = tr; }
      }
    }
    sync();
    // D: Gu-Eisenstat z (four lanes per value); the deflation rotations; the merged values
    for (int base = wid * 8; base < n; base += 8 * NW) {
      const int i = base + g;
      const bool in = i < n;
      const int q = in ? own[i] : 0, lo = nlo[q], it = i - lo, kk = S.nk[q];
      const bool live = in && it < kk;
      const double* dl = S.dl + lo;
      double prod = 1.0;
      if (live) {
        const double rho = S.nrho[q], di = dl[it];
        for (int j = t; j < kk; j += 4) {
          const double dij = (di - dl[S.org[lo + j]]) - S.troot[lo + j];
          prod *= lqm_div_normal(-dij, j == it ? rho : dl[j] - di);
        }
      }
      prod *= __shfl_xor_sync(FULL, prod, 1);
      prod *= __shfl_xor_sync(FULL, prod, 2);
      if (in && t == 0) {
        const double zh = sqrt(fabs(prod));
        if (live) S.zhat[i] = S.zl[i] < 0.0 ? -zh : zh;
        S.vals[i] = live ? dl[S.org[i]] + S.troot[i] : S.dval[lo + it - kk];
      }
    }
    if (vec) {
      for (int r = tid; r < n; r += NT) {
        const int q = own[r], lo = nlo[q], nr = S.nrot[q];
        for (int u = 0; u < nr; ++u) {
          const int x = r + pc[S.ri[lo + u]] * n, y = r + pc[S.rj[lo + u]] * n;
          const double c = S.rc[lo + u], s = S.rs[lo + u], qx = Q[x], qy = Q[y];
          Q[x] = c * qx + s * qy;
          Q[y] = c * qy - s * qx;
        }
      }
    } else {
      for (int u2 = tid; u2 < 2 * nn; u2 += NT) {
        const int q = u2 >> 1, lo = nlo[q], nr = S.nrot[q];
        double* row = (u2 & 1) ? LT : FT;
        for (int u = 0; u < nr; ++u) {
          const int x = S.ri[lo + u], y = S.rj[lo + u];
          const double c = S.rc[lo + u], s = S.rs[lo + u], rx = row[x], ry = row[y];
          row[x] = c * rx + s * ry;
          row[y] = c * ry - s * rx;
        }
      }
    }
    sync();
    for (int i = tid; i < n; i += NT) {
      const int q = own[i], lo = nlo[q], hi = nhi[q], it = i - lo, kk = S.nk[q];
      const double v = S.vals[i];
      int pos = lo;
      if (v == v)
        for (int j = lo; j < hi; ++j) { const double vj = S.vals[j]; pos += (vj < v) || (vj == v && j < i); }
      else  // NaN: after every number, by index
        for (int j = lo; j < hi; ++j) pos += S.vals[j] == S.vals[j] || j < i;
      S.newpos[i] = pos;
      ev[pos] = v;
      // the physical column of this value: a non-deflated value takes that of its place
      S.perm[pos] = pc[it < kk ? S.colnd[i] : S.dcol[lo + it - kk]];
    }
    sync();
    if (!vec) {
      for (int c = wid; c < n; c += NW) {
        const int q = own[c], lo = nlo[q], it = c - lo, kk = S.nk[q], dst = S.newpos[c];
        if (it < kk) {
          const double* dl = S.dl + lo;
          const double lorg = dl[S.org[c]], tq = S.troot[c];
          double ss = 0.0, f = 0.0, l = 0.0;
          for (int p = lane; p < kk; p += 32) {
            const double u = lqm_div_normal(S.zhat[lo + p], (dl[p] - lorg) - tq);
            const int col = S.colnd[lo + p];
            ss += u * u;
            f += FT[col] * u;
            l += LT[col] * u;
          }
          ss = warp_sum(ss);
          f = warp_sum(f);
          l = warp_sum(l);
          if (lane == 0) {
            const double sc = 1.0 / sqrt(ss);
            QF[dst] = f * sc;
            QL[dst] = l * sc;
          }
        } else if (lane == 0) {
          const int src = S.dcol[lo + it - kk];
          QF[dst] = FT[src];
          QL[dst] = LT[src];
        }
      }
      sync();
      continue;
    }
    if (root) occupation();
    // H: eight new columns of node q, from value c0 on, as R tiles of 8 rows (the upper
    // half's rows first): acc = Q U scaled to unit columns
    auto columns = [&](int q, int c0, auto& acc) {
      constexpr int R = sizeof(acc) / sizeof(acc[0]);
      const int lo = nlo[q], mid = nmid[q], hi = nhi[q], kk = S.nk[q], ku = k1[q], kum = k12[q];
      const int tu = (mid - lo + 7) >> 3;  // row tiles of the upper half
      const int it = c0 + g;
      const bool in = it < kk;
      const double* dl = S.dl + lo;
      const double lorg = in ? dl[S.org[lo + it]] : 0.0, tq = in ? S.troot[lo + it] : 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0.0;
      double ss = 0.0;
      for (int x = 0; x < kk; x += 4) {
        const bool px = x + t < kk;
        const int p = px ? pl[lo + x + t] : 0, col = px ? pq[lo + x + t] : lo;
        const double u = (in && px) ? lqm_div_normal(S.zhat[lo + p], (dl[p] - lorg) - tq) : 0.0;
        ss = fma(u, u, ss);
        const double* qc = Q + (size_t)col * n;
        const bool upper = x < kum, lower = x + 4 > ku;  // uniform
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool isup = r < tu;
          if (isup ? !upper : !lower) continue;
          const int row = isup ? lo + 8 * r + g : mid + 8 * (r - tu) + g;
          const bool have = px && row < (isup ? mid : hi);
          if (!isup && mid + 8 * (r - tu) >= hi) continue;
          dmma_884(acc[r][0], acc[r][1], have ? qc[row] : 0.0, u);
        }
      }
      ss += __shfl_xor_sync(FULL, ss, 1);
      ss += __shfl_xor_sync(FULL, ss, 2);
      const double sc = in ? 1.0 / sqrt(ss) : 0.0;
      const double sa = __shfl_sync(FULL, sc, 8 * t), sb = __shfl_sync(FULL, sc, 8 * t + 4);
#pragma unroll
      for (int r = 0; r < R; ++r) { acc[r][0] *= sa; acc[r][1] *= sb; }
    };
    if (!root) {
      // unit (node, eight columns): two per warp at most, as columns() of all nodes fill
      // n / 8 + nodes units
      double acc[SETS][RT][2];
      int uq[SETS], uc[SETS];
#pragma unroll
      for (int s = 0; s < SETS; ++s) {
        int u = wid + s * NW, q = 0;
        while (q < nn && u >= (S.nk[q] + 7) >> 3) { u -= (S.nk[q] + 7) >> 3; ++q; }
        uq[s] = q < nn ? q : -1;
        uc[s] = 8 * u;
        if (uq[s] >= 0) columns(q, 8 * u, acc[s]);
      }
      sync();
#pragma unroll
      for (int s = 0; s < SETS; ++s) {
        if (uq[s] < 0) continue;
        const int q = uq[s], lo = nlo[q], mid = nmid[q], hi = nhi[q], kk = S.nk[q], tu = (mid - lo + 7) >> 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int it = uc[s] + 2 * t + h;
          if (it >= kk) continue;
          double* dst = Q + (size_t)pc[S.colnd[lo + it]] * n;
#pragma unroll
          for (int r = 0; r < RT; ++r) {
            const int row = r < tu ? lo + 8 * r + g : mid + 8 * (r - tu) + g;
            if (row < (r < tu ? mid : hi)) dst[row] = acc[s][r][h];
          }
        }
      }
      sync();
      for (int i = tid; i < n; i += NT) pc[i] = S.perm[i];
      sync();
    } else {
      const int kk = S.nk[0], mid = nmid[0], tu = (mid + 7) >> 3;
      int i0 = 0, i1 = 0;  // non-deflated values among the needed columns: a range, as both ascend
      for (int p0 = 0; p0 < kk; p0 += 32) {
        const int p = p0 + lane, c = p < kk ? S.newpos[p] : n;
        i0 += __popc(__ballot_sync(FULL, p < kk && c < cbeg));
        i1 += __popc(__ballot_sync(FULL, p < kk && c < cend));
      }
      for (int c0 = i0 + 8 * wid; c0 < i1; c0 += 8 * NW) {
        double acc[RR][2];
        columns(0, c0, acc);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int it = c0 + 2 * t + h;
          if (it >= i1) continue;
          const int c = S.newpos[it];
          if (c < cbeg || c >= cend) continue;  // NaN among the values: the places do not ascend
          double* dst = Zk + (c - cbeg) * n;
#pragma unroll
          for (int r = 0; r < RR; ++r) {
            const int row = r < tu ? 8 * r + g : mid + 8 * (r - tu) + g;
            if (row < (r < tu ? mid : n)) dst[row] = acc[r][h];
          }
        }
      }
      for (int i = kk + wid; i < n; i += NW) {  // deflated
        const int c = S.newpos[i];
        if (c < cbeg || c >= cend) continue;
        const double* src = Q + (size_t)pc[S.dcol[i - kk]] * n;
        for (int r = lane; r < n; r += 32) Zk[(c - cbeg) * n + r] = src[r];
      }
    }
  }
  for (int i = tid; i < n; i += NT) a.bands[k * n + i] = ev[i] * scale;
  if (tid == 0 && vec) a.ncol[k] = cend - cbeg;
  if (a.phase_cycles && tid == 0) atomicAdd(&a.phase_cycles[PH_DC], (unsigned long long)(clock64() - t0));
}

// ---------------------------------------------------------------------------
// 3. Compact-WY factors, one warp per (k-point, block of kStNB reflectors).
// ---------------------------------------------------------------------------
struct StBackArgs {
  int n;
  int64_t nk;
  const double2* V;    // nk x (n x n)
  const double2* tau;  // nk x n
  double2* Tm;         // nk x P x (8 x 8), T(l, i) at l + 8 i, P = ceil((n - 1) / 8)
  const double* Z;     // nk x (n x n)
  const int* ncol;     // nk
  double2* U;          // nk x (n x n)
  int groups;          // column groups per k-point
  unsigned long long* phase_cycles;
};
__host__ __device__ inline int st_panels(int n) { return (n - 1 + kStNB - 1) / kStNB; }

// T of H_{j0} ... H_{j0+7} = I - V T V^H (LAPACK zlarft, forward): T(i, i) = tau_i,
// T(l, i) = -tau_i sum_{l <= q < i} T(l, q) (V^H V)(q, i).  Four warps per CTA.
__global__ void __launch_bounds__(128) st_tfac_kernel(StBackArgs a) {
  __shared__ double2 gs[4][kStNB * kStNB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = a.n, P = st_panels(n);
  const int64_t id = (int64_t)blockIdx.x * 4 + warp;
  if (id >= a.nk * P) return;
  const int64_t k = id / P;
  const int p = (int)(id - k * P), j0 = p * kStNB, nb = min(kStNB, n - 1 - j0);
  const double2* V = a.V + k * (int64_t)n * n + (int64_t)j0 * n;
  double2 acc[kStNB * (kStNB - 1) / 2];
#pragma unroll
  for (int q = 0; q < kStNB * (kStNB - 1) / 2; ++q) acc[q] = cmk(0.0, 0.0);
  for (int r = j0 + 1 + lane; r < n; r += 32) {
    double2 v[kStNB];
#pragma unroll
    for (int i = 0; i < kStNB; ++i) v[i] = (i < nb && r > j0 + i) ? V[r + (int64_t)i * n] : cmk(0.0, 0.0);
    int u = 0;
#pragma unroll
    for (int i = 1; i < kStNB; ++i)
#pragma unroll
      for (int q = 0; q < i; ++q, ++u) acc[u] = cfma_conj(acc[u], v[q], v[i]);
  }
  double2* G = gs[warp];
  {
    int u = 0;
#pragma unroll
    for (int i = 1; i < kStNB; ++i)
#pragma unroll
      for (int q = 0; q < i; ++q, ++u) {
        const double x = warp_sum(acc[u].x), y = warp_sum(acc[u].y);
        if (lane == 0) G[q + i * kStNB] = cmk(x, y);
      }
  }
  __syncwarp();
  if (lane < kStNB) {
    const int l = lane;
    double2 t[kStNB];
#pragma unroll
    for (int i = 0; i < kStNB; ++i) {
      const double2 ti = i < nb ? a.tau[k * n + j0 + i] : cmk(0.0, 0.0);
      double2 s = cmk(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < kStNB; ++q)
        if (q < i && q >= l) s = cfma(s, t[q], G[q + i * kStNB]);
      t[i] = (i == l) ? ti : (i > l) ? cmul(cmk(-ti.x, -ti.y), s) : cmk(0.0, 0.0);
    }
    double2* Tp = a.Tm + id * (kStNB * kStNB);
#pragma unroll
    for (int i = 0; i < kStNB; ++i) Tp[l + kStNB * i] = t[i];
  }
}

// ---------------------------------------------------------------------------
// 4. U = H_0 ... H_{n-2} Z.
// ---------------------------------------------------------------------------
// A warp holds eight columns of U for all rows as the accumulators of 8 x 8 tiles of
// U^T (re and im; RT row tiles cover n): lane (g, t) has U(8 i + 2 t + h, column g).  As
// the sum over rows may take them in any order, the same registers are the A operand of
// X^T = U^T conj(V) with k index t standing for row 8 i + 2 t + h, and X^T and Y^T = X^T
// T^T chain the same way into U^T -= Y^T V^T: between the products nothing moves.  V and
// T of the next block arrive by cp.async meanwhile.  In shared memory the block's
// reflectors are rows of 8 RT + 1 complex (== 1 mod 8 16-byte units: both fragment
// reads conflict-free).
constexpr int kStBackWarps = 6;
__host__ __device__ constexpr int st_back_pitch(int RT) { return 8 * RT + 1; }
__host__ __device__ constexpr size_t st_back_smem(int RT) {
  return (size_t)2 * (kStNB * st_back_pitch(RT) + kStNB * kStNB) * 16;
}
__device__ __forceinline__ void st_cp16(void* sdst, const void* gsrc, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  const int nbytes = valid ? 16 : 0;  // 0: zero-filled, nothing is read
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void st_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void st_cp_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// grid: groups column groups of 8 kStBackWarps of each k-point, one k-point after the other
template <int RT, int MINB>
__global__ void __launch_bounds__(32 * kStBackWarps, MINB) st_back_kernel(StBackArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int PT = st_back_pitch(RT), STG = kStNB * PT + kStNB * kStNB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n = a.n, P = st_panels(n);
  const int64_t k = blockIdx.x / a.groups;
  const int K = a.ncol[k];
  const int cb = (int)(blockIdx.x % a.groups) * 8 * kStBackWarps;
  if (cb >= K) return;
  const long long t0 = a.phase_cycles ? clock64() : 0;
  const int c = cb + 8 * warp + g;  // this lane's column of U
  const bool busy = cb + 8 * warp < K;
  const int64_t nn = (int64_t)n * n;
  const double2* V = a.V + k * nn;
  const double2* Tm = a.Tm + k * P * (kStNB * kStNB);
  double2* stg = (double2*)smem;
  auto issue = [&](int p, int b) {
    double2* dst = stg + b * STG;
    const int j0 = p * kStNB;
    for (int u = threadIdx.x; u < kStNB * 8 * RT; u += blockDim.x) {
      const int i = u / (8 * RT), r = u % (8 * RT);
      const bool ok = r < n && j0 + i < n - 1 && r > j0 + i;
      st_cp16(dst + i * PT + r, ok ? (const void*)(V + r + (int64_t)(j0 + i) * n) : (const void*)V, ok);
    }
    for (int u = threadIdx.x; u < kStNB * kStNB; u += blockDim.x)
      st_cp16(dst + kStNB * PT + u, Tm + p * (kStNB * kStNB) + u, true);
    st_cp_commit();
  };
  issue(P - 1, 0);
  double ur[RT][2], ui[RT][2];
  const double* Zc = a.Z + k * nn + (int64_t)c * n;
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * i + 2 * t + h;
      ur[i][h] = (c < K && r < n) ? Zc[r] : 0.0;
      ui[i][h] = 0.0;
    }
  for (int p = P - 1, b = 0; p >= 0; --p, b ^= 1) {
    st_cp_wait();
    __syncthreads();  // block p has landed; every warp is past block p + 1's buffer
    if (p > 0) issue(p - 1, b ^ 1);
    if (!busy) continue;
    const double2* vs = stg + b * STG;
    const double2* ts = vs + kStNB * PT;
    const int first = (p * kStNB + 1) >> 3;  // first row tile that the block touches
    // X^T = U^T conj(V): two partial sums per product (the tile's even and odd rows)
    double xr[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, xi[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    double yr[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, yi[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      if (i < first) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 v = vs[g * PT + 8 * i + 2 * t + h];
        dmma_884(xr[h][0], xr[h][1], ur[i][h], v.x);
        dmma_884(yr[h][0], yr[h][1], ui[i][h], v.y);
        dmma_884(xi[h][0], xi[h][1], ui[i][h], v.x);
        dmma_884(yi[h][0], yi[h][1], ur[i][h], -v.y);
      }
    }
    // X^T (column g; reflectors 2 t + h); Y^T = X^T T^T
    double zr[2] = {0.0, 0.0}, zi[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double ar = (xr[0][h] + xr[1][h]) + (yr[0][h] + yr[1][h]);
      const double ai = (xi[0][h] + xi[1][h]) + (yi[0][h] + yi[1][h]);
      const double2 tv = ts[g + kStNB * (2 * t + h)];  // T(g, 2 t + h)
      dmma_884(zr[0], zr[1], ar, tv.x);
      dmma_884(zr[0], zr[1], -ai, tv.y);
      dmma_884(zi[0], zi[1], ar, tv.y);
      dmma_884(zi[0], zi[1], ai, tv.x);
    }
    // U^T -= Y^T V^T
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      if (i < first) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 v = vs[(2 * t + h) * PT + 8 * i + g];
        dmma_884(ur[i][0], ur[i][1], -zr[h], v.x);
        dmma_884(ui[i][0], ui[i][1], -zr[h], v.y);
        dmma_884(ur[i][0], ur[i][1], zi[h], v.y);
        dmma_884(ui[i][0], ui[i][1], -zi[h], v.x);
      }
    }
  }
  if (busy && c < K) {
    double2* Uc = a.U + k * nn + (int64_t)c * n;
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 8 * i + 2 * t + h;
        if (r < n) Uc[r] = cmk(ur[i][h], ui[i][h]);
      }
  }
  if (a.phase_cycles && threadIdx.x == 0)
    atomicAdd(&a.phase_cycles[PH_BACK], (unsigned long long)(clock64() - t0));
}

// ---------------------------------------------------------------------------
// 5. rho_k = sum_c occ_c u_c u_c^H (+ I).
// ---------------------------------------------------------------------------
struct StRhoArgs {
  int n;
  int64_t nk;
  const double2* U;   // nk x (n x n), the packed columns from column first[k] on (null: 0)
  const int* first;
  const double* occ;  // nk x n
  const int* ncol;
  const int* comp;
  double2* rho;       // nk x (n x n)
  unsigned long long* phase_cycles;
};

// Occupations of all n columns of U for st_rho_kernel, a warp per k-point: the same choice
// of the columns that rho_k needs as the density passes make, and its band energy.
__global__ void __launch_bounds__(128) st_occ_kernel(int n, int64_t nk, const double* bands, double mu_val,
                                                     const double* mu_ptr, double T, const double* w, double* eband_k,
                                                     double* occ, int* first, int* ncol, int* comp) {
  const int lane = threadIdx.x & 31;
  const int64_t k = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (k >= nk) return;
  const double mu = mu_ptr ? *mu_ptr : mu_val;
  const double* bk = bands + k * n;
  double eb = 0.0;
  int full = 0, empty = 0, c0 = n, c1 = -1;
  for (int c = lane; c < n; c += 32) {
    const double e = bk[c], f = fermi(e - mu, T);
    eb += e * f;
    full += f == 1.0;
    empty += f == 0.0;
    if (f != 1.0) c0 = min(c0, c);
    if (f != 0.0) c1 = max(c1, c);
  }
  eb = warp_sum(eb);
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    full += __shfl_xor_sync(0xffffffffu, full, s);
    empty += __shfl_xor_sync(0xffffffffu, empty, s);
    c0 = min(c0, __shfl_xor_sync(0xffffffffu, c0, s));
    c1 = max(c1, __shfl_xor_sync(0xffffffffu, c1, s));
  }
  const bool cm = full > empty;
  const int cbeg = cm ? c0 : 0, cend = cm ? n : c1 + 1;
  for (int c = cbeg + lane; c < cend; c += 32) {
    const double f = fermi(bk[c] - mu, T);
    occ[k * n + (c - cbeg)] = cm ? f - 1.0 : f;
  }
  if (lane == 0) {
    eband_k[k] = w[k] * eb;
    first[k] = cbeg;
    ncol[k] = cend - cbeg;
    comp[k] = cm ? 1 : 0;
  }
}

// grid: the lower 32 x 32 blocks of each rho_k, one k-point after the other; four warps of
// one 16 x 16 quadrant each.
// The columns come in slices of 8 through shared memory, k-contiguous per row with a pitch
// of 12 complex (fragment reads conflict-free); a block below the diagonal is written
// together with its mirror image.
__global__ void __launch_bounds__(128) st_rho_kernel(StRhoArgs a) {
  constexpr int PT = 12, KS = 8;
  __shared__ __align__(16) double2 sa[2][32 * PT];
  __shared__ __align__(16) double2 sb[2][32 * PT];
  __shared__ double sw[2][KS];
  const int n = a.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nb = (n + 31) / 32, per = nb * (nb + 1) / 2;
  const int64_t k = blockIdx.x / per, nn = (int64_t)n * n;
  int I = 0, J = (int)(blockIdx.x % per);  // block (I, J), J <= I
  while (J > I) { J -= I + 1; ++I; }
  const int K = a.ncol[k];
  const long long t0 = a.phase_cycles ? clock64() : 0;
  const double2* U = a.U + k * nn + (a.first ? a.first[k] * n : 0);
  const double* w = a.occ + k * n;
  auto issue = [&](int c0, int b) {
    for (int u = threadIdx.x; u < 32 * KS; u += 128) {
      const int r = u & 31, c = c0 + (u >> 5);
      const int ra = 32 * I + r, rb = 32 * J + r;
      const bool oka = ra < n && c < K, okb = rb < n && c < K;
      st_cp16(&sa[b][r * PT + (u >> 5)], oka ? (const void*)(U + ra + (int64_t)c * n) : (const void*)U, oka);
      st_cp16(&sb[b][r * PT + (u >> 5)], okb ? (const void*)(U + rb + (int64_t)c * n) : (const void*)U, okb);
    }
    if (threadIdx.x < KS) sw[b][threadIdx.x] = c0 + threadIdx.x < K ? w[c0 + threadIdx.x] : 0.0;
    st_cp_commit();
  };
  const int wm = (warp & 1) * 16, wn = (warp >> 1) * 16;
  double re[2][2][2], im[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  if (K > 0) issue(0, 0);
  for (int c0 = 0, b = 0; c0 < K; c0 += KS, b ^= 1) {
    st_cp_wait();
    __syncthreads();
    if (c0 + KS < K) issue(c0 + KS, b ^ 1);
#pragma unroll
    for (int kk = 0; kk < KS; kk += 4) {
      const double f = sw[b][kk + t];
      double2 av[2], bv[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) av[i] = sa[b][(wm + 8 * i + g) * PT + kk + t];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = cscale(f, sb[b][(wn + 8 * j + g) * PT + kk + t]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {  // a conj(b)
          dmma_884(re[i][j][0], re[i][j][1], av[i].x, bv[j].x);
          dmma_884(re[i][j][0], re[i][j][1], av[i].y, bv[j].y);
          dmma_884(im[i][j][0], im[i][j][1], av[i].y, bv[j].x);
          dmma_884(im[i][j][0], im[i][j][1], -av[i].x, bv[j].y);
        }
    }
  }
  const double one = a.comp[k] ? 1.0 : 0.0;
  double2* R = a.rho + k * nn;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = 32 * I + wm + 8 * i + g;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 32 * J + wn + 8 * j + 2 * t + h;
        if (r >= n || c > r) continue;
        double2 v = cmk(re[i][j][h], im[i][j][h]);
        if (r == c) v = cmk(v.x + one, 0.0);
        R[r + (int64_t)c * n] = v;
        if (r != c) R[c + (int64_t)r * n] = cconj(v);
      }
  }
  if (a.phase_cycles && threadIdx.x == 0)
    atomicAdd(&a.phase_cycles[PH_OUT], (unsigned long long)(clock64() - t0));
}

}  // namespace lqm
