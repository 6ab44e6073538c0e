// pdg_conv.cuh -- the cell evaluation of the convection terms (pdg_conv.cu) and
// its block layout, shared by the kernels of pdg_conv.cu and pdg_conv_i.cu.
#pragma once

#include "pdg_ops.cuh"

namespace pdg {

template <int N>
struct CCfg {
  static constexpr int N2 = N * N, NB = N * N * N, TPC = N * N;
  static constexpr int CPB = (128 / TPC) > 0 ? (128 / TPC) : 1;
  static constexpr int THREADS = CPB * TPC;
  // S0..S3, then the face region: fluxes / face test results, own and
  // neighbour partial traces (the latter two reused for the partial tests)
  static constexpr int PER_CELL_RAW = 4 * NB + 18 * N2;
  // padding that puts the cells of a warp on different shared-memory banks
  // (counted wavefronts of the volume part's accesses, 4-byte elements)
  static constexpr int PAD = N == 2 ? 4 : N == 3 ? 27 : N == 4 ? 16 : N == 5 ? 3 : 0;
  // (FP32; FP64 keeps the raw stride)
  template <typename T>
  static constexpr int per_cell() { return sizeof(T) == 4 ? PER_CELL_RAW + PAD : PER_CELL_RAW; }
  static constexpr int TAB = 2 * N2;                 // B[q][a], D[q][a]
  static constexpr int VREC = 3 * NB;                // G_dir(q)
  static constexpr int FREC = 6 * N2;                // F_f(p)
};

// One block of cells: y += alpha C x (C^T when a.transpose) for the CPB cells of
// this block; smem_raw: CCfg<N>::TAB + CPB * per_cell values of T.
template <typename T, int N>
__device__ __forceinline__ void conv_block(const OpParams<T> &p, const ApplyArgs<T> &a,
                                           const T *__restrict__ vrec,
                                           const T *__restrict__ tabBD,
                                           unsigned char *smem_raw) {
  using C = CCfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  T *tB = reinterpret_cast<T *>(smem_raw);   // B[q][a]
  T *tD = tB + N2;                           // D[q][a] (xi-derivative)
  const int t = threadIdx.x, cs = t / TPC, l = t - cs * TPC;
  T *S0 = tB + C::TAB + cs * C::template per_cell<T>();
  T *S1 = S0 + NB, *S2 = S1 + NB, *S3 = S2 + NB;
  T *fl = S3 + NB;                           // [6][N2] fluxes, then face test results
  T *Ue = fl + 6 * N2, *Un = Ue + 6 * N2;    // [6][N2] partial traces (own, neighbour)
  if (a.skip && *a.skip) return;
  for (int i = t; i < C::TAB; i += blockDim.x) tB[i] = tabBD[i];
  const long li = (long)blockIdx.x * CPB + cs;
  const bool ranged = !a.cells && a.ncells > 0;
  const bool active = (a.cells || ranged) ? li < a.ncells : li < p.ncell;
  const long e = a.cells ? (active ? (long)a.cells[li] : 0) : (ranged ? (long)a.cell0 + li : li);
  const long ee = active ? e : 0;
  int ix[3];
  {
    long r = ee;
    ix[0] = (int)(r % p.nc[0]); r /= p.nc[0];
    ix[1] = (int)(r % p.nc[1]); r /= p.nc[1];
    ix[2] = (int)r;
  }
  const long stride[3] = {1, (long)p.nc[0], (long)p.nc[0] * p.nc[1]};
  const T *rec = vrec + ee * (C::VREC + C::FREC);
  const int tx = l % N, ty = l / N;
  T col[N];
  const T *xe = a.x + ee * NB;
#pragma unroll
  for (int z = 0; z < N; z++) {
    col[z] = xe[z * N2 + l];
    S3[z * N2 + l] = col[z];   // own values for the face traces
  }
  __syncthreads();

  // ---------------- volume ----------------
  T r[N];
  if (!a.transpose) {
    // u_q = (B (x) B (x) B) u
    T v[N];
#pragma unroll
    for (int qz = 0; qz < N; qz++) {
      T s = T(0);
#pragma unroll
      for (int z = 0; z < N; z++) s += tB[qz * N + z] * col[z];
      v[qz] = s;
    }
#pragma unroll
    for (int z = 0; z < N; z++) S0[z * N2 + l] = v[z];
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int b = 0; b < N; b++) s += tB[ty * N + b] * S0[z * N2 + b * N + tx];
      S1[z * N2 + l] = s;
    }
    __syncthreads();
    // point (qx=tx, qy=ty, qz): u_q, then F_dir = G_dir u_q -> S0 (x), S1 (y), S2 (z)
    T uq[N];
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int aa = 0; aa < N; aa++) s += tB[tx * N + aa] * S1[z * N2 + ty * N + aa];
      uq[z] = s;
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int q = z * N2 + l;
      S0[q] = rec[0 * NB + q] * uq[z];
      S1[q] = rec[1 * NB + q] * uq[z];
      S2[q] = rec[2 * NB + q] * uq[z];
    }
    __syncthreads();
    // x-step (node tx): Tx = Dt F_x, Ty = Bt F_y, Tz = Bt F_z
    T Tx[N], Ty[N], Tz[N];
#pragma unroll
    for (int z = 0; z < N; z++) {
      T sx = T(0), sy = T(0), sz = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) {
        const int i = z * N2 + ty * N + q;
        sx += tD[q * N + tx] * S0[i];
        sy += tB[q * N + tx] * S1[i];
        sz += tB[q * N + tx] * S2[i];
      }
      Tx[z] = sx; Ty[z] = sy; Tz[z] = sz;
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; z++) {
      S0[z * N2 + l] = Tx[z];
      S1[z * N2 + l] = Ty[z];
      S2[z * N2 + l] = Tz[z];
    }
    __syncthreads();
    // y-step (node ty): Sxy = Bt Tx + Dt Ty ; Sz = Bt Tz
    T Sxy[N], Sz[N];
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s1 = T(0), s2 = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) {
        const int i = z * N2 + q * N + tx;
        s1 += tB[q * N + ty] * S0[i] + tD[q * N + ty] * S1[i];
        s2 += tB[q * N + ty] * S2[i];
      }
      Sxy[z] = s1;
      Sz[z] = s2;
    }
    // z-step (registers): r = -(Bt Sxy + Dt Sz)
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) s += tB[q * N + z] * Sxy[q] + tD[q * N + z] * Sz[q];
      r[z] = -s;
    }
  } else {
    // gradient at the points: g_x = (B (x) B (x) D) u, g_y = (B (x) D (x) B) u,
    // g_z = (D (x) B (x) B) u; F = -(G_x g_x + G_y g_y + G_z g_z); r = (Bt (x) Bt (x) Bt) F
    T vb[N], vd[N];
#pragma unroll
    for (int qz = 0; qz < N; qz++) {
      T sb = T(0), sd = T(0);
#pragma unroll
      for (int z = 0; z < N; z++) {
        sb += tB[qz * N + z] * col[z];
        sd += tD[qz * N + z] * col[z];
      }
      vb[qz] = sb;
      vd[qz] = sd;
    }
#pragma unroll
    for (int z = 0; z < N; z++) {
      S0[z * N2 + l] = vb[z];   // z interpolated
      S1[z * N2 + l] = vd[z];   // z differentiated
    }
    __syncthreads();
    // y-step: A = B_y S0 (for x- and z-gradients use S0/S1 with B_y), Bd = D_y S0
#pragma unroll
    for (int z = 0; z < N; z++) {
      T sbb = T(0), sbd = T(0), sdb = T(0);
#pragma unroll
      for (int b = 0; b < N; b++) {
        const int i = z * N2 + b * N + tx;
        sbb += tB[ty * N + b] * S0[i];   // B_y B_z u
        sdb += tD[ty * N + b] * S0[i];   // D_y B_z u
        sbd += tB[ty * N + b] * S1[i];   // B_y D_z u
      }
      S2[z * N2 + l] = sbb;
      vb[z] = sdb;
      vd[z] = sbd;
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; z++) {
      S0[z * N2 + l] = vb[z];
      S1[z * N2 + l] = vd[z];
    }
    __syncthreads();
    T F[N];
#pragma unroll
    for (int z = 0; z < N; z++) {
      T gx = T(0), gy = T(0), gz = T(0);
#pragma unroll
      for (int aa = 0; aa < N; aa++) {
        const int i = z * N2 + ty * N + aa;
        gx += tD[tx * N + aa] * S2[i];   // D_x B_y B_z
        gy += tB[tx * N + aa] * S0[i];   // B_x D_y B_z
        gz += tB[tx * N + aa] * S1[i];   // B_x B_y D_z
      }
      const int q = z * N2 + l;
      F[z] = -(rec[q] * gx + rec[NB + q] * gy + rec[2 * NB + q] * gz);
    }
    __syncthreads();
    // test with Bt (x) Bt (x) Bt
#pragma unroll
    for (int z = 0; z < N; z++) S0[z * N2 + l] = F[z];
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) s += tB[q * N + tx] * S0[z * N2 + ty * N + q];
      S1[z * N2 + l] = s;
    }
    __syncthreads();
    T w[N];
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) s += tB[q * N + ty] * S1[z * N2 + q * N + tx];
      w[z] = s;
    }
#pragma unroll
    for (int z = 0; z < N; z++) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) s += tB[q * N + z] * w[q];
      r[z] = s;
    }
  }

  // ---------------- faces ----------------
  // Traces at the face points and the test with the face basis are
  // sum-factorised through shared memory (the volume part has released
  // S0..S2): thread l = (pa, pb) first contracts row pb of a node layer with
  // B[pa][.], then column pa of the partial results with B[pb][.].
  const int pa = l % N, pb = l / N;
  const int st[3] = {1, N, N2};
  long nbr[6];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    if (hi) nbr[f] = ix[dir] + 1 < p.nc[dir] ? ee + stride[dir] : -1;
    else nbr[f] = ix[dir] > 0 ? ee - stride[dir] : -1;
  }
  T Bp[N], Bq[N];   // B[pa][.] and B[pb][.] (face point -> node layer)
#pragma unroll
  for (int i = 0; i < N; i++) {
    Bp[i] = tB[pa * N + i];
    Bq[i] = tB[pb * N + i];
  }
  // per face, U[j][pa] = sum_i B[pa][i] layer[j][i] into Ue (own), Un (neighbour)
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const int od0 = dir == 0 ? 1 : 0, od1 = dir == 2 ? 1 : 2;   // tangential dirs
    const int lay_e = hi ? N - 1 : 0, lay_n = hi ? 0 : N - 1;
    // row j = pb of the own and the neighbour's node layer
    T se = T(0), sn = T(0);
    const int rowe = lay_e * st[dir] + pb * st[od1], rown = lay_n * st[dir] + pb * st[od1];
#pragma unroll
    for (int i = 0; i < N; i++) se += Bp[i] * S3[rowe + i * st[od0]];
    if (nbr[f] >= 0 && !a.diag_only) {
      const T *xn = a.x + nbr[f] * NB;
#pragma unroll
      for (int i = 0; i < N; i++) sn += Bp[i] * xn[rown + i * st[od0]];
    }
    Ue[f * N2 + pb * N + pa] = se;
    Un[f * N2 + pb * N + pa] = sn;
  }
  __syncthreads();
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    T ue = T(0), un = T(0);
#pragma unroll
    for (int j = 0; j < N; j++) {
      ue += Bq[j] * Ue[f * N2 + j * N + pa];
      un += Bq[j] * Un[f * N2 + j * N + pa];
    }
    const T bnw = rec[C::VREC + f * N2 + l];
    T flux = T(0);
    if (nbr[f] >= 0) {
      if (a.diag_only) un = T(0);
      if (!a.transpose) flux = (bnw >= T(0) ? ue : un) * bnw;
      else flux = bnw >= T(0) ? (ue - un) * bnw : T(0);
    } else {
      const int bc = p.bc[f];
      if (bc == PDG_BC_DIRICHLET) flux = bnw >= T(0) ? ue * bnw : T(0);
      else if (bc == PDG_BC_OUTFLOW) flux = ue * bnw;
    }
    fl[f * N2 + l] = flux;
  }
  __syncthreads();
  // test with the face basis: W[j][pa] = sum_i B[i][pa] flux[j][i] (into S2),
  // then R[pb][pa] = sum_j B[j][pb] W[j][pa] (into fl, in place per face)
  T Cp[N], Cq[N];   // B[.][pa] and B[.][pb]
#pragma unroll
  for (int i = 0; i < N; i++) {
    Cp[i] = tB[i * N + pa];
    Cq[i] = tB[i * N + pb];
  }
  T *Wt = Ue;       // [6][N2]; Ue's last reads were before the previous barrier
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    T w = T(0);
#pragma unroll
    for (int i = 0; i < N; i++) w += Cp[i] * fl[f * N2 + pb * N + i];
    Wt[f * N2 + pb * N + pa] = w;
  }
  __syncthreads();
  T Rf[6];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    T rr = T(0);
#pragma unroll
    for (int j = 0; j < N; j++) rr += Cq[j] * Wt[f * N2 + j * N + pa];
    Rf[f] = rr;
  }
  __syncthreads();
#pragma unroll
  for (int f = 0; f < 6; f++) fl[f * N2 + pb * N + pa] = Rf[f];   // R[f][n1][n0]
  __syncthreads();
  // node (tx, ty, z) on the layer of face f receives R[f][n1][n0]
#pragma unroll
  for (int z = 0; z < N; z++) {
    T s = T(0);
    const int node[3] = {tx, ty, z};
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const int dir = f >> 1, hi = f & 1;
      if (node[dir] != (hi ? N - 1 : 0)) continue;
      const int od0 = dir == 0 ? 1 : 0, od1 = dir == 2 ? 1 : 2;
      s += fl[f * N2 + node[od1] * N + node[od0]];
    }
    r[z] += s;
  }
  if (active) {
    T *ye = a.y + e * NB;
#pragma unroll
    for (int z = 0; z < N; z++) ye[z * N2 + l] += a.alpha * r[z];
  }
}

}  // namespace pdg
