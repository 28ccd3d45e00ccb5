// ib_jk.cu -- density digestion of ERI blocks: J/K energies and their nuclear
// gradient (the adjoint of the integral evaluation with respect to centres).
//
// Quartets are unique shell quartets (a>=b, c>=d, pair(ab)>=pair(cd) in the
// caller's ordering), each standing for its 8-fold permutation family with
// degeneracy deg = (a!=b ? 2:1)(c!=d ? 2:1)(ab!=cd ? 2:1).  With a real
// symmetric density P (Cartesian basis):
//   E_J = 1/2 sum_ijkl P_ij P_kl (ij|kl),   E_K = -1/4 sum_ijkl P_ik P_jl (ij|kl)
// so the symmetrised weight of one element is
//   D_ijkl = 1/2 P_ij P_kl - 1/8 (P_ik P_jl + P_il P_jk).
// Gradient: d/dA_x of a primitive x^ax y^ay z^az exp(-alpha r_A^2) is
//   2 alpha [a+1x] - ax [a-1x],
// so dE/dA_x = sum deg D (a~+1x b|cd) - ax D (a-1x b|cd), with a~ the shell with
// coefficients 2 alpha c and l+1.  The caller evaluates those auxiliary
// blocks with the ERI kernels; these kernels map every auxiliary element back
// to the component it differentiates and accumulate the atom's force, and
// the opposite contribution on centre D (translational invariance).
#include <cuda_runtime.h>

#include "../../include/intception_b200.h"
#include "ib_generic.cuh"

namespace {

__device__ __forceinline__ void jk_comp(int l, int k, int& x, int& y, int& z) {
  int s = 0;
  while ((s + 1) * (s + 2) / 2 <= k) ++s;
  z = k - s * (s + 1) / 2;
  y = s - z;
  x = l - s;
}

// y + z of component k
__device__ __forceinline__ int jk_yz(int k) {
  return (k >= 1) + (k >= 3) + (k >= 6) + (k >= 10) + (k >= 15) + (k >= 21);
}

__device__ __forceinline__ int jk_index(int x, int y, int z) { return z + (y + z) * (y + z + 1) / 2; }

// The six density values of an element (P is symmetric).  A warp's elements run
// through i, then j, and few k and l: rows k and l put their values into one line
// each, where rows i and j would take a line a value.
struct JkP {
  double ij, kl, ki, lj, li, kj;
};
__device__ __forceinline__ JkP jk_density(const double* __restrict__ P, int n, int i, int j, int k, int l) {
  const double* __restrict__ Pk = P + (size_t)k * n;
  const double* __restrict__ Pl = P + (size_t)l * n;
  return {__ldg(P + (size_t)i * n + j), __ldg(Pk + l), __ldg(Pk + i), __ldg(Pl + j), __ldg(Pl + i), __ldg(Pk + j)};
}
__device__ __forceinline__ double jk_weight(const double* __restrict__ P, int n, int i, int j, int k, int l) {
  const JkP p = jk_density(P, n, i, j, k, l);
  return 0.5 * p.ij * p.kl - 0.125 * (p.ki * p.lj + p.li * p.kj);
}

__device__ __forceinline__ double jk_deg(const int* s) {
  return (s[0] != s[1] ? 2.0 : 1.0) * (s[2] != s[3] ? 2.0 : 1.0) * ((s[0] != s[2] || s[1] != s[3]) ? 2.0 : 1.0);
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Compensated (double-double) sums: the energy of a large system is a sum of
// ~1e8 quartet terms, and a plain sum in an order that changes with the
// quartet list (atomics, a geometry's screening) moves it by ~1e-13
// relative -- enough to swamp a central difference with h = 1e-4.
// Block partials of the energy kernel (4 doubles per block), one array per
// device: calls on one device run in stream order (JKSystem uses one stream).
#define JK_MAX_PART_BLOCKS 4096
__device__ double ib_jk_part[4 * JK_MAX_PART_BLOCKS];

struct JkDD {
  double hi, lo;
};
__device__ __forceinline__ JkDD jk_dd_add(JkDD a, double b) {  // Knuth's TwoSum
  const double s = a.hi + b, bb = s - a.hi, e = (a.hi - (s - bb)) + (b - bb);
  return {s, a.lo + e};
}
__device__ __forceinline__ JkDD jk_dd_add(JkDD a, JkDD b) {
  JkDD r = jk_dd_add(a, b.hi);
  r.lo += b.lo;
  return r;
}

// e / n for the element indices of a block (e < 28^4 < 2^21, n <= 28): (e + 0.5) / n
// is at least 0.5 / n away from an integer, the two roundings are below that.
__device__ __forceinline__ int jk_quot(int e, float rn) { return (int)(((float)e + 0.5f) * rn); }

// One warp per quartet.  Each lane sums its shares in plain double (a few
// hundred terms, a fixed order), the warp, block and grid sums are
// double-double: block k writes its (E_J, E_K) partials to part[4k .. 4k+3]
// and ib_jk_energy_finish adds them in block order into e_out.  The result
// does not depend on scheduling.  27 atoms, l <= 2: 5.75 ms an energy, 6.22 with
// integer divisions and densities read along the rows of i and j, 6.24 with
// two quartets a warp (neighbours in the list differ in size).
__global__ void ib_jk_energy_kernel(const int* __restrict__ quartets, const long long* __restrict__ out_off, int nq,
                                    const int* __restrict__ shell_l, const int* __restrict__ fofs,
                                    const double* __restrict__ P, int nbf, const double* __restrict__ blocks,
                                    double* __restrict__ part) {
  __shared__ JkDD red[2][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  double sj = 0.0, sk = 0.0;  // this lane's plain sums: a few hundred terms in a fixed order
  for (int q = warp; q < nq; q += nwarp) {
    int s[4], n[4], f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = __ldg(quartets + 4 * (size_t)q + i);
      n[i] = ib_ncart(__ldg(shell_l + s[i]));
      f[i] = __ldg(fofs + s[i]);
    }
    const double deg = jk_deg(s);
    const double* __restrict__ blk = blocks + __ldg(out_off + q);
    const int tot = n[0] * n[1] * n[2] * n[3];
    const float rn0 = 1.0f / (float)n[0], rn1 = 1.0f / (float)n[1], rn2 = 1.0f / (float)n[2];
    double pj = 0.0, pk = 0.0;
    for (int e = lane; e < tot; e += 32) {
      const int r1 = jk_quot(e, rn0), r2 = jk_quot(r1, rn1), id = jk_quot(r2, rn2);
      const int i = f[0] + e - r1 * n[0], j = f[1] + r1 - r2 * n[1], k = f[2] + r2 - id * n[2], l = f[3] + id;
      const JkP p = jk_density(P, nbf, i, j, k, l);
      const double v = __ldg(blk + e);
      pj += p.ij * p.kl * v;
      pk += (p.ki * p.lj + p.li * p.kj) * v;
    }
    sj += 0.5 * deg * pj;
    sk -= 0.125 * deg * pk;
  }
  // the lanes' sums over the warp in double-double, in a fixed shuffle order
  JkDD ej = {sj, 0.0}, ek = {sk, 0.0};
  for (int o = 16; o > 0; o >>= 1) {
    ej = jk_dd_add(ej, JkDD{__shfl_xor_sync(0xffffffffu, ej.hi, o), __shfl_xor_sync(0xffffffffu, ej.lo, o)});
    ek = jk_dd_add(ek, JkDD{__shfl_xor_sync(0xffffffffu, ek.hi, o), __shfl_xor_sync(0xffffffffu, ek.lo, o)});
  }
  if (lane == 0) {
    red[0][wib] = ej;
    red[1][wib] = ek;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    JkDD a = {0.0, 0.0}, b = {0.0, 0.0};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a = jk_dd_add(a, red[0][w]);
      b = jk_dd_add(b, red[1][w]);
    }
    part[4 * blockIdx.x + 0] = a.hi;
    part[4 * blockIdx.x + 1] = a.lo;
    part[4 * blockIdx.x + 2] = b.hi;
    part[4 * blockIdx.x + 3] = b.lo;
  }
}

// One warp: e_out[0..1] += the partials of nb blocks (lane t takes blocks t,
// t + 32, ..., then the lanes' sums meet in a fixed shuffle order).
__global__ void ib_jk_energy_finish(const double* __restrict__ part, int nb, double* __restrict__ e_out) {
  const int lane = threadIdx.x;
  JkDD a = {0.0, 0.0}, b = {0.0, 0.0};
  for (int k = lane; k < nb; k += 32) {
    a = jk_dd_add(a, JkDD{part[4 * k], part[4 * k + 1]});
    b = jk_dd_add(b, JkDD{part[4 * k + 2], part[4 * k + 3]});
  }
  for (int o = 16; o > 0; o >>= 1) {
    a = jk_dd_add(a, JkDD{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)});
    b = jk_dd_add(b, JkDD{__shfl_xor_sync(0xffffffffu, b.hi, o), __shfl_xor_sync(0xffffffffu, b.lo, o)});
  }
  if (lane == 0) {
    e_out[0] += a.hi + a.lo;
    e_out[1] += b.hi + b.lo;
  }
}

// Gradient contribution of one auxiliary batch: centre `pos` (0..2) of each
// listed quartet carries level l+1 (sign > 0, shell coefficients 2 alpha c)
// or l-1 (sign < 0).  aux_off[k] locates the auxiliary block of quartet
// qidx[k] of the unique quartet list.  Forces accumulate in shared memory per
// atom and are flushed once per block.
//
// One warp per quartet.  When every shell has l <= JK_STAGE_L and the block has
// at least 128 elements, the six density
// blocks the quartet's weights read (P over the shell pairs ab, cd, ac, bd, ad,
// bc) are first copied to the warp's slice of shared memory with coalesced
// row loads, and every weight then reads shared memory: an element of the
// auxiliary block needs up to 3 weights of 6 density values each, which as
// global gathers dominated the kernel.
#define JK_STAGE_L 3
#define JK_STAGE_N 10  // ncart(JK_STAGE_L)
#define JK_WARPS 8

__device__ __forceinline__ void jk_stage(const double* __restrict__ P, int nbf, int r0, int nr, int c0, int nc,
                                         double* __restrict__ dst, int lane) {
  for (int e = lane; e < nr * nc; e += 32) {
    const int i = e / nc, j = e - i * nc;
    dst[i * JK_STAGE_N + j] = __ldg(P + (size_t)(r0 + i) * nbf + c0 + j);
  }
}

__global__ void ib_jk_force_kernel(const int* __restrict__ quartets, const int* __restrict__ qidx,
                                   const long long* __restrict__ aux_off, int naux, int pos, int sign,
                                   const int* __restrict__ shell_l, const int* __restrict__ fofs,
                                   const int* __restrict__ shell_atom, const double* __restrict__ P, int nbf,
                                   int natom, const double* __restrict__ blocks, double* __restrict__ force) {
  extern __shared__ double fs[];
  // [3 natom] force sums, then per warp 6 staged density blocks of JK_STAGE_N^2
  double* stage = fs + ((3 * natom + 1) & ~1);
  for (int i = threadIdx.x; i < 3 * natom; i += blockDim.x) fs[i] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double* __restrict__ st = stage + (size_t)wib * 6 * JK_STAGE_N * JK_STAGE_N;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int k = warp; k < naux; k += nwarp) {
    const int q = qidx[k];
    int s[4], l[4], n[4], f[4];
    for (int i = 0; i < 4; ++i) {
      s[i] = quartets[4 * q + i];
      l[i] = shell_l[s[i]];
      f[i] = fofs[s[i]];
      n[i] = ib_ncart(l[i]);
    }
    const int lx = l[pos] + (sign > 0 ? 1 : -1);
    int na[4] = {n[0], n[1], n[2], n[3]};
    na[pos] = ib_ncart(lx);
    const double deg = jk_deg(s);
    const double* blk = blocks + aux_off[k];
    const int tot = na[0] * na[1] * na[2] * na[3];
    // staged blocks: 0 ab, 1 cd, 2 ac, 3 bd, 4 ad, 5 bc (rows of the first shell)
    // staging pays for large blocks only: a block of a few elements needs fewer
    // gathers than the six density blocks hold (measured: staging every quartet
    // made the 60-atom gradient's digestion 1.69 -> 2.04 s)
    const bool staged = max(max(l[0], l[1]), max(l[2], l[3])) <= JK_STAGE_L && tot >= 128;
    const int SS = JK_STAGE_N * JK_STAGE_N;
    if (staged) {
      __syncwarp();
      jk_stage(P, nbf, f[0], n[0], f[1], n[1], st + 0 * SS, lane);
      jk_stage(P, nbf, f[2], n[2], f[3], n[3], st + 1 * SS, lane);
      jk_stage(P, nbf, f[0], n[0], f[2], n[2], st + 2 * SS, lane);
      jk_stage(P, nbf, f[1], n[1], f[3], n[3], st + 3 * SS, lane);
      jk_stage(P, nbf, f[0], n[0], f[3], n[3], st + 4 * SS, lane);
      jk_stage(P, nbf, f[1], n[1], f[2], n[2], st + 5 * SS, lane);
      __syncwarp();
    }
    double g[3] = {0.0, 0.0, 0.0};
    for (int e = lane; e < tot; e += 32) {
      int idx[4];
      int r = e;
      for (int i = 0; i < 4; ++i) {
        idx[i] = r % na[i];
        r /= na[i];
      }
      const double v = deg * blk[e];
      int cx, cy, cz;
      jk_comp(lx, idx[pos], cx, cy, cz);
      int c[3] = {cx, cy, cz};
      for (int d = 0; d < 3; ++d) {
        int o[3] = {c[0], c[1], c[2]};
        double coef;
        if (sign > 0) {
          if (o[d] == 0) continue;
          o[d] -= 1;
          coef = 1.0;
        } else {
          o[d] += 1;
          coef = -(double)o[d];
        }
        int li[4] = {idx[0], idx[1], idx[2], idx[3]};  // component indices within each shell
        li[pos] = jk_index(o[0], o[1], o[2]);
        double w;
        if (staged) {
          const int N = JK_STAGE_N;
          w = 0.5 * st[0 * SS + li[0] * N + li[1]] * st[1 * SS + li[2] * N + li[3]] -
              0.125 * (st[2 * SS + li[0] * N + li[2]] * st[3 * SS + li[1] * N + li[3]] +
                       st[4 * SS + li[0] * N + li[3]] * st[5 * SS + li[1] * N + li[2]]);
        } else {
          w = jk_weight(P, nbf, f[0] + li[0], f[1] + li[1], f[2] + li[2], f[3] + li[3]);
        }
        g[d] += coef * v * w;
      }
    }
    for (int d = 0; d < 3; ++d) g[d] = warp_sum(g[d]);
    if (lane == 0) {
      const int ax = shell_atom[s[pos]], ad = shell_atom[s[3]];
      for (int d = 0; d < 3; ++d) {
        atomicAdd(&fs[3 * ax + d], g[d]);
        atomicAdd(&fs[3 * ad + d], -g[d]);  // translational invariance: d/dD = -(d/dA + d/dB + d/dC)
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * natom; i += blockDim.x)
    if (fs[i] != 0.0) atomicAdd(force + i, fs[i]);
}

// All six auxiliary batches of a quartet list at once.  aux.off[b][q] locates
// quartet q's block in aux.blk[b] (b = 2 pos + (sign < 0); -1: the quartet has
// no block there, an l = 0 shell at pos for sign < 0).  The loop runs over the
// quartet's ORIGINAL elements o: its density weight W(o) is formed once, and
// for each centre pos and direction x
//   dE/dA_pos,x += deg W(o) [(o + 1x | raised at pos) - o_x (o - 1x | lowered at pos)],
// the adjoint of the derivative rule above; centre D takes the opposite sum.
//
// 20 atoms, l <= 2 (screen 1e-15): 14.6 ms of a gradient before, 10.8 now, by
// quotients in float instead of integer divisions, 16 exchanges a quartet
// instead of 45, one shared add a lane instead of 18 in turn, and densities read
// along the rows of k and l.  Staging the six density blocks in shared memory
// (ib_jk_force_kernel's way) made it 12.4: its 38 KB a block cost more
// occupancy than the gathers cost time.  Fetching the next quartet's indices
// early changed nothing (11.1).
struct JkAux {
  const long long* off[6];
  const double* blk[6];
};

__global__ void ib_jk_force_all_kernel(const int* __restrict__ quartets, int nq, const JkAux aux,
                                       const int* __restrict__ shell_l, const int* __restrict__ fofs,
                                       const int* __restrict__ shell_atom, const double* __restrict__ P, int nbf,
                                       int natom, double* __restrict__ force) {
  extern __shared__ double fs[];
  for (int i = threadIdx.x; i < 3 * natom; i += blockDim.x) fs[i] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int q = warp; q < nq; q += nwarp) {
    int s[4], l[4], n[4], f[4];
    long long off[6];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = __ldg(quartets + 4 * (size_t)q + i);
      l[i] = __ldg(shell_l + s[i]);
      f[i] = __ldg(fofs + s[i]);
      n[i] = ib_ncart(l[i]);
    }
#pragma unroll
    for (int b = 0; b < 6; ++b) off[b] = __ldg(aux.off[b] + q);
    const double deg = jk_deg(s);
    const int tot = n[0] * n[1] * n[2] * n[3];
    const float rn[3] = {1.0f / (float)n[0], 1.0f / (float)n[1], 1.0f / (float)n[2]};
    double g[16];  // [pos][x], zeros up to a power of two
#pragma unroll
    for (int k = 0; k < 16; ++k) g[k] = 0.0;
    for (int e = lane; e < tot; e += 32) {
      int r[4], idx[4];  // r[i]: index over shells i and later
      r[0] = e;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        r[i + 1] = jk_quot(r[i], rn[i]);
        idx[i] = r[i] - r[i + 1] * n[i];
      }
      idx[3] = r[3];
      const double w = deg * jk_weight(P, nbf, f[0] + idx[0], f[1] + idx[1], f[2] + idx[2], f[3] + idx[3]);
      int stride = 1;
#pragma unroll
      for (int pos = 0; pos < 3; ++pos) {
        // component k = t (t + 1) / 2 + z of x = l - t, y + z = t: one more x keeps
        // the index, one more y adds t + 1, one more z adds t + 2
        const int k = idx[pos], t = jk_yz(k), z = k - t * (t + 1) / 2;
        const int lo = e - stride * r[pos];
        const double* bp = aux.blk[2 * pos] + off[2 * pos] + lo + stride * (k + ib_ncart(l[pos] + 1) * r[pos + 1]);
        double v[3] = {__ldg(bp), __ldg(bp + stride * (t + 1)), __ldg(bp + stride * (t + 2))};
        if (off[2 * pos + 1] >= 0) {
          const double* bm =
              aux.blk[2 * pos + 1] + off[2 * pos + 1] + lo + stride * (k + ib_ncart(l[pos] - 1) * r[pos + 1]);
          if (l[pos] > t) v[0] -= (double)(l[pos] - t) * __ldg(bm);
          if (t > z) v[1] -= (double)(t - z) * __ldg(bm - stride * t);
          if (z > 0) v[2] -= (double)z * __ldg(bm - stride * (t + 1));
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) g[3 * pos + x] += w * v[x];
        stride *= n[pos];
      }
    }
    // sums over the lanes: each step halves the values that a lane holds, so
    // that lanes 2k and 2k + 1 end with the sum of value k (16 exchanges, not 45)
#pragma unroll
    for (int o = 16, m = 8; m > 0; o >>= 1, m >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < m; ++k) {
        const double give = up ? g[k] : g[k + m], keep = up ? g[k + m] : g[k];
        g[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    const double sum = g[0] + __shfl_xor_sync(0xffffffffu, g[0], 1);
    // even lanes add a value to its centre; odd lanes 1, 3, 5 the opposite of a
    // direction's three to centre D (one lane after the other took 18 adds in turn)
    const int k = lane >> 1, x = k % 3;
    const double dx = __shfl_sync(0xffffffffu, sum, 2 * x) + __shfl_sync(0xffffffffu, sum, 2 * x + 6) +
                      __shfl_sync(0xffffffffu, sum, 2 * x + 12);
    const bool centre_d = lane & 1;
    if (k < (centre_d ? 3 : 9)) {
      const int at = centre_d ? s[3] : k < 3 ? s[0] : k < 6 ? s[1] : s[2];
      atomicAdd(&fs[3 * shell_atom[at] + x], centre_d ? -dx : sum);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * natom; i += blockDim.x)
    if (fs[i] != 0.0) atomicAdd(force + i, fs[i]);
}

}  // namespace

extern "C" int intception_b200_jk_energy(const int* quartets, const long long* out_off, int nq, const int* shell_l,
                                         const int* fofs, const double* P, int nbf, const double* blocks,
                                         double* e_out, void* stream) {
  if (nq < 0 || (nq > 0 && (!quartets || !out_off || !shell_l || !fofs || !P || !blocks || !e_out)))
    return IB_ERR_ARG;
  if (nq == 0) return IB_OK;
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return IB_ERR_NODEVICE;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int threads = 256, wpb = threads / 32;
  int blocks_n = (nq + wpb - 1) / wpb;
  if (blocks_n > nsm * 16) blocks_n = nsm * 16;
  if (blocks_n > JK_MAX_PART_BLOCKS) blocks_n = JK_MAX_PART_BLOCKS;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  double* part = nullptr;  // this device's copy of the file-scope partials array
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&part), ib_jk_part) != cudaSuccess) return IB_ERR_CUDA;
  ib_jk_energy_kernel<<<blocks_n, threads, 0, s>>>(quartets, out_off, nq, shell_l, fofs, P, nbf, blocks, part);
  ib_jk_energy_finish<<<1, 32, 0, s>>>(part, blocks_n, e_out);
  return cudaGetLastError() == cudaSuccess ? IB_OK : IB_ERR_CUDA;
}

extern "C" int intception_b200_jk_force(const int* quartets, const int* qidx, const long long* aux_off, int naux,
                                        int pos, int sign, const int* shell_l, const int* fofs,
                                        const int* shell_atom, const double* P, int nbf, int natom,
                                        const double* blocks, double* force, void* stream) {
  if (naux < 0 || pos < 0 || pos > 2 || (sign != 1 && sign != -1) || natom < 1 || natom > 4096) return IB_ERR_ARG;
  if (naux == 0) return IB_OK;
  if (!quartets || !qidx || !aux_off || !shell_l || !fofs || !shell_atom || !P || !blocks || !force)
    return IB_ERR_ARG;
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return IB_ERR_NODEVICE;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem =
      sizeof(double) * (((3 * (size_t)natom + 1) & ~(size_t)1) + (size_t)JK_WARPS * 6 * JK_STAGE_N * JK_STAGE_N);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(ib_jk_force_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return IB_ERR_CUDA;
  const int threads = 32 * JK_WARPS, wpb = JK_WARPS;
  int blocks_n = (naux + wpb - 1) / wpb;
  if (blocks_n > nsm * 8) blocks_n = nsm * 8;
  ib_jk_force_kernel<<<blocks_n, threads, smem, static_cast<cudaStream_t>(stream)>>>(
      quartets, qidx, aux_off, naux, pos, sign, shell_l, fofs, shell_atom, P, nbf, natom, blocks, force);
  return cudaGetLastError() == cudaSuccess ? IB_OK : IB_ERR_CUDA;
}

extern "C" int intception_b200_jk_force_all(const int* quartets, int nq, const long long* const* aux_off,
                                            const double* const* aux_blocks, const int* shell_l, const int* fofs,
                                            const int* shell_atom, const double* P, int nbf, int natom,
                                            double* force, void* stream) {
  if (nq < 0 || natom < 1 || natom > 4096) return IB_ERR_ARG;
  if (nq == 0) return IB_OK;
  if (!quartets || !aux_off || !aux_blocks || !shell_l || !fofs || !shell_atom || !P || !force) return IB_ERR_ARG;
  JkAux aux;
  for (int b = 0; b < 6; ++b) {
    if (!aux_off[b] || !aux_blocks[b]) return IB_ERR_ARG;
    aux.off[b] = aux_off[b];
    aux.blk[b] = aux_blocks[b];
  }
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return IB_ERR_NODEVICE;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = sizeof(double) * 3 * (size_t)natom;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(ib_jk_force_all_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return IB_ERR_CUDA;
  const int threads = 32 * JK_WARPS, wpb = JK_WARPS;
  int blocks_n = (nq + wpb - 1) / wpb;
  if (blocks_n > nsm * 8) blocks_n = nsm * 8;
  ib_jk_force_all_kernel<<<blocks_n, threads, smem, static_cast<cudaStream_t>(stream)>>>(
      quartets, nq, aux, shell_l, fofs, shell_atom, P, nbf, natom, force);
  return cudaGetLastError() == cudaSuccess ? IB_OK : IB_ERR_CUDA;
}
