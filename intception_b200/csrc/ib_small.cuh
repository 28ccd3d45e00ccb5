// ib_small.cuh -- kernels for small batches of l <= 2 quartets.
//
// The batch pipeline (classify, sort, items, one kernel per class on its own
// side stream, joins) costs about a hundred microseconds of launches however
// little work there is.  A few hundred quartets take one kernel that does all
// of it (ib_small_kernel): a block takes quartet after quartet in the caller's
// order, puts it in canonical order and calls its class's function (the body
// of the class kernel).  A few thousand keep the sort, which brings quartets of
// one class together (warps of different classes evict one another's code) and
// the long ones to the front, and run every class in one kernel
// (ib_merged_kernel).  256 quartets of K <= 3: 107 us with a kernel per class, 29
// here, most of it the dependent loads of one quartet and the launch.  All classes
// share one register budget there (two blocks per SM), which is why larger batches
// keep a kernel per class.
#pragma once
#include "ib_eri_device.cuh"

struct IbSmallArgs {
  const int* quartets;
  const long long* out_off;
  const double* bounds;  // screening bounds, or null
  double skip_below;
  IbItem* items;         // [nq], for the redo launch
  int nq, lmax;
};

cudaError_t ib_small_prepare_cart();
cudaError_t ib_small_prepare_sph();
cudaError_t ib_small_launch_cart(int grid, cudaStream_t s, const IbLaunch& a, const IbSmallArgs& b);
cudaError_t ib_small_launch_sph(int grid, cudaStream_t s, const IbLaunch& a, const IbSmallArgs& b);

cudaError_t ib_merged_launch_cart(int grid, cudaStream_t s, const IbLaunch& a);
cudaError_t ib_merged_launch_sph(int grid, cudaStream_t s, const IbLaunch& a);

template <class Switch, bool SPH>
__global__ void __launch_bounds__(IB_BLOCK, 2) ib_small_kernel(const __grid_constant__ IbLaunch a,
                                                               const __grid_constant__ IbSmallArgs b) {
  __shared__ IbItem item;
  __shared__ int cls;
  for (int q = blockIdx.x; q < b.nq; q += gridDim.x) {  // the block's four warps share a quartet
    if (threadIdx.x == 0) {
      int s[4], l[4], st[4];
      bool bad = false;
      for (int i = 0; i < 4; ++i) {
        s[i] = b.quartets[4 * q + i];
        l[i] = a.shell_l[s[i]];
        bad |= (l[i] < 0) | (l[i] > b.lmax);
      }
      // block strides from the shells' own l, as the batch pipeline lays a
      // block out; a quartet with an l out of range is then evaluated as (ss|ss)
      int n = 1;
      for (int i = 0; i < 4; ++i) {
        const int li = min(max(l[i], 0), IB_LMAX);
        st[i] = n;
        n *= SPH ? 2 * li + 1 : ib_ncart_d(li);
      }
      int cid = -1 - n;  // screened out: n zeros
      if (!(b.bounds && b.bounds[q] < b.skip_below)) {
        if (bad)
          for (int i = 0; i < 4; ++i) l[i] = 0;
        ib_canon(s, l, st);
        ib_compact_first(a.shell_k, a.shell_ptr, a.prim_exp, s, l, st);
        const int pb = ib_pair_ext(l[0], l[1]), pk = ib_pair_ext(l[2], l[3]);
        cid = pb * (pb + 1) / 2 + pk;
      }
      if (bad) atomicExch(a.status, 1);  // IB_ERR_ARG
      IbItem it;
      for (int i = 0; i < 4; ++i) {
        it.s[i] = s[i];
        it.st[i] = st[i];
      }
      it.off = b.out_off[q];
      item = it;
      cls = cid;
      b.items[q] = it;
    }
    __syncthreads();
    const int cid = cls;
    if (cid < 0) {
      double* __restrict__ o = a.out + item.off;
      for (int x = threadIdx.x; x < -1 - cid; x += IB_BLOCK) o[x] = 0.0;
    } else {
      Switch::run(a, &item, q, IB_BLOCK / 32, cid);
    }
    __syncthreads();
  }
}

// The class kernels of a sorted l <= 2 batch as one kernel.  Quartets of the
// costliest class first; in a class the long ones come first (the sort key's
// order), so its range starts with those of at least 2^IB_MERGED_LONG_LOG2
// primitive quartets: whole blocks take these, one at a time, before single warps take
// the rest.
template <class Switch, bool SPH>
__global__ void __launch_bounds__(IB_BLOCK, 2) ib_merged_kernel(const __grid_constant__ IbLaunch a) {
  constexpr int NC = Switch::NC;
  __shared__ int beg[2][NC], first[2][NC + 1], grab[IB_BLOCK / 32];
  if (threadIdx.x < NC) {
    const int k = threadIdx.x, cid = Switch::cid(k);
    const int b = a.ranges[2 * cid], e = a.ranges[2 * cid + 1], h = max(b, a.ranges[IB_SLOT_LONG_END + cid]);
    beg[0][k] = b;
    first[0][k + 1] = h - b;
    beg[1][k] = h;
    first[1][k + 1] = e - h;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    int* f = first[threadIdx.x];
    f[0] = 0;
    for (int k = 0; k < NC; ++k) f[k + 1] += f[k];
  }
  __syncthreads();
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    const int n = first[part][NC];
    // few short quartets: more warps each
    const int W = part == 0 || n <= 2 * (int)gridDim.x ? 4 : n <= 8 * (int)gridDim.x ? 2 : 1;
    const int gid = threadIdx.x / 32, sg = gid / W, SG = 32 * W, r = (int)threadIdx.x - sg * SG;
    while (true) {
      if (r == 0) grab[sg] = atomicAdd(a.counter + part, 1);
      ib_sg_sync(SG, sg, 0xffffffffu);
      const int t = grab[sg];
      if (t >= n) break;  // uniform over the slot
      int k = 0;
      while (t >= first[part][k + 1]) ++k;
      const int p = beg[part][k] + t - first[part][k];
      Switch::run(a, a.items + p, p, W, Switch::cid(k));
      ib_sg_sync(SG, sg, 0xffffffffu);
    }
    __syncthreads();
  }
}

// smem: the largest class's; set once per device (ib_small_prepare_*).
template <class Switch, bool SPH>
cudaError_t ib_small_prepare(int smem) {
  const cudaError_t e =
      cudaFuncSetAttribute(ib_merged_kernel<Switch, SPH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(ib_small_kernel<Switch, SPH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
template <class Switch, bool SPH>
cudaError_t ib_small_go(int grid, int smem, cudaStream_t s, const IbLaunch& a, const IbSmallArgs& b) {
  ib_small_kernel<Switch, SPH><<<grid, IB_BLOCK, smem, s>>>(a, b);
  return cudaGetLastError();
}
template <class Switch, bool SPH>
cudaError_t ib_merged_go(int grid, int smem, cudaStream_t s, const IbLaunch& a) {
  ib_merged_kernel<Switch, SPH><<<grid, IB_BLOCK, smem, s>>>(a);
  return cudaGetLastError();
}
