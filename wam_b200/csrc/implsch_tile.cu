// IMPLSCH on tiles of 32 sea points (implsch_tile.cuh): launch shapes, the
// kernels and their batched form.
#include "implsch_tile.cuh"
#include <mutex>

namespace wamgpu {

template <int DPW, bool ST6, int KLT>
__device__ __forceinline__ void tile_cta(const DevTables<float>& T, const ImplArgs<float>& a, int blk,
                                         unsigned char* smem) {
  const TileShape& L = T.tile;
  float* sm = reinterpret_cast<float*>(smem);
  const int lane = threadIdx.x & 31, wid = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int ij0 = blk * 32, ij = min(ij0 + lane, a.nsea - 1);
  const bool real = ij0 + lane < a.nsea;
  // stage the tile: one 128-byte row of 32 points per bin and warp
  {
    const float* g = a.fl3_in + ij + (size_t)a.ld * wid;
    const size_t step = (size_t)a.ld * L.nw;
    unsigned sa = (unsigned)__cvta_generic_to_shared(sm + wid * 32 + lane);
    for (int b = wid; b < T.NS; b += L.nw) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(g) : "memory");
      g += step; sa += 128 * L.nw;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float* tab = sm + L.oTab;
  for (int i = threadIdx.x; i < T.lay.nreal; i += blockDim.x) {
    const int q = i - T.lay.RNLCOEF;
    const bool rnl = q >= 0 && q < RNL_STRIDE * T.MLSTHG;
    tab[rnl ? i - q % RNL_STRIDE + tile_rnl(q % RNL_STRIDE) : i] = T.small[i];
  }
  STabs<float> S;
  S.bind(tab, T.ismall, T.lay);
  WarpWS<float> w{};
  Src<float> src(T, S, w, lane, ij, a.indep[ij], a.u10[ij], a.udir[ij], a.roairn[ij], a.wstar[ij], a.depth[ij], a.enh, a.enh_ld);
  src.wncg = a.wncg ? a.wncg + (size_t)ij * 2 * T.ML : nullptr;
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  // the wind direction's cosine and sine: correctly rounded where LFACTOR's
  // decisions take them (ST6)
  const float cu = ST6 ? crcos(src.UDIR) : dcos(src.UDIR), su = ST6 ? crsin(src.UDIR) : dsin(src.UDIR);
  const Tile<DPW, ST6, KLT> t{T, a, S,      sm + lane, sm + L.oU + lane, sm + L.oRow + lane,
                         smem + (size_t)L.oLL * 4 + lane, reinterpret_cast<uint32_t*>(sm + L.oLL) + lane, lane, wid, ij, src.INDEP, real, src.U10, src.UDIR,
                         src.ROAIRN, src.WSTAR, src.DEPTH, cu, su, src};
  t.run();
}

template <int DPW, bool ST6, int KLT>
__global__ void __launch_bounds__(TILE_MAXW * 32, 1)
    implsch_tile_kernel(const __grid_constant__ DevTables<float> T, const __grid_constant__ ImplArgs<float> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  tile_cta<DPW, ST6, KLT>(T, a, blockIdx.x, smem);
}

// Batched form: CTA b works for member g with first[g] <= b < first[g + 1].
template <int DPW, bool ST6, int KLT>
__global__ void __launch_bounds__(TILE_MAXW * 32, 1)
    implsch_tile_batch_kernel(const __grid_constant__ DevTables<float> T, const ImplArgs<float>* __restrict__ mem,
                              const int* __restrict__ first, int nmem) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) unsigned char sraw[sizeof(ImplArgs<float>)];
  ImplArgs<float>& sa = *reinterpret_cast<ImplArgs<float>*>(sraw);
  int lo = 0, hi = nmem - 1;  // last g with first[g] <= blockIdx.x
  while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1; }
  const int nwords = (int)(sizeof(ImplArgs<float>) / sizeof(int));
  const int* src = reinterpret_cast<const int*>(mem + lo);
  for (int q = threadIdx.x; q < nwords; q += blockDim.x) reinterpret_cast<int*>(&sa)[q] = src[q];
  __syncthreads();
  tile_cta<DPW, ST6, KLT>(T, sa, (int)blockIdx.x - first[lo], smem);
}

// Shared-memory layout for these tables; smem = 0 where the tile kernel does
// not apply.
TileShape tile_shape(const DevTables<float>& T, int max_smem) {
  TileShape L{};
  if (T.lcflx || T.KL > 3 * TILE_MAXW) return L;
  L.dpw = (T.KL + TILE_MAXW - 1) / TILE_MAXW;
  L.nw = (T.KL + L.dpw - 1) / L.dpw;
  L.xcol = T.KL + L.dpw;
  const int ML = T.ML, st6 = T.iphys == 2;
  for (L.nbuf = 2; L.nbuf >= 1; --L.nbuf) {
    int u = 6 * L.xcol * L.nbuf;  // rows of 32 words
    u = std::max(u, 8 * ML);
    u = std::max(u, st6 ? 5 * T.NK10 + 24 + 3 * ML : 4 * ML + 3 * T.KL + 14 + (2 * ML + 31) / 32);
    u = std::max(u, 4 * ML + 22 + T.KL);
    L.oTab = T.NS * 32;
    L.oU = L.oTab + (T.lay.nreal + 31) / 32 * 32;
    L.oRow = L.oU + u * 32;
    L.oLL = L.oRow + (st6 ? 5 : 2) * ML * 32;
    const int bytes = L.oLL * 4 + ML * (st6 ? (T.KL + 31) / 32 * 128 : L.nw * 32);
    if (bytes <= max_smem) { L.smem = bytes; return L; }
  }
  L.smem = 0;
  return L;
}

namespace {
template <int DPW, bool ST6, int KLT> struct TileK {
  static cudaError_t limit(int bytes) {
    cudaError_t e = cudaFuncSetAttribute(implsch_tile_kernel<DPW, ST6, KLT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(implsch_tile_batch_kernel<DPW, ST6, KLT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  }
  static cudaError_t one(const DevTables<float>& T, const ImplArgs<float>& a, cudaStream_t s) {
    implsch_tile_kernel<DPW, ST6, KLT><<<(a.nsea + 31) / 32, T.tile.nw * 32, T.tile.smem, s>>>(T, a);
    return cudaGetLastError();
  }
  static cudaError_t batch(const DevTables<float>& T, const ImplArgs<float>* mem, const int* first,
                           int nmem, int nblocks, cudaStream_t s) {
    implsch_tile_batch_kernel<DPW, ST6, KLT><<<nblocks, T.tile.nw * 32, T.tile.smem, s>>>(T, mem, first, nmem);
    return cudaGetLastError();
  }
};
}  // namespace

#define TILE_PHYS(DPW, KLT, CALL) (T.iphys == 2 ? TileK<DPW, true, KLT>::CALL : TileK<DPW, false, KLT>::CALL)
#define TILE_DISPATCH(CALL)                       \
  (T.KL == 36   ? TILE_PHYS(3, 36, CALL)          \
   : T.KL == 30 ? TILE_PHYS(3, 30, CALL)          \
   : T.KL == 24 ? TILE_PHYS(2, 24, CALL)          \
   : T.KL == 12 ? TILE_PHYS(1, 12, CALL)          \
   : T.tile.dpw == 1 ? TILE_PHYS(1, 0, CALL)      \
   : T.tile.dpw == 2 ? TILE_PHYS(2, 0, CALL)      \
                     : TILE_PHYS(3, 0, CALL))

// The opt-in limit of a kernel is process state of the device: raised once to
// the device's maximum less the kernel's static part.
cudaError_t tile_set_max_smem(const DevTables<float>& T) {
  const TileShape& L = T.tile;
  static std::mutex mu;
  static int cur[64][7][2] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> lock(mu);
  int& c = cur[dev][T.KL == 36 ? 6 : T.KL == 30 ? 5 : T.KL == 24 ? 4 : T.KL == 12 ? 3 : L.dpw - 1][T.iphys == 2];
  if (L.smem <= c) return cudaSuccess;
  e = TILE_DISPATCH(limit(L.smem));
  if (e == cudaSuccess) c = L.smem;
  return e;
}

cudaError_t launch_implsch_tile(const DevTables<float>& T, const ImplArgs<float>& a, cudaStream_t s) {
  if (a.nsea == 0) return cudaSuccess;
  return TILE_DISPATCH(one(T, a, s));
}

cudaError_t launch_implsch_tile_batch(const DevTables<float>& T, const ImplArgs<float>* mem,
                                      const int* first, int nmem, int nblocks, cudaStream_t s) {
  if (nblocks == 0) return cudaSuccess;
  return TILE_DISPATCH(batch(T, mem, first, nmem, nblocks, s));
}

}  // namespace wamgpu
