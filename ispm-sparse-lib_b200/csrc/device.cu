// Device initialisation and device-resident sliced-ELL matrices.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "cuda_util.cuh"
#include "host_pool.h"
#include "operator.h"
#include "spmv_launch.h"

namespace ispm {

int device_sm_count()
{
  static std::mutex mu;
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return 148;
  std::lock_guard<std::mutex> g(mu);
  if (!cached[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
      v = 148;
    cached[dev] = v;
  }
  return cached[dev];
}

static size_t elm_size(int dtype) { return dtype == ISPM_F64 ? 8 : dtype == ISPM_F32 ? 4 : 2; }

// Round to BF16, nearest even (finite values).
static uint16_t to_bf16(float f)
{
  uint32_t u;
  std::memcpy(&u, &f, 4);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

// ---- staged-walk tile records ----------------------------------------------

void stage_records(const HostSlell &h, std::vector<int> &rec)
{
  rec.clear();
  const unsigned S = h.slice_height;
  if (!h.diags || h.var_height || h.hblock != 1 || S < 16 || kStageTileRows % S || !h.n_slices)
    return;
  const unsigned spt = kStageTileRows / S;  // <= 16 slices per tile
  const unsigned n_tiles = (h.n_slices + spt - 1) / spt;
  rec.assign((size_t)n_tiles * kStageRecInts, 0);
  const unsigned *sp = h.slice_ptr.data();
  const long long rows = kStageTileRows;
  std::vector<long long> win, all;
  for (unsigned t = 0; t < n_tiles; t++) {
    int *r = rec.data() + (size_t)t * kStageRecInts;
    const unsigned b0 = t * spt, nsl = std::min(spt, h.n_slices - b0);
    r[2] = (int)nsl;
    // window starts of every slice's diagonals (slice b: [elms_end, cols_end,
    // diag_ptr] at 3b, conversion.h:393-402): the x column that tile row 0
    // would read, so x[w + t] serves tile row t (diag_pos is absolute)
    all.clear();
    bool ok = true, ell = false;
    for (unsigned s = 0; s < nsl; s++) {
      const unsigned b = b0 + s;
      const unsigned e0 = sp[3 * b], c0 = sp[3 * b + 1], e1 = sp[3 * b + 3], c1 = sp[3 * b + 4];
      ell = ell || c1 != c0;
      const unsigned nd = (e1 - e0 - (c1 - c0)) / S, dd = sp[3 * b + 2];
      for (unsigned k = 0; k < nd; k++) {
        const long long w = (long long)sp[dd + k] - S - (long long)s * S;
        if (k && w <= all.back())
          ok = false;
        all.push_back(w);
      }
    }
    win = all;
    std::sort(win.begin(), win.end());
    win.erase(std::unique(win.begin(), win.end()), win.end());
    const int nu = (int)win.size();
    const long long e_first = sp[3 * b0], e_count = (long long)sp[3 * (b0 + nsl)] - e_first;
    if (!ok || nu < 1 || nu > kStageMaxDiag || e_first > INT32_MAX || e_count > INT32_MAX)
      continue;  // r[0] = 0
    // runs of window starts less than rows + gap apart share a band; a band
    // covers its windows' columns for all tile rows, 16-byte aligned
    long long lo[kStageMaxDiag], hi[kStageMaxDiag];
    int band[kStageMaxDiag], nb = 0;
    for (int u = 0; u < nu; u++) {
      const long long w = win[u];
      if (u == 0 || w - win[u - 1] > rows + kStageGap) {
        lo[nb] = w;
        nb++;
      }
      hi[nb - 1] = w + rows;
      band[u] = nb - 1;
    }
    if (nb > kStageMaxBands || lo[0] < INT32_MIN / 2 || hi[nb - 1] > INT32_MAX / 2)
      continue;
    long long words = 0, dst[kStageMaxBands], c0[kStageMaxBands];
    for (int q = 0; q < nb; q++) {
      c0[q] = lo[q] >= 0 ? lo[q] / 4 * 4 : -((-lo[q] + 3) / 4) * 4;
      const long long c1 = (hi[q] + 3) / 4 * 4;
      dst[q] = words;
      r[156 + 2 * q] = (int)c0[q];
      r[157 + 2 * q] = (int)(c1 - c0[q]);
      words += c1 - c0[q];
    }
    if (words > kStageMaxXWords)
      continue;
    r[1] = nu;
    for (int u = 0; u < nu; u++)
      r[8 + u] = (int)(dst[band[u]] + (win[u] - c0[band[u]]));
    // slice masks over the window starts, slice element offsets; uniform
    // when every slice carries all nu windows and no explicit columns
    bool uniform = !ell;
    for (unsigned s = 0; s < nsl; s++) {
      const unsigned b = b0 + s;
      const unsigned e0 = sp[3 * b], c0s = sp[3 * b + 1], e1 = sp[3 * b + 3],
                     c1s = sp[3 * b + 4];
      const unsigned nd = (e1 - e0 - (c1s - c0s)) / S, dd = sp[3 * b + 2];
      unsigned long long mask = 0;
      for (unsigned k = 0; k < nd; k++) {
        const long long w = (long long)sp[dd + k] - S - (long long)s * S;
        const int u = (int)(std::lower_bound(win.begin(), win.end(), w) - win.begin());
        mask |= 1ull << u;
      }
      uniform = uniform && (int)nd == nu;
      r[72 + 2 * s] = (int)(unsigned)(mask & 0xffffffffull);
      r[73 + 2 * s] = (int)(unsigned)(mask >> 32);
      r[104 + s] = (int)((long long)e0 + (c1s - c0s) - e_first);
      r[120 + s] = (int)((c1s - c0s) / S);
      r[136 + s] = (int)c0s;
    }
    r[0] = uniform ? 1 : 2;
    r[152] = (int)e_first;
    r[153] = (int)e_count;
    r[154] = nb;
    r[155] = (int)words;
  }
}


namespace {
struct StageEntry {
  const int *rec;
  int max_x_words;
  int max_elms;
  unsigned n_slices;
};
std::mutex g_stage_mu;
std::vector<std::pair<const unsigned *, StageEntry>> g_stage;  // few live matrices
}  // namespace

bool find_stage_records(const unsigned *slice_ptr, unsigned n_slices, StageInfo &out)
{
  std::lock_guard<std::mutex> g(g_stage_mu);
  for (const auto &e : g_stage)
    if (e.first == slice_ptr && e.second.n_slices == n_slices) {
      out.rec = e.second.rec;
      out.max_x_words = e.second.max_x_words;
      out.max_elms = e.second.max_elms;
      return true;
    }
  return false;
}

int DeviceSlell::attach_stage_records(const HostSlell &h)
{
  std::vector<int> rec;
  stage_records(h, rec);
  if (rec.empty())
    return ISPM_OK;
  int mx = 0, me = 0;
  for (size_t t = 0; t < rec.size(); t += kStageRecInts)
    if (rec[t]) {
      mx = std::max(mx, rec[t + 155]);
      me = std::max(me, rec[t + 153]);
    }
  cudaError_t e = cudaMalloc(&stage_rec, rec.size() * sizeof(int));
  if (e != cudaSuccess) {
    stage_rec = nullptr;
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? ISPM_ERR_NOMEM : ISPM_ERR_CUDA,
                "cudaMalloc(stage records): %s", cudaGetErrorString(e));
  }
  ISPM_CUDA_TRY(cudaMemcpy(stage_rec, rec.data(), rec.size() * sizeof(int),
                           cudaMemcpyHostToDevice));
  std::lock_guard<std::mutex> g(g_stage_mu);
  g_stage.push_back({slice_ptr, StageEntry{stage_rec, mx, me, meta.n_slices}});
  return ISPM_OK;
}

void DeviceSlell::release()
{
  if (stage_rec) {
    {
      std::lock_guard<std::mutex> g(g_stage_mu);
      for (size_t k = 0; k < g_stage.size(); k++)
        if (g_stage[k].second.rec == stage_rec) {
          g_stage.erase(g_stage.begin() + (long)k);
          break;
        }
    }
    cudaFree(stage_rec);
    stage_rec = nullptr;
  }
  if (slice_ptr)
    cudaFree(slice_ptr);
  if (cols)
    cudaFree(cols);
  if (elms)
    cudaFree(elms);
  slice_ptr = nullptr;
  cols = nullptr;
  elms = nullptr;
}

int DeviceSlell::upload(const HostSlell &h, bool bf16_values)
{
  release();
  meta = h.view();
  if (bf16_values && h.elm_dtype != ISPM_F32)
    return fail(ISPM_ERR_INVALID, "BF16 storage converts an FP32 element array");
  const int store = bf16_values ? ISPM_BF16 : h.elm_dtype;
  meta.elm_dtype = store;
  const size_t nsp = h.slice_ptr.size(), nc = h.cols.size(), ne = h.n_elms();
  // The reference zero-fills every device allocation (util/cuda/allocator.h:14-20);
  // here every byte is overwritten by the copy that follows.
  auto alloc = [](void **p, size_t bytes) -> int {
    cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
    if (e != cudaSuccess) {
      *p = nullptr;
      cudaGetLastError();
      return fail(e == cudaErrorMemoryAllocation ? ISPM_ERR_NOMEM : ISPM_ERR_CUDA,
                  "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    }
    return ISPM_OK;
  };
  int st;
  if ((st = alloc((void **)&slice_ptr, nsp * 4)) || (st = alloc((void **)&cols, nc * 4)) ||
      (st = alloc(&elms, ne * elm_size(store)))) {
    release();
    return st;
  }
  ISPM_CUDA_TRY(cudaMemcpy(slice_ptr, h.slice_ptr.data(), nsp * 4, cudaMemcpyHostToDevice));
  if (nc)
    ISPM_CUDA_TRY(cudaMemcpy(cols, h.cols.data(), nc * 4, cudaMemcpyHostToDevice));
  if (ne && bf16_values) {
    std::vector<uint16_t> b(ne);
    for (size_t k = 0; k < ne; k++)
      b[k] = to_bf16(h.elms_f[k]);
    ISPM_CUDA_TRY(cudaMemcpy(elms, b.data(), ne * 2, cudaMemcpyHostToDevice));
  } else if (ne) {
    ISPM_CUDA_TRY(
        cudaMemcpy(elms, h.elms_ptr(), ne * elm_size(h.elm_dtype), cudaMemcpyHostToDevice));
  }
  return attach_stage_records(h);
}

int DeviceSlell::upload_f16(const HostSlell &h)
{
  if (h.elm_dtype != ISPM_F32)
    return fail(ISPM_ERR_INVALID, "FP16 storage converts an FP32 element array");
  // the structure arrays travel unchanged, the elements as binary16
  std::vector<uint16_t> b(h.n_elms());
  for (size_t k = 0; k < b.size(); k++) {
    const double v = h.elms_f[k];
    b[k] = f16_bits(v);
    if (f16_value(b[k]) != v)
      return fail(ISPM_ERR_INVALID, "element %zu (%g) is not a binary16 value", k, v);
  }
  release();
  meta = h.view();
  meta.elm_dtype = ISPM_F16;
  const size_t nsp = h.slice_ptr.size(), nc = h.cols.size(), ne = b.size();
  auto alloc = [](void **p, size_t bytes) -> int {
    cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
    if (e != cudaSuccess) {
      *p = nullptr;
      cudaGetLastError();
      return fail(e == cudaErrorMemoryAllocation ? ISPM_ERR_NOMEM : ISPM_ERR_CUDA,
                  "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    }
    return ISPM_OK;
  };
  int st;
  if ((st = alloc((void **)&slice_ptr, nsp * 4)) || (st = alloc((void **)&cols, nc * 4)) ||
      (st = alloc(&elms, ne * 2))) {
    release();
    return st;
  }
  ISPM_CUDA_TRY(cudaMemcpy(slice_ptr, h.slice_ptr.data(), nsp * 4, cudaMemcpyHostToDevice));
  if (nc)
    ISPM_CUDA_TRY(cudaMemcpy(cols, h.cols.data(), nc * 4, cudaMemcpyHostToDevice));
  if (ne)
    ISPM_CUDA_TRY(cudaMemcpy(elms, b.data(), ne * 2, cudaMemcpyHostToDevice));
  return attach_stage_records(h);
}

int DeviceSlell::update_elms(const HostSlell &h)
{
  if (!elms && meta.n_elms)
    return fail(ISPM_ERR_INVALID, "device matrix not uploaded");
  if ((long long)h.n_elms() != meta.n_elms || h.elm_dtype != meta.elm_dtype)
    return fail(ISPM_ERR_INVALID, "element array shape changed (%zu vs %lld)", h.n_elms(),
                meta.n_elms);
  if (meta.n_elms)
    ISPM_CUDA_TRY(cudaMemcpy(elms, h.elms_ptr(), meta.n_elms * elm_size(h.elm_dtype),
                             cudaMemcpyHostToDevice));
  return ISPM_OK;
}

// elms[map[k]] = vals[k]: new values for an unchanged sparsity pattern,
// written straight into the device sliced-ELL array.  Padding slots are not
// in the map and keep their zeros.
template <class E, class V>
__global__ void refresh_values_kernel(E *__restrict__ elms, const unsigned *__restrict__ map,
                                      const V *__restrict__ vals, long long n)
{
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    elms[__ldcs(map + k)] = (E)__ldcs(vals + k);
}

template <class V>
__global__ void refresh_bf16_kernel(__nv_bfloat16 *__restrict__ elms,
                                    const unsigned *__restrict__ map, const V *__restrict__ vals,
                                    long long n)
{
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    elms[__ldcs(map + k)] = __float2bfloat16_rn((float)__ldcs(vals + k));
}

template <class E> __device__ __forceinline__ E element(double v, double)
{
  return (E)v;
}
template <> __device__ __forceinline__ __nv_bfloat16 element<__nv_bfloat16>(double v, double)
{
  return __float2bfloat16_rn((float)v);
}
template <> __device__ __forceinline__ __half element<__half>(double v, double scale)
{
  return __double2half(v * scale);
}

// The power of two that maps *amax into [2^13, 2^14) (1 for 0).
__device__ __forceinline__ double f16_scale(const double *amax)
{
  const double m = amax ? *amax : 0.0;
  return m > 0.0 ? scalbn(1.0, isfinite(m) ? 13 - ilogb(m) : 14) : 1.0;
}

// A scale whose inverse FP32 holds; with another the elements stay as they are
// and the caller, who reads *amax back, refuses the update.
__device__ __forceinline__ bool f16_scale_ok(double s) { return s >= 0x1p-126 && s <= 0x1p126; }

// Values through shared memory (SlotMap).  Bound by HBM: 8 bytes of value, 2
// of map and the element a slot.  61 x 75 x 83 27-point FP64 (10.0 M entries):
// 43 us (4.2 TB/s); gathering each slot's value from the CSR, 4 bytes of map a
// slot, took 49 us.
template <class E, class E2, class V>
__global__ void __launch_bounds__(256)
    refresh_chunks_kernel(E *__restrict__ elms, E2 *__restrict__ second,
                          const SlotChunk *__restrict__ chunk,
                          const unsigned short *__restrict__ idx, const V *__restrict__ vals,
                          const double *amax)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *sm = reinterpret_cast<V *>(smem_raw);
  pdl_wait();
  const uint4 c = __ldg(reinterpret_cast<const uint4 *>(chunk) + blockIdx.x);
  const V *v = vals + c.z;
  const int slots = (int)c.y, entries = (int)c.w;
  elms += c.x;
  idx += c.x;
  if (second)
    second += c.x;
#pragma unroll 8
  for (int i = threadIdx.x; i < entries; i += 256)
    sm[i] = __ldcs(v + i);
  const double scale = std::is_same<E, __half>::value ? f16_scale(amax) : 1.0;
  if (std::is_same<E, __half>::value && !f16_scale_ok(scale))
    return;
  __syncthreads();
  auto value = [&](unsigned k) { return k == 0xffffu ? 0.0 : (double)sm[k]; };
  if (((c.x | c.y) & 3) == 0) {  // four slots a thread
    struct __align__(sizeof(E) * 4) Q {
      E v[4];
    };
    struct __align__(sizeof(E2) * 4) Q2 {
      E2 v[4];
    };
#pragma unroll 2
    for (int i = 4 * threadIdx.x; i < slots; i += 1024) {
      const ushort4 k = __ldcs(reinterpret_cast<const ushort4 *>(idx + i));
      const double a = value(k.x), b = value(k.y), d = value(k.z), e = value(k.w);
      *reinterpret_cast<Q *>(elms + i) =
          Q{{element<E>(a, scale), element<E>(b, scale), element<E>(d, scale),
             element<E>(e, scale)}};
      if (second)
        *reinterpret_cast<Q2 *>(second + i) =
            Q2{{element<E2>(a, scale), element<E2>(b, scale), element<E2>(d, scale),
                element<E2>(e, scale)}};
    }
  } else {
    for (int i = threadIdx.x; i < slots; i += 256) {
      const double a = value(idx[i]);
      elms[i] = element<E>(a, scale);
      if (second)
        second[i] = element<E2>(a, scale);
    }
  }
  pdl_trigger();
}

template <class E, class E2, class V>
__global__ void refresh_gather_kernel(E *__restrict__ elms, E2 *__restrict__ second,
                                      const int *__restrict__ inv, const V *__restrict__ vals,
                                      long long n, const double *amax)
{
  pdl_wait();
  const double scale = std::is_same<E, __half>::value ? f16_scale(amax) : 1.0;
  if (std::is_same<E, __half>::value && !f16_scale_ok(scale))
    return;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const int src = __ldcs(inv + k);
    const double v = src >= 0 ? (double)__ldg(vals + src) : 0.0;
    elms[k] = element<E>(v, scale);
    if (second)
      second[k] = element<E2>(v, scale);
  }
  pdl_trigger();
}

template <class E>
__global__ void scatter_values_kernel(E *__restrict__ elms, const unsigned *__restrict__ map,
                                      const double *__restrict__ vals, long long n,
                                      const double *amax)
{
  pdl_wait();
  const double scale = std::is_same<E, __half>::value ? f16_scale(amax) : 1.0;
  if (std::is_same<E, __half>::value && !f16_scale_ok(scale))
    return;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    elms[__ldcs(map + k)] = element<E>(__ldg(vals + k), scale);
  pdl_trigger();
}

std::vector<unsigned> slice_begins(const HostSlell &h)
{
  const unsigned spe = 1 + (h.hblock > 1) + (h.var_height ? 1 : 0) + (h.diags ? 2 : 0);
  std::vector<unsigned> b(h.n_slices + 1, 0u);
  for (unsigned s = 0; s <= h.n_slices && h.n_slices; s++)
    b[s] = h.slice_ptr[(size_t)spe * s];
  return b;
}

void SlotMap::release()
{
  for (void *p : {(void *)chunk, (void *)idx, (void *)inv})
    if (p)
      cudaFree(p);
  chunk = nullptr;
  idx = nullptr;
  inv = nullptr;
  n_chunks = max_entries = 0;
  n_slots = 0;
}

constexpr int kChunkEntries = 8192;  // the most entries of a chunk

std::vector<SlotChunk> slot_chunks(const std::vector<unsigned> &slice_begin,
                                   const std::vector<int2> &span)
{
  // a chunk: slices up to 3,072 entries (24 KB of FP64 values, eight CTAs an
  // SM), a taller slice alone up to 8,192, unless such slices are under a third: then
  // every chunk's CTA pays for their shared memory, and the slots are gathered.
  // Slots past 8,192 of a chunk are dealt out by a CTA of their own that copies
  // the entries again (a long row among short ones makes a slice of mostly
  // padding).  FP64, 200,000 rows of 5 entries with every 2,000th of 8,000: 25.4
  // us a refresh with neither rule, 15.6 split, 11.2 gathered.
  constexpr int kFull = 3072;
  constexpr unsigned kSlots = 8192;
  std::vector<SlotChunk> ch;
  size_t tall = 0, runs = 0;
  int lo = 0, hi = -1;  // the open chunk's entries
  unsigned first = 0;
  auto close = [&](unsigned end) {
    const int n = hi >= lo ? hi - lo + 1 : 0;
    runs++;
    tall += n > kFull;
    while (first < end) {
      const unsigned slots = std::min(end - first, kSlots);
      ch.push_back(SlotChunk{first, slots, n ? lo : 0, n});
      first += slots;
    }
    lo = 0;
    hi = -1;
  };
  for (size_t s = 0; s < span.size(); s++) {
    const int l = span[s].x, h = span[s].y;
    if (h < l)
      continue;  // (padding alone joins the open chunk)
    if (h - l >= kChunkEntries)
      return {};
    if (hi >= lo && std::max(hi, h) - std::min(lo, l) >= kFull)
      close(slice_begin[s]);
    lo = hi >= lo ? std::min(lo, l) : l;
    hi = std::max(hi, h);
  }
  close(slice_begin.back());
  if (3 * tall < runs && tall)
    return {};
  return ch;
}

// A map's device array; no memory leaves no error behind for later launches.
template <class T> static int map_array(T **d, const T *h, size_t count)
{
  const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
  if (cudaMalloc(d, bytes) != cudaSuccess) {
    cudaGetLastError();
    *d = nullptr;
    return fail(ISPM_ERR_NOMEM, "value refresh map: cudaMalloc(%zu)", bytes);
  }
  if (count)
    ISPM_CUDA_TRY(cudaMemcpy(*d, h, count * sizeof(T), cudaMemcpyHostToDevice));
  return ISPM_OK;
}

int SlotMap::build(const std::vector<unsigned> &slice_begin, const std::vector<unsigned> &pos)
{
  release();
  n_slots = slice_begin.back();
  const size_t n = (size_t)n_slots;
  // Host passes over entries and slots, 65,536 of them a thread at least (a
  // thread's start-up costs as much); the pages of the arrays are first touched
  // in them.  slot -> entry + 1 (0: padding)
  constexpr long long kGrain = 65536;
  struct Free {
    void operator()(void *p) const { free(p); }
  };
  const std::unique_ptr<int[], Free> own((int *)calloc(std::max<size_t>(n, 1), sizeof(int)));
  int *const in = own.get();
  if (!in)
    return fail(ISPM_ERR_NOMEM, "host allocation while mapping values");
  parallel_for(
      (long long)pos.size(),
      [&](long long a, long long b) {
        for (long long k = a; k < b; k++)
          in[pos[(size_t)k]] = (int)k + 1;
      },
      kGrain);
  const auto grain = [&](size_t parts) {
    return std::max(1LL, (long long)(kGrain * (double)parts / std::max(1.0, (double)n)));
  };
  const long long n_sl = (long long)slice_begin.size() - 1;
  std::vector<int2> span((size_t)n_sl);  // first and last entry of a slice
  parallel_for(
      n_sl,
      [&](long long a, long long b) {
        for (long long s = a; s < b; s++) {
          int l = 0x7fffffff, h = -1;
          for (unsigned p = slice_begin[s]; p < slice_begin[s + 1]; p++)
            if (in[p]) {
              l = std::min(l, in[p] - 1);
              h = std::max(h, in[p] - 1);
            }
          span[(size_t)s] = make_int2(l, h);
        }
      },
      grain((size_t)n_sl));
  const std::vector<SlotChunk> ch = slot_chunks(slice_begin, span);
  if (!ch.empty()) {
    const std::unique_ptr<unsigned short[]> ix(new unsigned short[n]);
    parallel_for(
        (long long)ch.size(),
        [&](long long a, long long b) {
          for (long long q = a; q < b; q++) {
            const SlotChunk c = ch[(size_t)q];
            for (size_t p = c.first, end = p + c.slots; p < end; p++)
              ix[p] = in[p] ? (unsigned short)(in[p] - 1 - c.entry) : (unsigned short)0xffffu;
          }
        },
        grain(ch.size()));
    int e = map_array(&chunk, ch.data(), ch.size());
    if (!e)
      e = map_array(&idx, ix.get(), n);
    if (e) {
      release();
      return e;
    }
    n_chunks = (int)ch.size();
    for (const SlotChunk &c : ch)
      max_entries = std::max(max_entries, c.entries);
    return ISPM_OK;
  }
  parallel_for(
      n_slots,
      [&](long long a, long long b) {
        for (long long p = a; p < b; p++)
          in[p]--;
      },
      kGrain);
  return map_array(&inv, in, n);
}

namespace {

template <class E, class E2, class V>
int refresh_slots_t(E *elms, E2 *second, const SlotMap &m, const V *vals, const double *amax,
                    cudaStream_t s)
{
  cudaError_t e;
  if (m.chunk) {
    const size_t smem = (size_t)m.max_entries * sizeof(V);
    const auto kernel = refresh_chunks_kernel<E, E2, V>;
    // (one limit for every map: another thread may be about to launch a larger one)
    e = smem > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                kChunkEntries * (int)sizeof(V))
                         : cudaSuccess;
    if (e == cudaSuccess)
      e = launch_kernel(kernel, dim3(m.n_chunks), dim3(256), smem, s, true, elms, second,
                        (const SlotChunk *)m.chunk, (const unsigned short *)m.idx, vals, amax);
  } else {
    const long long blocks =
        std::min<long long>((m.n_slots + 255) / 256, (long long)device_sm_count() * 16);
    e = launch_kernel(refresh_gather_kernel<E, E2, V>, dim3((unsigned)blocks), dim3(256), 0, s, true,
                      elms, second, (const int *)m.inv, vals, m.n_slots, amax);
  }
  if (e == cudaSuccess)
    e = cudaPeekAtLastError();
  return e == cudaSuccess ? ISPM_OK
                          : fail(ISPM_ERR_CUDA, "value refresh: %s", cudaGetErrorString(e));
}

template <class V>
int refresh_slots_v(DeviceSlell &d, const SlotMap &m, const V *vals, const double *amax,
                    cudaStream_t s)
{
  switch (d.meta.elm_dtype) {
  case ISPM_F32: return refresh_slots_t((float *)d.elms, (float *)nullptr, m, vals, amax, s);
  case ISPM_F64: return refresh_slots_t((double *)d.elms, (double *)nullptr, m, vals, amax, s);
  case ISPM_BF16:
    return refresh_slots_t((__nv_bfloat16 *)d.elms, (__nv_bfloat16 *)nullptr, m, vals, amax, s);
  }
  return refresh_slots_t((__half *)d.elms, (__half *)nullptr, m, vals, amax, s);
}

}  // namespace

int refresh_slots(DeviceSlell &d, const SlotMap &map, const void *vals, int val_dtype,
                  cudaStream_t s, DeviceSlell *second, const double *amax)
{
  if (map.n_slots != d.meta.n_elms || (second && second->meta.n_elms != d.meta.n_elms))
    return fail(ISPM_ERR_INVALID, "a slot map of %lld slots for %lld elements", map.n_slots,
                d.meta.n_elms);
  if ((d.meta.elm_dtype == ISPM_F16) != (amax != nullptr))
    return fail(ISPM_ERR_INVALID, "FP16 elements (alone) are refreshed with their scale");
  if (!map.n_slots)
    return ISPM_OK;
  if (second) {  // an FP64 matrix and its FP32 or FP64 copy
    if (d.meta.elm_dtype != ISPM_F64 || val_dtype != ISPM_F64 ||
        (second->meta.elm_dtype != ISPM_F32 && second->meta.elm_dtype != ISPM_F64))
      return fail(ISPM_ERR_INVALID, "a joint refresh of element types %d and %d",
                  d.meta.elm_dtype, second->meta.elm_dtype);
    return second->meta.elm_dtype == ISPM_F32
               ? refresh_slots_t((double *)d.elms, (float *)second->elms, map,
                                 (const double *)vals, amax, s)
               : refresh_slots_t((double *)d.elms, (double *)second->elms, map,
                                 (const double *)vals, amax, s);
  }
  return val_dtype == ISPM_F32 ? refresh_slots_v(d, map, (const float *)vals, amax, s)
                               : refresh_slots_v(d, map, (const double *)vals, amax, s);
}

int scatter_values(DeviceSlell &d, const unsigned *map, const double *vals, long long n,
                   cudaStream_t s, const double *amax)
{
  if ((d.meta.elm_dtype == ISPM_F16) != (amax != nullptr))
    return fail(ISPM_ERR_INVALID, "FP16 elements (alone) are refreshed with their scale");
  if (!n)
    return ISPM_OK;
  const unsigned blocks =
      (unsigned)std::min<long long>((n + 255) / 256, (long long)device_sm_count() * 8);
  const auto launch = [&](auto *elms) {
    using E = typename std::remove_pointer<decltype(elms)>::type;
    return launch_kernel(scatter_values_kernel<E>, dim3(blocks), dim3(256), 0, s, true, elms, map,
                         vals, n, amax);
  };
  cudaError_t e = d.meta.elm_dtype == ISPM_F64    ? launch((double *)d.elms)
                  : d.meta.elm_dtype == ISPM_F32  ? launch((float *)d.elms)
                  : d.meta.elm_dtype == ISPM_BF16 ? launch((__nv_bfloat16 *)d.elms)
                                                  : launch((__half *)d.elms);
  if (e == cudaSuccess)
    e = cudaPeekAtLastError();
  return e == cudaSuccess ? ISPM_OK
                          : fail(ISPM_ERR_CUDA, "value scatter: %s", cudaGetErrorString(e));
}

// *out = max |v_k| as the bit pattern of a non-negative double (which orders
// like an unsigned integer); *out must start at 0.
__global__ void absmax_kernel(const double *__restrict__ v, long long n, unsigned long long *out)
{
  double m = 0.0;
#pragma unroll 4
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    m = fmax(m, fabs(__ldg(v + k)));
  for (int off = 16; off > 0; off >>= 1)
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0)
    atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

int absmax_async(const double *vals, long long n, double *out, cudaStream_t s)
{
  ISPM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double), s));
  if (!n)
    return ISPM_OK;
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)device_sm_count() * 8);
  absmax_kernel<<<blocks, 256, 0, s>>>(vals, n, (unsigned long long *)out);
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  return ISPM_OK;
}

int refresh_values(DeviceSlell &d, const unsigned *map, const void *vals, int val_dtype,
                   long long n, cudaStream_t s)
{
  if (d.meta.elm_dtype == ISPM_F16)
    return fail(ISPM_ERR_INVALID, "FP16 elements are refreshed with their scale");
  if (!n)
    return ISPM_OK;
  const int threads = 256;
  long long blocks = (n + threads - 1) / threads;
  blocks = std::min<long long>(blocks, (long long)device_sm_count() * 8);
  const bool e32 = d.meta.elm_dtype == ISPM_F32, v32 = val_dtype == ISPM_F32;
  if (d.meta.elm_dtype == ISPM_BF16 && v32)
    refresh_bf16_kernel<float><<<blocks, threads, 0, s>>>((__nv_bfloat16 *)d.elms, map,
                                                          (const float *)vals, n);
  else if (d.meta.elm_dtype == ISPM_BF16)
    refresh_bf16_kernel<double><<<blocks, threads, 0, s>>>((__nv_bfloat16 *)d.elms, map,
                                                           (const double *)vals, n);
  else if (e32 && v32)
    refresh_values_kernel<float, float><<<blocks, threads, 0, s>>>((float *)d.elms, map,
                                                                   (const float *)vals, n);
  else if (e32)
    refresh_values_kernel<float, double><<<blocks, threads, 0, s>>>((float *)d.elms, map,
                                                                    (const double *)vals, n);
  else if (v32)
    refresh_values_kernel<double, float><<<blocks, threads, 0, s>>>((double *)d.elms, map,
                                                                    (const float *)vals, n);
  else
    refresh_values_kernel<double, double><<<blocks, threads, 0, s>>>((double *)d.elms, map,
                                                                     (const double *)vals, n);
  cudaError_t e = cudaPeekAtLastError();
  return e == cudaSuccess ? ISPM_OK
                          : fail(ISPM_ERR_CUDA, "value refresh: %s", cudaGetErrorString(e));
}

static unsigned pow2_floor(unsigned v) { return v ? 1u << ilog2(v) : 0u; }
static unsigned pow2_ceil(unsigned v) { return v <= 1 ? 1u : 1u << (ilog2(v - 1) + 1); }

ispm_launch_params default_launch(int x_dtype, const ispm_slell_view &m)
{
  return register_walk_launch(x_dtype, m);
}

ispm_launch_params register_walk_launch(int x_dtype, const ispm_slell_view &m,
                                        long long rows)
{
  (void)x_dtype;
  ispm_launch_params p{};
  const double work_rows = rows ? (double)rows : (double)m.n_rows;
  const unsigned esz = m.elm_dtype == ISPM_F64 ? 8 : m.elm_dtype == ISPM_F32 ? 4 : 2;
  const unsigned hmax = m.var_height ? m.min_slice_height : m.slice_height;
  // one 128-bit load of elements per thread and step, at most 4 rows
  unsigned H = std::min(16u / esz, 4u);
  while (H > 1 && H > hmax)
    H >>= 1;
  const unsigned S = m.var_height ? m.max_slice_height : m.slice_height;
  unsigned R = S / H ? S / H : 1;
  // Enough threads to fill the GPU, split a row between several threads
  // only when rows alone do not.
  const double avg_width = m.n_rows ? (double)m.n_elms / (double)m.n_rows : 1.0;
  const double want_threads = 148.0 * 2048.0;
  const double row_threads = work_rows / H;
  unsigned P = 1;
  if (row_threads < want_threads)
    P = pow2_ceil((unsigned)(want_threads / (row_threads > 1 ? row_threads : 1)));
  unsigned pmax = pow2_floor((unsigned)(avg_width / (m.hblock ? m.hblock : 1)));
  if (pmax < 1)
    pmax = 1;
  if (P > pmax)
    P = pmax;
  while (R * P > 1024 && P > 1)
    P >>= 1;
  unsigned N = R * P;
  if (N < 4)
    N = 4;
  while (N > 1024 && H < 4 && H * 2 <= hmax) {  // very tall slices: more rows per thread
    H *= 2;
    N = (S / H) * P;
  }
  p.N = N;
  p.S = m.var_height ? N * H : m.slice_height;
  if (m.var_height && p.S < H)
    p.S = H;
  p.H = H;
  p.use_tex_sliceptr = 1;
  p.use_tex_x = 1;
  return p;
}

}  // namespace ispm

using namespace ispm;

extern "C" {

int ispm_initialize(void)
{
  clear_error();
  int dev = 0;
  ISPM_CUDA_TRY(cudaGetDevice(&dev));
  int major = 0, minor = 0;
  ISPM_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  ISPM_CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev));
  if (major != 10 || minor != 0)
    return fail(ISPM_ERR_ARCH, "compiled for sm_100a, device %d is sm_%d%d", dev, major, minor);
  // The reference sets cudaDeviceMapHost (initialize.cu:28).  Once a context is
  // active the flag can no longer change; mapped host memory is on by default
  // with unified addressing, so that refusal is not an error.
  cudaError_t e = cudaSetDeviceFlags(cudaDeviceMapHost);
  if (e != cudaSuccess && e != cudaErrorSetOnActiveProcess)
    return fail(ISPM_ERR_CUDA, "cudaSetDeviceFlags: %s", cudaGetErrorString(e));
  cudaGetLastError();
  return ISPM_OK;
}

int ispm_get_device_string(char *buf, int len)
{
  clear_error();
  if (!buf || len <= 0)
    return fail(ISPM_ERR_INVALID, "NULL buffer");
  int dev = 0;
  ISPM_CUDA_TRY(cudaGetDevice(&dev));
  cudaDeviceProp p;
  ISPM_CUDA_TRY(cudaGetDeviceProperties(&p, dev));
  snprintf(buf, (size_t)len, "%04x:%02x:%02x (%s)", p.pciDomainID, p.pciBusID, p.pciDeviceID,
           p.name);
  return ISPM_OK;
}

int ispm_refresh_chunks(int n_slices, const unsigned *slice_begin, const int *first_entry,
                        const int *last_entry, ispm_refresh_chunk *out, int cap)
{
  clear_error();
  if (n_slices < 0 || !slice_begin || (n_slices && (!first_entry || !last_entry)) ||
      (cap > 0 && !out))
    return -1;
  try {
    std::vector<int2> span;
    for (int s = 0; s < n_slices; s++)
      span.push_back(make_int2(first_entry[s], last_entry[s]));
    const std::vector<SlotChunk> ch =
        slot_chunks(std::vector<unsigned>(slice_begin, slice_begin + n_slices + 1), span);
    for (size_t k = 0; k < ch.size() && (int)k < cap; k++)
      out[k] = ispm_refresh_chunk{ch[k].first, ch[k].slots, ch[k].entry, ch[k].entries};
    return (int)ch.size();
  } catch (const std::bad_alloc &) {
    return -1;
  }
}

int ispm_dslell_upload(const ispm_slell *h, ispm_dslell **out)
{
  clear_error();
  if (!h || !out)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  *out = nullptr;
  ispm_dslell *d = new (std::nothrow) ispm_dslell;
  if (!d)
    return fail(ISPM_ERR_NOMEM, "host allocation");
  int st = d->d.upload(h->m);
  if (st) {
    delete d;
    return st;
  }
  *out = d;
  return ISPM_OK;
}

int ispm_dslell_upload_f16(const ispm_slell *h, ispm_dslell **out)
{
  clear_error();
  if (!h || !out)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  *out = nullptr;
  ispm_dslell *d = new (std::nothrow) ispm_dslell;
  if (!d)
    return fail(ISPM_ERR_NOMEM, "host allocation");
  int st = d->d.upload_f16(h->m);
  if (st) {
    delete d;
    return st;
  }
  *out = d;
  return ISPM_OK;
}

int ispm_slell_stage_records(const ispm_slell *m, int *out, long long cap, long long *n_ints)
{
  clear_error();
  if (!m || !n_ints || (cap > 0 && !out))
    return fail(ISPM_ERR_INVALID, "NULL argument");
  std::vector<int> rec;
  stage_records(m->m, rec);
  *n_ints = (long long)rec.size();
  for (long long k = 0; k < cap && k < (long long)rec.size(); k++)
    out[k] = rec[(size_t)k];
  return ISPM_OK;
}

int ispm_dslell_update_elms(ispm_dslell *d, const ispm_slell *h)
{
  clear_error();
  if (!d || !h)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  return d->d.update_elms(h->m);
}

int ispm_dslell_get_view(const ispm_dslell *d, ispm_slell_view *view)
{
  if (!d || !view)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  *view = d->d.view();
  return ISPM_OK;
}

void ispm_dslell_free(ispm_dslell *d) { delete d; }

int ispm_dslell_refresh_values(ispm_dslell *d, const unsigned *map, const void *vals,
                               int val_dtype, int n_nz, void *stream)
{
  clear_error();
  if (!d || (n_nz && (!map || !vals)) || n_nz < 0)
    return fail(ISPM_ERR_INVALID, "bad arguments");
  if (val_dtype != ISPM_F32 && val_dtype != ISPM_F64)
    return fail(ISPM_ERR_INVALID, "val_dtype %d", val_dtype);
  if (n_nz != d->d.meta.n_nz)
    return fail(ISPM_ERR_INVALID, "%d values for a matrix of %d non-zeros", n_nz,
                d->d.meta.n_nz);
  return refresh_values(d->d, map, vals, val_dtype, n_nz, (cudaStream_t)stream);
}

int ispm_default_launch(int x_dtype, const ispm_slell_view *m, ispm_launch_params *out)
{
  clear_error();
  if (!m || !out)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  *out = default_launch(x_dtype, *m);
  return check_launch(x_dtype, *out, *m);
}

}  // extern "C"
