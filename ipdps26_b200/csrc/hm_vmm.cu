// Growable device memory on CUDA virtual memory management (GrowSpace).
// The driver's VMM calls are looked up through the runtime's entry-point
// query, so the library does not link the driver library directly.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "hm_device.h"

namespace {

using FnCreate = CUresult (*)(CUmemGenericAllocationHandle*, size_t, const CUmemAllocationProp*, unsigned long long);
using FnRelease = CUresult (*)(CUmemGenericAllocationHandle);
using FnReserve = CUresult (*)(CUdeviceptr*, size_t, size_t, CUdeviceptr, unsigned long long);
using FnFree = CUresult (*)(CUdeviceptr, size_t);
using FnMap = CUresult (*)(CUdeviceptr, size_t, size_t, CUmemGenericAllocationHandle, unsigned long long);
using FnUnmap = CUresult (*)(CUdeviceptr, size_t);
using FnAccess = CUresult (*)(CUdeviceptr, size_t, const CUmemAccessDesc*, size_t);
using FnGran = CUresult (*)(size_t*, const CUmemAllocationProp*, CUmemAllocationGranularity_flags);
using FnAttr = CUresult (*)(int*, CUdevice_attribute, CUdevice);

struct Vmm {
  bool ok = false;
  FnCreate create = nullptr;
  FnRelease release = nullptr;
  FnReserve reserve = nullptr;
  FnFree free = nullptr;
  FnMap map = nullptr;
  FnUnmap unmap = nullptr;
  FnAccess access = nullptr;
  FnGran gran = nullptr;
  FnAttr attr = nullptr;
};

template <class F>
bool lookup(const char* name, F* fn) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q{};
  if (cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !p) {
    cudaGetLastError();
    return false;
  }
  *fn = reinterpret_cast<F>(p);
  return true;
}

const Vmm& vmm_api() {
  static Vmm v;
  static std::once_flag once;
  std::call_once(once, [] {
    v.ok = lookup("cuMemCreate", &v.create) && lookup("cuMemRelease", &v.release) &&
           lookup("cuMemAddressReserve", &v.reserve) && lookup("cuMemAddressFree", &v.free) &&
           lookup("cuMemMap", &v.map) && lookup("cuMemUnmap", &v.unmap) && lookup("cuMemSetAccess", &v.access) &&
           lookup("cuMemGetAllocationGranularity", &v.gran) && lookup("cuDeviceGetAttribute", &v.attr);
  });
  return v;
}

CUmemAllocationProp prop_of(int device) {
  CUmemAllocationProp p = {};
  p.type = CU_MEM_ALLOCATION_TYPE_PINNED;
  p.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  p.location.id = device;
  return p;
}

size_t round_up(size_t x, size_t g) { return (x + g - 1) / g * g; }

}  // namespace

namespace hm {

// Maps one chunk at va and opens it to the device.
static int map_one(const Vmm& v, int device, CUdeviceptr va, size_t size, unsigned long long handle) {
  if (v.map(va, size, 0, handle, 0) != CUDA_SUCCESS) return set_error(HM_ERR_CUDA, "cuMemMap of %zu bytes failed", size);
  CUmemAccessDesc d = {};
  d.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  d.location.id = device;
  d.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
  if (v.access(va, size, &d, 1) != CUDA_SUCCESS) {
    v.unmap(va, size);
    return set_error(HM_ERR_CUDA, "cuMemSetAccess failed");
  }
  return HM_OK;
}

// Unmaps chunks [i0, i1) of a reservation at va, one mapping at a time. The
// caller has waited for the context's stream: every kernel that reads the
// chunks runs on it, or was waited for by the call that launched it. (Waiting
// for the device would end the captures other contexts have under way, and
// fail itself while one is.)
static void unmap_chunks(const Vmm& v, CUdeviceptr va, const std::vector<size_t>& sizes, size_t i0, size_t i1) {
  size_t at = 0;
  for (size_t i = 0; i < i0; ++i) at += sizes[i];
  for (size_t i = i0; i < i1; ++i) {
    v.unmap(va + at, sizes[i]);
    at += sizes[i];
  }
}

// Physical memory is taken in chunks of at most kChunk bytes, so that shrink
// can give back all but the chunk the kept bytes end in.
constexpr size_t kChunk = size_t(1) << 30;

// A first allocation of up to this size comes from the context's pool, and
// moves to mapped chunks when it grows. Reserving, creating, mapping and
// opening chunks, and the device synchronisations around unmapping, cost a
// small graph that is built and counted more than its kernels (three arrays
// each; 20K hyperedges: 3.2 ms, 0.8 ms of it kernels). Sizes are rounded up to
// kGranule as mapped chunks are, so the budget is charged the same either way.
constexpr size_t kPooledMax = size_t(64) << 20, kGranule = size_t(2) << 20;

static bool vmm_supported(int device) {
  int ok = 0;
  const Vmm& v = vmm_api();
  return v.ok && v.attr(&ok, CU_DEVICE_ATTRIBUTE_VIRTUAL_MEMORY_MANAGEMENT_SUPPORTED, device) == CUDA_SUCCESS && ok;
}

int GrowSpace::grow(hm_ctx* c, size_t bytes) {
  if (bytes <= mapped) return HM_OK;
  ctx = c;
  HM_CUDA(cudaSetDevice(ctx->device));
  if (vmm) return grow_mapped(bytes);
  if (vmm_supported(ctx->device) && (mapped || bytes > kPooledMax)) return move_to_chunks(bytes);
  bytes = round_up(bytes, kGranule);
  void* q = nullptr;
  HM_TRY(dev_alloc(ctx, &q, bytes));
  if (mapped) {  // no VMM: allocate, copy, free
    HM_CUDA(cudaMemcpyAsync(q, base, mapped, cudaMemcpyDeviceToDevice, ctx->stream));
    dev_free(ctx, base, mapped);
  }
  base = static_cast<char*>(q);
  mapped = reserved = bytes;
  return HM_OK;
}

// From the pool (or nothing) to mapped chunks. The old block is freed only once
// the new one holds its contents, so a growth that fails leaves the space as it
// was, at the same address. While both exist the budget is charged for the new
// one alone: growth in chunks needs no second copy and a store it suits must
// still fit, and the old block is kPooledMax at most.
int GrowSpace::move_to_chunks(size_t bytes) {
  GrowSpace next;
  next.ctx = ctx;
  next.vmm = true;
  uncharge(ctx, mapped);
  int s = next.grow_mapped(bytes);
  if (s == HM_OK && mapped) {
    const cudaError_t e = cudaMemcpyAsync(next.base, base, mapped, cudaMemcpyDeviceToDevice, ctx->stream);
    if (e != cudaSuccess) s = set_error(HM_ERR_CUDA, "moving an arena to chunks: %s", cudaGetErrorString(e));
  }
  if (s < 0) {
    next.release();
    ctx->used.fetch_add(mapped);
    return s;
  }
  if (mapped) cudaFreeAsync(base, ctx->stream);
  base = next.base;
  mapped = next.mapped;
  reserved = next.reserved;
  vmm = true;
  handles.swap(next.handles);
  sizes.swap(next.sizes);
  next.base = nullptr;  // now held here
  return HM_OK;
}

int GrowSpace::grow_mapped(size_t bytes) {
  const Vmm& v = vmm_api();
  const CUmemAllocationProp prop = prop_of(ctx->device);
  size_t g = 0;
  if (v.gran(&g, &prop, CU_MEM_ALLOC_GRANULARITY_RECOMMENDED) != CUDA_SUCCESS || !g) g = 2u << 20;
  const size_t target = mapped + round_up(bytes - mapped, g);
  HM_TRY(charge(ctx, target - mapped));
  // the new chunks
  const size_t first = handles.size();
  int status = HM_OK;
  for (size_t at = mapped; at < target;) {
    const size_t sz = std::min(kChunk, target - at);
    CUmemGenericAllocationHandle h = 0;
    CUresult r = v.create(&h, sz, &prop, 0);
    if (r == CUDA_ERROR_OUT_OF_MEMORY) {  // the stream-ordered pool may hold freed blocks
      trim_pool(ctx);
      r = v.create(&h, sz, &prop, 0);
    }
    if (r != CUDA_SUCCESS) {
      status = set_error(r == CUDA_ERROR_OUT_OF_MEMORY ? HM_ERR_NOMEM : HM_ERR_CUDA,
                         "cuMemCreate of %zu bytes failed (%d)", sz, (int)r);
      break;
    }
    handles.push_back(h);
    sizes.push_back(sz);
    at += sz;
  }
  CUdeviceptr va = (CUdeviceptr)base;
  size_t va_size = reserved;
  const bool moved = target > reserved;
  if (status == HM_OK && moved) {
    // a new, larger reservation holding every chunk; the old one is dropped
    // once no kernel can still use it
    va_size = round_up(std::max(2 * reserved, 2 * target), g);
    va = 0;
    if (v.reserve(&va, va_size, g, 0, 0) != CUDA_SUCCESS) {
      va = 0;
      status = set_error(HM_ERR_NOMEM, "cuMemAddressReserve of %zu bytes failed", va_size);
    }
  }
  size_t n_mapped = 0;  // chunks mapped into va by this call, from index `from`
  const size_t from = moved ? 0 : first;
  if (status == HM_OK) {
    size_t at = 0;
    for (size_t i = 0; i < from; ++i) at += sizes[i];
    for (size_t i = from; i < handles.size(); ++i) {
      status = map_one(v, ctx->device, va + at, sizes[i], handles[i]);
      if (status != HM_OK) break;
      ++n_mapped;
      at += sizes[i];
    }
  }
  if (status != HM_OK) {
    unmap_chunks(v, va, sizes, from, from + n_mapped);
    if (moved && va) v.free(va, va_size);
    for (size_t i = first; i < handles.size(); ++i) v.release(handles[i]);
    handles.resize(first);
    sizes.resize(first);
    uncharge(ctx, target - mapped);
    return status;
  }
  if (moved) {
    if (base) {
      HM_CUDA(cudaStreamSynchronize(ctx->stream));
      unmap_chunks(v, (CUdeviceptr)base, sizes, 0, first);
      v.free((CUdeviceptr)base, reserved);
    }
    base = reinterpret_cast<char*>(va);
    reserved = va_size;
  }
  mapped = target;
  return HM_OK;
}

void GrowSpace::shrink(size_t bytes) {
  if (!base || !vmm || bytes >= mapped) return;
  const Vmm& v = vmm_api();
  size_t at = mapped;
  size_t k = handles.size();
  while (k > 0 && at - sizes[k - 1] >= bytes && at - sizes[k - 1] > 0) {
    at -= sizes[k - 1];
    --k;
  }
  if (k == handles.size()) return;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  unmap_chunks(v, (CUdeviceptr)base, sizes, k, handles.size());
  for (size_t i = k; i < handles.size(); ++i) v.release(handles[i]);
  uncharge(ctx, mapped - at);
  handles.resize(k);
  sizes.resize(k);
  mapped = at;
}

void GrowSpace::release() {
  if (!base) return;
  if (!vmm) {
    dev_free(ctx, base, mapped);
  } else {
    const Vmm& v = vmm_api();
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    unmap_chunks(v, (CUdeviceptr)base, sizes, 0, handles.size());
    v.free((CUdeviceptr)base, reserved);
    for (auto h : handles) v.release(h);
    uncharge(ctx, mapped);
  }
  handles.clear();
  sizes.clear();
  base = nullptr;
  mapped = reserved = 0;
  vmm = false;
  ctx = nullptr;
}

bool vmm_available() { return vmm_api().ok; }

}  // namespace hm
