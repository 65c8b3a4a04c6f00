// Host-side support for the C-ABI: device check, TMA tensor-map cache, error
// text.  Nothing here launches a kernel or allocates device memory.

#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "common.cuh"
#include "host.h"

namespace b200 {

static thread_local char g_detail[512] = "";

void set_detail(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_detail, sizeof(g_detail), fmt, ap);
  va_end(ap);
}
const char* get_detail() { return g_detail; }

int cuda_fail(cudaError_t e, const char* where) {
  set_detail("%s: %s", where, cudaGetErrorString(e));
  return -kErrCuda;
}

// Per-device facts and per-(kernel, device) attribute calls, remembered under one mutex so that concurrent
// first calls from several host threads neither race nor repeat the driver call.
struct DeviceFacts {
  int device, major, sm_count;
};
static std::mutex g_dev_mu;
static std::vector<DeviceFacts> g_devices;
struct KernelAttr {
  const void* kernel;
  int device, bytes;
};
static std::vector<KernelAttr> g_kernel_attrs;

static int device_facts(DeviceFacts* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  std::lock_guard<std::mutex> lock(g_dev_mu);
  for (const DeviceFacts& f : g_devices)
    if (f.device == dev) {
      *out = f;
      return 0;
    }
  DeviceFacts f{dev, 0, 0};
  e = cudaDeviceGetAttribute(&f.major, cudaDevAttrComputeCapabilityMajor, dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute(major)");
  e = cudaDeviceGetAttribute(&f.sm_count, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute(sm count)");
  g_devices.push_back(f);
  *out = f;
  return 0;
}

int check_device(int* device_out) {
  DeviceFacts f;
  int rc = device_facts(&f);
  if (rc) return rc;
  if (f.major != 10) {
    set_detail("device %d has compute capability %d.x; this library is built for sm_100a only", f.device,
               f.major);
    return -kErrUnsupported;
  }
  if (device_out) *device_out = f.device;
  return 0;
}

bool overlapped_launch_enabled() {
  static const bool enabled = [] {
    const char* v = getenv("B200_SERIAL_LAUNCH");
    return !(v && v[0] != '\0' && v[0] != '0');
  }();
  return enabled;
}

int device_sm_count(int* out) {
  DeviceFacts f;
  int rc = device_facts(&f);
  if (rc) return rc;
  *out = f.sm_count > 0 ? f.sm_count : 148;
  return 0;
}

int ensure_dynamic_smem(const void* kernel, int bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  std::lock_guard<std::mutex> lock(g_dev_mu);
  for (const KernelAttr& a : g_kernel_attrs)
    if (a.kernel == kernel && a.device == dev && a.bytes >= bytes) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(max dynamic shared memory)");
  g_kernel_attrs.push_back(KernelAttr{kernel, dev, bytes});
  return 0;
}

struct KernelResidency {
  const void* kernel;
  int device, threads;
  size_t smem;
  int ctas;
};
static std::vector<KernelResidency> g_residency;

int resident_ctas(const void* kernel, int threads, size_t smem, int* out) {
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_dev_mu);
  for (const KernelResidency& r : g_residency)
    if (r.kernel == kernel && r.device == dev && r.threads == threads && r.smem == smem) {
      *out = r.ctas;
      return 0;
    }
  cudaFuncAttributes attr;
  B200_CUDA(cudaFuncGetAttributes(&attr, kernel));
  int ctas = 0;
  if (threads <= attr.maxThreadsPerBlock)
    B200_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kernel, threads, smem));
  if (g_residency.size() < 256) g_residency.push_back(KernelResidency{kernel, dev, threads, smem, ctas});
  *out = ctas;
  return 0;
}

int many_form_pays(const void* few, const void* many, int threads, size_t few_smem, size_t many_smem, long long ctas, bool* out) {
  int held_few = 0, held_many = 0, sms = 0;
  int rc = resident_ctas(few, threads, few_smem, &held_few);
  if (!rc) rc = resident_ctas(many, threads, many_smem, &held_many);
  if (!rc) rc = device_sm_count(&sms);
  if (rc) return rc;
  *out = held_few == 0 || (held_many > held_few && ctas > static_cast<long long>(held_few) * sms);
  return 0;
}

// ------------------------------------------------------- tensor-map cache --
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct MapKey {
  int device;
  const void* base;
  uint64_t dim[4];  // innermost first
  int elem_bytes;
  uint32_t box[4];
  uint64_t stride[3];  // bytes, of dim[1..]
  bool operator==(const MapKey& o) const {
    if (base != o.base || device != o.device || elem_bytes != o.elem_bytes) return false;
    for (int i = 0; i < 4; ++i)
      if (dim[i] != o.dim[i] || box[i] != o.box[i] || (i < 3 && stride[i] != o.stride[i])) return false;
    return true;
  }
  size_t set() const {  // FNV-1a over the words, folded
    uint64_t h = 14695981039346656037ull;
    auto mix = [&h](uint64_t v) { h = (h ^ v) * 1099511628211ull; };
    mix(reinterpret_cast<uintptr_t>(base));
    mix(static_cast<uint64_t>(device) << 32 | static_cast<uint32_t>(elem_bytes));
    for (int i = 0; i < 4; ++i) mix(dim[i] << 9 ^ box[i]);
    for (int i = 0; i < 3; ++i) mix(stride[i]);
    return static_cast<size_t>((h ^ h >> 29 ^ h >> 47) % kMapSets);
  }
  static constexpr size_t kMapSets = 1024;
};
struct MapEntry {
  MapKey key;
  CUtensorMap map;
};
// Encoded maps in sets of eight, the oldest of a full set making room.  Every launch looks up a few, so a lookup must not depend
// on how many there are: a list that was searched from its start took 5 us a lookup with 4000 maps in it, and passes of
// few rows, whose launches the host issues one by one, are bound by that.
struct MapSet {
  MapEntry entry[8];
  uint32_t used = 0;  // entries ever put here
};

static std::mutex g_map_mu;
static MapSet* g_maps = nullptr;
static EncodeTiledFn g_encode = nullptr;

// Tensor of `rank` 2 to 4 dimensions.
static int get_tensor_map(int rank, MapKey key, CUtensorMap* out) {
  cudaError_t ce = cudaGetDevice(&key.device);
  if (ce != cudaSuccess) return cuda_fail(ce, "cudaGetDevice");
  std::lock_guard<std::mutex> lock(g_map_mu);
  if (g_maps == nullptr) g_maps = new MapSet[MapKey::kMapSets];
  MapSet& set = g_maps[key.set()];
  for (uint32_t i = 0; i < 8 && i < set.used; ++i) {
    if (set.entry[i].key == key) {
      *out = set.entry[i].map;
      return 0;
    }
  }
  if (g_encode == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    ce = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
    if (ce != cudaSuccess || fn == nullptr || qres != cudaDriverEntryPointSuccess) {
      set_detail("cuTensorMapEncodeTiled is not available from the driver");
      return -kErrTensorMap;
    }
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  const unsigned long long cols = key.dim[0], rows = key.dim[1];
  if (key.box[0] * static_cast<uint32_t>(key.elem_bytes) != 128u || key.box[1] == 0 || key.box[1] > 256 || key.box[2] == 0 ||
      key.box[2] > 256 || key.box[3] == 0 || key.box[3] > 256 || (reinterpret_cast<uintptr_t>(key.base) & 15) != 0 || key.stride[0] % 16 != 0) {
    set_detail("tensor map: base %p rows %llu cols %llu elem %d box %ux%ux%u is not encodable", key.base, rows, cols,
               key.elem_bytes, key.box[2], key.box[1], key.box[0]);
    return -kErrTensorMap;
  }
  cuuint64_t gdim[4] = {key.dim[0], key.dim[1], key.dim[2], key.dim[3]};
  cuuint64_t gstride[3] = {key.stride[0], key.stride[1], key.stride[2]};
  cuuint32_t box[4] = {key.box[0], key.box[1], key.box[2], key.box[3]};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  MapEntry entry;
  entry.key = key;
  CUresult r = g_encode(&entry.map,
                        key.elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8,
                        rank, const_cast<void*>(key.base), gdim, gstride, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_detail("cuTensorMapEncodeTiled failed with CUresult %d (base %p rows %llu cols %llu)", (int)r, key.base, rows, cols);
    return -kErrTensorMap;
  }
  set.entry[set.used % 8] = entry;
  if (++set.used == 16) set.used = 8;
  *out = entry.map;
  return 0;
}

int get_tensor_map_2d(const void* base, uint64_t rows, uint64_t cols, int elem_bytes,
                      uint32_t box_rows, uint32_t box_cols, CUtensorMap* out) {
  return get_tensor_map(2, MapKey{0, base, {cols, rows, 1, 1}, elem_bytes, {box_cols, box_rows, 1, 1}, {cols * elem_bytes, 0, 0}}, out);
}

int get_tensor_map_3d(const void* base, uint64_t planes, uint64_t rows, uint64_t cols, int elem_bytes, uint32_t box_planes,
                      uint32_t box_rows, uint32_t box_cols, CUtensorMap* out) {
  return get_tensor_map(3, MapKey{0, base, {cols, rows, planes, 1}, elem_bytes, {box_cols, box_rows, box_planes, 1},
                                  {cols * elem_bytes, cols * rows * elem_bytes, 0}}, out);
}

int get_tensor_map_atoms(const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out) {
  const uint64_t pitch = cols * 2;
  return get_tensor_map(4, MapKey{0, base, {64, 8, cols / 64, rows / 8}, 2, {64, 8, static_cast<uint32_t>(cols / 64), box_rows / 8},
                                  {pitch, 128, 8 * pitch}}, out);
}

int get_tensor_map_columns(const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out) {
  return get_tensor_map(3, MapKey{0, base, {64, rows, cols / 64, 1}, 2, {64, box_rows, static_cast<uint32_t>(cols / 64), 1},
                                  {cols * 2, 128, 0}}, out);
}

int get_tensor_map_atoms_of(const void* base, uint64_t planes, uint64_t rows, uint64_t cols, uint32_t box_planes, CUtensorMap* out) {
  const uint64_t pitch = cols * 2;
  return get_tensor_map(4, MapKey{0, base, {64, rows, cols / 64, planes}, 2, {64, 8, static_cast<uint32_t>(cols / 64), box_planes},
                                  {pitch, 128, rows * pitch}}, out);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_abi_version(void) { return 1; }

extern "C" const char* b200_strerror(int code) {
  switch (code < 0 ? -code : code) {
    case kErrOk: return "ok";
    case kErrBadArg: return "bad argument (null pointer, shape or alignment)";
    case kErrUnsupported: return "unsupported device or configuration (sm_100a required)";
    case kErrWorkspace: return "workspace too small";
    case kErrCuda: return "CUDA runtime error";
    case kErrTensorMap: return "TMA tensor map could not be encoded";
    case kErrDevBadBlockId: return "device: block table entry outside the pool";
    case kErrDevBadCtxLen: return "device: context length or position outside the block table";
    case kErrDevWaitTimeout: return "device: a bounded barrier wait ran out";
    case kErrDevBadExpert: return "device: expert id outside [0, num_experts)";
    case kErrDevPeerTimeout: return "device: a bounded wait for another rank's flag ran out";
    default: return "unknown error";
  }
}

extern "C" const char* b200_last_error_detail(void) { return get_detail(); }

// Copies the device status word back and returns it negated (0 = clean).
// This is the one entry point that synchronises the stream.
extern "C" int b200_read_status(const void* status_word, void* stream) {
  if (status_word == nullptr) {
    set_detail("read_status: null pointer");
    return -kErrBadArg;
  }
  int v = 0;
  cudaError_t e = cudaMemcpyAsync(&v, status_word, sizeof(int), cudaMemcpyDeviceToHost, as_stream(stream));
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(status)");
  e = cudaStreamSynchronize(as_stream(stream));
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
  return -v;
}
