// Host side of the TMA path: tensor-map encoding through the driver entry point (no link-time
// dependency on libcuda) and the pinned error word that kernels with bounded waits report into.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>
#include <memory>

#include "common.h"
#include "tma_utils.cuh"

namespace kutacc {
namespace dev {

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
        KUTACC_CHECK(e == cudaSuccess && q == cudaDriverEntryPointSuccess && p != nullptr,
                     "cuTensorMapEncodeTiled is not available from this driver");
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}
}  // namespace

namespace {
// A tensor map is a pure function of its arguments, and a program calls the operators with the same buffers again and
// again: the last maps of this thread are kept (one per slot of a small hash table) instead of encoded anew, 16 of them per
// gated-attention call at about half a microsecond each.
struct MapKey {
    const void *base;
    cuuint64_t dims[4], strides[3];
    cuuint32_t box[4];
    uint32_t rank, type, swizzle, pad;
};
struct MapSlot {
    MapKey key;
    CUtensorMap map;
    bool used;
};
constexpr uint32_t kMapSlots = 256;

bool encode(CUtensorMap *map, CUtensorMapDataType type, const void *base, uint32_t rank, const cuuint64_t *dims,
            const cuuint64_t *strides, const cuuint32_t *box, int swizzle_bytes)
{
    static thread_local MapSlot *slots = nullptr;
    static thread_local std::unique_ptr<MapSlot[]> owner;
    if (slots == nullptr) {
        owner.reset(new MapSlot[kMapSlots]());
        slots = owner.get();
    }
    MapKey key;
    std::memset(&key, 0, sizeof(key));
    key.base = base;
    for (uint32_t i = 0; i < rank; ++i) {
        key.dims[i] = dims[i];
        key.box[i] = box[i];
        if (i + 1 < rank) key.strides[i] = strides[i];
    }
    key.rank = rank;
    key.type = (uint32_t)type;
    key.swizzle = (uint32_t)swizzle_bytes;
    uint64_t words[sizeof(MapKey) / 8], h = 0;
    static_assert(sizeof(MapKey) % 8 == 0, "hashed word by word");
    std::memcpy(words, &key, sizeof(key));
    for (uint64_t w : words) h = (h ^ w) * 0x9E3779B97F4A7C15ull, h ^= h >> 29;
    MapSlot &slot = slots[h % kMapSlots];
    if (slot.used && std::memcmp(&slot.key, &key, sizeof(key)) == 0) {
        *map = slot.map;
        return true;
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle sw = swizzle_bytes == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                  : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                  : swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                        : CU_TENSOR_MAP_SWIZZLE_NONE;
    const CUresult r = fn(&slot.map, type, rank, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    slot.used = r == CUDA_SUCCESS;
    KUTACC_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with ", (int)r, " rank ", rank, " dims ", dims[0], "x", dims[1],
                 " strides in bytes ", strides[0], " box ", box[0], "x", box[1], " data type ", (int)type);
    if (!slot.used) return false;
    slot.key = key;
    *map = slot.map;
    return true;
}
}  // namespace

bool make_tensor_map_bf16_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                             uint64_t stride1, uint64_t stride2, uint32_t box0, uint32_t box1, int swizzle_bytes,
                             uint32_t box2)
{
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {stride1 * 2, stride2 * 2};
    const cuuint32_t box[3] = {box0, box1, box2};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 3, dims, strides, box, swizzle_bytes);
}

bool make_tensor_map_bf16_4d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3,
                             uint64_t stride1, uint64_t stride2, uint64_t stride3, uint32_t box0, uint32_t box1, uint32_t box3,
                             int swizzle_bytes)
{
    const cuuint64_t dims[4] = {d0, d1, d2, d3}, strides[3] = {stride1 * 2, stride2 * 2, stride3 * 2};
    const cuuint32_t box[4] = {box0, box1, 1, box3};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 4, dims, strides, box, swizzle_bytes);
}

bool make_tensor_map_f32_4d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3,
                            uint64_t stride1, uint64_t stride2, uint64_t stride3, uint32_t box0, uint32_t box1, uint32_t box3,
                            int swizzle_bytes)
{
    const cuuint64_t dims[4] = {d0, d1, d2, d3}, strides[3] = {stride1 * 4, stride2 * 4, stride3 * 4};
    const cuuint32_t box[4] = {box0, box1, 1, box3};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, 4, dims, strides, box, swizzle_bytes);
}

bool make_tensor_map_f32_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1,
                            uint64_t stride2, uint32_t box0, uint32_t box1, int swizzle_bytes)
{
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {stride1 * 4, stride2 * 4};
    const cuuint32_t box[3] = {box0, box1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, 3, dims, strides, box, swizzle_bytes);
}

bool make_tensor_map_2d(CUtensorMap *map, const void *base, int elem_bytes, uint64_t d0, uint64_t d1, uint64_t stride1,
                        uint32_t box0, uint32_t box1, int swizzle_bytes)
{
    if (elem_bytes != 2 && elem_bytes != 4) return false;
    const cuuint64_t dims[2] = {d0, d1}, strides[1] = {stride1 * (cuuint64_t)elem_bytes};
    const cuuint32_t box[2] = {box0, box1};
    return encode(map, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 2, dims,
                  strides, box, swizzle_bytes);
}

int sm_count()
{
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

// One pair of counters per STREAM: launches on one stream run one after another, so they can share a pair (the last CTA of a
// launch zeroes it again), while launches on different streams may overlap and must not. Up to 63 streams per device get a
// pair of their own; further streams share the last pair, which is only safe while they do not run attention kernels at
// the same time.
int *work_counter(cudaStream_t stream)
{
    constexpr int kCounters = 64;
    static int *counters[64] = {};                       // per device
    static cudaStream_t owner[64][kCounters] = {};
    static int owners[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return nullptr;
    if (counters[dev] == nullptr) {
        int *c = nullptr;
        KUTACC_CUDA(cudaMalloc(&c, 2 * kCounters * sizeof(int)));
        if (c == nullptr) return nullptr;
        KUTACC_CUDA(cudaMemset(c, 0, 2 * kCounters * sizeof(int)));
        KUTACC_CUDA(cudaStreamSynchronize(nullptr));     // the caller's stream may not wait for the default one
        counters[dev] = c;
    }
    int slot = -1;
    for (int i = 0; i < owners[dev]; ++i)
        if (owner[dev][i] == stream) {
            slot = i;
            break;
        }
    if (slot < 0) {
        if (owners[dev] < kCounters - 1) {
            slot = owners[dev]++;
            owner[dev][slot] = stream;
        } else {
            slot = kCounters - 1;
        }
    }
    return counters[dev] + 2 * slot;
}

KernelErrorWord &kernel_error_word()
{
    static KernelErrorWord w;
    if (w.host == nullptr) {
        void *h = nullptr;
        cudaError_t e = cudaHostAlloc(&h, sizeof(int), cudaHostAllocMapped);
        KUTACC_CHECK(e == cudaSuccess, "cannot allocate the kernel error word: ", cudaGetErrorString(e));
        if (e == cudaSuccess) {
            w.host = static_cast<int *>(h);
            *w.host = 0;
            void *d = nullptr;
            e = cudaHostGetDevicePointer(&d, h, 0);
            KUTACC_CHECK(e == cudaSuccess, "cannot map the kernel error word: ", cudaGetErrorString(e));
            w.device = static_cast<int *>(d);
        }
    }
    return w;
}

}  // namespace dev
}  // namespace kutacc
