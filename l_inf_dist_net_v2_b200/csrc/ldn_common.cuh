// Shared definitions for the sm_100a L_p-distance kernels: tile geometry, kernel parameter blocks,
// mbarrier / TMA primitives (inline PTX, no multicast), and the host-side context.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace ldn {

// ---------------------------------------------------------------------------------------------
// Status codes returned by every C-ABI entry point (0 = success).  Values >= 1000 wrap a
// cudaError_t (code - 1000).
// ---------------------------------------------------------------------------------------------
enum Status : int {
    kOk = 0,
    kBadArgument = 1,      // null pointer, non-positive size, CI or CO not divisible by G, p <= 0 ...
    kNoDevice = 2,         // no CUDA device / driver entry point missing
    kWorkspace = 3,        // workspace allocation failed or fixed scratch too small
    kDeviceTimeout = 4,    // a bounded wait inside a kernel gave up (status word set by the device)
    kTensorMap = 5,        // cuTensorMapEncodeTiled rejected a descriptor
    kCaptureGrowth = 6,    // the scratch arena would have to grow while its stream is being captured
    kCudaBase = 1000
};

// ---------------------------------------------------------------------------------------------
// Tile geometry.  One CTA of 256 threads owns a 128 x 128 output tile; every thread owns an
// 8 x 8 register block.  The reduction dimension advances 32 elements per pipeline stage.
// ---------------------------------------------------------------------------------------------
constexpr int kTileM = 128;
constexpr int kTileN = 128;
constexpr int kTileK = 32;
constexpr int kThreads = 256;
constexpr int kRegM = 8;
constexpr int kRegN = 8;
constexpr int kTileElems = kTileM * kTileN;            // outputs per tile
constexpr int kOperandTileBytes = kTileM * kTileK * 4;  // 16 KiB, both operand tile shapes

// Bounded waits: a poll loop gives up after this many failed polls (each followed by a short
// nanosleep once the fast polls are used up), writes kDeviceTimeout into the status word and the
// CTA returns.  2^22 polls * >= 64 ns is far beyond any legitimate TMA latency.
constexpr uint32_t kFastPolls = 1u << 14;
constexpr uint32_t kMaxPolls = 1u << 22;

// One operand as the generic (non-TMA) code sees it: element (row r, inner index c, group g)
// lives at ptr[c + r * stride_row + g * stride_group].
struct Operand {
    const float* ptr;
    long long stride_row;
    long long stride_group;
};

struct Shape {
    int B, CO, CI, G, HW;
    int CIg, COg;
    long long M;  // B * HW
    // A range of output channels of a wider layer (G == 1 only): grad_output / output rows are co_src channels long and
    // this problem's channel o is their channel co_off + o.  co_src == CO, co_off == 0: the whole layer.
    int co_src, co_off;
};

// Output addressing shared by all kernels:
//   offset(m, n, g) = (m / hw_div) * s_b + (m % hw_div) * s_hw + g * s_g + n * s_n
struct OutAddr {
    long long s_b, s_hw, s_g, s_n;
    int hw_div;
};

struct TileParams {
    int M, N, K, G;             // per-group extents of the tile problem
    int tiles_m, tiles_n, kt;   // kt = ceil(K / 32)
    long long total_iters;      // G * tiles_m * tiles_n * kt
    int a_row_coord;            // which TMA coordinate (1 or 2) is the row/k index of A; the other is g
    int b_row_coord;            // same for B
    int b_group_mod;            // > 0: B's group coordinate is (engine group) % b_group_mod; 0: the engine group
    Operand a0, a1, b, pres;    // generic views (rescan of argmax chunks, resident per-output operand)
    OutAddr out;
    float* out_f0;
    float* out_f1;
    int* out_i0;
    int* out_i1;
    float p;                    // the exponent the op was called with
    float q;                    // op specific (p - 1 for backward)
    const float* norm_rows;     // FwdPowNorm with a separable normaliser M[m, n] = max(norm_rows[g][m] + norm_cols[g'][n], 1e-10)
    const float* norm_cols;     //   (row-wise largest magnitudes of the two operands: an upper bound of max |t|); else null
    int* guard;                 // raised by that form when a sum comes out too small for the normaliser to have been adequate
    const float* col_sub;       // optional per-output-channel epilogue of the no-grad p = inf kernels:
    const float* col_add;       //   stored value = (result - col_sub[channel]) + col_add[channel]; either may be null
    const int* gate;            // not null: the kernel returns at once unless (*gate != 0) == (gate_invert == 0)
    int gate_invert;
    int pres_vec;               // backward kernels: elements n .. n + 3 (n a multiple of 4) of a row of the resident operand,
                                //   which has the output's layout, are one aligned 16-byte piece
    int accumulate_out;         // backward kernels: add to the output instead of overwriting it
    float* side_out;            // fused backward: per-row-tile column sums [tile_m][g][k][n] (else null)
    float* partials;            // stream-K scratch: [grid][2][arrays][kTileElems]
    int* status;                // device status word (0 = ok)
    unsigned long long* trace;  // optional per-CTA trace: {sm id, start ns, end ns, iterations}; may be null
};

// ---------------------------------------------------------------------------------------------
// Device primitives
// ---------------------------------------------------------------------------------------------
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  Returns false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < kMaxPolls; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i >= kFastPolls) __nanosleep(64);
    }
    return false;
}

// Tiled TMA load of one 3-D box into shared memory (no multicast), completion on an mbarrier.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)),
          "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// Start of every kernel that is launched with launch_after(): lets the next kernel of the stream be set up while this one
// runs, and waits until everything in front of it on the stream is complete and visible.  Nothing may be read or written
// before it, and every block executes it: a grid that was complete before its predecessor would let its successor run too
// early.  (Pointers of these kernels carry no __restrict__: a load that is known not to change could be moved up across it.)
// A launch behind another costs 1 us less: 200 x 1001 -> 777, p = 3, forward + input gradient (10 launches) 121 -> 107 us,
// 128 x 64 x 16 x 16 convolution step at p = inf 400 -> 391, 512 x 3072 -> 5120 certification 1982 -> 1972.
__device__ __forceinline__ void stream_order_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void stream_order_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void stream_order_begin() {
    stream_order_release();
    stream_order_wait();
}

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned sm_id() {
    unsigned s;
    asm volatile("mov.u32 %0, %smid;" : "=r"(s));
    return s;
}

// `bytes` of BYTES (4 or 16) from global into shared memory, in the background; zeros for the rest
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src, int bytes) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// Order-preserving code of a float (0 is below all of them); a not-a-number of either sign is above infinity in the code of
// the value or of its negative.
__device__ __forceinline__ unsigned ordered(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float from_ordered(unsigned c) {
    return __uint_as_float((c & 0x80000000u) ? c & 0x7fffffffu : ~c);
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
#endif  // __CUDACC__

// ---------------------------------------------------------------------------------------------
// Host-side context (ldn_context.cu)
// ---------------------------------------------------------------------------------------------
struct DeviceCtx {
    int device;
    int sm_count;
    int max_smem_optin;
};

// Cached per-device properties for the current device; nullptr + status on failure.
int get_device_ctx(const DeviceCtx** out);

// Per-(device, stream) scratch arena owned by the library.  The block grows on demand (never while the stream is
// being captured) and is 256-byte aligned.  The arena also carries the device status word.
struct Arena {
    char* base;
    size_t capacity;
    int* status;   // device int, zeroed at creation
    int* status_host;  // pinned host mirror used when checking
    void* call_mutex;  // std::mutex*: held for the length of one entry-point call, so that two host threads that
                       // use the same stream cannot interleave launches that share the scratch block
    bool graph_used;   // a call was issued on this arena while its stream was being captured
    void* retired;     // std::vector<void*>*: earlier blocks that captured graphs may still refer to
    bool reserved = false;  // the caller chose the size (ldn_reserve_scratch): it grows only for what a call cannot do without
    const int* extreme_words = nullptr;  // device words of the last call, if that started from the extreme channels
    const int* power_words[2] = {};  // device words of the last call, if that began with the matrix products of an even p or with
                                     // power lists: one that is not 0 (either may be null) says that the general kernels ran
    size_t refused = 0;     // not 0: the smallest size that could not be had for a growth that a call can do without
};
int find_arena(cudaStream_t stream, Arena** out);
int ensure_arena(Arena* arena, cudaStream_t stream, size_t bytes);  // caller holds call_mutex
// The same for scratch that a call can do without: false leaves the arena as it is.
bool extend_arena(Arena* arena, cudaStream_t stream, size_t bytes);

// Bump allocator over an arena (256-byte granularity).
struct Bump {
    char* base;
    size_t off;
    size_t cap;
    template <class T>
    T* take(size_t count) {
        size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
        if (off + bytes > cap) return nullptr;
        T* p = reinterpret_cast<T*>(base + off);
        off += bytes;
        return p;
    }
};
inline size_t pad256(size_t bytes) { return (bytes + 255) & ~size_t(255); }

// Tiled 3-D tensor map over fp32 data.  dims/strides are in elements, innermost first; `swizzle128`
// selects the 128-byte swizzle (inner box must then be 32 floats).
int make_tensor_map(CUtensorMap* map, const float* base, const unsigned long long dims[3],
                    const unsigned long long strides_elems[2], const unsigned box[3], bool swizzle128);

// optional CUDA-event pair around the most recent tile-kernel launch (ldn_diag.cu); no-ops unless enabled
void timing_before(cudaStream_t st);
void timing_after(cudaStream_t st);
void timing_forget();  // there is no launch to report until the next pair

// host-side launch counter and optional per-CTA trace buffer (ldn_diag.cu)
unsigned long long* trace_buffer();
void count_launches(int n);

inline int cuda_status(cudaError_t e) { return e == cudaSuccess ? kOk : kCudaBase + static_cast<int>(e); }

// What a launcher sets up once per device (static in it), such as its kernels' shared memory: by whichever thread comes first, or
// by several (it does no harm).
class OncePerDevice {
    std::atomic<bool> done_[64] = {};

public:
    template <class F>
    int operator()(F set_up) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 64 && done_[dev].load(std::memory_order_acquire)) return kOk;
        const cudaError_t e = set_up();
        if (e == cudaSuccess && dev < 64) done_[dev].store(true, std::memory_order_release);
        return cuda_status(e);
    }
};
template <class K>
cudaError_t allow_smem(K* kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Launches a kernel that begins with stream_order_begin(): its blocks may be placed on the SMs that the kernel in front of it
// on the stream leaves, instead of after that kernel's end and a launch's latency.
template <class... P, class... A>
int launch_after_in_clusters(void (*kernel)(P...), unsigned cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                             A&&... args) {
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e == cudaSuccess) count_launches(1);
    else cudaGetLastError();
    return cuda_status(e);
}
template <class... P, class... A>
int launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    return launch_after_in_clusters(kernel, 1, grid, block, smem, st, args...);
}

}  // namespace ldn
