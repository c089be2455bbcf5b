// pack.cu - field validation, rigid-pose validation and corner-replicated field copies.
//
// One pass over the field (reference kernels/projection_checks.py:20-56 field scan) also
// writes the layout the sampling kernels read: for the FP32 and FP64 arithmetic a float4
// "quad" per voxel holding the (x, x+1) x (y, y+1) corners of its z plane; for the
// compensated form (FP32, FP16 or BF16 storage) the eight polynomial coefficients of the
// cell.  A sample then needs two 16-byte loads instead of eight gathers.  Corner indices
// clamp to n-1 exactly like
// corner_index (reference kernels/projection.py:217-222), so every sample sees the same
// values as a direct gather.
#include "launch.h"

namespace dpt {
namespace {

__device__ __forceinline__ float half_bits_to_float(uint16_t h)
{
    return __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ float bf16_bits_to_float(uint16_t b)
{
    return __uint_as_float((uint32_t)b << 16);
}

// Exact quotient of a 31-bit index by a fixed divisor: (umulhi(i, m) + i) >> s with
// s = ceil(log2 d) and m = floor(2^32 (2^s - d) / d) + 1 (Granlund and Montgomery's round-up
// method for one bit less than the word, so the sum does not overflow).
struct Divisor {
    unsigned d, m, s;
    void init(unsigned divisor)
    {
        d = divisor;
        s = 0;
        while ((1ull << s) < d) ++s;
        m = (unsigned)((((1ull << s) - d) << 32) / d + 1);
    }
    __device__ __forceinline__ unsigned of(unsigned i) const { return (__umulhi(i, m) + i) >> s; }
};

struct PackArgs {
    int nx, ny, nz;
    Divisor by_nx, by_ny;
    int signed_domain;  // DPT_DOMAIN_SIGNED: only non-finite values are flagged
    unsigned voxels;    // below 2^31
    int views;
    const double* poses;
    int32_t* status;
};

__device__ __forceinline__ void flag_field(bool bad, int32_t* status)
{
    const unsigned any = __ballot_sync(0xffffffffu, bad);
    if (any && (threadIdx.x & 31) == 0) atomicOr(status, 8);
}

// Rigid-pose check of every view, a view per thread of the launch.
__device__ __forceinline__ void check_poses(const PackArgs& a)
{
    for (unsigned view = blockIdx.x * blockDim.x + threadIdx.x; view < (unsigned)a.views; view += gridDim.x * blockDim.x) {
        double p[12];
        for (int k = 0; k < 12; ++k) p[k] = a.poses[12 * (int64_t)view + k];
        if (!rigid_pose(p)) atomicOr(a.status + view, 1);
    }
}

template <int kDtype>
__device__ __forceinline__ float decode(const void* field, int64_t index)
{
    if constexpr (kDtype == DPT_F32) return static_cast<const float*>(field)[index];
    else if constexpr (kDtype == DPT_BF16) return bf16_bits_to_float(static_cast<const uint16_t*>(field)[index]);
    else return half_bits_to_float(static_cast<const uint16_t*>(field)[index]);
}

__device__ __forceinline__ bool out_of_domain(const PackArgs& a, float v)
{
    return !isfinite(v) || (!a.signed_domain && v < 0.0f);
}

// Voxels per thread: 16 independent loads in flight per thread keep HBM busy.  Bound by HBM: with
// one voxel and two 64-bit divisions per thread the check of a 76 x 507 x 512 FP32 field took 115
// us and its quads 148 us, now 22 us (3.5 TB/s) and 70 us (5.7 TB/s); the coefficients of a 512^3
// BF16 field 1062 -> 853 us (5.3 TB/s).
constexpr int kCheckVoxels = 16, kQuadVoxels = 4, kPolyVoxels = 2;
constexpr int kPackBlock = 256;

// Field and pose check without a copy.
template <int kDtype>
__global__ void __launch_bounds__(kPackBlock) k_check_field(PackArgs a, const void* __restrict__ field)
{
    check_poses(a);
    const unsigned first = blockIdx.x * (unsigned)(kPackBlock * kCheckVoxels) + threadIdx.x;
    float v[kCheckVoxels];
#pragma unroll
    for (int k = 0; k < kCheckVoxels; ++k) {
        const unsigned index = first + k * kPackBlock;
        v[k] = index < a.voxels ? decode<kDtype>(field, index) : 0.0f;
    }
    bool bad = false;
#pragma unroll
    for (int k = 0; k < kCheckVoxels; ++k) bad = bad || out_of_domain(a, v[k]);
    flag_field(bad, a.status);
}

// The corners (x, x+1) x (y, y+1) of voxel `index` at its z plane and, with kBoth, at the next.
template <int kDtype, bool kBoth>
__device__ __forceinline__ void load_corners(const PackArgs& a, const void* field, unsigned index, float* v)
{
    const unsigned row = a.by_nx.of(index), z = a.by_ny.of(row);
    const unsigned x = index - row * a.by_nx.d, y = row - z * a.by_ny.d;
    const int64_t right = x + 1 < (unsigned)a.nx ? 1 : 0, down = y + 1 < (unsigned)a.ny ? a.nx : 0;
    const int64_t i = index;
    v[0] = decode<kDtype>(field, i);
    v[1] = decode<kDtype>(field, i + right);
    v[2] = decode<kDtype>(field, i + down);
    v[3] = decode<kDtype>(field, i + down + right);
    if constexpr (kBoth) {
        const int64_t j = i + (z + 1 < (unsigned)a.nz ? (int64_t)a.nx * a.ny : 0);
        v[4] = decode<kDtype>(field, j);
        v[5] = decode<kDtype>(field, j + right);
        v[6] = decode<kDtype>(field, j + down);
        v[7] = decode<kDtype>(field, j + down + right);
    }
}

// FP32 corner quads of any storage type (half values decoded exactly).
struct QuadRecord {
    static constexpr int kVoxels = kQuadVoxels;
    static constexpr bool kBoth = false;
    using Type = float4;
    static __device__ __forceinline__ void write(float4* to, unsigned index, const float* v)
    {
        to[index] = make_float4(v[0], v[1], v[2], v[3]);
    }
};

// Polynomial copy of the compensated precision form: per cell the coefficients of
// f = c0 + c1 x + c2 y + c3 z + c4 xy + c5 xz + c6 yz + c7 xyz from its eight decoded corner
// values (clamped like corner_index), in the order and FP32 arithmetic of PolyCache.
struct PolyRecord {
    static constexpr int kVoxels = kPolyVoxels;
    static constexpr bool kBoth = true;
    using Type = float4;
    static __device__ __forceinline__ void write(float4* to, unsigned index, const float* v)
    {
        const float c1 = v[1] - v[0], c2 = v[2] - v[0], c3 = v[4] - v[0];
        const float c4 = (v[3] - v[2]) - c1, c5 = (v[5] - v[4]) - c1, c6 = (v[6] - v[4]) - c2;
        const float c7 = ((v[7] - v[6]) - (v[5] - v[4])) - c4;
        float4* at = to + 2 * (int64_t)index;
        // one 32-byte store where the copy starts on its boundary (the ABI asks for 16): two
        // 16-byte ones each fill half of every sector
        if ((reinterpret_cast<uintptr_t>(to) & 31) == 0) {
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "f"(v[0]), "f"(c1),
                         "f"(c2), "f"(c3), "f"(c4), "f"(c5), "f"(c6), "f"(c7)
                         : "memory");
        } else {
            at[0] = make_float4(v[0], c1, c2, c3);
            at[1] = make_float4(c4, c5, c6, c7);
        }
    }
};

template <int kDtype, class Record>
__global__ void __launch_bounds__(kPackBlock) k_pack(PackArgs a, const void* __restrict__ field,
                                                     typename Record::Type* __restrict__ copy)
{
    check_poses(a);
    const unsigned first = blockIdx.x * (unsigned)(kPackBlock * Record::kVoxels) + threadIdx.x;
    float v[Record::kVoxels][8];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < Record::kVoxels; ++k) {
        const unsigned index = first + k * kPackBlock;
        if (index < a.voxels) load_corners<kDtype, Record::kBoth>(a, field, index, v[k]);
    }
#pragma unroll
    for (int k = 0; k < Record::kVoxels; ++k) {
        const unsigned index = first + k * kPackBlock;
        if (index < a.voxels) {
            bad = bad || out_of_domain(a, v[k][0]);
            Record::write(copy, index, v[k]);
        }
    }
    flag_field(bad, a.status);
}

template <int kDtype>
void launch_pack(const dpt_problem& p, const PackArgs& a, const void* field, void* copy, cudaStream_t stream)
{
    auto blocks = [&](int voxels) { return (unsigned)(((int64_t)a.voxels + kPackBlock * voxels - 1) / (kPackBlock * voxels)); };
    if (!copy)
        k_check_field<kDtype><<<blocks(kCheckVoxels), kPackBlock, 0, stream>>>(a, field);
    else if (p.arith == DPT_ARITH_F32C)
        k_pack<kDtype, PolyRecord><<<blocks(kPolyVoxels), kPackBlock, 0, stream>>>(a, field, static_cast<float4*>(copy));
    else
        k_pack<kDtype, QuadRecord><<<blocks(kQuadVoxels), kPackBlock, 0, stream>>>(a, field, static_cast<float4*>(copy));
}

}  // namespace

cudaError_t launch_prepare_field(const dpt_problem& p, const void* field, void* packed,
                                 const double* poses, int32_t* status, cudaStream_t stream)
{
    PackArgs a;
    a.nx = p.nx;
    a.ny = p.ny;
    a.nz = p.nz;
    a.by_nx.init((unsigned)p.nx);
    a.by_ny.init((unsigned)p.ny);
    a.voxels = (unsigned)((int64_t)p.nx * p.ny * p.nz);
    a.signed_domain = p.field_domain == DPT_DOMAIN_SIGNED;
    a.views = p.views;
    a.poses = poses;
    a.status = status;
    if (p.field_dtype == DPT_F32)
        launch_pack<DPT_F32>(p, a, field, packed, stream);
    else if (p.field_dtype == DPT_BF16)
        launch_pack<DPT_BF16>(p, a, field, packed, stream);
    else
        launch_pack<DPT_F16>(p, a, field, packed, stream);
    return cudaGetLastError();
}

}  // namespace dpt
