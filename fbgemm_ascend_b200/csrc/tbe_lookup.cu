// Quantized table-batched-embedding lookup for B200 (sm_100a).
//
// Replaces the device side of int_nbit_split_embedding_codegen_lookup_function
// (reference: c310/op_kernel/int_nbit_split_embedding_pooling_kernel.h:44-394 and
// int_nbit_split_embedding_nobag_kernel.h:31-398).  The path is a gather and a
// reduction, bounded by the instructions issued per row and by HBM/L2 bandwidth.  Codes as operands of mma.sync with bags as
// its columns measured slower than the packed FMAs: the instruction runs at one per 64 cycles and SM quarter here.
//
// Pooled kernel (SUM / MEAN), in three tiers chosen per table:
//   * aligned rows of INT8 / INT4 / FP8 / FP16 / FP32 with D a multiple of 16 up to 512 (FP32: from 80) (pool_run_stream): LPR lanes
//     share a row, 16 fp32 accumulators per lane, so a warp has 32/LPR lane groups.  The rows of a warp's bags are
//     cut into equal ranges, one per group, and every group streams its range through a small ring in shared
//     memory: asynchronous 16-byte copies through L1 (which holds the hot head of a Zipf-distributed table), several
//     rows per group in flight, consumed in order; bags that straddle two ranges are combined through shared memory.  Codes
//     are multiplied by the row's fp16 scale and accumulated in fp32 where they lie in their words (see kCodeScale).  INT8/INT4 rows start with a 4-byte header, which shifts the payload off the
//     16-byte grid; the lane that reads the header chunk has 4 / 8 free slots, which take the row's last
//     elements, so D = 16*LPR rows keep every lane busy with exactly 16 elements;
//   * aligned rows of the same types and any other D that is a multiple of 4 (pool_run_steps): a warp sums its bags one after
//     the other, eight rows per step, every unit of a row by four lanes;
//   * anything else (row_alignment 1, odd D, INT2 or BF16 rows, unaligned tables): a byte-wise path.
// Sequence mode (pooling NONE): tbe_nobag_kernel, 64 consecutive positions per warp.
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>

#include <atomic>

#include "tbe_common.cuh"

namespace tbe {

namespace {

constexpr unsigned kFull = 0xffffffffu;

struct LookupParams {
    const uint8_t* dev_weights;
    const int64_t* weights_offsets;
    const uint8_t* weights_tys;
    const int32_t* D_offsets;
    const void* indices;
    const void* offsets;
    const float* pw;
    void* output;
    const int64_t* out_cols;
    void* const* dests;
    int32_t* error_flag;
    int64_t B;
    int64_t num_bags;
    int64_t num_indices;
    int64_t out_stride;
    int64_t rows_per_dest;
    int64_t span;        // bags per warp
    int32_t T;
    uint32_t B32;        // B when T*B < 2^32, else 0
    int32_t pooling_mode;
    int32_t out_ty;
    int32_t row_alignment;
    uint32_t fp8_shift;  // 16 + exponent bits
    float fp8_mult;      // 2^(127 - bias)
    int64_t dev_weights_bytes;   // size of dev_weights, 0 = unknown
    int32_t idx64;       // indices and offsets are 64-bit
};

__host__ __device__ inline int64_t row_bytes_of(int ty, int D, int align)
{
    int64_t b;
    switch (ty) {
        case TBE_B200_FP32: b = 4ll * D; break;
        case TBE_B200_FP16: b = 2ll * D; break;
        case TBE_B200_BF16: b = 2ll * D; break;
        case TBE_B200_FP8: b = D; break;
        case TBE_B200_INT8: b = D + 4ll; break;
        case TBE_B200_INT4: b = (D + 1) / 2 + 4ll; break;
        case TBE_B200_INT2: b = (D + 3) / 4 + 4ll; break;
        default: return 0;
    }
    if (align > 1) b = (b + align - 1) / align * align;
    return b;
}

// ---- output ----------------------------------------------------------------

// Two finished elements as 16-bit ones.
__device__ __forceinline__ uint32_t pack_out(float a, float b, int out_ty)
{
    if (out_ty == TBE_B200_FP16) {
        const __half2 x = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&x);
    }
    const __nv_bfloat162 x = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&x);
}

// Converts and stores four consecutive finished elements, from element e0 of `seg` on; `vec` says that the address is
// aligned for one store.
__device__ __forceinline__ void store_out4(void* seg, int e0, const float* v, int out_ty, bool vec)
{
    if (out_ty == TBE_B200_FP32) {
        float* p = static_cast<float*>(seg) + e0;
        if (vec) {
            st_stream16(p, make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3])));
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = v[j];
        }
    } else {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = (out_ty == TBE_B200_FP16) ? f32_to_f16_bits(v[j]) : f32_to_bf16_bits(v[j]);
        unsigned short* p = static_cast<unsigned short*>(seg) + e0;
        if (vec) {
            st_stream8(p, make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16)));
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = static_cast<unsigned short>(h[j]);
        }
    }
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// 16-byte asynchronous copy global -> shared through L1 (the line stays cached for the rows that are fetched again and
// again); `bytes` = 16, or 0 to write zeros without reading.
__device__ __forceinline__ void cp_async16_ca(uint32_t dst, const void* src, int bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
#ifdef TBE_L2_HINTS
// Experiment (TBE_L2_HINTS builds only): the row copies carry an L2 evict-last policy.  Measured on benchmark
// configurations 2 and 4 (scaled): L2 hit rate, DRAM bytes and kernel time all unchanged (31.8 -> 31.9 % and
// 45.5 -> 45.5 %; the hottest rows never reach L2, they hit L1, and the rest of the Zipf head stays in L2 anyway),
// so the plain form is what is built.
__device__ __forceinline__ uint64_t l2_policy_evict_last()
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void cp_async16_ca_hint(uint32_t dst, const void* src, int bytes, uint64_t pol)
{
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(dst), "l"(src), "r"(bytes), "l"(pol) : "memory");
}
#endif
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, int bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint4 lds16(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds8(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds4(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// ---- dequantisation arithmetic ------------------------------------------------
//
// Integer -> float conversion instructions run at 16 lanes per clock per SM on sm_100a, which would cap a 128-element INT8
// row at 8 cycles, so neither mode uses them.  Pooled sums take codes where they lie (see kCodeScale).  Sequence mode
// turns codes into exact fp16 values with one byte permute (or mask) and one half2 subtract per pair -- 0x6400 | q is the
// half 1024 + q -- and adds them to the bias with the sm_100 mixed-precision FMA (fp16 * fp16 + fp32 -> fp32): the
// row scale is stored as fp16, so code * scale + bias is rounded once, as by an fp32 FMA.

// Two exact fp16 values (as a half2 bit pattern) from two codes already or'ed into the mantissas of
// the half2 `magic` (0x6400: 1024, 0x5400: 64 with the code in mantissa bits 4..7).
__device__ __forceinline__ uint32_t codes_to_half2(uint32_t packed, uint32_t magic)
{
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&packed), *reinterpret_cast<const __half2*>(&magic));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// a0, a1 += pair (half2 bits) * scale (fp16 bits), a mixed FMA each.
__device__ __forceinline__ void add_pair(float& a0, float& a1, uint32_t pair, unsigned short scale_h)
{
    asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; fma.rn.f32.f16 %0, l, %3, %0; fma.rn.f32.f16 %1, h, %3, %1; }"
        : "+f"(a0), "+f"(a1)
        : "r"(pair), "h"(scale_h));
}

// Description of the table a bag belongs to; reloaded only when the warp moves on to another table.
struct TableMeta {
    const uint8_t* table;   // first row
    int64_t stride;         // bytes per row
    int64_t col;            // output column of the table
    int64_t avail;          // bytes of dev_weights the table's rows may occupy (a row past them is not read)
    int32_t ty;
    int32_t D;
    bool rows_aligned;      // table start and row stride are multiples of 16 bytes
};

__device__ __forceinline__ TableMeta load_meta(const LookupParams& p, int t)
{
    TableMeta m;
    m.ty = p.weights_tys[t];
    const int d0 = p.D_offsets[t];
    m.D = p.D_offsets[t + 1] - d0;
    m.table = p.dev_weights + p.weights_offsets[t];
    m.col = p.out_cols ? p.out_cols[t] : static_cast<int64_t>(d0);
    m.stride = row_bytes_of(m.ty, m.D, p.row_alignment);
    m.rows_aligned = ((reinterpret_cast<uintptr_t>(m.table) | static_cast<uint64_t>(m.stride)) & 15) == 0;
    // The table ends where the next one starts (tables laid out in order) or, failing that, where dev_weights ends.
    m.avail = 0x7fffffffffffffffll;
    if (p.dev_weights_bytes > 0) {
        const int64_t start = p.weights_offsets[t];
        int64_t end = p.dev_weights_bytes;
        if (t + 1 < p.T) {
            const int64_t next = p.weights_offsets[t + 1];
            if (next > start && next < end) end = next;
        }
        m.avail = end > start ? end - start : 0;
    }
    return m;
}

// ---- byte-wise path (any alignment, any D, every type) ----------------------

__device__ __forceinline__ float decode_elem(const uint8_t* row, int ty, int e, float scale, float bias,
                                             uint32_t fp8_shift, float fp8_mult)
{
    switch (ty) {
        case TBE_B200_INT8: return fmaf(static_cast<float>(row[4 + e]), scale, bias);
        case TBE_B200_INT4: return fmaf(static_cast<float>((row[4 + (e >> 1)] >> ((e & 1) * 4)) & 0xf), scale, bias);
        case TBE_B200_INT2: return fmaf(static_cast<float>((row[4 + (e >> 2)] >> ((e & 3) * 2)) & 0x3), scale, bias);
        case TBE_B200_FP8: {
            const uint32_t b = row[e];
            const float mag = __uint_as_float((b & 0x7fu) << fp8_shift) * fp8_mult;
            return __uint_as_float(__float_as_uint(mag) | ((b & 0x80u) << 24));
        }
        case TBE_B200_FP16: return half_bits_to_float(row[2 * e] | (static_cast<uint32_t>(row[2 * e + 1]) << 8));
        case TBE_B200_BF16:
            return __uint_as_float((row[2 * e] | (static_cast<uint32_t>(row[2 * e + 1]) << 8)) << 16);
        default: {
            const uint32_t u = row[4 * e] | (static_cast<uint32_t>(row[4 * e + 1]) << 8) |
                               (static_cast<uint32_t>(row[4 * e + 2]) << 16) | (static_cast<uint32_t>(row[4 * e + 3]) << 24);
            return __uint_as_float(u);
        }
    }
}

__device__ __forceinline__ void read_header(const uint8_t* row, int ty, float& scale, float& bias)
{
    scale = 1.0f;
    bias = 0.0f;
    if (ty == TBE_B200_INT8 || ty == TBE_B200_INT4 || ty == TBE_B200_INT2) {
        scale = half_bits_to_float(row[0] | (static_cast<uint32_t>(row[1]) << 8));
        bias = half_bits_to_float(row[2] | (static_cast<uint32_t>(row[3]) << 8));
    }
}

__device__ __forceinline__ void store_scalar(void* seg, int e, float v, int out_ty)
{
    if (out_ty == TBE_B200_FP32) static_cast<float*>(seg)[e] = v;
    else static_cast<unsigned short*>(seg)[e] =
        static_cast<unsigned short>(out_ty == TBE_B200_FP16 ? f32_to_f16_bits(v) : f32_to_bf16_bits(v));
}

constexpr int kByteAcc = 4;   // accumulators per lane in the byte-wise path

template <typename IdxT>
__device__ __noinline__ void pool_bag_bytewise(const IdxT* indices, const float* pw, int32_t* error_flag,
                                               const uint8_t* table, int64_t stride, int L, int D, void* seg,
                                               float mean_mul, int ty, int out_ty, uint32_t fp8_shift,
                                               float fp8_mult, int lane, int64_t avail)
{
    for (int e_blk = 0; e_blk < D; e_blk += kByteAcc * kWarp) {
        float acc[kByteAcc];
#pragma unroll
        for (int j = 0; j < kByteAcc; ++j) acc[j] = 0.0f;
        for (int n = 0; n < L; ++n) {
            const int64_t idx = static_cast<int64_t>(indices[n]);
            if (idx < 0) {
                if (idx < -1 && lane == 0 && error_flag && e_blk == 0) atomicOr(error_flag, 1);
                continue;
            }
            if (idx > 0x7fffffffll || static_cast<uint64_t>(idx + 1) * static_cast<uint64_t>(stride) > static_cast<uint64_t>(avail)) {
                if (lane == 0 && error_flag && e_blk == 0) atomicOr(error_flag, idx > 0x7fffffffll ? 1 : 4);
                continue;
            }
            const float w = pw ? pw[n] : 1.0f;
            const uint8_t* row = table + idx * stride;
            float scale, bias;
            read_header(row, ty, scale, bias);
#pragma unroll
            for (int j = 0; j < kByteAcc; ++j) {
                const int e = e_blk + j * kWarp + lane;
                if (e < D) acc[j] = fmaf(w, decode_elem(row, ty, e, scale, bias, fp8_shift, fp8_mult), acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < kByteAcc; ++j) {
            const int e = e_blk + j * kWarp + lane;
            if (e < D) store_scalar(seg, e, acc[j] * mean_mul, out_ty);
        }
    }
}

// ---- the common shapes: rows streamed through a shared-memory ring, groups of lanes -----------------

// Read-once streams (indices, per-sample weights): not kept in L1.
__device__ __forceinline__ int32_t ld_once32(const void* p) { return ld_stream(static_cast<const int32_t*>(p)); }
__device__ __forceinline__ float ld_once_f32(const void* p) { return ld_stream(static_cast<const float*>(p)); }
__device__ __forceinline__ uint2 ld_once_2x32(const void* p)
{
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ void sts16(uint32_t a, float x, float y, float z, float w)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t a, int32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ float4 lds16f(uint32_t a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int32_t lds4i(uint32_t a)
{
    int32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// Two packed fp32 numbers, and a + b on them.
__device__ __forceinline__ unsigned long long pack2(uint32_t lo, uint32_t hi)
{
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    return v;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b)
{
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
// a * b on them.
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b)
{
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
// c0 += a0 * b and c1 += a1 * b in one instruction.
__device__ __forceinline__ void fma2(float& c0, float& c1, unsigned long long a, float b)
{
    asm("{ .reg .b64 c, d; mov.b64 c, {%0, %1}; mov.b64 d, {%3, %3}; fma.rn.f32x2 c, %2, d, c; mov.b64 {%0, %1}, c; }"
        : "+f"(c0), "+f"(c1)
        : "l"(a), "f"(b));
}

// (a0 * b0 + c, a1 * b1 + c) in one instruction.
__device__ __forceinline__ float2 fma2_value(float a0, float a1, float b0, float b1, float c)
{
    float2 v;
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%6, %6}; fma.rn.f32x2 x, x, y, z; mov.b64 {%0, %1}, x; }"
        : "=f"(v.x), "=f"(v.y)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c));
    return v;
}

// Codes as fp32 numbers.  A code is used where it lies: masked out of its word and read as fp32 it is a subnormal
// (q * 2^8 * 2^-149 for the second byte), which is exact, and so is its product with the row's scale times kCodeScale; one
// packed FMA adds two of them with one rounding each, as a mixed FMA per code did, and what the place of a code
// multiplied is undone when the bag is stored (code_unit).  With per-sample weights scale * weight may have any magnitude, so
// the codes are made ordinary numbers first: a nibble that lies at bit k becomes 2^(23 - k) + q in the masking instruction, less
// 2^(23 - k) in half a packed addition (a byte 2^23 + q by a byte permute); the sums are then those of the codes themselves, and
// overflow where fp32 does.
// Against a byte permute and a mixed FMA per code, and with the row loop inlined (see the kernel): 64 INT8 tables of 128, batch
// 65536: 4.05 -> 3.38 ms; INT4 of 64/128/256, batch 16384: 1.73 -> 1.24 ms.
constexpr float kCodeScale = 0x1p111f;
template <int TY, bool WEIGHTED>
__device__ constexpr float code_unit(int slot)
{
    constexpr float kBase = 0x1p38f;                   // 1 / (2^-149 * kCodeScale)
    if (WEIGHTED) return 1.0f;
    if (TY == TBE_B200_INT8) return kBase * (slot % 4 == 1 ? 0x1p-8f : slot % 4 == 2 ? 0x1p-16f : 1.0f);
    if (TY == TBE_B200_INT4)
        return kBase * (slot % 8 == 1 || slot % 8 == 7 ? 0x1p-4f : slot % 8 == 2 ? 0x1p-8f : slot % 8 == 3 ? 0x1p-12f : slot % 8 == 4 ? 0x1p-16f
                        : slot % 8 == 5 ? 0x1p-20f : 1.0f);
    return 1.0f;
}

// The codes of a word, two at a time: where they lie, or, with per-sample weights, as the numbers they are.
// Nibbles at bits K and K + 4 (K at most 8 with weights).
template <bool WEIGHTED, int K>
__device__ __forceinline__ unsigned long long two_nibbles(uint32_t word)
{
    constexpr uint32_t kLo = 0xFu << K, kHi = 0xF0u << K;
    if constexpr (!WEIGHTED) return pack2(word & kLo, word & kHi);
    constexpr uint32_t kMagicLo = (150u - K) << 23, kMagicHi = (146u - K) << 23;      // 2^(23 - K) and 2^(19 - K)
    return add2(pack2((word & kLo) | kMagicLo, (word & kHi) | kMagicHi), pack2(kMagicLo | 0x80000000u, kMagicHi | 0x80000000u));
}
// Bytes J and J + 1.  With weights a byte permute each: 24 tables of 512 INT8, 3.1 M rows: 338 us, 404 with masks and a shift.
template <bool WEIGHTED, int J>
__device__ __forceinline__ unsigned long long two_bytes(uint32_t word)
{
    if constexpr (WEIGHTED)
        return add2(pack2(__byte_perm(word, 0x4B000000u, 0x7440u + J), __byte_perm(word, 0x4B000000u, 0x7441u + J)), pack2(0xCB000000u, 0xCB000000u));
    else if constexpr (J == 0) return pack2(word & 0xFFu, word & 0xFF00u);
    else return pack2(word & 0xFF0000u, word >> 24);
}

// Adds NW 32-bit words of INT8 (4 per word) or INT4 (8 per word) codes, times `s`, to consecutive slots of `acc`.
template <int TY, bool WEIGHTED, int NW>
__device__ __forceinline__ void accum_codes(const uint32_t (&words)[NW], float s, float* acc)
{
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t x = words[i], y = x >> 16;
        if constexpr (TY == TBE_B200_INT8) {
            fma2(acc[4 * i], acc[4 * i + 1], two_bytes<WEIGHTED, 0>(x), s);
            fma2(acc[4 * i + 2], acc[4 * i + 3], two_bytes<WEIGHTED, 2>(x), s);
        } else {
            fma2(acc[8 * i], acc[8 * i + 1], two_nibbles<WEIGHTED, 0>(x), s);
            fma2(acc[8 * i + 2], acc[8 * i + 3], two_nibbles<WEIGHTED, 8>(x), s);
            fma2(acc[8 * i + 4], acc[8 * i + 5], WEIGHTED ? two_nibbles<WEIGHTED, 0>(y) : two_nibbles<false, 16>(x), s);
            fma2(acc[8 * i + 6], acc[8 * i + 7], WEIGHTED ? two_nibbles<WEIGHTED, 8>(y) : two_nibbles<false, 0>(x >> 24), s);
        }
    }
}

// Adds NW 32-bit words of FP8 bytes, two bytes at a time as bf16: sign to the top, the rest to exponent and mantissa
// (reference: c310/op_kernel/common.h:120-167); a bf16 is the upper half of an fp32.  What is placed lacks a factor of
// fp8_mult, a power of two.  Unweighted sums get it at the bag's end (placed values are whole multiples of 2^-132 at least,
// so nothing is lost below the normal range).  A weight may have any magnitude: there the values get it before they
// meet the weight `w`.
// Against placing, scaling and signing every byte by itself, 24 tables, 3.1 M rows: 128 elements 200 -> 132 us, 256 elements with
// weights 364 -> 251 us.
template <bool WEIGHTED, int NW>
__device__ __forceinline__ void accum_fp8(const uint32_t (&words)[NW], uint32_t fp8_shift, float fp8_mult, float w, float* acc)
{
    const unsigned long long mult = pack2(__float_as_uint(fp8_mult), __float_as_uint(fp8_mult));
    auto two = [&](uint32_t a, uint32_t b) { return WEIGHTED ? mul2(pack2(a, b), mult) : pack2(a, b); };
    const uint32_t sh = fp8_shift - 16;                // exponent bits
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t x = words[i], y = x >> 8;
        const uint32_t even = ((x & 0x007F007Fu) << sh) | ((x & 0x00800080u) << 8), odd = ((y & 0x007F007Fu) << sh) | ((y & 0x00800080u) << 8);
        fma2(acc[4 * i], acc[4 * i + 1], two(even << 16, odd << 16), w);
        fma2(acc[4 * i + 2], acc[4 * i + 3], two(even & 0xffff0000u, odd & 0xffff0000u), w);
    }
}

// Output address of element 0 of bag `b` of the table at column `col`, when the result is scattered
// over per-destination buffers (bag b belongs to destination b / rows_per_dest).
__device__ __forceinline__ char* dest_segment(const LookupParams& p, int64_t b, int64_t col, int esz)
{
    int64_t which, rem;
    if (p.B32) {
        const uint32_t w = static_cast<uint32_t>(b) / static_cast<uint32_t>(p.rows_per_dest);
        which = w;
        rem = static_cast<uint32_t>(b) - w * static_cast<uint32_t>(p.rows_per_dest);
    } else {
        which = b / p.rows_per_dest;
        rem = b - which * p.rows_per_dest;
    }
    return static_cast<char*>(p.dests[which]) + (rem * p.out_stride + col) * esz;
}

// Shared memory of one warp in the streaming kernel: the partial sums that lane groups hand to one another
// (up to 32 floats per lane), the run's bag offsets, and the ring of rows in flight.
constexpr int kPartBytes = kWarp * 128;
constexpr int kMaxRunBags = 31;                        // bags of one run: their nb + 1 offsets are held one per lane
constexpr int kRelBytes = 128;                         // kMaxRunBags + 1 offsets
#ifndef TBE_RING_BYTES
#define TBE_RING_BYTES 4352                            // four stages of rows with up to 32 bytes per lane
#endif
#ifndef TBE_MAX_STAGES
#define TBE_MAX_STAGES 4
#endif
constexpr int kRingBytes = TBE_RING_BYTES;
constexpr int kStreamSmemBytes = kPartBytes + kRelBytes + kRingBytes;

__host__ __device__ constexpr int floor_pow2(int x) { return x >= 8 ? 8 : x >= 4 ? 4 : x >= 2 ? 2 : 1; }
__host__ __device__ constexpr int min3(int a, int b, int c) { return a < b ? (a < c ? a : c) : (b < c ? b : c); }

// A run of nb <= kMaxRunBags consecutive bags of ONE table whose rows are D = 16 * n <= 512 elements, 16-byte
// aligned.  Lane l <= nb brings the offset of bag l relative to the run's first row, R0, as `rel`.  LPR lanes share a row, 16 elements per lane, so a warp has G = 32 / LPR lane groups.
//
// Work split.  The run's rows -- positions [R0, R1) of `indices` -- are cut into G equal ranges, one per
// group, whatever the bag lengths are, so the groups finish together.  A group walks its range row by row
// and keeps the sum of the bag it is in; when the walk reaches the end of a bag the group stores the bag
// and starts the next one (a divergent branch, taken once per bag and group).  A bag that straddles a range
// boundary is summed in pieces: the group in whose range the bag STARTS owns it; every later group that holds
// a piece writes its partial sum to shared memory, and the owner adds those pieces at the end of the run.
// Empty bags are written (zeros) by the group whose walk passes their position.
//
// Row fetch.  Lane k of a group reads the index of the group's row c * LPR + k (chunk c of the range; the indices
// of a chunk are requested two chunks ahead).  Rows travel through a ring of NS stages in the warp's shared memory:
// in step q the group consumes row q - NS out of stage q mod NS and then requests row q into the same stage with
// asynchronous copies (cp.async through L1, 16 bytes per lane, completion counted per step with commit / wait
// groups), so NS rows per group are in flight all the time, whatever the compiler does with registers -- a ring of
// registers filled by ordinary loads measured twice as slow, because a warp has only six scoreboards and a row
// about to be consumed ended up waiting for loads that had just been issued.  A lane reads back only the bytes it
// copied itself, so no barrier is involved.  A row that is not to be added (index -1, out of range, past the end
// of the group's range) is zero-filled in the stage without being read.
template <int TY, int LPR, int EPL, bool WEIGHTED>
__device__ __forceinline__ void pool_run_stream(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b0, int lane,
                                             uint32_t wsm)
{
    static_assert(EPL == 16 || (EPL == 32 && (TY == TBE_B200_INT8 || TY == TBE_B200_INT4)), "32 elements per lane: INT8 / INT4 only");
    constexpr bool kHdr = (TY == TBE_B200_INT8 || TY == TBE_B200_INT4);
    constexpr bool k8 = (TY == TBE_B200_INT8);
    // A lane holds NCH chunks of CH bytes of a row; chunk c is unit k + c * nunits of the row (a unit = UE elements),
    // so one copy instruction of a group covers nunits * CH contiguous bytes.
    constexpr int NCH = (TY == TBE_B200_FP16) ? 2 : (TY == TBE_B200_FP32) ? 4 : (k8 ? EPL / 16 : 1);
    constexpr int CH = (TY == TBE_B200_INT4) ? EPL / 2 : 16;           // bytes per chunk
    constexpr int UE = EPL / NCH;                      // elements per unit
    constexpr int HS = k8 ? 4 : (TY == TBE_B200_INT4 ? 8 : 0);         // slots of the header lane that hold the row's tail
    constexpr int G = kWarp / LPR;                     // lane groups
    constexpr int LOG_G = G == 1 ? 0 : G == 2 ? 1 : G == 4 ? 2 : 3;
    constexpr int LANEB = CH * NCH;                                    // bytes of a row that one lane holds
    constexpr int STAGE = kWarp * LANEB + (kHdr ? 32 : 0);             // one row per group, and the groups' tail words
    constexpr int NS = floor_pow2(min3(kRingBytes / STAGE, LPR, TBE_MAX_STAGES));   // stages of the ring (rows in flight per group)
    static_assert(NS >= 1 && NS * STAGE <= kRingBytes, "the ring does not fit");
    static_assert(G <= 8, "at least 4 lanes per row");
    const int k = lane % LPR;
    const int g = lane / LPR;
    const unsigned gmask = (LPR == 32) ? kFull : (((1u << (LPR & 31)) - 1u) << (g * LPR));
    const int D = m.D;
    const int nunits = D / EPL;                        // lanes that hold a piece of the row
    const bool head_lane = kHdr && (k == 0);
    const bool act = k < nunits;                       // lanes past the row's last unit have nothing to add (D < EPL * LPR)
    const uint32_t stride = static_cast<uint32_t>(m.stride);
    const uint8_t* lane_base = m.table + k * CH;
    const uint32_t tail_off = k8 ? D : D / 2;          // header lane (k = 0): where the row's last HS elements are
    const uint32_t chunk_step = static_cast<uint32_t>(nunits) * CH;    // distance between a lane's chunks
    const bool idx64 = p.idx64 != 0;
    const int isz = idx64 ? 8 : 4;
    const uint32_t sm_rel = wsm + kPartBytes;

    const int n = __shfl_sync(kFull, rel, nb);
    __syncwarp();                                      // the previous run's reads of this memory are over
    if (lane <= nb) sts4(sm_rel + 4 * lane, rel);
    __syncwarp();

    // This group's range of rows, and the bag its first row is in.
    const int per = (n + G - 1) >> LOG_G;
    const int lo = min(n, g * per);
    const int hi = min(n, lo + per);
    int cur = 0;
    if constexpr (G > 1) {
#pragma unroll
        for (int gg = 1; gg < G; ++gg) {
            const int lo_gg = min(n, gg * per);
            const unsigned started = __ballot_sync(kFull, lane >= 1 && lane <= nb && rel <= lo_gg);
            if (g == gg) cur = __popc(started);
        }
    }
    const bool active = (g == 0) || (lo < hi);         // group 0 also writes the empty bags at the front of the run
    int bag_start = lds4i(sm_rel + 4 * cur);
    int bag_end = (active && cur < nb) ? lds4i(sm_rel + 4 * (cur + 1)) : -1;
    int pos = lo;

    // Element a slot stands for: slot s belongs to the lane's chunk s / UE, which is unit k + (s / UE) * nunits of the
    // row.  INT8 / INT4 units are shifted by the header (unit u covers elements [UE * u - HS, UE * u + UE - HS)), and
    // the header lane's first HS slots are the row's last HS elements.
    auto elem_of = [&](int slot) -> int {
        if (kHdr && head_lane && slot < HS) return D - HS + slot;
        return UE * (k + (slot / UE) * nunits) - HS + (slot % UE);
    };

    float acc[EPL];
#pragma unroll
    for (int s = 0; s < EPL; ++s) acc[s] = 0.0f;
    float bias_acc = 0.0f;

    char* const out0 = static_cast<char*>(p.output) + (b0 * p.out_stride + m.col) * ((p.out_ty == TBE_B200_FP32) ? 4 : 2);   // bag 0 of the run
    // Makes sums of elements of the sums of codes (or of placed FP8 bytes): what their place multiplied is undone and the
    // biases are added.  Done before a bag is stored and before a piece of one is handed over: the codes of a piece are
    // many times what is left of them beside their biases, and would round the other pieces' sums away.
    auto settle = [&]() {
        if constexpr (kHdr || (TY == TBE_B200_FP8 && !WEIGHTED)) {
#pragma unroll
            for (int s = 0; s < EPL; s += 2) {
                const float u0 = TY == TBE_B200_FP8 ? p.fp8_mult : code_unit<TY, WEIGHTED>(s);
                const float u1 = TY == TBE_B200_FP8 ? p.fp8_mult : code_unit<TY, WEIGHTED>(s + 1);
                const float2 v = fma2_value(acc[s], acc[s + 1], u0, u1, bias_acc);
                acc[s] = v.x;
                acc[s + 1] = v.y;
            }
        }
    };
    // Stores the settled bag `bag` of L rows (times 1/L for MEAN).  Executed by whole groups.
    auto store_bag = [&](int bag, int L) {
        if (p.pooling_mode == TBE_B200_POOL_MEAN && L > 0) {
            const float mm = 1.0f / static_cast<float>(L);
#pragma unroll
            for (int s = 0; s < EPL; s += 2) {
                const float2 v = fma2_value(acc[s], acc[s + 1], mm, mm, 0.0f);
                acc[s] = v.x;
                acc[s + 1] = v.y;
            }
        }
        // (computed here, once per bag, rather than kept in registers across the row loop)
        const int esz = (p.out_ty == TBE_B200_FP32) ? 4 : 2;
        char* seg = p.dests ? dest_segment(p, b0 + bag, m.col, esz) : out0 + static_cast<int64_t>(bag) * (p.out_stride * esz);
        const bool vec = (reinterpret_cast<uintptr_t>(seg) & 15) == 0;
        bool stored = false;
        if constexpr (k8) {
            // INT8 with a 16-bit output.  A unit's 16 elements start 4 elements before a 32-byte boundary.
            // Its first 4 go to the unit before it (unit 0's, the row's tail, to the last unit), after which every
            // unit is 16 elements from a 32-byte boundary on: two aligned 16-byte stores, whole sectors.  The unit after
            // lane k's chunk c is lane k + 1's chunk c, or, for the last lane, lane 0's NEXT chunk.  `vec` is the same
            // for all lanes of the group, so the group takes the shuffles together.
            if (vec && esz == 2) {
                uint32_t h[EPL / 2];
#pragma unroll
                for (int q = 0; q < EPL / 2; ++q) h[q] = pack_out(acc[2 * q], acc[2 * q + 1], p.out_ty);
                const int from = (k + 1 == nunits) ? 0 : k + 1;
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    const int cn = (c + 1) % NCH;
                    const uint32_t s0 = (k == 0) ? h[8 * cn] : h[8 * c];
                    const uint32_t s1 = (k == 0) ? h[8 * cn + 1] : h[8 * c + 1];
                    const uint32_t up0 = __shfl_sync(gmask, s0, from, LPR);
                    const uint32_t up1 = __shfl_sync(gmask, s1, from, LPR);
                    if (act) {
                        char* dst = seg + 32 * (k + c * nunits);
                        st_stream16(dst, make_uint4(h[8 * c + 2], h[8 * c + 3], h[8 * c + 4], h[8 * c + 5]));
                        st_stream16(dst + 16, make_uint4(h[8 * c + 6], h[8 * c + 7], up0, up1));
                    }
                }
                stored = true;
            }
        }
        if (!stored && act) {
#pragma unroll
            for (int q = 0; q < EPL / 4; ++q) store_out4(seg, elem_of(4 * q), &acc[4 * q], p.out_ty, vec);
        }
    };
    // Hands this group's settled piece of a bag that started in an earlier group's range to that bag's owner.
    auto write_partial = [&]() {
#pragma unroll
        for (int q = 0; q < EPL / 4; ++q)
            sts16(wsm + static_cast<uint32_t>(q * kWarp + lane) * 16u, acc[4 * q + 0], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
    };
    // Finishes every bag that ends at the group's position (the one being summed, then the empty ones after it).
    auto drain = [&]() {
        while (pos == bag_end) {
            settle();
            if (bag_start < lo) write_partial();
            else store_bag(cur, bag_end - bag_start);
#pragma unroll
            for (int s = 0; s < EPL; ++s) acc[s] = 0.0f;
            bias_acc = 0.0f;
            ++cur;
            bag_start = bag_end;
            bag_end = (cur < nb) ? lds4i(sm_rel + 4 * (cur + 1)) : -1;
        }
    };
    drain();

    // Index stream of the group: lane k reads the index (and weight) of row c * LPR + k of the range (chunk c).
    const char* ipb = static_cast<const char*>(p.indices) + (R0 + lo + k) * isz;
    const float* wpb = WEIGHTED ? p.pw + R0 + lo + k : nullptr;
    // The index is kept exactly as loaded (one or two 32-bit words; nothing is computed from it before `narrow` looks
    // at it two chunks later: even a sign extension right after the load would make the warp wait for the load).
    auto load_raw = [&](int c, uint2& raw, float& w) {
        raw = make_uint2(0xffffffffu, 0xffffffffu);
        w = 0.0f;
        if (lo + c * LPR + k < hi) {
            const char* ip = ipb + static_cast<int64_t>(c) * (LPR * isz);
            if (idx64) raw = ld_once_2x32(ip);
            else raw.x = static_cast<uint32_t>(ld_once32(ip));
            if constexpr (WEIGHTED) w = ld_once_f32(wpb + c * LPR);
        }
    };
    // Row number narrowed to 32 bits; -1 = nothing to add.  A row outside [-1, 2^31) or past the end of the
    // table is reported and skipped.  `max_rows` (once per run) folds both limits into one unsigned compare.
    const uint64_t rows_avail = static_cast<uint64_t>(m.avail) / stride;
    const uint64_t max_rows = rows_avail < 0x80000000ull ? rows_avail : 0x80000000ull;
    auto narrow = [&](uint2 words) -> int32_t {
        const int64_t raw = idx64 ? static_cast<int64_t>((static_cast<uint64_t>(words.y) << 32) | words.x)
                                  : static_cast<int64_t>(static_cast<int32_t>(words.x));
        if (static_cast<uint64_t>(raw) >= max_rows) {          // -1 and every other negative number included
            if (raw != -1 && p.error_flag) atomicOr(p.error_flag, (raw < 0 || raw > 0x7fffffffll) ? 1 : 4);
            return -1;
        }
        return static_cast<int32_t>(raw);
    };

    // The ring of rows in flight: stage s holds one row per group; a lane copies and reads back its own chunk(s)
    // only (chunk c of lane l at (c * 32 + l) * 16), the header lane also the group's tail word.
#ifdef TBE_L2_HINTS
    const uint64_t row_policy = l2_policy_evict_last();
#endif
    const uint32_t ring = wsm + kPartBytes + kRelBytes;
    const uint32_t my_main = ring + static_cast<uint32_t>(lane) * CH;   // chunk c of lane l at (c * 32 + l) * CH
    const uint32_t my_tail = ring + kWarp * LANEB + static_cast<uint32_t>(g) * 4u;
    // Requests row `idx` of the table into stage `st` (byte offset): asynchronous copies through L1, zero-filled
    // without reading for a row that is not to be added.
    auto request = [&](uint32_t st, int32_t idx) {
        const bool ok = act && idx >= 0;   // the lanes past the row's last unit zero-fill their slots as well
        const uint8_t* src = lane_base + static_cast<uint64_t>(static_cast<uint32_t>(max(idx, 0))) * stride;
        const int sz = ok ? CH : 0;
        if constexpr (CH == 8) {
            cp_async8(my_main + st, src, sz);
        } else {
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
#ifdef TBE_L2_HINTS
                cp_async16_ca_hint(my_main + st + c * (kWarp * 16), src + c * chunk_step, sz, row_policy);
#else
                cp_async16_ca(my_main + st + c * (kWarp * 16), src + c * chunk_step, sz);
#endif
            }
        }
        if constexpr (kHdr) {
            if (head_lane) cp_async4(my_tail + st, src + tail_off, ok ? 4 : 0);
        }
        cp_async_commit();
    };
    // Adds the row in stage `st`, with weight w.
    auto consume = [&](uint32_t st, float w) {
        constexpr int NW = LANEB / 4;      // 32-bit words of the row in this lane
        uint32_t r[NW];
        if constexpr (CH == 8) {
            const uint2 v = lds8(my_main + st);
            r[0] = v.x;
            r[1] = v.y;
        } else {
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const uint4 v = lds16(my_main + st + c * (kWarp * 16));
                r[4 * c + 0] = v.x;
                r[4 * c + 1] = v.y;
                r[4 * c + 2] = v.z;
                r[4 * c + 3] = v.w;
            }
        }
        if constexpr (kHdr) {
            const uint32_t hdr = __shfl_sync(kFull, r[0], 0, LPR);   // zero for a row that was not copied
            if (head_lane) r[0] = lds4(my_tail + st);                // the header lane's first HS slots: the row's tail
            // the header: fp16 scale, fp16 bias
            const float sc = half_bits_to_float(hdr & 0xffffu), bi = half_bits_to_float(hdr >> 16);
            bias_acc = WEIGHTED ? fmaf(bi, w, bias_acc) : bias_acc + bi;
            accum_codes<TY, WEIGHTED, NW>(r, WEIGHTED ? sc * w : sc * kCodeScale, acc);
        } else if constexpr (TY == TBE_B200_FP8) {
            accum_fp8<WEIGHTED, NW>(r, p.fp8_shift, p.fp8_mult, w, acc);
        } else if constexpr (TY == TBE_B200_FP16 && !WEIGHTED) {
            // value * 1.0 + acc in one mixed FMA
#pragma unroll
            for (int i8 = 0; i8 < 8; ++i8) add_pair(acc[2 * i8], acc[2 * i8 + 1], r[i8], 0x3c00u);
        } else if constexpr (TY == TBE_B200_FP16) {
#pragma unroll
            for (int i8 = 0; i8 < 8; ++i8) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r[i8]));
                fma2(acc[2 * i8], acc[2 * i8 + 1], pack2(__float_as_uint(f.x), __float_as_uint(f.y)), w);
            }
        } else {
#pragma unroll
            for (int s = 0; s < 8; ++s) fma2(acc[2 * s], acc[2 * s + 1], pack2(r[2 * s], r[2 * s + 1]), w);
        }
    };

    // Step q requests row q of the range and consumes row q - NS (copied NS steps ago into the same stage), so NS rows
    // per group are in flight; rows per .. per + NS - 1 do not exist and only drain the ring.  The step loop is kept
    // rolled on purpose: unrolled over the stages (constant stage addresses, one copy of the end-of-bag code per stage)
    // it measured 5-10 % slower, and twice as slow with eight stages -- the loop no longer fits the instruction cache.
    const int total = per + NS;
    uint2 raw_a, raw_b;                    // the indices of the next chunk and of the one after it, as loaded
    float w_a = 0.0f, w_b = 0.0f;
    int32_t idx_c;                         // lane k: index of row c * LPR + k of the chunk being requested
    float w_c = 0.0f, w_prev = 0.0f;       // weights of the chunk being requested / of the one before it
    {
        uint2 raw0;
        load_raw(0, raw0, w_c);
        load_raw(1, raw_a, w_a);
        load_raw(2, raw_b, w_b);
        idx_c = narrow(raw0);
        if (idx_c < 0) w_c = 0.0f;
    }
    int q = 0;
#pragma unroll 1
    for (int c = 0; q < total; ++c) {
        if (c > 0) {
            w_prev = w_c;
            idx_c = narrow(raw_a);
            w_c = (idx_c >= 0) ? w_a : 0.0f;
            raw_a = raw_b;
            w_a = w_b;
            load_raw(c + 2, raw_b, w_b);
        }
        const int u_end = min(LPR, total - q);
#pragma unroll 1
        for (int u = 0; u < u_end; ++u, ++q) {
            const uint32_t st = static_cast<uint32_t>(q & (NS - 1)) * STAGE;
            if (q >= NS) {
                float w = 1.0f;
                if constexpr (WEIGHTED) w = __shfl_sync(kFull, u >= NS ? w_c : w_prev, (u - NS) & (LPR - 1), LPR);
                cp_async_wait<NS - 1>();
                consume(st, w);
                pos = min(pos + 1, hi);
                if (pos == bag_end) drain();
            }
            request(st, __shfl_sync(kFull, idx_c, u, LPR));
        }
    }
    cp_async_wait<0>();                    // nothing of this run is still on its way when the ring is handed on

    // A bag that the range ended in the middle of: a piece for its owner, or, when it started in this range, the
    // owner's own piece, completed with the pieces of the groups after it.
    const bool open = active && bag_end >= 0 && bag_start < pos && pos < bag_end;
    if (open) {
        settle();
        if (bag_start < lo) write_partial();
    }
    __syncwarp();
    if (open && bag_start >= lo) {
        for (int gg = g + 1; gg < G && gg * per < bag_end; ++gg) {
#pragma unroll
            for (int q = 0; q < EPL / 4; ++q) {
                const float4 v = lds16f(wsm + static_cast<uint32_t>(q * kWarp + gg * LPR + k) * 16u);
                acc[4 * q + 0] += v.x;
                acc[4 * q + 1] += v.y;
                acc[4 * q + 2] += v.z;
                acc[4 * q + 3] += v.w;
            }
        }
        store_bag(cur, bag_end - bag_start);
    }
}

template <int TY, bool WEIGHTED>
__device__ __forceinline__ void pool_run_stream_by_width(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b,
                                                         int lane, uint32_t wsm)
{
    // INT8 / INT4 rows of 128 elements or more that divide into 32-element pieces: 32 elements per lane, so that twice
    // as many bags share a warp and the per-row work that does not depend on the width is shared twice as widely.
    if constexpr (TY == TBE_B200_INT8 || TY == TBE_B200_INT4) {
        if (m.D >= 128 && (m.D & 31) == 0) {
            const int n32 = m.D / 32;
            if (n32 <= 4) pool_run_stream<TY, 4, 32, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
            else if (n32 <= 8) pool_run_stream<TY, 8, 32, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
            else pool_run_stream<TY, 16, 32, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
            return;
        }
    }
    const int nunits = m.D / 16;
    if (nunits <= 4) pool_run_stream<TY, 4, 16, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
    else if (nunits <= 8) pool_run_stream<TY, 8, 16, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
    else if (nunits <= 16) pool_run_stream<TY, 16, 16, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
    else pool_run_stream<TY, 32, 16, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
}

template <bool WEIGHTED>
__device__ __forceinline__ void pool_run_stream_by_type(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b,
                                                        int lane, uint32_t wsm)
{
    switch (m.ty) {
        case TBE_B200_INT8:
            pool_run_stream_by_width<TBE_B200_INT8, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
            return;
        case TBE_B200_INT4: pool_run_stream_by_width<TBE_B200_INT4, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm); return;
        case TBE_B200_FP8: pool_run_stream_by_width<TBE_B200_FP8, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm); return;
        case TBE_B200_FP16: pool_run_stream_by_width<TBE_B200_FP16, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm); return;
        default: pool_run_stream_by_width<TBE_B200_FP32, WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm); return;
    }
}


// ---- bags summed in steps of eight rows -----------------------------------------------------------------
//
// A warp takes its run's bags in order, a bag in steps of up to eight rows.  Lane 8 j + g owns unit g (and g + 8) of rows
// j and j + 4 of the step, so a unit is summed by four lanes, each over its quarter of the bag's rows, and what is left
// of a bag at its end is one exchange through shared memory: every lane takes one quad of elements from the four
// that have summed it and stores it, 32 lanes one contiguous piece.  All of that is warp-uniform and runs once per bag, where
// pool_run_stream runs its end of a bag once per bag AND lane group.  No row of another bag shares a step, so
// nothing is masked: a step's missing rows are zero-filled.
//
// Row fetch.  Rows travel through a ring of NS stages in the warp's shared memory with asynchronous copies through L1, each
// lane copying and reading back only its own bytes.  CB bytes per lane and row: 4, 8, 16 or 32, so that narrow rows keep
// all lanes busy and one pass covers up to 256 bytes (INT4: 128); wider rows take several passes over the run, each
// over its own columns.  Any D that is a multiple of 4 will do: a row's last unit may reach into the row's padding,
// whose sums are not stored.

// Asynchronous 4-byte copy by the lanes that `on` selects, predicated instead of branched around.
__device__ __forceinline__ void cp_async4_if(bool on, uint32_t dst, const void* src, int bytes)
{
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %3, 0; @p cp.async.ca.shared.global [%0], [%1], 4, %2; }" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(static_cast<int>(on))
                 : "memory");
}

constexpr int kIndexRing = 128;                        // rows whose numbers (and weights) are at hand: a power of two above what is in flight

template <int TY, int CB, bool WEIGHTED>
__device__ __noinline__ void pool_run_steps(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b0, int lane, uint32_t wsm)
{
    static_assert(CB == 4 || CB == 8 || CB == 16 || (CB == 32 && TY != TBE_B200_INT4), "at most 32 elements per lane and pass");
    constexpr bool k8 = (TY == TBE_B200_INT8), k4 = (TY == TBE_B200_INT4), k16 = (TY == TBE_B200_FP16), kF8 = (TY == TBE_B200_FP8),
                   k32 = (TY == TBE_B200_FP32);
    constexpr bool kHdr = k8 || k4;
    static_assert((!k16 || CB >= 8) && (!k32 || CB >= 16), "four elements at least");
    constexpr int EPW = k4 ? 8 : k16 ? 2 : k32 ? 1 : 4;   // elements of a 32-bit word of the row
    constexpr int HS = kHdr ? EPW : 0;                    // element slots of the first unit that the header takes
    constexpr int NCH = (CB == 32) ? 2 : 1;               // units per lane and pass
    constexpr int CHB = CB / NCH;                         // bytes of a unit: one asynchronous copy
    constexpr int WPU = CHB / 4;                          // 32-bit words of a unit
    constexpr int NW = CB / 4;                            // words per lane and row
    constexpr int NQ = NW * EPW / 4;                      // quads: four elements each
    constexpr int EPU = WPU * EPW;                        // elements of a unit
    constexpr int HALF = kWarp * CB;                      // four rows of a stage
    constexpr int STAGE = 2 * HALF + 32;                  // eight rows and their side words
    constexpr int XQ = NQ < 4 ? NQ : 4;                   // quads exchanged at a time
    constexpr int XROW = 32 + 8 / XQ;                     // (so that eight lanes' reads fall on different banks)
    constexpr int XCHG = XQ * XROW * 16;
    constexpr int RING = kStreamSmemBytes - kRelBytes - 2 * kIndexRing * 4 - XCHG;
    constexpr int NS = RING / STAGE < 6 ? RING / STAGE : 6;   // stages: steps in flight
    static_assert(NS >= 2 && NS * 8 + 2 * kWarp + 8 <= kIndexRing, "the rings do not fit");
    const int j = lane >> 3, g = lane & 7;             // row of the step, unit: a copy instruction covers whole pieces of four rows
    const int D = m.D;
    const uint32_t stride = static_cast<uint32_t>(m.stride);
    const int payload = k32 ? 4 * D : k16 ? 2 * D : k4 ? D / 2 : D;     // bytes
    // A row that is a whole number of units without its header: the header's place in the first unit takes the row's last
    // four bytes (the side word), so that no unit is spent on them.
    const bool wrap = kHdr && payload % CHB == 0;
    const int units = wrap ? payload / CHB : (payload + (kHdr ? 4 : 0) + CHB - 1) / CHB;
    const bool idx64 = p.idx64 != 0;
    const int isz = idx64 ? 8 : 4;
    const uint32_t sm_rel = wsm, sm_idx = wsm + kRelBytes, sm_w = sm_idx + kIndexRing * 4, sm_x = sm_w + kIndexRing * 4, ring = sm_x + XCHG;

    const int n = __shfl_sync(kFull, rel, nb);
    __syncwarp();                                      // the previous run's reads of this memory are over
    if (lane <= nb) sts4(sm_rel + 4 * lane, rel);
    const int next_rel = __shfl_down_sync(kFull, rel, 1);
    const int total_steps = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(lane < nb ? (next_rel - rel + 7) >> 3 : 0)));
    __syncwarp();

    const char* ipb = static_cast<const char*>(p.indices) + (R0 + lane) * isz;
    const float* wpb = WEIGHTED ? p.pw + R0 + lane : nullptr;
    const uint64_t rows_avail = static_cast<uint64_t>(m.avail) / stride;
    const uint64_t max_rows = rows_avail < 0x80000000ull ? rows_avail : 0x80000000ull;
    const int esz = (p.out_ty == TBE_B200_FP32) ? 4 : 2;
    const float unit_base = kF8 && !WEIGHTED ? p.fp8_mult : 1.0f;

    for (int u0 = 0; u0 < units; u0 += 8 * NCH) {
        const bool first_pass = (u0 == 0);
        // The side word (lanes 0, 8, 16 and 24, one per row): the row's tail in the first pass of a wrapped row, the header in later ones.
        const bool side_lane = kHdr && g == 0 && (wrap || !first_pass);
        const uint8_t* lane_base = m.table + (u0 + g) * CHB;
        const uint8_t* side_base = m.table + (first_pass ? payload : 0);
        const int size0 = u0 + g < units ? CHB : 0, size1 = u0 + g + 8 < units ? CHB : 0;

        float acc[4 * NQ];
#pragma unroll
        for (int i = 0; i < 4 * NQ; ++i) acc[i] = 0.0f;
        float bias_acc = 0.0f;

        // Indices are loaded 32 at a time, two chunks ahead, kept as loaded until their chunk's turn (anything computed from
        // them earlier would wait for the load), then narrowed and put into the ring.  -1 = nothing to add; a row outside
        // [-1, 2^31) or past the end of the table is reported and skipped.
        uint2 raw_a, raw_b;
        float w_a = 0.0f, w_b = 0.0f;
        auto load_raw = [&](int c, uint2& raw, float& w) {
            raw = make_uint2(0xffffffffu, 0xffffffffu);
            if (c * kWarp + lane < n) {
                const char* ip = ipb + static_cast<int64_t>(c) * (kWarp * isz);
                if (idx64) raw = ld_once_2x32(ip);
                else raw.x = static_cast<uint32_t>(ld_once32(ip));
                if constexpr (WEIGHTED) w = ld_once_f32(wpb + c * kWarp);
            }
        };
        auto put_chunk = [&](int c, uint2 words, float w) {
            const int64_t raw = idx64 ? static_cast<int64_t>((static_cast<uint64_t>(words.y) << 32) | words.x)
                                      : static_cast<int64_t>(static_cast<int32_t>(words.x));
            int32_t idx = static_cast<int32_t>(raw);
            if (static_cast<uint64_t>(raw) >= max_rows) {          // -1 and every other negative number included
                if (raw != -1 && p.error_flag) atomicOr(p.error_flag, (raw < 0 || raw > 0x7fffffffll) ? 1 : 4);
                idx = -1;
            }
            const uint32_t at = static_cast<uint32_t>((c * kWarp + lane) & (kIndexRing - 1)) * 4u;
            sts4(sm_idx + at, idx);
            if constexpr (WEIGHTED) sts4(sm_w + at, __float_as_int(idx >= 0 ? w : 0.0f));
            __syncwarp();
        };

        const uint32_t my_main = ring + static_cast<uint32_t>(lane) * CHB;
        const uint32_t my_side = ring + 2 * HALF + static_cast<uint32_t>(j) * 4u;
        // Requests this lane's bytes of row `idx` into half h of the stage; a row that is not to be added is zero-filled.
        auto request_row = [&](uint32_t st, int h, int32_t idx) {
            const uint64_t at = static_cast<uint64_t>(static_cast<uint32_t>(max(idx, 0))) * stride;
            const uint32_t dst = my_main + st + h * HALF;
            // (lanes past the row's last unit zero-fill as well: no branch)
            if constexpr (CHB == 4) cp_async4(dst, lane_base + at, idx >= 0 ? size0 : 0);
            else if constexpr (CHB == 8) cp_async8(dst, lane_base + at, idx >= 0 ? size0 : 0);
            else cp_async16_ca(dst, lane_base + at, idx >= 0 ? size0 : 0);
            if constexpr (NCH == 2) cp_async16_ca(dst + kWarp * 16, lane_base + at + 128, idx >= 0 ? size1 : 0);
            if constexpr (kHdr) cp_async4_if(side_lane, my_side + st + h * 16, side_base + at, idx >= 0 ? 4 : 0);
        };

        // Adds this lane's words of one row.  `hdr` is the row's header, w its weight.
        auto add_row = [&](const uint32_t (&r)[NW], uint32_t hdr, float w) {
            if constexpr (kHdr) {
                const float sc = half_bits_to_float(hdr & 0xffffu), bi = half_bits_to_float(hdr >> 16);
                bias_acc = WEIGHTED ? fmaf(bi, w, bias_acc) : bias_acc + bi;
                accum_codes<TY, WEIGHTED, NW>(r, WEIGHTED ? sc * w : sc * kCodeScale, acc);
            } else if constexpr (kF8) {
                accum_fp8<WEIGHTED, NW>(r, p.fp8_shift, p.fp8_mult, w, acc);
            } else if constexpr (k32) {
#pragma unroll
                for (int i = 0; i < NW / 2; ++i) fma2(acc[2 * i], acc[2 * i + 1], pack2(r[2 * i], r[2 * i + 1]), w);
            } else {
#pragma unroll
                for (int i = 0; i < NW; ++i) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r[i]));
                    fma2(acc[2 * i], acc[2 * i + 1], pack2(__float_as_uint(f.x), __float_as_uint(f.y)), w);
                }
            }
        };

        // Adds the (up to) eight rows in stage `st`, rows pos .. min(pos + 8, end) - 1 of the run.
        auto consume = [&](uint32_t st, int pos, int end) {
            uint32_t r[2][NW];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t src = my_main + st + h * HALF;
                if constexpr (CHB == 4) {
                    r[h][0] = lds4(src);
                } else if constexpr (CHB == 8) {
                    const uint2 v = lds8(src);
                    r[h][0] = v.x;
                    r[h][1] = v.y;
                } else {
#pragma unroll
                    for (int c = 0; c < NCH; ++c) {
                        const uint4 v = lds16(src + c * (kWarp * 16));
                        r[h][4 * c + 0] = v.x;
                        r[h][4 * c + 1] = v.y;
                        r[h][4 * c + 2] = v.z;
                        r[h][4 * c + 3] = v.w;
                    }
                }
            }
            uint32_t hdr[2] = {0u, 0u};
            if constexpr (kHdr) {
                uint32_t word[2] = {r[0][0], r[1][0]};
                // read by every lane (no branch); the tails take the headers' places in a wrapped row's first pass
                const uint32_t s0 = lds4(my_side + st), s1 = lds4(my_side + st + 16);
                if (side_lane) {
                    word[0] = first_pass ? word[0] : s0;
                    word[1] = first_pass ? word[1] : s1;
                    r[0][0] = first_pass ? s0 : r[0][0];
                    r[1][0] = first_pass ? s1 : r[1][0];
                }
                hdr[0] = __shfl_sync(kFull, word[0], lane & 24);   // from the lane of unit 0; zero for a row that was not copied
                hdr[1] = __shfl_sync(kFull, word[1], lane & 24);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float w = 1.0f;
                if constexpr (WEIGHTED) {
                    const int at = pos + 4 * h + j;
                    w = __int_as_float(lds4i(sm_w + static_cast<uint32_t>(at & (kIndexRing - 1)) * 4u));
                    w = at < end ? w : 0.0f;                       // (what is found past the bag's end belongs to another bag)
                }
                add_row(r[h], hdr[h], w);
            }
        };

        // Stores bag `bag` of L rows, and clears the sums.
        auto finish_bag = [&](int bag, int L) {
            bias_acc += __shfl_xor_sync(kFull, bias_acc, 8);
            bias_acc += __shfl_xor_sync(kFull, bias_acc, 16);
            const float mm = (p.pooling_mode == TBE_B200_POOL_MEAN && L > 0) ? 1.0f / static_cast<float>(L) : 1.0f;
            char* seg = p.dests ? dest_segment(p, b0 + bag, m.col, esz) : static_cast<char*>(p.output) + ((b0 + bag) * p.out_stride + m.col) * esz;
            const bool vec = (reinterpret_cast<uintptr_t>(seg) & (4 * esz - 1)) == 0;     // element positions are multiples of 4
#pragma unroll
            for (int x0 = 0; x0 < NQ; x0 += XQ) {
                __syncwarp();                          // the previous exchange has been read
#pragma unroll
                for (int i = 0; i < XQ; ++i)
                    sts16(sm_x + static_cast<uint32_t>(i * XROW + lane) * 16u, acc[4 * (x0 + i)], acc[4 * (x0 + i) + 1], acc[4 * (x0 + i) + 2], acc[4 * (x0 + i) + 3]);
                __syncwarp();
                const int xu = lane / XQ, q = x0 + lane % XQ;     // the unit (of eight) and the quad this lane finishes
                if (xu < 8) {
                    const uint32_t from = sm_x + static_cast<uint32_t>((lane % XQ) * XROW + xu) * 16u;
                    const float4 a = lds16f(from), b = lds16f(from + 128), c = lds16f(from + 256), d = lds16f(from + 384);
                    // what a code's place in its word multiplied
                    const bool upper = k4 && (q & 1);  // nibbles 4 .. 7 of the word
                    const float m0 = unit_base * (upper ? code_unit<TY, WEIGHTED>(4) : code_unit<TY, WEIGHTED>(0));
                    const float m1 = unit_base * (upper ? code_unit<TY, WEIGHTED>(5) : code_unit<TY, WEIGHTED>(1));
                    const float m2 = unit_base * (upper ? code_unit<TY, WEIGHTED>(6) : code_unit<TY, WEIGHTED>(2));
                    const float m3 = unit_base * (upper ? code_unit<TY, WEIGHTED>(7) : code_unit<TY, WEIGHTED>(3));
                    // the mean is taken of the finished sum: codes and biases that cancel do so before anything is rounded
                    const float v[4] = {fmaf((a.x + b.x) + (c.x + d.x), m0, bias_acc) * mm, fmaf((a.y + b.y) + (c.y + d.y), m1, bias_acc) * mm,
                                        fmaf((a.z + b.z) + (c.z + d.z), m2, bias_acc) * mm, fmaf((a.w + b.w) + (c.w + d.w), m3, bias_acc) * mm};
                    constexpr int QPU = EPU / 4;       // quads of a unit
                    const int unit = u0 + xu + 8 * (q / QPU);
                    int e0 = EPU * unit - HS + 4 * (q % QPU);
                    if (kHdr && unit == 0 && q % QPU < HS / 4) e0 = wrap ? D - HS + 4 * q : -1;
                    if (unit < units && e0 >= 0 && e0 < D) store_out4(seg, e0, v, p.out_ty, vec);
                }
            }
#pragma unroll
            for (int i = 0; i < 4 * NQ; ++i) acc[i] = 0.0f;
            bias_acc = 0.0f;
        };

        load_raw(0, raw_a, w_a);
        load_raw(1, raw_b, w_b);
        int chunks = 0;                                // chunks in the index ring
        // the walk of the requests, and that of the sums NS steps behind it: bag, next row, end of the bag
        int r_bag = 0, r_pos = 0, r_end = lds4i(sm_rel + 4);
        int c_bag = 0, c_pos = 0, c_end = r_end;
        uint32_t st = 0;
#pragma unroll 1
        for (int q = 0; q < total_steps + NS; ++q) {
            if (q >= NS) {
                while (c_pos == c_end) {               // empty bags
                    finish_bag(c_bag, 0);
                    c_end = lds4i(sm_rel + 4 * (++c_bag + 1));
                }
                cp_async_wait<NS - 1>();
                consume(st, c_pos, c_end);
                c_pos = min(c_pos + 8, c_end);
                if (c_pos == c_end) {
                    finish_bag(c_bag, c_end - lds4i(sm_rel + 4 * c_bag));
                    ++c_bag;
                    c_end = c_bag < nb ? lds4i(sm_rel + 4 * (c_bag + 1)) : -1;
                }
            }
            if (q < total_steps) {
                while (r_pos == r_end) r_end = lds4i(sm_rel + 4 * (++r_bag + 1));
                while (chunks * kWarp < min(r_pos + 8, n)) {
                    put_chunk(chunks, raw_a, w_a);
                    raw_a = raw_b;
                    w_a = w_b;
                    ++chunks;
                    load_raw(chunks + 1, raw_b, w_b);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int at = r_pos + 4 * h + j;
                    int32_t idx = lds4i(sm_idx + static_cast<uint32_t>(at & (kIndexRing - 1)) * 4u);
                    idx = at < r_end ? idx : -1;
                    request_row(st, h, idx);
                }
                r_pos = min(r_pos + 8, r_end);
            }
            cp_async_commit();
            st = (st + STAGE == NS * STAGE) ? 0u : st + STAGE;
        }
        cp_async_wait<0>();                            // nothing of this pass is still on its way when the ring is handed on
        while (c_bag < nb) finish_bag(c_bag++, 0);     // empty bags at the end
        __syncwarp();
    }
}

template <int TY, bool WEIGHTED>
__device__ __forceinline__ void pool_run_steps_by_width(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b0, int lane,
                                                        uint32_t wsm)
{
    // The narrowest unit with which eight lanes cover the row, so that narrow rows keep all of them busy.
    constexpr int kHead = (TY == TBE_B200_INT8 || TY == TBE_B200_INT4) ? 4 : 0;
    const int bytes = TY == TBE_B200_FP32 ? 4 * m.D : TY == TBE_B200_FP16 ? 2 * m.D : TY == TBE_B200_INT4 ? m.D / 2 : m.D;
    auto covers = [&](int unit) { return bytes <= 8 * unit && (bytes % unit == 0 || bytes + kHead <= 8 * unit); };
    if constexpr (kHead != 0 || TY == TBE_B200_FP8) {
        if (covers(4)) { pool_run_steps<TY, 4, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return; }
    }
    if constexpr (TY != TBE_B200_FP32) {
        if (covers(8)) { pool_run_steps<TY, 8, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return; }
    }
    if constexpr (TY == TBE_B200_INT4) {
        pool_run_steps<TY, 16, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm);
    } else {
        if (covers(16)) pool_run_steps<TY, 16, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm);
        else pool_run_steps<TY, 32, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm);
    }
}

template <bool WEIGHTED>
__device__ __forceinline__ void pool_run_steps_by_type(const LookupParams& p, const TableMeta& m, int64_t R0, int rel, int nb, int64_t b0, int lane,
                                                       uint32_t wsm)
{
    switch (m.ty) {
        case TBE_B200_INT8: pool_run_steps_by_width<TBE_B200_INT8, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return;
        case TBE_B200_INT4: pool_run_steps_by_width<TBE_B200_INT4, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return;
        case TBE_B200_FP8: pool_run_steps_by_width<TBE_B200_FP8, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return;
        case TBE_B200_FP16: pool_run_steps_by_width<TBE_B200_FP16, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return;
        default: pool_run_steps_by_width<TBE_B200_FP32, WEIGHTED>(p, m, R0, rel, nb, b0, lane, wsm); return;
    }
}

// A run of bags of one table through the byte-wise code.
template <typename IdxT>
__device__ __noinline__ void pool_run_bytewise(const LookupParams& p, const TableMeta& m, int64_t i0, int nb, int64_t b, int lane)
{
    const IdxT* offsets = static_cast<const IdxT*>(p.offsets) + i0;
    const IdxT* indices = static_cast<const IdxT*>(p.indices);
    const int esz = (p.out_ty == TBE_B200_FP32) ? 4 : 2;
    int64_t start = static_cast<int64_t>(offsets[0]);
    for (int i = 0; i < nb; ++i, ++b) {
        const int64_t end = static_cast<int64_t>(offsets[i + 1]);
        const int L = static_cast<int>(end - start);
        const float mean_mul = (p.pooling_mode == TBE_B200_POOL_MEAN && L > 0) ? 1.0f / static_cast<float>(L) : 1.0f;
        char* seg = p.dests ? dest_segment(p, b, m.col, esz) : static_cast<char*>(p.output) + (b * p.out_stride + m.col) * esz;
        // positions outside `indices` are not read: the bag is written as if it were empty, and reported
        const bool sane = L >= 0 && start >= 0 && end <= p.num_indices;
        if (!sane && lane == 0 && p.error_flag) atomicOr(p.error_flag, 8);
        pool_bag_bytewise<IdxT>(indices + start, p.pw ? p.pw + start : nullptr, p.error_flag, m.table, m.stride, sane ? L : 0, m.D, seg, mean_mul,
                                m.ty, p.out_ty, p.fp8_shift, p.fp8_mult, lane, m.avail);
        start = end;
    }
}

// ---- kernels -----------------------------------------------------------------

// Warps per block.  With 8 (two blocks per SM) or 16 (one) the warps of an SM work on fewer tables at a time, which
// helps launches whose tables differ in type or width (their loops compete for the instruction cache): measured
// +4.5 % / +2.7 % on benchmark configuration 3 and +1.6 % / +0.4 % on configuration 5, but -0.9 % / -4.6 % on the
// single-shape configuration 4 (a finished block leaves its SM emptier for longer), so 4 it is.
#ifndef TBE_WARPS_PER_BLOCK
#define TBE_WARPS_PER_BLOCK 4
#endif
constexpr int kWarpsPerBlock = TBE_WARPS_PER_BLOCK;
#ifndef TBE_SPAN_LARGE
#define TBE_SPAN_LARGE 31
#endif
#ifndef TBE_STREAM_BLOCKS_PER_SM
#define TBE_STREAM_BLOCKS_PER_SM (16 / TBE_WARPS_PER_BLOCK)   // 16 resident warps per SM at up to 128 registers (32 accumulators per lane); measured best
#endif
constexpr int kStreamBlocksPerSM = TBE_STREAM_BLOCKS_PER_SM;

// The T*B bags (bag i = t*B + b) are cut into spans of `span` consecutive bags, one span per warp, so a
// warp walks `offsets`, `indices` and the per-sample weights front to back.  A span is processed as runs
// of consecutive bags of one table: the table's description is read once per run and the run is handed
// to the code specialised for its row shape.  pool_run_stream is inlined here (in a function of its own every memory
// instruction has its descriptor moved into uniform registers again and the arguments are read through a pointer); what a run
// does not need is not kept across it but computed anew behind it, which leaves the row loop without spills (with them the
// loop is slower than the function was).  What this and the arithmetic at kCodeScale gave together stands there.
template <bool WEIGHTED>
__global__ void __launch_bounds__(kWarpsPerBlock* kWarp, kStreamBlocksPerSM) tbe_pooled_kernel(const __grid_constant__ LookupParams p)
{
    extern __shared__ __align__(128) uint8_t smem[];      // kWarpsPerBlock * kStreamSmemBytes bytes, given at launch
    int lane = threadIdx.x & 31;
    uint32_t wsm = smem_u32(smem) + (threadIdx.x >> 5) * kStreamSmemBytes;
    // Kept in registers: made from the thread's number again and again inside the loops otherwise (179 instructions per step of
    // eight 128-byte rows; 64 INT8 tables of 128, batch 8192: 499 us, 441 us this way; INT4 of 64/128/256, batch 4096: 409, 360).
    asm volatile("" : "+r"(lane), "+r"(wsm));
    {
        const int64_t gw = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
        const int64_t lo = gw * p.span;
        if (lo >= p.num_bags) return;
        // The span's first offsets are needed right after the table description: ask for their line(s) now, so the two
        // latencies overlap.
        if (lane < 2) {
            const char* o = static_cast<const char*>(p.offsets) + (lane == 0 ? lo : min(p.num_bags, lo + p.span)) * (p.idx64 ? 8 : 4);
            asm volatile("prefetch.global.L1 [%0];" ::"l"(o));
        }
        // The last offset has to be the number of indices (the reference kernel asserts the same:
        // c310/op_kernel/int_nbit_split_embedding_pooling_kernel.h:149-150); here it is reported, not trapped.
        if (gw == 0 && lane == 0 && p.error_flag) {
            const int64_t last = p.idx64 ? static_cast<const int64_t*>(p.offsets)[p.num_bags]
                                         : static_cast<int64_t>(static_cast<const int32_t*>(p.offsets)[p.num_bags]);
            if (last != p.num_indices) atomicOr(p.error_flag, 8);
        }
    }

#pragma unroll 1
    for (int done = 0; done < p.span;) {
        uint32_t block;                                    // (read anew for every run)
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block));
        const int64_t i = (static_cast<int64_t>(block) * kWarpsPerBlock + (threadIdx.x >> 5)) * p.span + done;
        if (i >= p.num_bags) break;
        int t;
        int64_t b;
        if (p.B32) {
            t = static_cast<int>(static_cast<uint32_t>(i) / p.B32);
            b = static_cast<uint32_t>(i) - static_cast<uint32_t>(t) * p.B32;
        } else {
            t = static_cast<int>(i / p.B);
            b = i - static_cast<int64_t>(t) * p.B;
        }
        // the bags left in the span, in table t and at all
        const int nb = static_cast<int>(min(min(p.span - done, p.B - b), p.num_bags - i));
        // The run's nb + 1 offsets, one per lane.
        int64_t off = 0;
        if (lane <= nb) {
            const char* o = static_cast<const char*>(p.offsets) + (i + lane) * (p.idx64 ? 8 : 4);
            off = p.idx64 ? __ldg(reinterpret_cast<const int64_t*>(o)) : static_cast<int64_t>(__ldg(reinterpret_cast<const int32_t*>(o)));
        }
        const TableMeta m = load_meta(p, t);
        // A run with an offset that goes backwards or points outside `indices` (or one of 2^31 rows) is taken byte by byte, which
        // looks at every bag: the bad ones are reported and left empty, the others come out as ever.
        const int64_t R0 = __shfl_sync(kFull, off, 0), before = __shfl_up_sync(kFull, off, 1);
        const bool sane = !__any_sync(kFull, lane <= nb && (off < before || off < 0 || off > p.num_indices || off - R0 > 0x7fffff00ll));
        const int rel = static_cast<int>(off - R0);
        const bool aligned = sane && m.D > 0 && m.rows_aligned && (m.D & 3) == 0 && m.stride < (1ll << 32) &&
                             (m.ty == TBE_B200_INT8 || m.ty == TBE_B200_INT4 || m.ty == TBE_B200_FP16 || m.ty == TBE_B200_FP32 ||
                              (m.ty == TBE_B200_FP8 && p.fp8_shift <= 23));
        // Aligned widths of 16 n <= 512 elements go through the streams, fp32 rows of up to 64 elements and all other widths in
        // steps.  24 tables of 200 K rows, batch 4096, bags of 32, fp16 result, streams against steps in us: INT8 of 16, 48, 128,
        // 144, 512 elements 72, 76, 127, 187, 322 against 126, 134, 154, 197, 494; FP16 75, 97, 134, 200, 490 against 106, 121, 155,
        // 310, 585; FP8 97, 88, 132, 226, 412 against 119, 128, 152, 230, 446; INT4 85, 79, 108, 194, 267 against 143, 134, 150, 185, 393
        // (144 and 208 INT4 elements alone would be 4 % faster in steps); FP32 of 16, 32, 48, 64, 80, 128 elements 120, 124, 140, 138,
        // 210, 253 against 107, 109, 137, 134, 267, 263.
        const bool stream = aligned && (m.D & 15) == 0 && m.D <= 512 && !(m.ty == TBE_B200_FP32 && m.D <= 64);
        if (stream) pool_run_stream_by_type<WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
        else if (aligned) pool_run_steps_by_type<WEIGHTED>(p, m, R0, rel, nb, b, lane, wsm);
        else if (m.D > 0 && p.idx64) pool_run_bytewise<int64_t>(p, m, i, nb, b, lane);
        else if (m.D > 0) pool_run_bytewise<int32_t>(p, m, i, nb, b, lane);
        done += nb;
    }
}

// ---- pooling NONE (sequence mode) --------------------------------------------------------------
//
// Row n of the output gets the dequantised row indices[n] of the table that position n belongs to (the t with
// offsets[t*B] <= n < offsets[(t+1)*B]), zero-filled from D_t up to max_D.  A warp takes kNobagChunk consecutive
// positions: the table is found once by binary search and then followed.
//
// The output is larger than the input here, so the work is cut by OUTPUT: a lane makes one 16-byte piece (8 elements of
// 16 bits or 4 of 32) at a time and consecutive lanes take consecutive pieces, so every store instruction writes 512
// contiguous bytes straight from registers.  The few row bytes behind a piece are fetched with 4-byte (INT8: two)
// loads that neighbouring lanes coalesce, the header with one more that hits L1.  Value = code * scale + bias in one mixed
// FMA.  1.6 M rows of 128 INT8 codes to fp16 (26 tables of a million rows, 410 MB of output): 160 us with the rows put
// together in shared memory first, 128 us this way (a copy of the same bytes: 76 us).

constexpr int kNobagChunk = 64;

// One position through the byte-wise decoder (any type, alignment and width).
template <typename IdxT>
__device__ __noinline__ void nobag_position_bytewise(const LookupParams& p, const TableMeta& m, const IdxT* indices, int64_t n, int max_D,
                                                     int lane)
{
    const int esz = (p.out_ty == TBE_B200_FP32) ? 4 : 2;
    void* seg = static_cast<char*>(p.output) + n * p.out_stride * esz;
    const int64_t idx = static_cast<int64_t>(indices[n]);
    const bool bad = idx < -1 || idx > 0x7fffffffll;
    const bool past = !bad && idx >= 0 && static_cast<uint64_t>(idx + 1) * static_cast<uint64_t>(m.stride) > static_cast<uint64_t>(m.avail);
    if (idx < 0 || bad || past) {
        if ((bad || past) && lane == 0 && p.error_flag) atomicOr(p.error_flag, bad ? 1 : 4);
        for (int e = lane; e < max(m.D, max_D); e += kWarp) store_scalar(seg, e, 0.0f, p.out_ty);
        return;
    }
    const uint8_t* row = m.table + idx * m.stride;
    float scale, bias;
    read_header(row, m.ty, scale, bias);
    for (int e = lane; e < m.D; e += kWarp)
        store_scalar(seg, e, decode_elem(row, m.ty, e, scale, bias, p.fp8_shift, p.fp8_mult), p.out_ty);
    for (int e = m.D + lane; e < max_D; e += kWarp) store_scalar(seg, e, 0.0f, p.out_ty);
}

// Stores 16 bytes with the widest stores that their address takes.  (Output rows need not start on 16 bytes: 128 elements
// beside a table of 130 or 132, say.)
__device__ __forceinline__ void store_piece(char* dst, const uint32_t (&h)[4])
{
    const uint32_t low = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst)) & 15u;
    if (low == 0) {
        st_stream16(dst, make_uint4(h[0], h[1], h[2], h[3]));
    } else if ((low & 7) == 0) {
        st_stream8(dst, make_uint2(h[0], h[1]));
        st_stream8(dst + 8, make_uint2(h[2], h[3]));
    } else if ((low & 3) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) st_stream4(dst + 4 * q, h[q]);
    } else {                                           // 16-bit elements: the words in between start two bytes on
        *reinterpret_cast<unsigned short*>(dst) = static_cast<unsigned short>(h[0]);
#pragma unroll
        for (int q = 0; q < 3; ++q) st_stream4(dst + 4 * q + 2, __funnelshift_r(h[q], h[q + 1], 16));
        *reinterpret_cast<unsigned short*>(dst + 14) = static_cast<unsigned short>(h[3] >> 16);
    }
}

// `cnt` consecutive positions [n, n + cnt), cnt <= kNobagChunk, of one table with 16-byte aligned rows of D elements, D a
// multiple of EP: EP elements are one 16-byte piece of the output.  RAGGED: output rows start anywhere.  (Kernels of their own: with
// the stores for such rows in the same loop, 1.6 M rows of 128 to fp16 took 131 to 134 us instead of 129.5.)
template <int TY, int EP, bool RAGGED>
__device__ __forceinline__ void nobag_pieces(const LookupParams& p, const TableMeta& m, int64_t n, int cnt, int max_D, int lane)
{
    constexpr bool kHdr = (TY == TBE_B200_INT8 || TY == TBE_B200_INT4);
    // bytes and 32-bit words of a row behind one piece
    constexpr int PB = (TY == TBE_B200_INT4) ? EP / 2 : (TY == TBE_B200_FP16) ? 2 * EP : (TY == TBE_B200_FP32) ? 4 * EP : EP;
    constexpr int RW = (PB + 3) / 4;
    constexpr int U = RW <= 2 ? 4 : 2;                 // pieces per lane in flight
    const int D = m.D, width = max(D, max_D);
    const int per_row = (width + EP - 1) / EP;         // pieces of an output row (below 8192: the division by it is exact)
    const uint32_t inv = 0xffffffffu / static_cast<uint32_t>(per_row) + 1u;
    const int total = cnt * per_row;
    constexpr int esz = 16 / EP;
    const bool vec = !RAGGED && (reinterpret_cast<uintptr_t>(p.output) & 15) == 0 && (p.out_stride * esz) % 16 == 0;
    char* out = static_cast<char*>(p.output) + n * p.out_stride * esz;
    const int64_t out_row_bytes = p.out_stride * esz;
    // The positions' row numbers, checked once: lane l holds positions l and l + 32.
    auto checked = [&](int pos) -> int32_t {
        if (pos >= cnt) return -1;
        const int64_t idx = p.idx64 ? __ldg(static_cast<const int64_t*>(p.indices) + n + pos)
                                    : static_cast<int64_t>(__ldg(static_cast<const int32_t*>(p.indices) + n + pos));
        if ((idx < -1 || idx > 0x7fffffffll) && p.error_flag) atomicOr(p.error_flag, 1);
        if (idx > 0x7fffffffll || idx < 0) return -1;
        if (static_cast<uint64_t>(idx + 1) * static_cast<uint64_t>(m.stride) > static_cast<uint64_t>(m.avail)) {
            if (p.error_flag) atomicOr(p.error_flag, 4);
            return -1;
        }
        return static_cast<int32_t>(idx);
    };
    const int32_t idx_lo = checked(lane), idx_hi = checked(lane + 32);
#pragma unroll 1
    for (int i0 = 0; i0 < total; i0 += kWarp * U) {
        uint32_t raw[U][RW], hdr[U];
        int row_u[U], k_u[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = static_cast<uint32_t>(i0 + u * kWarp + lane);
            // (one piece per row: the reciprocal does not fit 32 bits)
            const int row = per_row == 1 ? static_cast<int>(i) : static_cast<int>(__umulhi(i, inv));
            const int k = static_cast<int>(i) - row * per_row;
            const int32_t a = __shfl_sync(kFull, idx_lo, row & 31), b = __shfl_sync(kFull, idx_hi, row & 31);
            const int32_t idx = row < 32 ? a : b;
            row_u[u] = row;
            k_u[u] = k;
            hdr[u] = 0u;
#pragma unroll
            for (int w = 0; w < RW; ++w) raw[u][w] = 0u;
            if (row < cnt && idx >= 0 && k * EP < D) {
                const uint8_t* base = m.table + static_cast<int64_t>(idx) * m.stride;
                if constexpr (kHdr) hdr[u] = ldg4(base);
                const uint8_t* q = base + (kHdr ? 4 : 0) + k * PB;
                if constexpr (PB == 2) {
                    raw[u][0] = __ldg(reinterpret_cast<const unsigned short*>(q));
                } else if constexpr (PB >= 16) {
#pragma unroll
                    for (int w = 0; w < RW; w += 4) {
                        const uint4 v = ldg16(q + 4 * w);
                        raw[u][w] = v.x; raw[u][w + 1] = v.y; raw[u][w + 2] = v.z; raw[u][w + 3] = v.w;
                    }
                } else if constexpr (PB == 8 && !kHdr) {
                    const uint2 v = ldg8(q);
                    raw[u][0] = v.x; raw[u][1] = v.y;
                } else {                               // behind the header only 4-byte alignment is left
#pragma unroll
                    for (int w = 0; w < RW; ++w) raw[u][w] = ldg4(q + 4 * w);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (row_u[u] >= cnt) continue;
            float v[EP];
            if constexpr (kHdr) {
                const unsigned short scale_h = static_cast<unsigned short>(hdr[u] & 0xffffu);
                const float bias = half_bits_to_float(hdr[u] >> 16);
#pragma unroll
                for (int s = 0; s < EP; ++s) v[s] = bias;
                if constexpr (TY == TBE_B200_INT8) {
#pragma unroll
                    for (int w = 0; w < RW; ++w) {
                        const uint32_t c = raw[u][w];
                        const uint32_t even = codes_to_half2((c & 0x00FF00FFu) | 0x64006400u, 0x64006400u);
                        const uint32_t odd = codes_to_half2(__byte_perm(c, 0x64646464u, 0x4341), 0x64006400u);
                        add_pair(v[4 * w + 0], v[4 * w + 2], even, scale_h);
                        add_pair(v[4 * w + 1], v[4 * w + 3], odd, scale_h);
                    }
                } else {
                    // nibble pairs (j, j + EP / 2) are brought 16 bits apart
                    const uint32_t c = EP == 8 ? raw[u][0] : ((raw[u][0] & 0xffu) | ((raw[u][0] & 0xff00u) << 8));
                    const uint32_t y = c >> 8;
                    const uint32_t p0 = codes_to_half2((c & 0x000F000Fu) | 0x64006400u, 0x64006400u);
                    const uint32_t p1 = codes_to_half2((c & 0x00F000F0u) | 0x54005400u, 0x54005400u);
                    add_pair(v[0], v[EP / 2], p0, scale_h);
                    add_pair(v[1], v[EP / 2 + 1], p1, scale_h);
                    if constexpr (EP == 8) {
                        const uint32_t p2 = codes_to_half2((y & 0x000F000Fu) | 0x64006400u, 0x64006400u);
                        const uint32_t p3 = codes_to_half2((y & 0x00F000F0u) | 0x54005400u, 0x54005400u);
                        add_pair(v[2], v[6], p2, scale_h);
                        add_pair(v[3], v[7], p3, scale_h);
                    }
                }
            } else if constexpr (TY == TBE_B200_FP8) {
#pragma unroll
                for (int s = 0; s < EP; ++s) {
                    const uint32_t by = (raw[u][s >> 2] >> (8 * (s & 3))) & 0xffu;
                    const float mag = __uint_as_float((by & 0x7fu) << p.fp8_shift) * p.fp8_mult;
                    v[s] = __uint_as_float(__float_as_uint(mag) | ((by & 0x80u) << 24));
                }
            } else if constexpr (TY == TBE_B200_FP16) {
#pragma unroll
                for (int s = 0; s < EP; ++s) v[s] = half_bits_to_float((raw[u][s >> 1] >> (16 * (s & 1))) & 0xffffu);
            } else {
#pragma unroll
                for (int s = 0; s < EP; ++s) v[s] = __uint_as_float(raw[u][s]);
            }
            char* dst = out + row_u[u] * out_row_bytes + k_u[u] * 16;
            if (RAGGED && (k_u[u] + 1) * EP <= width) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) h[q] = EP == 4 ? __float_as_uint(v[q]) : pack_out(v[(2 * q) % EP], v[(2 * q + 1) % EP], p.out_ty);
                store_piece(dst, h);
            } else if (vec && (k_u[u] + 1) * EP <= width) {
                if constexpr (EP == 4) {
                    store_out4(dst, 0, v, TBE_B200_FP32, true);
                } else {
                    uint32_t h[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) h[q] = pack_out(v[2 * q], v[2 * q + 1], p.out_ty);
                    st_stream16(dst, make_uint4(h[0], h[1], h[2], h[3]));
                }
            } else {
                for (int s = 0; s < EP && k_u[u] * EP + s < width; ++s) store_scalar(dst, s, v[s], p.out_ty);
            }
        }
    }
}

template <int TY, bool RAGGED>
__device__ __forceinline__ void nobag_pieces_by_output(const LookupParams& p, const TableMeta& m, int64_t n, int cnt, int max_D, int lane)
{
    if (p.out_ty == TBE_B200_FP32) nobag_pieces<TY, 4, RAGGED>(p, m, n, cnt, max_D, lane);
    else nobag_pieces<TY, 8, RAGGED>(p, m, n, cnt, max_D, lane);
}

template <typename IdxT, bool RAGGED>
__global__ void __launch_bounds__(kWarpsPerBlock* kWarp)
tbe_nobag_kernel(const __grid_constant__ LookupParams p, int64_t num_indices, int max_D)
{
    const int lane = threadIdx.x & 31;
    const int64_t gw = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
    int64_t n = gw * kNobagChunk;
    const int64_t n_end = min(num_indices, n + kNobagChunk);
    if (n >= n_end) return;
    const IdxT* offsets = static_cast<const IdxT*>(p.offsets);
    const IdxT* indices = static_cast<const IdxT*>(p.indices);
    // Binary search over the T+1 table boundaries offsets[t*B]: the table of the chunk's first position.
    int lo = 0, hi = p.T;   // invariant: boundary(lo) <= n < boundary(hi)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (static_cast<int64_t>(offsets[static_cast<int64_t>(mid) * p.B]) <= n) lo = mid;
        else hi = mid;
    }
    int t = lo;
    while (n < n_end) {
        // positions [n, stop) belong to table t (skip tables without positions)
        int64_t stop = static_cast<int64_t>(offsets[static_cast<int64_t>(t + 1) * p.B]);
        while (stop <= n && t + 1 < p.T) {
            ++t;
            stop = static_cast<int64_t>(offsets[static_cast<int64_t>(t + 1) * p.B]);
        }
        stop = (t + 1 >= p.T) ? n_end : min(stop, n_end);
        if (stop <= n) stop = n_end;   // offsets that do not cover every position: the last table takes the rest
        const TableMeta m = load_meta(p, t);
        const int cnt = static_cast<int>(stop - n);
        // whole pieces of 8 (16-bit output) or 4 elements; an output row of fewer than 8192 of them
        const int ep = p.out_ty == TBE_B200_FP32 ? 4 : 8;
        const bool fast = m.rows_aligned && m.D > 0 && m.D % ep == 0 && max(m.D, max_D) < 8191 * ep;
        bool done = fast;
        if (fast) {
            switch (m.ty) {
                case TBE_B200_INT8: nobag_pieces_by_output<TBE_B200_INT8, RAGGED>(p, m, n, cnt, max_D, lane); break;
                case TBE_B200_INT4: nobag_pieces_by_output<TBE_B200_INT4, RAGGED>(p, m, n, cnt, max_D, lane); break;
                case TBE_B200_FP8: nobag_pieces_by_output<TBE_B200_FP8, RAGGED>(p, m, n, cnt, max_D, lane); break;
                case TBE_B200_FP16: nobag_pieces_by_output<TBE_B200_FP16, RAGGED>(p, m, n, cnt, max_D, lane); break;
                case TBE_B200_FP32: nobag_pieces_by_output<TBE_B200_FP32, RAGGED>(p, m, n, cnt, max_D, lane); break;
                default: done = false; break;
            }
        }
        if (!done)
            for (int64_t q = n; q < stop; ++q) nobag_position_bytewise<IdxT>(p, m, indices, q, max_D, lane);
        n = stop;
    }
}

constexpr int kSpanLarge = TBE_SPAN_LARGE;   // bags per warp when there is plenty of work: the more, the fewer bags straddle lane groups

// Blocks of a kernel that fit on one SM of the current device (occupancy query, once per device and kernel).
template <typename Kernel>
int resident_blocks(Kernel kernel, int variant, int fallback, int smem_bytes = 0)
{
    constexpr int kMaxDev = 64, kVariants = 2;
    static std::atomic<int> cached[kMaxDev][kVariants];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return fallback;
    int n = cached[dev][variant].load(std::memory_order_relaxed);
    if (n == 0) {
        if (smem_bytes > 48 * 1024) (void)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kWarpsPerBlock * kWarp, smem_bytes) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            n = fallback;
        }
        cached[dev][variant].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Environment switches, read once: TBE_B200_L2_POLICY (0 = nothing, the default; 2 = access-policy window, see
// apply_l2_window) and TBE_B200_SPAN (bags per warp, for experiments; 0 = automatic).
int env_int(const char* name, int dflt)
{
    const char* v = getenv(name);
    return (v && *v) ? atoi(v) : dflt;
}
int l2_policy_mode()
{
    static const int mode = env_int("TBE_B200_L2_POLICY", 0);
    return mode;
}

// TBE_B200_L2_POLICY=2: an access-policy window over dev_weights on the caller's stream, with part of L2 set aside for
// persisting lines (per-context state that ends with the process).  Off by default: the hot rows of a table are
// scattered over it, so the window cannot single them out (it keeps a random fraction of the table's lines), and it
// measured 3-6 % slower with the L2 hit rate unchanged.
void apply_l2_window(const void* base, int64_t bytes, cudaStream_t s)
{
    static std::atomic<int> prepared[64];
    int dev = 0;
    if (bytes <= 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    int max_window = 0, max_persist = 0;
    cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, dev);
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, dev);
    if (max_window <= 0 || max_persist <= 0) return;
    if (prepared[dev].exchange(1) == 0) (void)cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, static_cast<size_t>(max_persist));
    cudaStreamAttrValue attr{};
    const size_t win = static_cast<size_t>(bytes < max_window ? bytes : max_window);
    attr.accessPolicyWindow.base_ptr = const_cast<void*>(base);
    attr.accessPolicyWindow.num_bytes = win;
    const float ratio = static_cast<float>(max_persist) / static_cast<float>(win);
    attr.accessPolicyWindow.hitRatio = ratio < 1.0f ? ratio : 1.0f;
    attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    (void)cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &attr);
    (void)cudaGetLastError();
}
int forced_span()
{
    static const int span = env_int("TBE_B200_SPAN", 0);
    return span;
}

template <bool WEIGHTED>
int launch_pooled(LookupParams p, cudaStream_t s)
{
    constexpr int kSmemBytes = kWarpsPerBlock * kStreamSmemBytes;
    const int resident = resident_blocks(tbe_pooled_kernel<WEIGHTED>, WEIGHTED ? 1 : 0, kStreamBlocksPerSM, kSmemBytes);
    // Plenty of bags: fixed spans, as many blocks as that takes; the hardware block scheduler evens out the load.
    // Otherwise the spans are sized so that the warps fill a whole number of waves of resident warps.
    const int64_t slots = static_cast<int64_t>(sm_count()) * resident * kWarpsPerBlock;
    const int64_t waves = (p.num_bags + slots * kSpanLarge - 1) / (slots * kSpanLarge);
    if (waves >= 4) {
        p.span = kSpanLarge;
    } else {
        const int64_t per = (p.num_bags + slots * waves - 1) / (slots * waves);
        p.span = per < 1 ? 1 : (per > kSpanLarge ? kSpanLarge : per);
    }
    const int fs = forced_span();
    if (fs > 0) p.span = fs > kMaxRunBags ? kMaxRunBags : fs;
    const int64_t warps = (p.num_bags + p.span - 1) / p.span;
    const int64_t blocks = (warps + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (blocks > 0x7fffffffll) return fail(TBE_B200_ERR_UNSUPPORTED, "lookup: too many bags for one launch");
    tbe_pooled_kernel<WEIGHTED><<<static_cast<unsigned>(blocks), kWarpsPerBlock * kWarp, kSmemBytes, s>>>(p);
    return check_launch("tbe_pooled_kernel");
}

}  // namespace

}  // namespace tbe

extern "C" int tbe_b200_int_nbit_lookup(const tbe_b200_lookup_args* a, tbe_b200_stream_t stream)
{
    using namespace tbe;
    if (!a) return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: args is NULL");
    if (a->T <= 0) return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: T must be positive, got %d", a->T);
    if (a->B < 0) return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: B must be non-negative");
    if (a->index_bits != 32 && a->index_bits != 64)
        return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: index_bits must be 32 or 64, got %d", a->index_bits);
    if (a->pooling_mode < TBE_B200_POOL_SUM || a->pooling_mode > TBE_B200_POOL_NONE)
        return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: pooling_mode must be 0 (SUM), 1 (MEAN) or 2 (NONE), got %d",
                    a->pooling_mode);
    if (a->output_dtype != TBE_B200_FP32 && a->output_dtype != TBE_B200_FP16 && a->output_dtype != TBE_B200_BF16)
        return fail(TBE_B200_ERR_UNSUPPORTED, "lookup: output_dtype %d is not supported (0 FP32, 1 FP16, 5 BF16)",
                    a->output_dtype);
    if (!a->dev_weights || !a->weights_offsets || !a->weights_tys || !a->D_offsets || !a->offsets || !a->output)
        return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: a required pointer is NULL");
    if (a->num_indices > 0 && !a->indices) return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: indices is NULL");
    if (a->row_alignment < 1) return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: row_alignment must be >= 1");
    if (a->dest_outputs && a->rows_per_dest <= 0)
        return fail(TBE_B200_ERR_INVALID_ARGUMENT, "lookup: rows_per_dest must be positive with dest_outputs");

    LookupParams p;
    p.dev_weights = a->dev_weights;
    p.weights_offsets = a->weights_offsets;
    p.weights_tys = a->weights_tys;
    p.D_offsets = a->D_offsets;
    p.indices = a->indices;
    p.offsets = a->offsets;
    p.pw = a->indice_weights;
    p.output = a->output;
    p.out_cols = a->output_col_offsets;
    p.dests = a->dest_outputs;
    p.error_flag = a->error_flag;
    p.B = a->B;
    p.num_bags = static_cast<int64_t>(a->T) * a->B;
    p.num_indices = a->num_indices;
    p.out_stride = a->output_stride;
    p.rows_per_dest = a->rows_per_dest;
    p.span = 1;
    p.T = a->T;
    p.B32 = (p.num_bags < (1ll << 32) && a->B > 0) ? static_cast<uint32_t>(a->B) : 0u;
    p.pooling_mode = a->pooling_mode;
    p.out_ty = a->output_dtype;
    p.row_alignment = a->row_alignment;
    p.dev_weights_bytes = a->dev_weights_bytes > 0 ? a->dev_weights_bytes : 0;
    p.idx64 = a->index_bits == 64 ? 1 : 0;
    const int ebits = a->fp8_exponent_bits > 0 ? a->fp8_exponent_bits : 4;
    const int ebias = a->fp8_exponent_bias >= 0 ? a->fp8_exponent_bias : 7;
    p.fp8_shift = static_cast<uint32_t>(16 + ebits);
    const uint32_t mult_bits = static_cast<uint32_t>(254 - ebias) << 23;
    memcpy(&p.fp8_mult, &mult_bits, 4);

    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (a->pooling_mode == TBE_B200_POOL_NONE) {
        if (a->num_indices <= 0) return TBE_B200_OK;
        const int64_t chunks = (a->num_indices + kNobagChunk - 1) / kNobagChunk;
        const int64_t blocks = (chunks + kWarpsPerBlock - 1) / kWarpsPerBlock;
        if (blocks > 0x7fffffffll) return fail(TBE_B200_ERR_UNSUPPORTED, "lookup: too many indices for one launch");
        const int64_t row_bytes = a->output_stride * (a->output_dtype == TBE_B200_FP32 ? 4 : 2);
        const bool ragged = ((reinterpret_cast<uintptr_t>(a->output) | static_cast<uint64_t>(row_bytes)) & 15) != 0;
        auto* const kernel = a->index_bits == 32 ? (ragged ? tbe_nobag_kernel<int32_t, true> : tbe_nobag_kernel<int32_t, false>)
                                                 : (ragged ? tbe_nobag_kernel<int64_t, true> : tbe_nobag_kernel<int64_t, false>);
        kernel<<<static_cast<unsigned>(blocks), kWarpsPerBlock * kWarp, 0, s>>>(p, a->num_indices, a->max_D);
        return check_launch("tbe_nobag_kernel");
    }
    if (p.num_bags == 0) return TBE_B200_OK;
    if (l2_policy_mode() == 2) apply_l2_window(a->dev_weights, a->dev_weights_bytes, s);
    return p.pw ? launch_pooled<true>(p, s) : launch_pooled<false>(p, s);
}
