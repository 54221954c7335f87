// Predicates of the compaction kernels: a row of consecutive elements to a mask of the kept ones.
#pragma once

#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "runtime.hpp"

namespace pxb {

template <typename T>
struct PredDev {
    PredKind kind;
    bool negate;
    T c, m, r;
    FastMod32 fm;           // 32-bit element types: m as an invariant divisor
    FastMod64 fm64;         // 64-bit integers: m and r
    const uint8_t* fl;      // FLAGS: one byte per element, written by a registered image
    __device__ __forceinline__ bool operator()(T x) const {
        bool v;
        switch (kind) {
            case PredKind::GT: v = x > c; break;
            case PredKind::GE: v = x >= c; break;
            case PredKind::LT: v = x < c; break;
            case PredKind::LE: v = x <= c; break;
            case PredKind::EQ: v = x == c; break;
            case PredKind::NE: v = x != c; break;
            case PredKind::NONZERO: v = x != T(0); break;
            case PredKind::MOD:
                v = mod_eq(x);
                break;
            default: v = false; break;
        }
        return v != negate;
    }
    // Flag bits of one row whose first element has global index gi: the switch on the
    // (CTA-uniform) kind is taken once per row. A bit costs its comparison and one predicated
    // OR; the negation is one XOR of the row.
    template <int ITEMS>
    __device__ __forceinline__ uint32_t flags(const T (&x)[ITEMS], uint64_t gi) const {
        uint32_t f = 0;
        switch (kind) {
            case PredKind::FLAGS:
                // rows start at multiples of ITEMS (28 or 14), so the row's flag bytes are
                // 4-byte (or 2-byte) aligned; the array is padded to the end of the last
                // tile of every kernel (compact_flags_padding)
                if constexpr (ITEMS % 4 == 0) {
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(fl + gi);
#pragma unroll
                    for (int v = 0; v < ITEMS / 4; ++v) {
                        const uint32_t b = w[v];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if ((b >> (8 * k)) & 0xffu) f |= 1u << (4 * v + k);
                    }
                } else {
                    static_assert(ITEMS % 2 == 0, "rows of an even number of elements");
                    const uint16_t* w = reinterpret_cast<const uint16_t*>(fl + gi);
#pragma unroll
                    for (int v = 0; v < ITEMS / 2; ++v) {
                        const uint32_t b = w[v];
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            if ((b >> (8 * k)) & 0xffu) f |= 1u << (2 * v + k);
                    }
                }
                break;
#define PXB_ROW(KIND, EXPR)                                              \
            case PredKind::KIND:                                          \
                _Pragma("unroll") for (int j = 0; j < ITEMS; ++j)          \
                    if (EXPR) f |= 1u << j;                                \
                break;
            PXB_ROW(GT, x[j] > c)
            PXB_ROW(GE, x[j] >= c)
            PXB_ROW(LT, x[j] < c)
            PXB_ROW(LE, x[j] <= c)
            PXB_ROW(EQ, x[j] == c)
            PXB_ROW(NE, x[j] != c)
            PXB_ROW(NONZERO, x[j] != T(0))
            case PredKind::MOD:
                if constexpr (std::is_integral<T>::value && sizeof(T) == 4) {
                    if (r == T(0)) {  // divisibility: a multiply and a compare per element
                        if (fm.am == 0) break;
#pragma unroll
                        for (int j = 0; j < ITEMS; ++j)
                            if (fm.divides0(x[j])) f |= 1u << j;
                        break;
                    }
                }
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if (mod_eq(x[j])) f |= 1u << j;
                break;
#undef PXB_ROW
            default: return 0u;
        }
        return negate ? ~f & ((1u << ITEMS) - 1u) : f;
    }
    // x % m == r with C semantics, without a division
    __device__ __forceinline__ bool mod_eq(T x) const {
        if constexpr (std::is_integral<T>::value && sizeof(T) == 4) {
            return fm.eq(x, r);
        } else if constexpr (std::is_integral<T>::value) {
            return fm64.eq(x);
        } else {
            return false;
        }
    }
};

template <typename T, int ITEMS, int V>
__device__ __forceinline__ void load_row(const T* row_ptr, T (&x)[ITEMS]) {
    const uint4* row = reinterpret_cast<const uint4*>(row_ptr);
#pragma unroll
    for (int v = 0; v < ITEMS / V; ++v) {
        const uint4 r = row[v];
        const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
        for (int k = 0; k < V; ++k) x[v * V + k] = e[k];
    }
}

template <typename T>
inline PredDev<T> make_pred(const Pred& p) {
    PredDev<T> e;
    e.kind = p.kind;
    e.negate = p.negate;
    if (std::is_floating_point<T>::value) e.c = (T)p.f;
    else if (std::is_signed<T>::value) e.c = (T)p.i;
    else e.c = (T)p.u;
    e.m = (T)p.mod_m;
    e.r = (T)p.mod_r;
    if constexpr (std::is_integral<T>::value && sizeof(T) == 4) e.fm = FastMod32::make((int64_t)e.m);
    if constexpr (std::is_integral<T>::value && sizeof(T) == 8) e.fm64 = FastMod64::make(e.m, e.r);
    e.fl = p.flags;
    return e;
}

}  // namespace pxb
