// Rows of any length between global memory and padded rows in shared memory: `total` bytes of consecutive rows of `row_bytes`, the
// first of them word aligned, whole words on the global side, single elements of type T on the other (a word may hold the end of one
// row and the start of the next).  One division a word.
#pragma once
#include "common.cuh"

namespace espdl {

template <typename T>
__device__ __forceinline__ void deal_rows(const uint32_t *src, int total, int row_bytes, uint32_t *rows, int pitch)
{
    const int nr = total / row_bytes;
    for (int w = threadIdx.x; 4 * w < total; w += blockDim.x) {
        uint32_t v = 0;
        if (4 * w + 4 <= total)
            v = src[w];
        else
            for (int k = 0; 4 * w + k < total; k++) v |= (uint32_t)((const uint8_t *)src)[4 * w + k] << (8 * k);
        int rr = 4 * w / row_bytes, o = 4 * w - rr * row_bytes;
#pragma unroll
        for (int k = 0; k < 4; k += (int)sizeof(T)) {
            if (rr < nr)
                *(T *)((uint8_t *)(rows + rr * pitch) + o) = (T)(v >> (8 * k));
            o += (int)sizeof(T);
            if (o == row_bytes)
                o = 0, rr++;
        }
    }
}

template <typename T>
__device__ __forceinline__ void collect_rows(uint32_t *dst, int total, int row_bytes, const uint32_t *rows, int pitch)
{
    constexpr uint32_t MASK = sizeof(T) == 1 ? 0xffu : 0xffffu;
    const int nr = total / row_bytes;
    for (int w = threadIdx.x; 4 * w < total; w += blockDim.x) {
        int rr = 4 * w / row_bytes, o = 4 * w - rr * row_bytes;
        uint32_t v = 0;
#pragma unroll
        for (int k = 0; k < 4; k += (int)sizeof(T)) {
            if (rr < nr)
                v |= ((uint32_t)(int)*(const T *)((const uint8_t *)(rows + rr * pitch) + o) & MASK) << (8 * k);
            o += (int)sizeof(T);
            if (o == row_bytes)
                o = 0, rr++;
        }
        if (4 * w + 4 <= total)
            dst[w] = v;
        else
            for (int k = 0; 4 * w + k < total; k++) ((uint8_t *)dst)[4 * w + k] = (uint8_t)(v >> (8 * k));
    }
}

} // namespace espdl
