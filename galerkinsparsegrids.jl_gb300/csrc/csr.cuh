// csr.cuh -- the lane reduction of the CSR row kernels (kernels.cu, csr_step.cu).
#pragma once
#include <cuda_runtime.h>

namespace sgdg {

// Sum of s[0..NV) over the VS lanes of a row group.  With NV = 2 or 4 the
// first steps exchange halves of the vector set instead of every value (a
// lane keeps the half selected by its lane bit and adds its partner's copy),
// so a row costs log2(VS) + NV - 2 FP64 additions per lane instead of
// NV log2(VS); each vector's sum has the pairing, and therefore the value, of
// the all-lane butterfly.  On return vector j's sum is in s[0] of the lanes
// whose group index has j in its top bits (csr_owner), or in s[j] of every
// lane when there was nothing to exchange (NV = 1 or 3, or VS too small).
template <int VS, int NV>
__device__ __forceinline__ void csr_reduce(double (&s)[NV], int lane) {
    if constexpr ((NV == 4 && VS >= 4) || (NV == 2 && VS >= 2)) {
        constexpr int o1 = VS / 2;
        const bool up1 = lane & o1;
        double h[NV / 2];
#pragma unroll
        for (int i = 0; i < NV / 2; i++) {
            const double keep = up1 ? s[NV / 2 + i] : s[i];
            const double give = up1 ? s[i] : s[NV / 2 + i];
            h[i] = keep + __shfl_xor_sync(0xffffffffu, give, o1);
        }
        double r;
        int o;
        if constexpr (NV == 4) {
            constexpr int o2 = VS / 4;
            const bool up2 = lane & o2;
            const double keep = up2 ? h[1] : h[0];
            const double give = up2 ? h[0] : h[1];
            r = keep + __shfl_xor_sync(0xffffffffu, give, o2);
            o = VS / 8;
        } else {
            r = h[0];
            o = VS / 4;
        }
        for (; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        s[0] = r;
    } else {
#pragma unroll
        for (int j = 0; j < NV; j++)
#pragma unroll
            for (int o = VS / 2; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    }
}

// Which vector's sum the lane holds after csr_reduce (-1: all of them, in
// s[j]); only lanes whose low bits are zero store it.
template <int VS, int NV>
__device__ __forceinline__ int csr_owner(int lane, bool& stores) {
    if constexpr ((NV == 4 && VS >= 4) || (NV == 2 && VS >= 2)) {
        constexpr int per = VS / NV;  // lanes holding one vector's sum
        stores = lane % per == 0;
        // vector index: bit VS/2 selects the upper half of the set, then bit VS/4 within it
        if constexpr (NV == 4)
            return ((lane & (VS / 2)) ? 2 : 0) + ((lane & (VS / 4)) ? 1 : 0);
        else
            return (lane & (VS / 2)) ? 1 : 0;
    } else {
        stores = lane == 0;
        return -1;
    }
}

}  // namespace sgdg
