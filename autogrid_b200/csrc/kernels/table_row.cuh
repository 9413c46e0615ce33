// Table rows of 8 columns.
#pragma once

namespace agb {

// 8 consecutive floats of a 32-byte aligned table row.  One 32-byte gather of
// a warp takes one L1 wavefront per lane, half of what two 16-byte ones take.
struct Row8 {
    float2 p[4];
};
__device__ __forceinline__ Row8 load_row8(const float *p)
{
    Row8 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.p[0].x), "=f"(r.p[0].y), "=f"(r.p[1].x), "=f"(r.p[1].y), "=f"(r.p[2].x), "=f"(r.p[2].y),
          "=f"(r.p[3].x), "=f"(r.p[3].y)
        : "l"(p));
    return r;
}

}  // namespace agb
