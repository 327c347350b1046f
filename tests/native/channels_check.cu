// Host-side check of the channel accesses (channels.cuh) with the local array at every 4-byte offset from a
// 16-byte boundary, as a compiler may place a plain float array; built with the alignment sanitizer, which
// ends the program at the first wider access that is not on its boundary.  Prints values that differ.
#include <cstdio>
#include "../../water_flow_simulation_b200/csrc/channels.cuh"
using namespace wfs;

template <int OFFSET>
struct alignas(16) Placed {
    float before[OFFSET];
    float v[8];
};
template <>
struct alignas(16) Placed<0> {
    float v[8];
};

static int differ = 0;

template <int OFFSET>
static void one()
{
    alignas(16) float in[8];
    alignas(16) float back[8];
    alignas(16) __nv_bfloat16 half[8];
    for (int j = 0; j < 8; ++j) in[j] = 1.0f + 0.125f * (float)(OFFSET * 8 + j);
    Placed<OFFSET> a;
    load_n<8>(a.v, in);
    store_n<8>(back, a.v);
    store_n<8>(half, a.v);
    for (int j = 0; j < 8; ++j) differ += a.v[j] != in[j] || back[j] != in[j] || __bfloat162float(half[j]) != in[j];
    float single[1];
    load_n<1>(single, in + 3);
    differ += single[0] != in[3];
}

int main()
{
    one<0>();
    one<1>();
    one<2>();
    one<3>();
    std::printf("%d\n", differ);
    return 0;
}
