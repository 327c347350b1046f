// Host-side check of the special cells' addresses (d3q19.cuh: pull_element) against the pull rule
// written out in coordinates and 64 bits: the neighbour's population, at a wall the cell's own
// opposite one, across an x end its own, under the lid the mirrored one of the row it came from.
// Prints cells times directions compared, addresses that differ, addresses outside the array.
#include <cstdio>
#include <cstdint>
#include <random>
#include <utility>
#include "../../water_flow_simulation_b200/csrc/d3q19.cuh"
using namespace wfs;

struct Size {
    long long pitch, ny, nz;
};

static long long rule(const Size& s, int i, long long x, long long y, long long z, long long nx, bool wall)
{
    const long long S = s.pitch * s.ny * s.nz, own = x + s.pitch * (y + s.ny * z);
    if (wall) return opp(i) * S + own;
    const long long xs = x - cx(i), ys = y - cy(i), zs = z - cz(i);
    if (xs < 0 || xs >= nx) return i * S + own;
    if (zs >= s.nz) return mirz(i) * S + xs + s.pitch * (ys + s.ny * z);
    return i * S + xs + s.pitch * (ys + s.ny * zs);
}

static long long compared = 0, differ = 0, outside = 0;

template <int I>
static void one(const Size& s, long long x, long long y, long long z, long long nx, bool wall)
{
    // rows past the y ends and below the bed are walls always; a wall bit is never set across an x end
    const long long xs = x - cx(I), ys = y - cy(I), zs = z - cz(I), S = s.pitch * s.ny * s.nz;
    wall = I > 0 && xs >= 0 && xs < nx && (wall || ys < 0 || ys >= s.ny || zs < 0);
    const long long got = pull_element<I>(x + s.pitch * (y + s.ny * z), s.pitch * s.ny, (int)s.pitch, S,
                                          wall ? 1u << I : 0u, z == s.nz - 1, x == 0, x == nx - 1);
    ++compared;
    differ += got != rule(s, I, x, y, z, nx, wall);
    outside += got < 0 || got >= Q * S;
}
template <int... Is>
static void all(std::integer_sequence<int, Is...>, const Size& s, long long x, long long y, long long z, long long nx, bool wall)
{
    (one<Is>(s, x, y, z, nx, wall), ...);
}

int main()
{
    // 60, 2^30 less and more than a layer, 1.14e9, 1.5e9 and 4.3e9 cells
    const Size sizes[] = {{4, 5, 3}, {1024, 1024, 1023}, {1024, 1024, 1025}, {4096, 2048, 136}, {8192, 4096, 45}, {4096, 4096, 257}};
    std::mt19937_64 rng(3);
    for (const Size& s : sizes)
        for (int n = 0; n < 4000; ++n) {
            const long long nx = s.pitch - (long long)(rng() % 4);
            const auto at = [&](long long m) {                 // ends as often as the inside
                const int k = (int)(rng() % 3);
                return k == 0 ? 0 : k == 1 ? m - 1 : (long long)(rng() % (uint64_t)m);
            };
            all(std::make_integer_sequence<int, Q>{}, s, at(nx < 1 ? 1 : nx), at(s.ny), at(s.nz), nx < 1 ? 1 : nx, rng() % 2);
        }
    std::printf("%lld %lld %lld\n", compared, differ, outside);
    return 0;
}
