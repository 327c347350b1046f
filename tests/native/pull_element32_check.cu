// Host-side check of the 32-bit form of the special cells' addresses (d3q19.cuh: pull_element<I, int>), which
// batches take, against the 64-bit one, on lattices of up to 2^30 cells, the most a batch case can have; built
// with the sanitizer that ends the program at a signed overflow.  Prints addresses compared and those that differ.
#include <cstdio>
#include <cstdint>
#include <random>
#include <utility>
#include "../../water_flow_simulation_b200/csrc/d3q19.cuh"
using namespace wfs;

static long long compared = 0, differ = 0;

template <int... Is>
static void all(std::integer_sequence<int, Is...>, int own, int plane, int pitch, long long S, bool wall, bool lid,
                bool first, bool last, bool (&row_out)[Q])
{
    const auto one = [&](auto I) {
        constexpr int i = decltype(I)::value;
        const bool edge = cx(i) == 1 ? first : cx(i) == -1 ? last : false;
        const uint32_t fk = i > 0 && !edge && (wall || row_out[i]) ? 1u << i : 0u;
        ++compared;
        differ += pull_element<i, int>(own, plane, pitch, S, fk, lid, first, last) !=
                  pull_element<i>((long long)own, (long long)plane, pitch, S, fk, lid, first, last);
    };
    (one(std::integral_constant<int, Is>{}), ...);
}

int main()
{
    const int sizes[][3] = {{8, 5, 3}, {64, 70, 14}, {4096, 1024, 255}, {8192, 4096, 32}};    // pitch, ny, nz; 2^30 cells
    std::mt19937_64 rng(7);
    for (const auto& s : sizes) {
        const int pitch = s[0], ny = s[1], nz = s[2], plane = pitch * ny;
        const long long S = (long long)plane * nz;
        for (int n = 0; n < 4000; ++n) {
            const auto at = [&](int m) {                   // ends as often as the inside
                const int k = (int)(rng() % 3);
                return k == 0 ? 0 : k == 1 ? m - 1 : (int)(rng() % (uint64_t)m);
            };
            const int nx = pitch - (int)(rng() % 4), x = at(nx), y = at(ny), z = at(nz);
            bool row_out[Q];
            for (int i = 0; i < Q; ++i) row_out[i] = y - cy(i) < 0 || y - cy(i) >= ny || z - cz(i) < 0;
            all(std::make_integer_sequence<int, Q>{}, x + pitch * y + plane * z, plane, pitch, S, rng() % 2, z == nz - 1,
                x == 0, x == nx - 1, row_out);
        }
    }
    std::printf("%lld %lld\n", compared, differ);
    return 0;
}
