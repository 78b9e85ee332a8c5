// How many candidates each ray of a batch lists (host code without CUDA).
#pragma once
#include <algorithm>
#include <cstddef>

namespace jbg {

// 256 while the lists of 8 bytes an entry stay within 512 MB, else as many as do, at least 8; never
// more than the world has bodies.
inline int ray_list_cap(int rays, int bodies) {
    const size_t fit = ((size_t)1 << 26) / (size_t)std::max(rays, 1);
    return std::max(1, std::min(bodies, (int)std::min<size_t>(256, std::max<size_t>(8, fit))));
}

// The entries a ray gets: the cap, halved as often as the device has no room for that many (a ray that
// finds more goes through k_ray_long).  held: entries there are now; grow(n) makes it n, or 0 and
// returns false.  0: no room for one entry a ray.
template <class Grow>
int ray_list_fit(int rays, int bodies, const size_t& held, Grow&& grow) {
    for (int cap = ray_list_cap(rays, bodies); cap > 0; cap /= 2)
        if (held >= (size_t)rays * cap || grow((size_t)rays * cap)) return cap;
    return 0;
}

}  // namespace jbg
