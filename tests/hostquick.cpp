// Host build of the quick HEALPix index beside the general one.
#include <stdint.h>

#include "hcg_math.cuh"

extern "C" long hq_compare(uint64_t nside, long n, const double *theta, const double *phi) {
    hcg::HpxParams h{};
    h.nside = nside;
    while ((1ULL << (h.order + 1)) <= nside) ++h.order;
    h.ncap = (nside * nside - nside) << 1;
    h.npix = 12 * nside * nside;
    h.fact2 = 4. / h.npix;
    h.fact1 = (nside << 1) * h.fact2;
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        int a, b;
        bad += hcg::ang2pix_quick(h, theta[i], phi[i], a) != hcg::ang2pix(h, theta[i], phi[i], b);
    }
    return bad;
}
