// route_cost.h -- estimates (us of 8 steps) behind the choice of a kernel for the smaller
// instances of a batch or a server: the persistent kernels, one CTA per instance, all
// instances side by side, against launches of the whole GPU one after another (packed
// one-CTA-per-trotter sweeps; the per-instance bipartite kernels).  Either gives the same
// results.  The constants are fits to measured times; what they decide, ms:
//                                          persistent   packed
//   batch, 16 steps, 150 x N = 64, m = 4         1.22     0.54
//                                  m = 16        1.29     1.21
//                                  m = 64        1.42     7.13
//                                  m = 256       2.51    50.0
//   60 instances of 100 to 200, m = 64           4.47     3.51;  m = 256  19.7, 19.4
//   150 of 200 to 400, m = 16                    7.36     2.76;  m = 128  26.8, 29.7
//   server, 32 steps, 60 x N = 64, m = 256      11.0     44.0
//   32 bipartite requests 20 x 20, m = 2         3.7      9.1
//                         200 x 200, m = 64     12.1      9.8
#pragma once

#include <algorithm>
#include <vector>

namespace sq103 {

constexpr int kPackInstances = 64;  // instances per packed launch (sq103_dense_anneal_pack)

// one packed launch of `ctas` trotters in all, rows of up to N spins and up to m trotters an
// instance; up to two CTAs per SM (perSm2), or four
inline double pack_us(int N, int m, int ctas, int perSm2) {
    return ctas <= perSm2 ? 60. + 0.4 * N + 0.15 * m : 100. + 0.8 * N + 0.9 * m;
}

// a dense instance in the persistent kernel, its spins and fields in shared memory or not
inline double dense_persistent_us(int N, int m, bool staged) {
    return 8. * N * (staged ? 1. + 0.004 * m : 1. + m * (0.013 + 0.00003 * N));
}

// a bipartite instance in the persistent kernel: its field tiles, one after another
inline double bipartite_persistent_us(int N0, int N1, int m) {
    const double rows = (m + 15) / 16;
    return 8. * (6. + rows * (((N0 + 31) / 32) * (2.6 + 0.0065 * N1) + ((N1 + 31) / 32) * (2.6 + 0.0065 * N0)));
}

struct DenseRoute {
    int N, m, cap;  // cap: resident trotters of a packed launch (0: only the persistent kernel takes it)
    double us;      // in the persistent kernel
    bool packed;    // is in the packed launches already
};

// The size N from which the instances go to the packed launches for the least time of all,
// which is the sum of the packed launches and the persistent kernel's: its CTAs fill the
// shared memory of their SMs, where the packed launches wait for the whole GPU.
// noLimit: a size above every instance's.
inline int dense_route_limit(std::vector<DenseRoute> &items, int perSm2, int noLimit) {
    std::sort(items.begin(), items.end(), [](const DenseRoute &a, const DenseRoute &b) { return a.N < b.N; });
    int best = noLimit;
    double bestUs = 0.;
    for (int limit : {noLimit, 1024, 768, 512, 384, 256, 192, 128, 96, 64}) {
        double us = 0., longest = 0., total = 0.;
        int n = 0, ctas = 0, maxM = 0, lastN = 0;
        auto flush = [&]() {
            if (n > 0) us += pack_us(lastN, maxM, ctas, perSm2);
            n = ctas = maxM = 0;
        };
        for (const DenseRoute &it : items) {
            if (it.cap == 0 || (it.N < limit && !it.packed)) {
                longest = std::max(longest, it.us);
                total += it.us;
                continue;
            }
            if (n == kPackInstances || ctas + it.m > it.cap) flush();
            ++n;
            ctas += it.m;
            maxM = std::max(maxM, it.m);
            lastN = it.N;
        }
        flush();
        if (longest > 0.) us += 40. + std::max(longest, total / perSm2);  // (two CTAs per SM staged)
        if (limit == noLimit || us < bestUs) {
            best = limit;
            bestUs = us;
        }
    }
    return best;
}

// the per-instance bipartite kernels: the host's 32 launches an instance, and the first's latency
constexpr double kBipLaunchesUs = 72., kBipLatencyUs = 70.;

// The least persistent time from which bipartite requests take the per-instance kernels,
// for the shortest tick: `us` their persistent times, `running` the longest of those that
// run there already, `there` the requests already on the per-instance kernels, `room` how
// many more may be.
inline double bipartite_route_cut(std::vector<double> &us, double running, int there, int room) {
    std::sort(us.begin(), us.end(), [](double a, double b) { return a > b; });
    double best = 0., cut = 1e300;
    for (int k = 0; k <= std::min<int>((int)us.size(), room); ++k) {
        const double rest = std::max(running, k < (int)us.size() ? us[k] : 0.);
        const double t = std::max(rest, k + there > 0 ? kBipLatencyUs + kBipLaunchesUs * (k + there) : 0.);
        if (k == 0 || t < best) {
            best = t;
            cut = k > 0 ? us[k - 1] : 1e300;
        }
    }
    return cut;
}

}  // namespace sq103
