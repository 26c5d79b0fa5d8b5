// Prints, for every dimension and bin count given as "dims bins" on stdin,
// whether the channel step stages a channel's tables (single-integrand and
// grouped launches), the shared memory that it asks for and its threads.
#include <cstdio>

#include "phase_dev.cuh"

int main() {
    int d, b;
    while (std::scanf("%d %d", &d, &b) == 2) {
        const chili_dev::ChannelShape s = chili_dev::channel_shape(d, b, true),
                                      g = chili_dev::grouped_channel_shape(d, b, true);
        std::printf("%d %zu %d %d %zu %d\n", s.tables, s.smem, s.threads, g.tables, g.smem, g.threads);
    }
}
