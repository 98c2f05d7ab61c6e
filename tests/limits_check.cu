// Host check of the fused FP64 render's rules (mk_sample_pair.cuh).  Prints one
// line a check, "name 1" if it holds.
#include <stdio.h>

#include "mk_sample_pair.cuh"

int main() {
    // a block's last rays: all of them find a lane, on one warp a sub-partition
    // if they fit, and a block without rays keeps a number of warps to divide by
    bool ok = true;
    for (int warps = 4; warps <= 8; warps += 4)
        for (int rays = 0; rays <= 32 * warps; rays++) {
            const int w = mk::warps_for(rays, warps);
            ok = ok && w >= 4 && w <= warps && w % 4 == 0 && 32 * w >= rays && (rays == 0 || rays > 128 || w == 4);
        }
    printf("warps_for %d\n", ok);
    return 0;
}
