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

    // requests for the pairs, and those that binary64 renders more exactly
    struct View {
        double inc, distance, div;
        bool pairs;
    };
    const View views[] = {{60, 1000, 40, true},  {5, 1000, 40, true},    {85, 1000, 40, true},  {17, 1000, 10, true},
                          {95, 1000, 40, true},  {60, 1000, 400, true},  {0, 1000, 40, false},  {90, 1000, 40, false},
                          {88, 1000, 40, false}, {180, 1000, 40, false}, {60, 100, 40, false},  {60, 1000, 9, false},
                          {60, 1000, 1, false},  {60, 0, 40, false},     {60, NAN, 40, false},  {NAN, 1000, 40, false}};
    ok = true;
    for (const View &v : views) {
        mk_request R = {};
        R.camera = {};
        R.camera.kind = MK_CAMERA_GRID;
        R.camera.bhspin = 0.94;
        R.camera.distance = v.distance;
        R.camera.cos_inc = cos(v.inc * M_PI / 180);
        R.camera.sin_inc = sin(v.inc * M_PI / 180);
        R.camera.fov_lower = -20;
        R.camera.fov_upper = 20;
        R.policy.div = v.div;
        R.policy.tol = 1e-4;
        R.fluid_gamma = 13.0 / 9;
        R.r_low = 1;
        R.r_high = 40;
        R.electron_gamma_m1 = 1.0 / 3;
        R.ion_gamma_m1 = 2.0 / 3;
        R.sigma_cut = 100;
        R.Ne_unit = 2e5;
        R.B_unit = 60;
        R.L_unit = 1e15;
        R.nnu = 1;
        R.nu[0] = 230e9;
        if (mk::pair_request(R) != v.pairs) {
            ok = false;
            printf("view_%g_%g_%g 0\n", v.inc, v.distance, v.div);
        }
        R.camera.kind = MK_CAMERA_EQUATOR;
        ok = ok && !mk::pair_request(R);
    }
    printf("pair_request %d\n", ok);
    return 0;
}
