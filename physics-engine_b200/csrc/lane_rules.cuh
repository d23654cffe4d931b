// How many lanes of a warp share a slot's list in each pair pass (lane_group.cuh).
// Plain C++: a function of the particle counts.
//
// G lanes shorten a list's serial walk G-fold, and cost every slot of the world,
// those without work in the pass too, its G threads: about S / G + c G slots, least
// where G^2 slots = S / c. So each rule takes the lanes that suit the slots with
// work, and fewer while G^2 slots is above the pass's bound (2,197 fluid particles
// among 540,002 boundary samples, us with 1 / 4 / 8 / 16 / 32 lanes: density
// 82/40/26/41/78, forces 182/59/39/50/89, XSPH 74/59/56/99/183, boundary
// 50/28/43/78/144; 15,625 among 1,100,002: 107/50/69/113/203, 212/86/95/140/233,
// 106/84/127/221/412, 54/55/96/175/336).
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define PE_LANES_HD __host__ __device__ __forceinline__
#else
#define PE_LANES_HD inline
#endif

namespace pe {

// The slot of a thread of a launch with G lanes a slot. The thread's number in the
// launch does not fit 32 bits for all worlds (2^27 slots of 32 lanes); this does.
template <int G>
PE_LANES_HD uint32_t lane_slot(uint32_t block, uint32_t block_threads, uint32_t thread) {
    return block * (block_threads / G) + thread / G;
}

// Lanes in each pass: 1, 4, 8, 16 or 32 (f64), 1, 8 or 32 (f32).
struct PassLanes {
    uint32_t density = 1, forces = 1, boundary = 1, xsph = 1;
};

// `lanes`, or the most of 32, 16, 8, 4, 1 (few: 32, 8, 1) below it with lanes^2 slots <= most.
inline uint32_t fit_lanes(uint32_t lanes, uint64_t slots, uint64_t most, bool few = false) {
    while (lanes > 1u && (uint64_t)lanes * lanes * slots > most)
        lanes = few ? (lanes == 32u ? 8u : 1u) : (lanes == 4u ? 1u : lanes / 2u);
    return lanes;
}

// f64 passes, from the slots that have work and the pairs each has (~250 in 3-D, ~50
// in 2-D). More lanes shorten a slot's serial chain; fewer waste less on the exchange
// of terms once the slots alone fill the SMs.
// us a pass, 1 / 4 / 8 / 16 / 32 lanes, dam-break tanks of fluid particles:
//   fluid      density            forces              XSPH                boundary (slots)
//   2,197      83/31/19/15/15     187/53/35/24/19     70/32/25/19/20      46/23/15/12/11
//   4,096      83/31/19/17/17     168/56/37/27/29     69/33/25/22/24      46/23/15/11/11 (10,170)
//   8,000      88/32/25/23/25     168/62/45/43/41     71/36/30/29/36      48/23/15/13/12 (17,130)
//   15,625     89/36/31/33/39     180/73/69/63/69     73/39/39/44/57      48/23/16/13/15 (29,551)
//   32,768     97/73/59/63/74     214/129/116/120/138 96/92/71/82/109     52/29/19/17/21 (55,034)
//   46,656     101/85/79/86/102   248/168/161/165/192 96/109/103/108/153  53/29/21/21/26 (74,766)
//   125,000    219/203/190        445/357/382         197/229/222         58/33/31 (176,472)
//   151,686    228/-/230          488/-/459           205/-/267           61/-/33 (210,648)
//     (Wendland) 255/233/236      627/515/549         208/258/272
//   166,375    230/-/254          512/-/504           210/-/296           61/-/35 (229,377)
//   185,193    236/269/272        578/507/549         212/297/317         61/37/36 (252,227)
//   512,000    579/732/736        1344/1319/1468      507/793/841         74/63/67
//   681,472    768/954/968        1658/1732/1948      670/1026/1099       79/74/81 (840,094)
//   1,000,000  1102/1387/1415     2345/2505/2841      953/1488/1609       87/95/122 (1,396,802)
// and without boundary samples 11/29/52/97/187 for the boundary pass of 1,000,000.
// In 2-D: 10,000 fluid particles density 23/13/11/13/15, forces 33/17/15/17/23,
// boundary 15/9/8/9/9 (10,680 slots); 40,000 25/19/19/25/35, 40/30/33/39/64, 15/11/9/11/13;
// 160,000 50/52/59/80/131, 86/93/113/148/259, 17/13/15/20/31; 490,000 boundary 19/22/31/52/94.
inline PassLanes pass_lanes(int dim, uint64_t fluid, uint64_t slots) {
    struct Limits {
        uint64_t l32, l16, l8, l4;  // the most slots each lane count is taken for
    };
    const auto pick = [](uint64_t n, const Limits& m) -> uint32_t {
        return n <= m.l32 ? 32u : n <= m.l16 ? 16u : n <= m.l8 ? 8u : n <= m.l4 ? 4u : 1u;
    };
    const bool d3 = dim == 3;
    const uint64_t most = 48000000;
    PassLanes r;
    r.density = fit_lanes(pick(fluid, d3 ? Limits{3000, 10000, 158000, 158000} : Limits{600, 10000, 40000, 100000}), slots, most);
    r.forces = fit_lanes(pick(fluid, d3 ? Limits{8000, 20000, 64000, 600000} : Limits{1000, 3000, 12000, 80000}), slots, most);
    r.xsph = fit_lanes(pick(fluid, d3 ? Limits{1500, 10000, 45000, 45000} : Limits{1000, 3000, 12000, 25000}), slots, most);
    r.boundary = fluid == slots ? 1u : fit_lanes(32u, slots, d3 ? 16000000 : 4000000);
    return r;
}

// Single-precision passes. One lane a particle streams its rows best once the
// particles alone fill the chip; below that the walk of one list is the pass's
// length, and 8 lanes (32 for the smallest scenes) shorten it. us a pass, 1 / 8 / 32
// lanes (four were slower than one or eight at every size):
//   fluid       density          forces           XSPH
//         216   56 / 21 / 13     101 / 31 / 20    51 / 21 / 16
//       2,197   62 / 22 / 18     112 / 32 / 27    61 / 22 / 20
//       6,859   64 / 28 / 30     112 / 40 / 40    64 / 26 / 31
//      32,768   73 / 62 / 100    132 / 83 / 119   74 / 56 / 94
//      68,921   91 / 110 / 198   171 / 144 / 228  100 / 98 / 181
//      79,507   99 / 126         194 / 163        102 / 111
//     125,000   134 / 186 / 351  250 / 242 / 401  111 / 161 / 320
//     157,464   167 / 230        299 / 298        181 / 197
//     195,112   183 / 281        330 / 363        187 / 239
//   2-D   900   17 / 10 / 9      33 / 18 / 14     18 / 12 / 13
//       6,400   18 / 11 / 13     34 / 18 / 22     21 / 13 / 17
//      32,400   19 / 18          35 / 28          21 / 20
//      48,400   19 / 23          37 / 35          23 / 24
//      90,000   23 / 35          43 / 50          24 / 36
//   2,197 among 540,002 boundary samples: 63 / 27 / 76, 112 / 40 / 89, 73 / 48 / 153;
//   15,625 among 1,100,002: 79 / 58, 154 / 83, 89 / 103
inline PassLanes pass_lanes_f32(int dim, uint64_t fluid, uint64_t slots) {
    const bool d2 = dim == 2;
    const uint64_t few = d2 ? 2048 : 4096;
    const auto rule = [&](uint64_t eight, uint64_t most) {
        return fit_lanes(fluid <= few ? 32u : fluid <= eight ? 8u : 1u, slots, most, true);
    };
    PassLanes r;
    r.density = rule(d2 ? 32768 : 49152, 100000000);
    r.forces = rule(d2 ? 65536 : 150000, 100000000);
    r.xsph = rule(d2 ? 40960 : 70000, 48000000);
    return r;
}

// PBF's constraint passes, 1 or 8 lanes on a list of ~33 entries, shared out while the
// slots do not fill the chip. ms for ten steps with 1 / 8 lanes: 6^3 fluid particles
// 3.7 / 2.4, 20^3 5.4 / 4.1, 30^3 6.0 / 5.3, 40^3 7.4 / 7.5, 50^3 11.4 / 11.7, 70^3
// 25.4 / 29.2; three steps of 2,197 particles among 60,002 boundary samples 1.17 /
// 0.79, among 540,002 2.74 / 2.96, of 27,000 among 540,002 3.03 / 3.40.
inline uint32_t pbf_lanes(uint64_t fluid, uint64_t slots) {
    return fit_lanes(fluid <= 48000 ? 8u : 1u, slots, 16000000, true);
}

// DFSPH's pair passes, 1, 8 or 32 lanes: many while the slots do not fill the chip,
// one where they do. ms for two steps with 1 / 8 / 32 lanes a fluid slot: 16^3 fluid
// particles 15.0 / 4.2 / 2.7, 36^3 24.1 / 13.0 / 14.1, 64^3 50.9 / 52.1 / 65.9, 90^3
// 102 / 130 / 172; for three steps of 2,197 particles among 60,002 boundary samples
// 8.9 / 2.4 / 1.7, among 540,002 12.1 / 4.5 / 7.9, of 27,000 among 18,358 16.6 / 5.6 /
// 6.0, among 540,002 18.4 / 7.5 / 14.9. The boundary slots' lists are few and long
// (all candidates of the cells), so these take more: 36^3 20.6 / 12.4 / 11.5, 64^3
// 49.9 / 42.0 / 42.6.
inline uint32_t dfsph_lanes(uint64_t fluid, uint64_t slots) {
    return fit_lanes(fluid <= 20000 ? 32u : fluid <= 230000 ? 8u : 1u, slots, 100000000, true);
}
inline uint32_t dfsph_boundary_lanes(uint64_t fluid, uint64_t slots) {
    return fluid == slots ? 1u : fit_lanes(fluid <= 150000 ? 32u : 8u, slots, 100000000, true);
}

}  // namespace pe
