// Over how many CTAs of a thread-block cluster K is split: by the kernels with the weights on the M side (gemm_rows.cu,
// gemm_small.cu) and by the 128-row kernel (gemm.cu).  Plain C++ without CUDA: what a GPU holds comes in as counts, so that the rules can be tested for any.
#pragma once
#include <stdint.h>

namespace sglb200 {

constexpr int kMostClusterCtas = 16;

// Clusters of s CTAs that a GPU holds at once: with one CTA on an SM, and with two on every SM.
struct ClusterFits {
  int64_t alone[kMostClusterCtas + 1], paired[kMostClusterCtas + 1];
};

// `ask(s, per_sm)` is the driver's answer for s CTAs with `per_sm` of them on an SM; 0 or less: it refuses or does not say,
// and then eight CTAs or fewer (the portable sizes) are taken to fit everywhere and more not at all.  A cluster stays within
// a GPC, whose number of SMs differs from GPC to GPC and from GPU to GPU, and the count for two an SM does not follow from
// the one for one: a B200 holds 148 74 45 33 26 22 15 15 15 11 7 7 7 7 7 7 clusters of 1 to 16 CTAs alone and 296 148 93 71
// 56 45 37 33 30 26 21 21 17 14 14 14 paired.  Counted as those of half the size (74 of four, 22 of twelve, 15 of sixteen), a
// few clusters had to wait for the others to end: with 64 rows, 9344 x 9600 32.5 us and now 27.0, 2816 x 16768 25.0 and 17.3;
// one row, 1920 x 9984 12.7 and 9.0.  For odd sizes twice the count for one an SM is kept where it is the smaller: in several
// rounds they fall behind what the larger one promises (23680 x 4352 with 55 rows: three CTAs in two rounds 33.5 us, one
// 23.7).
template <class Ask>
inline ClusterFits cluster_fits_of(const Ask& ask, int64_t sms) {
  ClusterFits f{};
  f.alone[1] = sms, f.paired[1] = 2 * sms;
  for (int s = 2; s <= kMostClusterCtas; ++s) {
    int64_t a = ask(s, 1), b = ask(s, 2);
    if (a <= 0) a = s <= 8 ? sms / s : 0;
    if (b <= 0) b = s <= 8 ? 2 * sms / s : 0;
    if (a == 0) b = 0;
    f.alone[s] = a;
    f.paired[s] = s % 2 != 0 && b > 2 * a ? 2 * a : b;
  }
  return f;
}

// CTAs per cluster for a dense problem of `tiles` tiles and `kb` slabs: the split that finishes first, counted in
// quarters of the time of a slab in a CTA that has an SM to itself (0.41 us with 64 rows).  A CTA's start and end are three
// slabs and the exchange of a cluster two more.  Where CTAs share SMs a slab takes 7/4 and start, end and exchange a little
// longer (a cluster or two too many for one CTA an SM still count as alone); clusters beyond what two CTAs an SM hold
// wait for a whole round.
// Measured with 64 rows over splits of 1 to 8: 4096 x 4096 four CTAs 10.0 us, eight (sharing SMs) 10.9; K 7168 with N 2112
// six 10.7, eight 11.0; 4096 x 14336 eight 16.1, four 18.1; 10240 x 8192 three 19.8, two 23.4, four 26.8 (a second round);
// 4616 x 1920 three 9.0, eight 14.1 (296 CTAs, but 37 clusters of eight do not fit); 14944 x 768 one 7.2, two 8.8.  More than
// eight CTAs, for few tiles and a long K: 512 x 8192 sixteen 8.6, eight 9.5; 768 x 18432 sixteen 11.1, eight 14.0; 1024 x
// 8192 ten 9.6, eight 9.9, sixteen 10.8; where that gains no whole slab, eight (1536 x 7168 with 20 rows eight 7.3, nine
// 7.5).  With up to 32 rows, whose partial sums are not pushed, they have to gain more than one (32 rows: 1280 x 5120 eight
// 7.0, ten 7.2; 576 x 7168 eight 7.4, fourteen 7.2; 640 x 12288 eight 8.6, sixteen 7.8).  Both hold where CTAs share SMs as well
// (64 rows: 19200 x 16128 five CTAs 68.2, nine 80.7; 3840 x 4352 four 11.5, nine 12.3; 3200 x 9856 five 14.4, ten 15.5; 32
// rows: 2560 x 13696 six 12.6, twelve 13.2), but for even clusters with 33 to 48 rows, which exchange less (35 rows: 3072 x
// 10240 five 13.9, ten 13.3; 39 rows: 2688 x 12288 six 14.1, twelve 13.7).  Still the better ones: ten for 3072 x 14720 with
// 52 rows (16.7, five 17.2) and 3072 x 10240 with 49 (13.7, five 14.1).
inline int rows_splits(int64_t tiles, int kb, int64_t rows, const ClusterFits& fits) {
  const int large = rows > 32 ? 1 : 5;  // (more than 32 rows: partial sums are pushed)
  int best = 1;
  int64_t best_cost = -1;
  for (int s = 1; s <= kMostClusterCtas && s <= kb; ++s) {
    const int64_t per = (kb + s - 1) / s, spread = fits.alone[s], fit = fits.paired[s];
    if (fit == 0) continue;
    const int64_t rounds = (tiles + fit - 1) / fit;
    const bool alone = tiles <= (s == 1 ? spread : spread + spread / 16);
    const bool charged = s > 8 && (alone || s % 2 != 0 || rows <= 32 || rows > 48);
    const int64_t cost = s == 1 ? rounds * per * (alone ? 4 : 7) + 12
                                : (alone ? 4 * per + 20 : rounds * (7 * per + (s > 4 ? 28 : 22))) + (charged ? large : 0);
    if (best_cost < 0 || cost <= best_cost) best = s, best_cost = cost;
  }
  return best;
}

// The same for the one-launch linear, whose CTAs hold all their slabs (at most `most_slabs`) at once, two CTAs an SM, and
// whose clusters all run at once; 0 = there is none.  The cheapest, in hundredths of a microsecond: 45 for a slab of a CTA,
// one for a CTA of the grid (they share the SMs, the L2 and the launch), 60 for a CTA without a cluster, 20 for an odd
// cluster (half of a pair of SMs idles), 15 for a cluster of more than eight and ten for each of its CTAs beyond the eighth.
// Measured with 16 rows over all splits: 512 x 512 one CTA 5.2 us, four 3.6; 4096 x 1024 two 5.3, four 4.8, eight 6.1;
// 7168 x 2048 three 8.0, four 6.9, five 8.2; 2048 x 2048 four 5.0, eight 4.8; 1024 x 8192 eleven 7.1, sixteen 5.8; 4368 x 4352
// six 8.7, eight 12.8 (35 clusters of eight do not fit), quantised in a launch of its own 10.6.
inline int small_splits(int64_t tiles, int kb, int most_slabs, const ClusterFits& fits) {
  int best = 0;
  int64_t best_cost = -1;
  for (int s = 1; s <= kMostClusterCtas && s <= kb; ++s) {
    const int slabs = (kb + s - 1) / s;
    if (slabs > most_slabs || tiles > fits.paired[s]) continue;
    const int64_t cost = 45 * slabs + tiles * s + (s == 1 ? 60 : s % 2 != 0 ? 20 : 0) + (s > 8 ? 15 + 10 * (s - 8) : 0);
    if (best_cost < 0 || cost < best_cost) best = s, best_cost = cost;
  }
  return best;
}

// The same for the 128-row kernel, one CTA an SM, on `tiles` tiles of 128 x 128: 1, or two, three, four, six or eight CTAs (what
// five and seven would have to exchange does not fit beside their operands).  Counted in slabs (0.25 us): the exchange is six and one
// for every 32 rows of a tile, and one for every 48 CTAs of the grid, which share DRAM and L2.  Measured over all of them, us of the
// layer: 128 x 4096 x 7168 one 20.6, two 16.1, three 15.4, four 14.2; 128 x 1536 x 16384 four 17.4, six 16.9, eight 15.0; 80 x 2048 x
// 7168 four 12.0, six 11.5; 80 x 4096 x 2048 one 10.4, two 9.8, four 9.7; 128 x 4096 x 2048 one 10.6, two 10.5, four 10.9; 128 x 7168 x
// 2048 one 10.9, two 11.1; 192 x 4096 x 1024 one 8.6, two 9.7; 128 x 9216 x 4096 one 15.1, two 15.1.
inline int tile_splits(int64_t tiles, int kb, int64_t rows, const ClusterFits& fits) {
  const int exchange = 6 + (int)((rows < 128 ? rows + 31 : 128) / 32);
  int best = 1;
  int64_t best_cost = kb;
  for (int s = 2; s <= 8; ++s) {
    if (s == 5 || s == 7 || s > kb || tiles > fits.alone[s]) continue;
    const int64_t cost = (kb + s - 1) / s + exchange + tiles * s / 48;
    if (cost < best_cost) best = s, best_cost = cost;
  }
  return best;
}

}  // namespace sglb200
