// Tiles of one window DFT launch over up to WIN_MAX_SIZES mask sizes: per size an extent that
// its splits share out in chunks, the blocks across it, the splits, the first image in the
// shared partial array and the first tile; tiles are numbered size after size, then image, block
// and split.  (imaging_fold.cu: the extent is the base rows, a chunk one of them, and the blocks
// are column blocks.)  Plain C++ (host and device), so the numbering is also checked on the CPU.
#pragma once

#ifdef __CUDACC__
#define LITHO_WT_HD __host__ __device__
#else
#define LITHO_WT_HD
#endif

namespace litho {

constexpr int WIN_MAX_SIZES = 4;  // mask sizes one window launch takes

struct WinTiles {
  int n;                              // mask sizes
  int Lx[WIN_MAX_SIZES];              // extent
  int rows[WIN_MAX_SIZES];            // blocks
  int ncs[WIN_MAX_SIZES];             // splits
  int img0[WIN_MAX_SIZES];            // first image in the partial array
  int tile0[WIN_MAX_SIZES + 1];       // first tile (tile0[n]: all tiles)
};

// tile t -> (size g, image, block, split) and its range [c0, c1) of chunks of `chunk`
LITHO_WT_HD inline void win_tile(const WinTiles& T, int t, int chunk, int& g, int& img, int& rb, int& cs, int& c0,
                                 int& c1) {
  g = 0;
  while (g + 1 < T.n && t >= T.tile0[g + 1]) ++g;
  const int l = t - T.tile0[g], rows = T.rows[g], ncs = T.ncs[g];
  const int nch = (T.Lx[g] + chunk - 1) / chunk;
  img = l / (rows * ncs);
  const int r = l - img * rows * ncs;
  rb = r / ncs;
  cs = r - rb * ncs;
  c0 = (int)((long long)nch * cs / ncs);
  c1 = (int)((long long)nch * (cs + 1) / ncs);
}

}  // namespace litho
