// Host build of the lower-star tile (msceer_gb300/csrc/lstar_tile.cuh) for the CPU tests:
// the phases the kernel runs with a block, run here by one thread over every tile of a
// volume, with the arrays at exactly their sizes.
#include <cstdint>
#include <vector>

#include "../msceer_gb300/csrc/lstar_tile.cuh"

template <int ND>
static void run(const float* f, const int64_t v[3], uint8_t* g, uint32_t enc_map) {
  using T = msc::LstarTile<ND>;
  using N = msc::Nb<ND>;
  const int64_t cs1 = 2 * v[0] - 1, cs2 = cs1 * (2 * v[1] - 1);
  int16_t off[N::NPOS];
  for (int p = 0; p < N::NPOS; p++) off[p] = (int16_t)T::off(p);
  for (int64_t z0 = 0; z0 < v[2]; z0 += T::BZ)
    for (int64_t y0 = 0; y0 < v[1]; y0 += T::BY)
      for (int64_t x0 = 0; x0 < v[0]; x0 += T::BX) {
        std::vector<float> sf(T::NF, 0.f);
        std::vector<msc::LatKey> lat(T::NL);
        std::vector<uint8_t> bytes(T::NL, 0);
        for (int i = 0; i < T::NF; i++) {
          const int64_t x = x0 - 1 + i % T::FX, y = y0 - 1 + (i / T::FX) % T::FY,
                        z = ND == 3 ? z0 - 1 + i / (T::FX * T::FY) : 0;
          if (x >= 0 && x < v[0] && y >= 0 && y < v[1] && z >= 0 && z < v[2])
            sf[i] = msc::plain_zero(f[x + v[0] * (y + v[1] * z)]);
        }
        for (int z = ND == 3 ? -1 : 0; z < T::BZ; z++)
          for (int y = -1; y < T::BY; y++)
            for (int x = -1; x < T::BX; x++) msc::tile_cell_keys<ND>(sf.data(), lat.data(), x, y, z);
        const bool rim = x0 == 0 || y0 == 0 || x0 + T::BX >= v[0] || y0 + T::BY >= v[1] ||
                         (ND == 3 && (z0 == 0 || z0 + T::BZ >= v[2]));
        for (int t = 0; t < T::NV; t++) {
          int x, y, z;
          T::vertex(t, x, y, z);
          if (x0 + x >= v[0] || y0 + y >= v[1] || z0 + z >= v[2]) continue;
          uint32_t lower = msc::tile_lower_mask<ND>(sf.data(), x, y, z);
          if (rim) lower &= msc::inside_mask<ND>(x0 + x, y0 + y, z0 + z, v);
          msc::tile_expand<ND>(msc::lower_star_mask<ND>(lower), t, rim, x0 + x, y0 + y, z0 + z, v, lat.data(),
                               bytes.data(), off, enc_map);
        }
        for (int i = 0; i < T::NL; i++)
          if (bytes[i])
            g[(2 * x0 - 1 + i % T::LX) + (2 * y0 - 1 + (i / T::LX) % T::LY) * cs1 +
              (ND == 3 ? 2 * z0 - 1 + i / (T::LX * T::LY) : 0) * cs2] = bytes[i];
      }
}

extern "C" void tile_pairs(int nd, const float* f, int64_t X, int64_t Y, int64_t Z, uint8_t* g, uint32_t enc_map) {
  const int64_t v[3] = {X, Y, Z};
  if (nd == 3) run<3>(f, v, g, enc_map); else run<2>(f, v, g, enc_map);
}
