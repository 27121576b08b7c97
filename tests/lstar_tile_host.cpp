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

// The conforming re-pairing: rlab holds the restriction label of every cell.  Returns the
// number of re-paired vertices.
extern "C" int64_t tile_conform(const float* f, int64_t X, int64_t Y, int64_t Z, const uint8_t* rlab, uint8_t* g,
                                uint32_t enc_map) {
  using T = msc::LstarTile<3>;
  using N = msc::Nb<3>;
  const int64_t v[3] = {X, Y, Z}, d[3] = {2 * X - 1, 2 * Y - 1, 2 * Z - 1};
  int16_t off[N::NPOS];
  for (int p = 0; p < N::NPOS; p++) off[p] = (int16_t)T::off(p);
  int64_t touched = 0;
  for (int64_t z0 = 0; z0 < Z; z0 += T::BZ)
    for (int64_t y0 = 0; y0 < Y; y0 += T::BY)
      for (int64_t x0 = 0; x0 < X; x0 += T::BX) {
        std::vector<float> sf(T::NF, 0.f);
        std::vector<msc::LatKey> lat(T::NL);
        std::vector<uint8_t> bytes(T::NL, 0xEE);
        for (int i = 0; i < T::NF; i++) {
          const int64_t x = x0 - 1 + i % T::FX, y = y0 - 1 + (i / T::FX) % T::FY, z = z0 - 1 + i / (T::FX * T::FY);
          if (x >= 0 && x < X && y >= 0 && y < Y && z >= 0 && z < Z) sf[i] = msc::plain_zero(f[x + X * (y + Y * z)]);
        }
        for (int z = -1; z < T::BZ; z++)
          for (int y = -1; y < T::BY; y++)
            for (int x = -1; x < T::BX; x++) {
              msc::tile_cell_keys<3>(sf.data(), lat.data(), x, y, z);
              uint32_t word = 0;
              if (x0 + x >= 0 && y0 + y >= 0 && z0 + z >= 0)
                for (int s = 0; s < 8; s++) {
                  const int64_t c[3] = {2 * (x0 + x) + (s & 1), 2 * (y0 + y) + ((s >> 1) & 1), 2 * (z0 + z) + (s >> 2)};
                  if (c[0] >= d[0] || c[1] >= d[1] || c[2] >= d[2]) continue;
                  const uint32_t r = rlab[c[0] + d[0] * (c[1] + d[1] * c[2])];
                  word |= (r & 1u) << s | (r >> 1) << (8 + s);
                }
              msc::tile_restrict(word, bytes.data(), x, y, z);
            }
        const bool rim = x0 == 0 || y0 == 0 || z0 == 0 || x0 + T::BX >= X || y0 + T::BY >= Y || z0 + T::BZ >= Z;
        for (int t = 0; t < T::NV; t++) {
          int x, y, z;
          T::vertex(t, x, y, z);
          if (x0 + x >= X || y0 + y >= Y || z0 + z >= Z) continue;
          uint32_t lower = msc::tile_lower_mask<3>(sf.data(), x, y, z), r1, r2;
          if (rim) lower &= msc::inside_mask<3>(x0 + x, y0 + y, z0 + z, v);
          const uint32_t L = msc::lower_star_mask<3>(lower);
          if (!msc::tile_labels(L, t, bytes.data(), off, r1, r2)) continue;
          touched++;
          msc::tile_expand_restricted(L, r1, r2, t, rim, x0 + x, y0 + y, z0 + z, v, lat.data(), bytes.data(), off,
                                      enc_map);
        }
        for (int i = 0; i < T::NL; i++)
          if (bytes[i] & 1)
            g[(2 * x0 - 1 + i % T::LX) + (2 * y0 - 1 + (i / T::LX) % T::LY) * d[0] +
              (2 * z0 - 1 + i / (T::LX * T::LY)) * d[0] * d[1]] = bytes[i];
      }
  return touched;
}
