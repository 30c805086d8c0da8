// Host harness of the PNG chunk checksum (test infrastructure).
//
// Compiles rohditor_gb300/csrc/deflate.cuh for the CPU and checksums bytes the way
// png_chunk_kernel does, its 256 threads played one after another: the same
// shares, four-byte steps and tree of advances within and across warps.
//
//   crc_host FILE LEN...   prints the CRC-32 of FILE's first LEN bytes, per LEN
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../rohditor_gb300/csrc/deflate.cuh"

using namespace rd::png;

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  std::FILE* f = std::fopen(argv[1], "rb");
  if (!f) return 2;
  std::vector<uint8_t> data(SEG_CAP + 64);
  data.resize(std::fread(data.data(), 1, data.size(), f));
  std::fclose(f);
  static uint32_t table[4][256];
  for (uint32_t v = 0; v < 256; ++v) table[0][v] = crc_byte_entry(v);
  for (int k = 1; k < 4; ++k)
    for (uint32_t v = 0; v < 256; ++v) table[k][v] = crc_zero_bytes(table[0], table[0][v], k);
  static constexpr CrcTree tree = crc_tree();
  for (int a = 2; a < argc; ++a) {
    const int len = std::atoi(argv[a]);
    if (len < 1 || (size_t)len > data.size()) return 2;
    uint32_t reg[CRC_SHARES];
    for (int t = 0; t < CRC_SHARES; ++t)
      reg[t] = crc_share(table, len, t, [&](int k) { return (uint32_t)data[k]; },
                         [&](int k) {
                           return (uint32_t)data[k] | (uint32_t)data[k + 1] << 8 | (uint32_t)data[k + 2] << 16 |
                                  (uint32_t)data[k + 3] << 24;
                         });
    // A lane takes the register 2^j lanes below it, its own where there is none (a shuffle up).
    auto level = [&](uint32_t* lanes, int n, int distance, const uint32_t (&t)[8][16]) {
      for (int l = n - 1; l >= 0; --l)
        lanes[l] = crc_advance(t, lanes[l >= distance ? l - distance : l]) ^ lanes[l];
    };
    uint32_t warp[CRC_SHARES / 32];
    for (int w = 0; w < CRC_SHARES / 32; ++w) {
      for (int j = 0; j < 5; ++j) level(reg + 32 * w, 32, 1 << j, tree.t[j]);
      warp[w] = reg[32 * w + 31];
    }
    for (int j = 0; j < 3; ++j) level(warp, CRC_SHARES / 32, 1 << j, tree.t[5 + j]);
    std::printf("%u\n", warp[CRC_SHARES / 32 - 1] ^ 0xFFFFFFFFu);
  }
  return 0;
}
