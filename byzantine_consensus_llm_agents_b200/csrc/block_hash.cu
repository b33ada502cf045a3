// Hash chain over a prompt's full token blocks, on the host: hash of a block = BLAKE2b (RFC 7693, 16-byte digest) of the previous
// block's hash followed by the block's tokens, little endian.  64 prompts of 900 tokens are 3,600 blocks per call; hashed one
// by one from Python they kept the GPU waiting for 5 ms, packed and hashed here for 2.
#include <string.h>

#include "common.cuh"
#include "kernels.h"

namespace bcg {

static const uint64_t kIv[8] = {0x6a09e667f3bcc908ull, 0xbb67ae8584caa73bull, 0x3c6ef372fe94f82bull, 0xa54ff53a5f1d36f1ull,
                                0x510e527fade682d1ull, 0x9b05688c2b3e6c1full, 0x1f83d9abfb41bd6bull, 0x5be0cd19137e2179ull};
static const uint8_t kSigma[10][16] = {
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
    {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
    {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
    {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
    {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0}};

static inline uint64_t rotr(uint64_t x, int n) { return x >> n | x << (64 - n); }
static inline void mix(uint64_t& a, uint64_t& b, uint64_t& c, uint64_t& d, uint64_t x, uint64_t y) {
  a += b + x;
  d = rotr(d ^ a, 32);
  c += d;
  b = rotr(b ^ c, 24);
  a += b + y;
  d = rotr(d ^ a, 16);
  c += d;
  b = rotr(b ^ c, 63);
}
// The only, and therefore last, input block of a message of `count` bytes
static void compress(uint64_t (&h)[8], const uint8_t* block, uint64_t count) {
  uint64_t v[16], m[16];
  memcpy(m, block, 128);
  for (int i = 0; i < 8; ++i) {
    v[i] = h[i];
    v[i + 8] = kIv[i];
  }
  v[12] ^= count;
  v[14] = ~v[14];
  for (int r = 0; r < 12; ++r) {
    const uint8_t* s = kSigma[r % 10];
    mix(v[0], v[4], v[8], v[12], m[s[0]], m[s[1]]);
    mix(v[1], v[5], v[9], v[13], m[s[2]], m[s[3]]);
    mix(v[2], v[6], v[10], v[14], m[s[4]], m[s[5]]);
    mix(v[3], v[7], v[11], v[15], m[s[6]], m[s[7]]);
    mix(v[0], v[5], v[10], v[15], m[s[8]], m[s[9]]);
    mix(v[1], v[6], v[11], v[12], m[s[10]], m[s[11]]);
    mix(v[2], v[7], v[8], v[13], m[s[12]], m[s[13]]);
    mix(v[3], v[4], v[9], v[14], m[s[14]], m[s[15]]);
  }
  for (int i = 0; i < 8; ++i) h[i] ^= v[i] ^ v[i + 8];
}

int block_hashes(const int* tokens, int n_blocks, int block, unsigned char* out) {
  // a block's tokens and the hash in front of them are one input block of BLAKE2b
  if (n_blocks < 0 || block <= 0 || 16 + 4 * static_cast<long long>(block) > 128 || (n_blocks > 0 && (!tokens || !out))) {
    set_last_error("bcg_block_hashes", "null pointer, or not 1 to 28 tokens per block");
    return BCG_ERR_ARG;
  }
  uint8_t in[128];
  memset(in, 0, sizeof(in));
  for (int i = 0; i < n_blocks; ++i) {
    memcpy(in + 16, tokens + static_cast<size_t>(i) * block, 4 * static_cast<size_t>(block));
    uint64_t h[8];
    for (int k = 0; k < 8; ++k) h[k] = kIv[k];
    h[0] ^= 0x01010000ull ^ 16u;     // no key, 16 bytes of digest
    compress(h, in, static_cast<uint64_t>(16 + 4 * block));
    memcpy(in, h, 16);
    memcpy(out + static_cast<size_t>(i) * 16, h, 16);
  }
  return BCG_OK;
}

}  // namespace bcg
