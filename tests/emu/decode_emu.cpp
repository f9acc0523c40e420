// Runs the zstd decoder's kernels under the CPU SIMT emulation on a call of
// several launch sets -- TEST INFRASTRUCTURE ONLY.  Built with small limits
// (CHUCKY_ZSTD_SCRATCH, CHUCKY_ZSTD_FRAMES) by tests/test_decode_emu.py.
//
// usage: decode_emu <chunk_bytes> <n_chunks> <seed>
// Frames of the stock libzstd at several levels; every fifth chunk is one that
// the block-parallel decoder leaves: two frames, a skippable one in front, cut
// short, a byte too long.  Prints the number of kernels launched.
#include "simt.hpp"

#include "../../chucky_gb300/csrc/zstd_decode.cu"

#include <dlfcn.h>

static unsigned launches;
namespace chucky {
void note_launches(unsigned n) { launches += n; }
int device_sm_count() { return 152; }
} // namespace chucky

static uint64_t rng_state;
static uint32_t rnd()
{
  rng_state = rng_state * 6364136223846793005ull + 1442695040888963407ull;
  return uint32_t(rng_state >> 33);
}

int main(int argc, char** argv)
{
  if (argc != 4)
    return 2;
  const size_t chunk = std::stoul(argv[1]), n = std::stoul(argv[2]);
  rng_state = std::stoull(argv[3]);
  void* z = dlopen("libzstd.so.1", RTLD_NOW);
  if (!z)
    return 3;
  auto zc = (size_t(*)(void*, size_t, const void*, size_t, int))dlsym(z, "ZSTD_compress");
  auto zb = (size_t(*)(size_t))dlsym(z, "ZSTD_compressBound");
  auto ze = (unsigned (*)(size_t))dlsym(z, "ZSTD_isError");
  std::vector<uint8_t> raw(n * chunk), in;
  std::vector<uint64_t> off, size;
  std::vector<uint32_t> want;
  auto frame = [&](const uint8_t* p, size_t k, int level) {
    std::vector<uint8_t> b(zb(k));
    const size_t got = zc(b.data(), b.size(), p, k, level);
    if (ze(got))
      std::exit(3);
    b.resize(got);
    return b;
  };
  for (size_t c = 0; c < n; ++c) {
    uint8_t* p = raw.data() + c * chunk;
    for (size_t i = 0; i < chunk; ++i) // words, noise, runs, few values
      switch (c % 4) {
        case 0: p[i] = uint8_t('a' + (i < 40 ? rnd() % 26 : p[i - 1 - rnd() % 2 * 7 - i / 9 % 30] - 'a')); break;
        case 1: p[i] = uint8_t(rnd()); break;
        case 2: p[i] = uint8_t(i / 50 % 7); break;
        default: p[i] = uint8_t(rnd() % 9 + rnd() % 9); break;
      }
    std::vector<uint8_t> b = frame(p, chunk, c % 3 == 0 ? 1 : c % 3 == 1 ? 5 : 19);
    uint32_t st = 0;
    if (c % 5 == 2)
      switch (c / 5 % 4) {
        case 0: { // two frames
          b = frame(p, chunk / 3, 3);
          const auto more = frame(p + chunk / 3, chunk - chunk / 3, 3);
          b.insert(b.end(), more.begin(), more.end());
          break;
        }
        case 1: { // a skippable frame in front
          const uint8_t skip[] = { 0x53, 0x2A, 0x4D, 0x18, 3, 0, 0, 0, 1, 2, 3 };
          b.insert(b.begin(), skip, skip + sizeof skip);
          break;
        }
        case 2:
          b.resize(b.size() - 1);
          st = 1;
          break;
        default:
          b.push_back(0);
          st = 1;
          break;
      }
    off.push_back(in.size());
    size.push_back(b.size());
    want.push_back(st);
    in.insert(in.end(), b.begin(), b.end());
  }
  const size_t stride = chunk + 5;
  std::vector<uint8_t> out(n * stride, 0xA5);
  std::vector<uint32_t> status(n, 99);
  if (chucky::launch_zstd_decode(in.data(), off.data(), size.data(), n, out.data(), stride, chunk,
                                 status.data(), nullptr) != cudaSuccess)
    return 1;
  for (size_t c = 0; c < n; ++c) {
    const bool bytes = std::memcmp(out.data() + c * stride, raw.data() + c * chunk, chunk) == 0;
    bool past = false;
    for (size_t i = chunk; i < stride; ++i)
      past |= out[c * stride + i] != 0xA5;
    if ((want[c] == 0) != (status[c] == 0) || (want[c] == 0 && !bytes) || past) {
      std::fprintf(stderr, "chunk %zu: status %u, bytes %s\n", c, status[c],
                   past ? "past its end" : bytes ? "right" : "wrong");
      return 1;
    }
  }
  std::printf("ok %u\n", launches);
  return 0;
}
