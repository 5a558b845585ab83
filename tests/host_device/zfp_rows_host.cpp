// The device ZFP codec as a host program, for the address sanitizer: random blocks
// whose bits run out, at every rate, coded by zfp_encode_block and decoded from
// words with no more room behind them than zfp_decode_staged asks for.
#include "cuda_host_shim.h"
#include "zfp_device.cuh"

#include <stdio.h>

#include <memory>
#include <random>

int main()
{
    std::mt19937 gen(7);
    // either sign, nearly the same size: the bits run out at every rate, though at 32
    // in one block of ten thousand only
    std::uniform_real_distribution<float> value(1.0f - 1.0f / 128.0f, 1.0f);
    for (uint32_t rate = 1; rate <= 32; ++rate)
        for (int b = 0; b < (rate == 32 ? 100000 : 1000); ++b) {
            float f[64], out[64];
            for (float& x : f) x = gen() & 1u ? value(gen) : -value(gen);
            std::unique_ptr<unsigned long long[]> words(new unsigned long long[rate]());
            bcmc::BitWriter bw;
            bw.init(words.get(), 0);
            bcmc::zfp_encode_block(f, 64u * rate, bw);
            bw.finish();
            std::unique_ptr<uint32_t[]> w(new uint32_t[2u * rate + 3u]());
            memcpy(w.get(), words.get(), 8u * rate);
            alignas(16) uint32_t pl[64];
            bcmc::zfp_decode_staged(w.get(), 64u * rate, pl, out);
            for (int i = 0; rate >= 16 && i < 64; ++i)
                if (!(fabsf(out[i] - f[i]) < 1e-2f)) {
                    printf("rate %u: %g for %g\n", rate, out[i], f[i]);
                    return 1;
                }
        }
    return 0;
}
