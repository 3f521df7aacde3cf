// Hand-over words of the kernel on pairs of SMs (q8_pair.cu), from a program that has the scratch itself: whatever way
// cut tiles are finished, every word is zero after the launch, no status bit is set, and launches that follow right
// behind, or run beside those of another stream, give the same bits.
//
// Prints "pass" at the end; exits 1 on the first failure.
#include <cuda_fp16.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "q8_launch.h"
#include "q8_schedule.cuh"
#include "q8_tile.cuh"

#define CHECK_CUDA(call)                                                                       \
    do {                                                                                       \
        cudaError_t err_ = (call);                                                             \
        if (err_ != cudaSuccess) {                                                             \
            std::fprintf(stderr, "%s: %s\n", #call, cudaGetErrorString(err_));                 \
            std::exit(1);                                                                      \
        }                                                                                      \
    } while (0)

static uint32_t next_random(uint32_t &state)
{
    state = state * 1664525u + 1013904223u;
    return state >> 8;
}

template <typename T>
static T *on_device(const std::vector<T> &from)
{
    T *to = nullptr;
    CHECK_CUDA(cudaMalloc(&to, from.size() * sizeof(T)));
    CHECK_CUDA(cudaMemcpy(to, from.data(), from.size() * sizeof(T), cudaMemcpyHostToDevice));
    return to;
}

// The scratch of a context, as aotx_q8_init makes it: two sets that launches take in turn.
struct Scratch {
    q8::UmmaScratch use = {};
    unsigned int words;

    explicit Scratch(unsigned int sm_count)
    {
        use.blocks = 2u * sm_count;
        use.tile_floats = 128ull * 256ull;
        words = 2u * use.blocks * q8::kFlagWords + 1u;
        CHECK_CUDA(cudaMalloc(&use.partial, 2ull * use.blocks * use.tile_floats * sizeof(float)));
        CHECK_CUDA(cudaMalloc(&use.flags, words * sizeof(unsigned int)));
        CHECK_CUDA(cudaMemset(use.flags, 0, words * sizeof(unsigned int)));
        use.status = use.flags + words - 1u;
    }
    Scratch(const Scratch &) = delete;
    ~Scratch()
    {
        cudaFree(use.partial);
        cudaFree(use.flags);
    }
    bool all_zero() const
    {
        std::vector<unsigned int> now(words);
        CHECK_CUDA(cudaMemcpy(now.data(), use.flags, words * sizeof(unsigned int), cudaMemcpyDeviceToHost));
        for (unsigned int i = 0; i < words; ++i) {
            if (now[i] != 0u) {
                std::printf("word %u of %u is %u\n", i, words, now[i]);
                return false;
            }
        }
        return true;
    }
};

struct Product {
    unsigned int n, k, m;
    unsigned char *w;
    __half *x;
    unsigned int *live;
    float *y;

    Product(unsigned int n_, unsigned int k_, unsigned int m_, unsigned int live_) : n(n_), k(k_), m(m_)
    {
        uint32_t state = n + m;
        std::vector<unsigned char> rows((size_t)n * (k / 32u) * 34u);
        for (size_t at = 0; at < rows.size(); at += 34u) {
            const __half d = __float2half(1e-4f + 1e-7f * (float)(next_random(state) & 0xFFFu));
            std::memcpy(&rows[at], &d, 2);
            for (size_t i = 2; i < 34u; ++i) {
                rows[at + i] = (unsigned char)next_random(state);
            }
        }
        std::vector<__half> in((size_t)m * k);
        for (auto &v : in) {
            v = __float2half((float)(int)(next_random(state) & 0x7FFu) / 1024.0f - 1.0f);
        }
        w = on_device(rows);
        x = on_device(in);
        live = on_device(std::vector<unsigned int>(1, live_));
        CHECK_CUDA(cudaMalloc(&y, (size_t)m * n * sizeof(float)));
    }
    Product(const Product &) = delete;
    ~Product()
    {
        cudaFree(w);
        cudaFree(x);
        cudaFree(live);
        cudaFree(y);
    }
    void launch(cudaStream_t stream, const Scratch &scratch, unsigned int sm_count, unsigned int set)
    {
        CHECK_CUDA(q8::launch_umma(stream, scratch.use, sm_count, w, n, k, x, 0, m, live, y, 0, set, true));
    }
    std::vector<float> result() const
    {
        std::vector<float> got((size_t)m * n);
        CHECK_CUDA(cudaMemcpy(got.data(), y, got.size() * sizeof(float), cudaMemcpyDeviceToHost));
        return got;
    }
    void forget() { CHECK_CUDA(cudaMemset(y, 0xFF, (size_t)m * n * sizeof(float))); }
};

// Say of every cut tile of a launch on set 0 that may be finished by all its holders that one of them came to wait before
// all had begun: the one that began it finishes it then.  Returns how many tiles that are.
static unsigned int leave_to_the_first(const Scratch &scratch, const Product &p, unsigned int sm_count)
{
    const unsigned int ntok = q8::pair_token_tile(p.m);
    const unsigned int tiles = (p.n + 255u) / 256u * ((p.m + ntok - 1u) / ntok), segs = p.k / 256u;
    const unsigned int pairs = tiles * segs < sm_count / 2u ? tiles * segs : sm_count / 2u;
    unsigned int found = 0;
    for (unsigned int id = 0; id < pairs; ++id) {
        q8::PairWork work;
        q8::pair_deal(&work, id, pairs, tiles, segs);
        const unsigned int from = q8::pair_share_from(work);
        while (work.next()) {
            if (work.s0 != 0u || work.s1 == segs || q8::pair_last_holder(work, id, work.tile) + 1u - id < from) {
                continue;
            }
            found += 1u;
            for (unsigned int rank = 0; rank < 2u; ++rank) {
                // the second holder's slot, behind its four flags
                std::vector<unsigned int> alone(4u, q8::kPairAlone);
                CHECK_CUDA(cudaMemcpy(scratch.use.flags + q8::kFlagWords * (2u * (id + 1u) + rank) + 4u, alone.data(), 16u,
                                      cudaMemcpyHostToDevice));
            }
        }
    }
    return found;
}

static int fail(const char *what, const Product &p, unsigned int live)
{
    std::printf("%s: %u x %u, %u rows, %u live\n", what, p.n, p.k, p.m, live);
    return 1;
}

int main()
{
    int sms = 0;
    CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0));
    const unsigned int sm_count = (unsigned int)sms;
    cudaStream_t stream;
    CHECK_CUDA(cudaStreamCreate(&stream));
    Scratch scratch(sm_count);
    // many holders and few; rows of w that leave quarters of a tile empty; live batches with fewer runs of rows than a
    // block has warps to finish them, and none
    const unsigned int shapes[][3] = {{1000, 2048, 200}, {256, 16384, 150}, {130, 16384, 257}, {130, 4096, 129},
                                      {2560, 2560, 300}, {300, 16384, 140}, {300, 256, 700},   {5000, 1024, 161}};
    unsigned int shared = 0;
    for (const auto &shape : shapes) {
        for (unsigned int live : {shape[2], 129u, 9u, 1u, 0u}) {
            Product p(shape[0], shape[1], shape[2], live);
            p.forget();
            p.launch(stream, scratch, sm_count, 0u);
            CHECK_CUDA(cudaStreamSynchronize(stream));
            const std::vector<float> first = p.result();
            if (!scratch.all_zero()) {
                return fail("words left after a launch", p, live);
            }
            for (unsigned int repeat = 0; repeat < 20u; ++repeat) {
                p.launch(stream, scratch, sm_count, repeat + 1u);
            }
            CHECK_CUDA(cudaStreamSynchronize(stream));
            if (!scratch.all_zero()) {
                return fail("words left after launches", p, live);
            }
            if (std::memcmp(first.data(), p.result().data(), first.size() * sizeof(float)) != 0) {
                return fail("another result", p, live);
            }
            if (live == shape[2]) {
                p.forget();
                shared += leave_to_the_first(scratch, p, sm_count);
                p.launch(stream, scratch, sm_count, 0u);
                CHECK_CUDA(cudaStreamSynchronize(stream));
                if (!scratch.all_zero()) {
                    return fail("words left by the first holder", p, live);
                }
                if (std::memcmp(first.data(), p.result().data(), first.size() * sizeof(float)) != 0) {
                    return fail("another result by the first holder", p, live);
                }
            }
        }
    }
    if (shared < 20u) {
        std::printf("only %u tiles of many holders\n", shared);
        return 1;
    }
    // two streams, one of them of a higher priority, a scratch each
    int low = 0, high = 0;
    CHECK_CUDA(cudaDeviceGetStreamPriorityRange(&low, &high));
    cudaStream_t other;
    CHECK_CUDA(cudaStreamCreateWithPriority(&other, cudaStreamNonBlocking, high));
    Scratch scratch2(sm_count);
    Product deep(256u, 16384u, 150u, 150u), many(1000u, 2048u, 200u, 200u);
    deep.launch(stream, scratch, sm_count, 0u);
    CHECK_CUDA(cudaDeviceSynchronize());
    many.launch(other, scratch2, sm_count, 0u);
    CHECK_CUDA(cudaDeviceSynchronize());
    const std::vector<float> want_deep = deep.result(), want_many = many.result();
    for (unsigned int repeat = 0; repeat < 200u; ++repeat) {
        deep.launch(stream, scratch, sm_count, repeat);
        many.launch(other, scratch2, sm_count, 2u * repeat);
        many.launch(other, scratch2, sm_count, 2u * repeat + 1u);
        if (repeat % 20u != 19u) {
            continue;
        }
        CHECK_CUDA(cudaDeviceSynchronize());
        if (!scratch.all_zero() || !scratch2.all_zero()) {
            return fail("words left beside another stream", deep, deep.m);
        }
        if (std::memcmp(want_deep.data(), deep.result().data(), want_deep.size() * sizeof(float)) != 0
            || std::memcmp(want_many.data(), many.result().data(), want_many.size() * sizeof(float)) != 0) {
            return fail("another result beside another stream", deep, deep.m);
        }
        deep.forget();
        many.forget();
        CHECK_CUDA(cudaDeviceSynchronize());
    }
    std::printf("pass\n");
    return 0;
}
