// Calls rb2_film_develop from one thread per job, each on its own stream, `iters`
// times; returns how many calls failed.
#include "rb2_render.h"

#include <atomic>
#include <thread>
#include <vector>

struct FilmJob {
    rb2_filter filter;
    uint32_t width, height, spp;
    const float* xy;
    const float* L;
    float* rgb;
    void* stream;
};

using Develop = int (*)(const rb2_filter*, uint32_t, uint32_t, uint32_t, const float*, const float*, float*, void*);

extern "C" int film_threads(Develop develop, const FilmJob* jobs, int n, int iters)
{
    std::atomic<int> ready{0}, failed{0};
    std::vector<std::thread> threads;
    for (int i = 0; i < n; i++)
        threads.emplace_back([&, i] {
            const FilmJob& j = jobs[i];
            ready++;
            while (ready.load() < n) {}
            for (int k = 0; k < iters; k++)
                if (develop(&j.filter, j.width, j.height, j.spp, j.xy, j.L, j.rgb, j.stream)) failed++;
        });
    for (std::thread& t : threads) t.join();
    return failed.load();
}
