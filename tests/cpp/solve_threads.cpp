// Host threads that solve 2D problems of two widths, each on its own stream, for
// a time: "<calls> calls, <errors> errors", and the first error's text.
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "sil_b200.h"

int main(int argc, char** argv)
{
    if (argc != 7) return 2;
    int const threads = std::atoi(argv[5]);
    double const seconds = std::atof(argv[6]);
    std::atomic<long> calls {0}, errors {0};
    std::mutex mutex;
    std::string first;
    auto const start = std::chrono::steady_clock::now();
    auto work = [&](int nx, int ny) {
        cudaStream_t stream;
        if (cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) std::exit(3);
        std::vector<double> mu(static_cast<size_t>(nx) * ny, 1.0), b(mu.size(), 0.0);
        for (int j = 1; j + 1 < ny; ++j)
            for (int i = 1; i + 1 < nx; ++i) b[i + static_cast<size_t>(nx) * j] = (7 * i + 13 * j) % 11 - 5.0;
        double* dev[3];
        for (double*& p : dev)
            if (cudaMalloc(&p, mu.size() * sizeof(double)) != cudaSuccess) std::exit(3);
        cudaMemcpy(dev[0], mu.data(), mu.size() * sizeof(double), cudaMemcpyHostToDevice);
        cudaMemcpy(dev[1], b.data(), b.size() * sizeof(double), cudaMemcpyHostToDevice);
        sil_mag2d_problem const problem {nx, ny, dev[0], dev[1], dev[2]};
        sil_solve_settings settings {};
        settings.solver = SIL_SOLVER_CG_F64;
        settings.max_iterations = 1;
        settings.relative_tolerance = 1e-2;
        while (std::chrono::duration<double>(std::chrono::steady_clock::now() - start).count() < seconds) {
            sil_solve_diagnostics diag {};
            ++calls;
            if (sil_mag2d_solve_batch(&problem, 1, &settings, &diag, stream) == SIL_OK) continue;
            ++errors;
            std::lock_guard<std::mutex> lock(mutex);
            if (first.empty()) first = sil_last_error();
        }
    };
    std::vector<std::thread> all;
    for (int t = 0; t < threads; ++t) {
        all.emplace_back(work, std::atoi(argv[1]), std::atoi(argv[2]));
        all.emplace_back(work, std::atoi(argv[3]), std::atoi(argv[4]));
    }
    for (std::thread& t : all) t.join();
    std::printf("%ld calls, %ld errors %s\n", calls.load(), errors.load(), first.c_str());
    return 0;
}
