// A user model whose log-likelihood is +infinity for one particle, stepped
// through the fused FP32 filter.  Built and called by
// tests/test_model_infinite_weight_gpu.py.
#include <vsmc_cuda_filter.cuh>

#include <cstdint>

namespace
{

// x[0] moves, x[1] is the particle's number
struct Spike {
    static constexpr int dim = 2;
    static constexpr int monitor_dim = 1;
    struct step_type {
    };
    float which; // this particle has an infinite log-likelihood

    __device__ step_type step(uint32_t) const { return {}; }

    __device__ void init(
        const step_type &, vsmc_cuda::ParticleRng &rng, float (&x)[2]) const
    {
        float b;
        rng.normal_pair(x[0], b);
        x[1] = static_cast<float>(rng.particle());
    }

    __device__ void move(
        const step_type &, vsmc_cuda::ParticleRng &rng, float (&x)[2]) const
    {
        float a, b;
        rng.normal_pair(a, b);
        x[0] += 0.1f * a;
    }

    __device__ float log_likelihood(
        const step_type &, const float (&x)[2]) const
    {
        return x[1] == which ? INFINITY : -x[0] * x[0];
    }
};

} // namespace

// status of T steps of n particles, threshold 0 (no resampling)
extern "C" int infinite_weight_run(size_t n, size_t T, float which)
{
    vsmc_cuda_pf *pf = nullptr;
    int rc = vsmc_cuda_pf_create_model(&pf, n, Spike::dim, Spike::monitor_dim,
        VSMC_CUDA_SYSTEMATIC, 0.0, 5, T, nullptr);
    if (rc != VSMC_CUDA_OK)
        return rc;
    const Spike m = {which};
    for (size_t t = 0; rc == VSMC_CUDA_OK && t < T; ++t) {
        vsmc_cuda_pf_step_desc d;
        rc = vsmc_cuda_pf_step_desc_get(pf, &d);
        if (rc == VSMC_CUDA_OK)
            rc = vsmc_cuda::pf_step_launch(d, m);
        if (rc == VSMC_CUDA_OK)
            rc = vsmc_cuda_pf_step_commit(pf);
    }
    if (rc == VSMC_CUDA_OK)
        rc = vsmc_cuda_pf_history(pf, T, nullptr, nullptr, nullptr, nullptr);
    vsmc_cuda_pf_destroy(pf);
    return rc;
}
