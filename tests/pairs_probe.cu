// The paired and float-pair forms against the operations they stand for, on every
// float, for tests/test_gpu_every_float.py.
#include "../lattibol_0.3.31f_gb300/csrc/lb_pairs.cuh"

namespace {

__device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}

// form 0: pair_rcp, 1: pair_rcp2, 2: pair_psi_exp1, each on the floats i and i + 2^31;
// 3: ff_psi_ref where it decides
__global__ void compare(int form, const lb::PairConst c, unsigned long long *wrong) {
    const uint32_t n = gridDim.x * blockDim.x;
    unsigned long long bad = 0;
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (1u << 31); i += n) {
        const float a = __uint_as_float((uint32_t)i), b = __uint_as_float((uint32_t)i + (1u << 31));
        const float2 x = make_float2(a, b);
        if (form == 0) {
            const float2 y = lb::pair_rcp(c, x);
            bad += !same(y.x, 1.f / a) + !same(y.y, 1.f / b);
        } else if (form == 1) {
            float2 p = x, q = make_float2(b, a);
            lb::pair_rcp2(c, p, q);
            bad += !same(p.x, 1.f / a) + !same(p.y, 1.f / b) + !same(q.x, 1.f / b) +
                   !same(q.y, 1.f / a);
        } else if (form == 2) {
            const float2 y = lb::pair_psi_exp1(c, x);
            bad += !same(y.x, lb::psi_exp1(a)) + !same(y.y, lb::psi_exp1(b));
        } else {
            float y;
            if (lb::ff_psi_ref(a, y)) bad += !same(y, (float)(4. * exp(-200. / (double)a)));
            if (lb::ff_psi_ref(b, y)) bad += !same(y, (float)(4. * exp(-200. / (double)b)));
        }
    }
    if (bad) atomicAdd(wrong, bad);
}

}  // namespace

// how many floats differ; negative: a CUDA error
extern "C" long probe_every_float(int form) {
    unsigned long long *wrong = nullptr, h = 0;
    cudaError_t e = cudaMalloc(&wrong, sizeof(h));
    if (e == cudaSuccess) e = cudaMemset(wrong, 0, sizeof(h));
    if (e == cudaSuccess) {
        compare<<<152 * 8, 256>>>(form, lb::pair_constants(), wrong);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&h, wrong, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(wrong);
    return e == cudaSuccess ? (long)h : -(long)e;
}
