// line_rcp against __drcp_rn over a range of exponents: out[d] counts the
// arguments whose results lie d units in the last place apart (3: more).
// Mantissas are random, or (near) within 7 units of a power of two.
#include "line_stage.cuh"

__global__ void compare(unsigned long long seed, int low, int high, int near, int n, unsigned long long* out) {
    unsigned long long s = seed + 0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1), count[4] = {0, 0, 0, 0};
    for (int i = 0; i < n; ++i) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        unsigned long long m = s >> 12;
        if (near) m = (s >> 33) & 1 ? m & 7 : ~(m & 7);
        const unsigned long long e = 1023 + low + static_cast<int>((s >> 34) % (high - low + 1));
        const double x = __longlong_as_double(static_cast<long long>(((s >> 20) & 1) << 63 | e << 52 | (m & 0xfffffffffffffull)));
        long long d = __double_as_longlong(ndg::dev::line_rcp(x)) - __double_as_longlong(__drcp_rn(x));
        if (d < 0) d = -d;
        ++count[d > 3 ? 3 : d];
    }
    for (int d = 0; d < 4; ++d) atomicAdd(out + d, count[d]);
}

extern "C" int compare_reciprocals(unsigned long long seed, int low, int high, int near, int n, unsigned long long* out) {
    compare<<<592, 256>>>(seed, low, high, near, n, out);
    return static_cast<int>(cudaDeviceSynchronize());
}
