// Test-only build of the library's host layer with a kernel that waits for a
// bulk copy nobody issues (tests/test_gpu_lost_copy.py): the wait runs out after
// its bound, and the library has to say so.
#include "qlskum_host.cpp"
#include "qlskum_ring.cuh"

namespace {

// One warp, two barriers that expect bytes which never come: the ring's wait
// gives up on the chunk it is at and on the one in flight behind it.
__global__ void k_lost_copy(DevCloud c, int *returned)
{
    __shared__ unsigned long long bars[mixed::kRingChunks];
    mixed::EdgeRing<1> R;
    R.bar = smem_addr(bars);
    if (threadIdx.x == 0)
        for (int s = 0; s < mixed::kRingChunks; s++) {
            mbar_init(R.bar + 8 * s, 1);
            mbar_expect(R.bar + 8 * s, 16);
        }
    __syncwarp();
    const bool arrived = R.wait(c);
    if (threadIdx.x == 0) *returned = arrived ? 1 : 2;
}

int launch(const DevCloud &c, cudaStream_t stream)
{
    int *d = nullptr, h = 0;
    if (cudaMalloc(&d, sizeof(int)) != cudaSuccess) return -1;
    k_lost_copy<<<1, 32, 0, stream>>>(c, d);
    cudaError_t e = cudaMemcpyAsync(&h, d, sizeof h, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    cudaFree(d);
    return e == cudaSuccess ? h : -1;
}

}  // namespace

extern "C" {

// 2: the wait gave up; 1: it returned as if the copy had arrived; -1: a CUDA error.
int qlskum_test_lost_copy(qlskum_handle *h) { return launch(h->dc, h->L.stream); }
int qlskum_test_lost_copy_batch(qlskum_batch *b) { return launch(b->sc, b->L.stream); }
int qlskum_test_lost_copy_partition(qlskum_partition *P)
{
    return launch(P->parts.back()->G.dc, P->parts.back()->L.stream);
}

}
