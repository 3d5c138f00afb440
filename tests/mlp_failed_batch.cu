// Training with the error flag of the network's kernels set from the host, as a
// wait that gave up sets it: built by test_gpu_mlp.py from the library's sources.
#define private public
#include "guess.cpp"
#undef private
#include "mlp.cu"

namespace cfdg {
void cuda_check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw Failure{CFDG_ERR_CUDA, what};
}
}  // namespace cfdg

// One epoch over `rows` samples; with `fail` every batch finds the flag set.  The
// parameters go to p; returns the Adam steps that the network counts, -1 when a
// failure is not reported or one is that should not be.
extern "C" int train(int rows, int batch, int fail, const uint16_t* x, const float* t, float* p) {
    using namespace cfdg;
    try {
        Mlp net(0, 5, 1);
        Dataset ds(0, 5, rows);
        ds.append_host(x, t, rows);
        const int flag = fail;
        cuda_check(cudaMemcpy(net.err_, &flag, sizeof(int), cudaMemcpyHostToDevice), "H2D");
        bool reported = false;
        try {
            net.train(ds, 1, batch, 1e-2f, 7, nullptr);
        } catch (const Failure&) {
            reported = true;
        }
        cuda_check(cudaDeviceSynchronize(), "sync");
        net.get_params(p);
        return reported == (fail != 0) ? net.step_ : -1;
    } catch (const Failure&) {
        return -1;
    }
}
