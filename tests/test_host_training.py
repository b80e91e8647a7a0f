"""A training epoch whose blocks' wait for one another ran out, with the CUDA runtime
and the kernels faked on the CPU: the call reports it, and weights, moments and the
count of Adam steps are those of the last whole epoch."""
import ctypes as C

import numpy as np
import pytest

import host_build
import n_body_sim_pro_b200 as nb

NP, STEPS, CTAS = 64 * 10 + 64 + 64 * 64 + 64 + 3 * 64 + 3, 5, 2
# an epoch adds its steps' first bias terms to every weight; a failing one leaves
# half of its results behind and the flag set
FAKES = r"""
enum { NP = %d, ROWS = 128 };
int fake_fail_epoch; /* epochs until one fails (0: none) */
EXPORT void fake_fail_after(int epochs) { fake_fail_epoch = epochs; }
int nbsp_mlp_param_count(void) { return NP; }
int nbsp_mlp_slot_floats(void) { return NP; }
int nbsp_mlp_rows_per_cta(void) { return ROWS; }
int nbsp_mlp_epoch_ctas(void) { return 32; }
size_t nbsp_mlp_frags_bytes(void) { return NP * sizeof(float); }
size_t nbsp_mlp_net_bytes(void) { return NP * sizeof(float); }
void nbsp_mlp_adam_bias(int step, float* bias) { bias[0] = bias[1] = (float)step; }
void nbsp_mlp_build_frags(const float* params, void* frags, void* net, cudaStream_t stream) {
    memcpy(frags, params, NP * sizeof(float));
    if (net != NULL) memcpy(net, params, NP * sizeof(float));
}
EXPORT NBodySimProCudaCorrection* fake_correction(size_t rows) {
    NBodySimProCudaCorrection* c = n_body_sim_pro_cuda_correction_create(3, NULL);
    c->rows = c->train_rows = rows;
    cudaMalloc((void**)&c->order, rows * sizeof(int));
    return c;
}
EXPORT void fake_state(NBodySimProCudaCorrection* c, float* out) {
    const void* parts[5] = {c->params, c->m, c->v, c->frags, c->net};
    for (int k = 0; k < 5; ++k) memcpy(out + k * NP, parts[k], NP * sizeof(float));
    out[5 * NP] = (float)c->adam_step;
}
"""
EPOCH = r"""
int nbsp_mlp_train_epoch(const uint32_t* x, const float* y, const int* order, int rows_total,
                         int steps, int ctas, float inv_batch3, void* frags, float* slots,
                         const float* params, const float* m, const float* v, float* next_params,
                         float* next_m, float* next_v, float lr, const void* bias, int* sync,
                         cudaStream_t stream) {
    const int fails = fake_fail_epoch > 0 && --fake_fail_epoch == 0;
    for (int k = 0; k < NP; ++k) {
        if (fails && k >= NP / 2) continue;
        float sum = 0.f;
        for (int s = 0; s < steps; ++s) sum += ((const float*)bias)[2 * s];
        next_params[k] = params[k] + sum;
        next_m[k] = m[k] + 1.f;
        next_v[k] = v[k] + 2.f;
        ((float*)frags)[k] = next_params[k];
    }
    sync[1] = fails;
    return 0;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = host_build.build(str(tmp_path_factory.mktemp("host")), "mlp_host.c", FAKES % NP + EPOCH)
    lib.fake_correction.restype = C.c_void_p
    lib.fake_correction.argtypes = [C.c_size_t]
    lib.fake_state.argtypes = [C.c_void_p, C.c_void_p]
    lib.n_body_sim_pro_cuda_correction_destroy.argtypes = [C.c_void_p]
    lib.n_body_sim_pro_cuda_correction_train.argtypes = [
        C.c_void_p, C.c_int, C.c_int, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    return lib


def train(host, c, epochs):
    err = nb.Error()
    return host.n_body_sim_pro_cuda_correction_train(c, epochs, CTAS * 128, 1e-3, None, None, C.byref(err))


def state(host, c):
    out = np.zeros(5 * NP + 1, dtype=np.float32)
    host.fake_state(c, out.ctypes.data)
    return out[:-1].reshape(5, NP), int(out[-1])


def test_failed_epoch_leaves_the_last_whole_one(host):
    c = host.fake_correction(STEPS * CTAS * 128)
    try:
        first, step = state(host, c)
        assert step == 0
        biases = np.arange(1, 1 + STEPS).sum()
        host.fake_fail_after(1)
        assert train(host, c, 1) == nb.Status.INVALID_STATE
        after, step = state(host, c)
        np.testing.assert_array_equal(after, first)
        assert step == 0
        host.fake_fail_after(3)  # two whole epochs, then a failing one
        assert train(host, c, 4) == nb.Status.INVALID_STATE
        after, step = state(host, c)
        assert step == 2 * STEPS
        biases += np.arange(1 + STEPS, 1 + 2 * STEPS).sum()
        np.testing.assert_allclose(after[0], first[0] + biases, rtol=1e-6)
        np.testing.assert_array_equal(after[1:3], first[1:3] + np.array([[2.0], [4.0]]))
        np.testing.assert_array_equal(after[3:], [after[0], after[0]])  # fragments and network follow
        assert train(host, c, 1) == nb.Status.OK
        assert state(host, c)[1] == 3 * STEPS
    finally:
        host.fake_fail_after(0)
        host.n_body_sim_pro_cuda_correction_destroy(c)
