"""What an evaluation's phase timings count, with the launchers and the GPU's clock
faked on the CPU: a launcher's work takes 1 us times a power of two, so that a sum
of them says which ones a phase holds."""
import ctypes as C

import pytest

import host_build
import n_body_sim_pro_b200 as nb

WORK = {"bounds": 1, "clear": 2, "keys": 4, "sort": 8, "gather": 16, "build": 32, "moments": 64,
        "walk": 128, "unsort": 256}
FAKES = "enum {%s};" % ", ".join(f"W_{k.upper()} = {1000 * v}" for k, v in WORK.items()) + r"""
static unsigned long long now = 5000;
static void stamp(unsigned long long* at) { if (at != NULL) *at = now; }
void nbsp_bh_bounds(double* x, double* y, double* z, const double* m, size_t n, double* partial,
                    double* geometry, int* status, const double* ax, const double* ay,
                    const double* az, int rms, const NbspLeapfrogFusion* lf,
                    unsigned long long* at, unsigned long long* end, cudaStream_t stream) {
    stamp(at);
    now += W_BOUNDS;
    if (geometry != NULL) stamp(end);
}
void nbsp_bh_keys(const double* x, const double* y, const double* z, const double* m, size_t n,
                  const double* geometry, uint64_t* keys, uint32_t* index, void* unsorted,
                  uint32_t* scratch, const double* ax, const double* ay, const double* az,
                  double tol_scale, float* tol, void* tree, unsigned long long* counters,
                  cudaStream_t stream) {
    now += W_CLEAR + W_KEYS;
}
void nbsp_bh_small_keys(const double* x, const double* y, const double* z, const double* m,
                        size_t n, const double* partial, double* geometry, uint64_t* keys,
                        uint32_t* index, void* unsorted, const double* ax, const double* ay,
                        const double* az, double tol_scale, float* tol, void* tree,
                        unsigned long long* counters, unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_KEYS;
}
void nbsp_bh_small_merge(const uint64_t* ki, const uint32_t* ii, size_t n, uint64_t* k, uint32_t* i,
                         const void* u, void* p, const float* tu, float* t, int* status,
                         unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_SORT;
}
void nbsp_bh_sort(uint64_t* k, uint32_t* i, uint64_t* ka, uint32_t* ia, size_t n, uint32_t* s,
                  int* status, unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_SORT;
}
int fake_gathers;
EXPORT int fake_gather_count(void) { return fake_gathers; }
void nbsp_bh_gather(const void* u, const uint32_t* perm, size_t n, void* pos4, const float* tu,
                    float* t, int* status, unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_GATHER;
    ++fake_gathers;
}
void nbsp_bh_build(const uint64_t* keys, const uint32_t* perm, const double* x, const double* y,
                   const double* z, size_t n, int leaf, void* tree, int* status,
                   unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_BUILD;
}
void nbsp_bh_moments(const void* p, const uint64_t* k, size_t n, const double* geo, double theta,
                     double start, int opening, int quad, void* tree, int* status,
                     unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_MOMENTS;
}
void nbsp_bh_walk(const void* p, const float* tol, size_t n, const void* tree, int order, int mode,
                  const void* corr, const NbspCorrectionLists* lists, float eps2,
                  const uint32_t* perm, void* acc, unsigned long long* counters, int* status,
                  unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_WALK;
}
void nbsp_bh_unsort(const void* acc, size_t n, double g, double* ax, double* ay, double* az,
                    const NbspLeapfrogFusion* lf, const void* tree, unsigned long long* counters,
                    unsigned long long* at, cudaStream_t stream) {
    stamp(at);
    now += W_UNSORT;
    if (at != NULL) at[NBSP_BH_END - NBSP_BH_INTEGRATE] = now;
}
size_t nbsp_bh_sort_scratch_words(size_t n) { return 1; }
size_t nbsp_bh_tree_bytes(size_t n) { return 1; }
EXPORT int fake_evaluate(size_t n, int order_only, NBodySimProCudaTimings* timings) {
    static NbspBarnesHut* b;
    double one[1] = {0};
    int status = 0;
    NbspBarnesHutState s = {.x = one, .y = one, .z = one, .m = one, .ax = one, .ay = one, .az = one, .n = n};
    if (order_only) return nbsp_bh_morton(&b, &s, &status, NULL, NULL, NULL, NULL, NULL);
    NbspBarnesHutParams p = {.gravitational_constant = 1, .theta = 0.7, .multipole_order = 1, .leaf_capacity = 16};
    NBodySimProBarnesHutStats stats;
    size_t restarts, corrected;
    int rc = nbsp_bh_accelerations(&b, &s, &p, &status, NULL, &stats, timings, NULL);
    nbsp_bh_collect(b, &stats, timings, &restarts, &corrected);
    return rc;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = host_build.build(str(tmp_path_factory.mktemp("host")), "bh_host.c", FAKES)
    lib.fake_evaluate.argtypes = [C.c_size_t, C.c_int, C.c_void_p]
    return lib


def held(ms):
    """The launchers whose work a phase of `ms` holds."""
    us = round(ms * 1e3)
    assert abs(ms * 1e3 - us) < 1e-6
    return {k for k, v in WORK.items() if us & v}


@pytest.mark.parametrize("n", [2, 98304, 98305])
def test_each_launcher_counts_in_its_own_phase(host, n):
    t = nb.Timings()
    assert host.fake_evaluate(n, 0, C.addressof(t)) == nb.Status.OK
    large = n > 98304
    assert held(t.bounds_ms) == {"bounds"}
    assert held(t.keys_ms) == ({"clear", "keys"} if large else {"keys"})  # the sort's scratch is cleared for the keys
    assert held(t.sort_ms) == {"sort"}
    assert held(t.build_ms) == ({"gather", "build"} if large else {"build"})
    assert held(t.moments_ms) == {"moments"}
    assert held(t.walk_ms) == {"walk"}
    assert held(t.integrate_ms) == {"unsort"}
    assert held(t.total_ms) == set(WORK) - (set() if large else {"clear", "gather"})


@pytest.mark.parametrize("n", [2, 98305])
def test_an_order_alone_gathers_no_records(host, n):
    before = host.fake_gather_count()
    assert host.fake_evaluate(n, 1, None) == nb.Status.OK
    assert host.fake_gather_count() == before
