"""How a plugin call reaches the caller's arrays, with the CUDA runtime and the
kernels faked on the CPU: a kernel may only be given what it can reach from the
first element to the last, and every other call takes the copies, whose checks
decide."""
import ctypes as C

import numpy as np
import pytest

import host_build
import n_body_sim_pro_b200 as nb

# kernels: accelerations are twice the positions; small_force_kernel's place
# counts arrays that a GPU could not read or write through the given addresses
FAKES = r"""
EXPORT int fake_faults, fake_small_calls;
EXPORT void fake_fail_host_alloc(int on) { fake_host_alloc_fails = on; }
EXPORT int fake_error_left(void) { return cudaGetLastError(); }
int nbsp_allpairs_small(const double* x, const double* y, const double* z, const double* m,
                        size_t n, float eps2, double g, void* packed, double* ax, double* ay,
                        double* az, double* ox, double* oy, double* oz, int* report,
                        cudaStream_t stream) {
    const double* arrays[7] = {x, y, z, m, ox, oy, oz};
    for (int k = 0; k < 7; ++k)
        if (!fake_reachable(arrays[k], n * sizeof(double))) {
            ++fake_faults;
            return 0;
        }
    ++fake_small_calls;
    for (size_t i = 0; i < n; ++i) {
        ox[i] = 2 * x[i];
        oy[i] = 2 * y[i];
        oz[i] = 2 * z[i];
    }
    *report = 0;
    return 0;
}
static NBodySimProCudaContext* fake_context;
EXPORT void fake_watch(NBodySimProCudaContext* c) { fake_context = c; }
void nbsp_allpairs_finalize(const void* hi, const void* lo, size_t n, int chunks, double g,
                            double* ax, double* ay, double* az, cudaStream_t stream) {
    for (size_t i = 0; i < n; ++i) {
        ax[i] = 2 * fake_context->x[i];
        ay[i] = 2 * fake_context->y[i];
        az[i] = 2 * fake_context->z[i];
    }
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = host_build.build(str(tmp_path_factory.mktemp("host")), "api.c", FAKES)
    lib.n_body_sim_pro_cuda_context_create.restype = C.c_void_p
    for f in ("fake_register", "fake_unregister", "fake_watch", "n_body_sim_pro_cuda_context_destroy"):
        getattr(lib, f).argtypes = [C.c_void_p] + ([C.c_size_t] if f == "fake_register" else [])
    lib.n_body_sim_pro_gravity_compute_acceleration_cuda.argtypes = [C.c_void_p] * 4
    return lib


FIELDS = ("positions_x", "positions_y", "positions_z", "masses", "accelerations_x",
          "accelerations_y", "accelerations_z")


class Call:
    """An all-pairs plugin call of n particles whose seven arrays start `shift` bytes
    behind a page's start; `locked` byte ranges of each (or of the fields `only`) are page-locked."""

    def __init__(self, host, n, locked=(), shift=0, only=None):
        self.host, self.n = host, n
        self.keep, self.registered = [], []
        self.view = nb.View(n)
        rng = np.random.default_rng(n)
        self.arrays = {}
        for k, f in enumerate(FIELDS):
            raw = np.zeros(8 * n + 8192 + shift, dtype=np.uint8)
            at = raw.ctypes.data
            off = -at % 4096 + shift
            a = raw[off:off + 8 * n].view(np.float64)
            if k < 4:
                a[:] = rng.standard_normal(n)
            self.keep.append(raw)
            self.arrays[f] = a
            setattr(self.view, f, C.cast(at + off, C.POINTER(C.c_double)))
            if only is None or f in only:
                for first, end in locked:
                    host.fake_register(at + off + first, end - first)
                    self.registered.append(at + off + first)
        self.host.fake_watch(None)

    def run(self, context):
        self.host.fake_watch(context)
        err, g = nb.Error(), nb.gravity_init(1.0, 0.01)
        faults = C.c_int.in_dll(self.host, "fake_faults")
        small = C.c_int.in_dll(self.host, "fake_small_calls")
        faults.value = small.value = 0
        status = self.host.n_body_sim_pro_gravity_compute_acceleration_cuda(
            C.addressof(self.view), C.addressof(g), context, C.addressof(err))
        for at in self.registered:
            self.host.fake_unregister(at)
        if status == nb.Status.OK:
            for a, x in zip(FIELDS[4:], FIELDS[:3]):
                np.testing.assert_array_equal(self.arrays[a], 2 * self.arrays[x])
        return status, faults.value, small.value


@pytest.fixture()
def context(host):
    c = host.n_body_sim_pro_cuda_context_create(None)
    assert c
    yield c
    host.fake_fail_host_alloc(0)
    host.n_body_sim_pro_cuda_context_destroy(c)


@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1000, 2047])
@pytest.mark.parametrize("locked", [False, True])
def test_whole_arrays_take_the_two_kernels(host, context, n, locked):
    call = Call(host, n, [(0, 8 * n)] if locked else ())
    assert call.run(context) == (nb.Status.OK, 0, 1)


@pytest.mark.parametrize("n", [2, 600, 2047])
@pytest.mark.parametrize("field", ["positions_x", "masses", "accelerations_z"])
def test_partly_locked_arrays_are_the_copies_to_judge(host, context, n, field):
    """A part of the array page-locked: refused by the copies, never a kernel's."""
    size = 8 * n
    parts = [[(0, size // 2)], [(size // 2, size)], [(0, size - 8)], [(8, size)]]
    if n == 2047:  # a hole of a page, both ends locked
        parts.append([(0, 4096), (8192, size)])
    for part in parts:
        status, faults, small = Call(host, n, part, only=[field]).run(context)
        assert (faults, small) == (0, 0)
        assert status == nb.Status.INVALID_STATE


@pytest.mark.parametrize("n", [1, 700, 2047])
@pytest.mark.parametrize("shift", [1, 4, 12])
def test_unaligned_arrays_go_through_the_rows(host, context, n, shift):
    """Page-locked or pageable, arrays that are not on 8-byte boundaries are served
    (the copies never asked for it), but not by a kernel's own loads and stores."""
    for locked in ([], [(0, 8 * n)]):
        for only in (None, ["masses"], ["accelerations_y"]):
            assert Call(host, n, locked, shift, only).run(context) == (nb.Status.OK, 0, 1)


@pytest.mark.parametrize("n", [5, 1000, 2047])
def test_calls_survive_a_failing_page_lock(host, context, n):
    """No page-locked memory for the rows: the copies serve the call, and the rows are
    there again when it can be had."""
    assert Call(host, 3).run(context) == (nb.Status.OK, 0, 1)
    host.fake_fail_host_alloc(1)
    served = Call(host, n).run(context)
    assert served == (nb.Status.OK, 0, int(n < 1024))  # (the first call's rows hold 1024)
    assert host.fake_error_left() == 0
    assert Call(host, 7).run(context)[0] == nb.Status.OK
    host.fake_fail_host_alloc(0)
    assert Call(host, n).run(context) == (nb.Status.OK, 0, 1)


def test_first_call_without_rows(host, context):
    host.fake_fail_host_alloc(1)
    assert Call(host, 100).run(context) == (nb.Status.OK, 0, 0)
    assert Call(host, 100, [(0, 800)]).run(context) == (nb.Status.OK, 0, 0)
