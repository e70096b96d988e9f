"""What the plain correlation refuses, on a fake CUDA runtime (no kernel runs): the shared memory of the general kernel
limits psi angles and CTAs per particle where that kernel runs, and not where the register form does."""
from .fakes.runtime import run_on_fake

CALLS = r"""
context = C.c_void_p()
ok(lib.gisapr_context_create(0, C.byref(context)), "context")
def single(n, crop, psi, bank=p):
    return lib.gisapr_correlate(context, None, bank, p, p, p, 3, psi, n, crop, p, p, p)
def batch(n, crop, psi, bank=p):
    return lib.gisapr_correlate_batch(context, None, bank, n * n * 4, 2, p, p, p, 3, 9, psi, n, crop, p, p, p)
calls = (single, batch)
odd = C.c_void_p(p.value + 8)  # a bank that does not start on 16 bytes is left to the general kernel
"""


def test_psi_angles_and_clusters(native_lib, tmp_path):
    run_on_fake(CALLS + r"""
for call in calls:
    for n in (64, 96, 128, 192, 256):
        for crop in (8, 12, 16):
            for cluster in range(9):
                ok(lib.gisapr_set_tuning(context, 1, n, cluster), "tuning")
                for psi in (1, 3, 40):
                    ok(call(n, crop, psi), (n, crop, cluster, psi))
                # the general kernel where the window or the alignment asks for it: a tuned number of CTAs that
                # its shared memory does not allow gives way to the default
                ok(call(n, 6, 1), (n, 6, cluster))
                ok(call(n, crop, 1, odd), (n, crop, cluster, "odd"))
            assert call(n, 6, 40) == 4 and b"too many psi" in lib.gisapr_last_error()
            assert call(n, crop, 40, odd) == 4 and b"too many psi" in lib.gisapr_last_error()
    for cluster in range(9):
        ok(lib.gisapr_set_tuning(context, 1, 48, cluster), "tuning")
        ok(call(48, 12, 3), "general size")
        assert call(48, 12, 400) == 4
""", tmp_path)
