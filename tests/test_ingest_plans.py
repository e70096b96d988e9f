"""The transforms that a context keeps for the particle preparation, on a fake CUDA runtime (no kernel runs)."""
from .fakes.runtime import run_on_fake

CALLS = r"""
context = C.c_void_p()
ok(lib.gisapr_context_create(0, C.byref(context)), "context")
def call(n, size, stream=None, flags=7):
    ok(lib.gisapr_ingest_stack(context, stream, p, n, size, size, None, size, size, flags, p, p, p, 9, p, p, p), "ingest")
"""


def test_every_call_waits_for_the_one_before(native_lib, tmp_path):
    """The work area is shared by all calls. A stream made where a destroyed one was has its handle, so an equal
    handle does not order the two."""
    run_on_fake(CALLS + r"""
for k in range(1, 6):
    call(4, 64, C.c_void_p(4096))
    assert fake.fake_recorded() == k
assert fake.fake_waited() >= 4, fake.fake_waited()
""", tmp_path)
