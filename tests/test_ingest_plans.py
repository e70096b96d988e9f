"""The transforms that a context keeps for the particle preparation, on a fake CUDA runtime (no kernel runs)."""
from .fakes.runtime import run_on_fake

CALLS = r"""
context = C.c_void_p()
ok(lib.gisapr_context_create(0, C.byref(context)), "context")
def call(n, size, stream=None, flags=7):
    ok(lib.gisapr_ingest_stack(context, stream, p, n, size, size, None, size, size, flags, p, p, p, 9, p, p, p), "ingest")
"""


def test_a_call_on_another_stream_waits_for_the_one_before(native_lib, tmp_path):
    """The work area is shared by all calls. A stream made where a destroyed one was has its handle, so an equal
    handle does not order the two."""
    run_on_fake(CALLS + r"""
for k in range(1, 11):
    fake.fake_new_stream()
    for again in range(2):
        call(4, 64, C.c_void_p(4096))
    assert fake.fake_recorded() == 2 * k
    assert fake.fake_waited() >= k, fake.fake_waited()
""", tmp_path)


def test_kept_transforms_share_one_work_area(native_lib, tmp_path):
    """Calls of many shapes leave one work area behind, as large as the largest took, whatever the order (and a few kB
    of notes on their tables); one above 1 GB is gone after the call, and so is everything with the context."""
    run_on_fake(CALLS + r"""
fake.fake_held.restype = C.c_longlong
fake.fake_plan_bytes.argtypes = [C.c_longlong]
MB = 1 << 20
call(1, 32, flags=2)
empty = fake.fake_held()
for turn in range(3):
    for n, size, take in ((5, 64, 100), (6, 64, 120), (7, 32, 40), (8, 48, 300), (9, 50, 20), (10, 64, 200)):
        fake.fake_plan_bytes(take * MB)
        call(n, size)
        assert fake.fake_held() - empty <= 301 * MB, (turn, n, (fake.fake_held() - empty) // MB)
fake.fake_plan_bytes(3000 * MB)
call(11, 64)
assert fake.fake_held() - empty <= 301 * MB, (fake.fake_held() - empty) // MB
fake.fake_plan_bytes(100 * MB)
call(12, 64)
call(12, 64, flags=1)
assert fake.fake_held() - empty <= 301 * MB
ok(lib.gisapr_context_destroy(context), "destroy")
assert fake.fake_held() == 0, fake.fake_held()
""", tmp_path)
