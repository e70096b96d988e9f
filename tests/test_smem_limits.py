"""The dynamic shared memory a kernel may take belongs to a device, and a process may hold contexts on several: every
launcher raises it on the device it launches on, and never lowers it (another thread's larger launch may be on its
way). Run on a fake CUDA runtime of two devices (fakes/cuda_two_devices.cpp), no kernel runs."""
from .fakes.runtime import run_on_fake

CHILD = r"""
contexts = []
for dev in (0, 1):
    c = C.c_void_p()
    ok(lib.gisapr_context_create(dev, C.byref(c)), "context")
    contexts.append(c)
def calls(c):
    for box in (32, 64, 96, 128, 192, 256):
        yield "particles", lib.gisapr_prepare_particles(c, None, p, 2, 3, p, p, None, p, box, box, p)
        yield "templates", lib.gisapr_project_templates(c, None, p, box, p, p, 2, p, None, p, box, p)
        if box not in (96, 192):
            yield "volume", lib.gisapr_volume_spectrum_blocked(c, None, p, box)
        for crop in (6, 10, 12):
            for psi in (1, 3):
                yield "correlate", lib.gisapr_correlate(c, None, p, p, p, p, 3, psi, box, crop, p, p, p)
        for precision in range(4):
            yield "tensor cores", lib.gisapr_correlate_tc_batch_ex(c, None, p, box * box * 4, 2, 2, p, p, p, p, p, 1, 3,
                                                                   3, box, 12, precision, None, None, 0, p, p, p, None)
    for size in (256, 64, 128, 512):  # larger before smaller
        for flags in (2, 3, 4, 7):
            yield "ingest", lib.gisapr_ingest_stack(c, None, p, 2, size, size, None, size, size, flags, p, p, p, 9, p, p, p)
    for box in (1024, 64, 256):
        yield "distance", lib.gisapr_restraint_edt(c, None, p, box, 1.0, p, p, p)
        yield "deposit", lib.gisapr_deposit(c, None, p, p, 5, p, box, 6, 1.0, 1.0, 1.0)
count = 0
for turn in range(2):
    for c in contexts:
        for what, rc in calls(c):
            ok(rc, what)
            count += 1
assert fake.fake_refused() == 0 and fake.fake_launched() > count, (fake.fake_refused(), fake.fake_launched())
assert fake.fake_lowered() == 0, fake.fake_lowered()
print("calls", count)
"""


def test_every_launcher_raises_the_limit_on_its_device(native_lib, tmp_path):
    assert run_on_fake(CHILD, tmp_path).startswith("calls ")
