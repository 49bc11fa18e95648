"""What the library's host code decides, over a CUDA runtime without a GPU
(fake_runtime.py)."""
import ctypes
import os
import subprocess

import pytest

from gpusharesat_gb300 import build

from fake_runtime import Fake, i64, vp


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


@pytest.fixture(autouse=True)
def clean(fake):
    fake.reset()
    yield
    fake.reset()


@pytest.mark.parametrize("what", ["malloc_host", "malloc"])
def test_engine_that_cannot_be_made_leaves_no_stream(fake, what):
    before = fake.lib.fake_streams()
    for after in range(3):
        fake.fail(what, after)
        rc, h = fake.engine()
        if rc == 0:  # fewer such allocations than that
            assert fake.lib.gss_engine_destroy(h) == 0
        else:
            assert h.value is None
        assert fake.lib.fake_streams() == before
    fake.fail(what)
    assert fake.engine()[0] != 0


def _noalloc(fake, lits=0, offsets=0, state=0, start=0, sow=0, out=0, counts=0, n=100):
    """One pass over buffers shifted by so many bytes; nothing is read."""
    room = ctypes.create_string_buffer(1 << 16)
    base = (ctypes.addressof(room) + 255) // 256 * 256
    p = [vp(base + 4096 * k + s) for k, s in enumerate((lits, offsets, state, start, sow, out, counts))]
    fake.reset()
    rc = fake.lib.gss_check_noalloc(p[0], p[1], n, p[2], 10, 1, p[3], p[4], p[5], 4, 16, p[6], None)
    return rc, [l.split()[1] for l in fake.log() if l.startswith("launch")], fake.log()


def test_noalloc_queue_address_picks_the_stores(fake):
    """A 16-byte store needs a queue on 16 bytes; a gss_report needs 4."""
    rc, wide, _ = _noalloc(fake)
    assert rc == 0 and len(wide) == 2 and "check_wide_persist" in wide[0]
    assert _noalloc(fake, out=16)[1] == wide and _noalloc(fake, out=32)[1] == wide
    by_word = set()
    for shift in (4, 8, 12, 20):
        rc, names, _ = _noalloc(fake, out=shift)
        assert rc == 0 and "check_wide_persist" in names[0]
        by_word.add(names[0])
    assert len(by_word) == 1 and wide[0] not in by_word


def test_noalloc_refuses_what_the_kernel_cannot_read(fake):
    for kw in ({"state": 8}, {"state": 16}, {"lits": 2}, {"offsets": 4}, {"start": 1}, {"sow": 2}, {"out": 2}):
        rc, names, _ = _noalloc(fake, **kw)
        assert rc == -1 and not names, kw
        assert _noalloc(fake, n=0, **kw)[0] == 0  # nothing to read
    rc, names, log = _noalloc(fake, counts=1)  # copied, not stored by a kernel
    assert rc == 0 and len(names) == 1 and any(l.startswith("copy2d") for l in log)


def test_staged_records_lie_on_16_bytes_by_type(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-I", os.path.join(build.ROOT, "include"), "-I",
                    build.CSRC, "-c", os.path.join(here, "cpp", "stage_alignment.cu"), "-o",
                    str(tmp_path / "stage_alignment.o")], check=True)
