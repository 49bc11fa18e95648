"""What the library's host code decides, over a CUDA runtime without a GPU
(fake_runtime.py)."""
import pytest

from fake_runtime import Fake


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
