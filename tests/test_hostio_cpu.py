"""What the field transfers (csrc/hostio.cu) promise their callers, over a CUDA
runtime of host memory (tests/fake_cuda) whose streams run when they are waited
for: a copy that is still queued shows as one, on any machine."""
import pathlib
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "gpu-comcot_b200" / "csrc"


@pytest.fixture(scope="module")
def scenario(tmp_path_factory):
    exe = tmp_path_factory.mktemp("hostio") / "hostio"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{HERE / 'fake_cuda'}", f"-I{CSRC}",
                    f"-I{HERE.parent / 'include'}", str(HERE / "fake_cuda" / "hostio_main.cpp"), "-o", str(exe)],
                   check=True)

    def run(*args):
        p = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=60)
        assert p.returncode == 0, (args, p.stdout, p.stderr)

    return run


# below the staging threshold, one staged piece, several with an odd last one
@pytest.mark.parametrize("nx,ny", [(33, 17), (200, 200), (300, 300), (2401, 2001)])
@pytest.mark.parametrize("kind", ["pageable", "locked", "managed"])
def test_source_may_change_after_an_upload(scenario, kind, nx, ny):
    scenario(kind, nx, ny)


@pytest.mark.parametrize("nx,ny", [(300, 300), (1201, 1001), (2401, 801)])   # a quarter of a slot, one slot, nearly one
@pytest.mark.parametrize("kind", ["beside-read", "beside-queued-read", "beside-upload"])
def test_transfers_do_not_wait_for_another_streams_work(scenario, kind, nx, ny):
    scenario(kind, nx, ny)


@pytest.mark.parametrize("nx,ny", [(33, 17), (300, 300), (2401, 2001)])
def test_transfers_on_a_device_that_is_not_current(scenario, nx, ny):
    scenario("foreign-device", nx, ny)


@pytest.mark.parametrize("nx,ny", [(33, 17), (300, 300), (2401, 2001)])
def test_callers_device_memory_is_left_to_the_runtime(scenario, nx, ny):
    scenario("device-caller", nx, ny)


def test_copy_without_memory_for_threads(scenario):
    scenario("no-memory")


@pytest.mark.parametrize("nx,ny", [(33, 17), (300, 300), (2401, 2001)])
@pytest.mark.parametrize("kind", ["ordered-locked", "ordered-managed", "ordered-device"])
def test_transfers_follow_earlier_work_on_their_stream(scenario, kind, nx, ny):
    scenario(kind, nx, ny)
