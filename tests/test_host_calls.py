"""The calls that the library's host code makes, on a runtime without a GPU
(fake_gpu.py): what a projector writes is in place before a stream reads it."""
import pytest

import fake_gpu


@pytest.fixture(scope="module")
def gpu(tmp_path_factory):
    so = fake_gpu.build(tmp_path_factory.mktemp("fake"))
    return lambda script: fake_gpu.run(so, script)


GEOMS = '''
G3 = (ImageGeom(32, 32, 21, 2.0, 2.0, 2.0), Sino3DGeom.span1(16, 40, 11, 33.0, 22.0, 100.0, 1))
G2 = (ImageGeom(32, 32, 1, 2.0, 2.0, 2.0), Sino2DGeom(16, 40, 33.0, 100.0))
'''


def waited(log):
    """The legacy stream was waited for after the last write on it."""
    writes = [i for i, l in enumerate(log) if l.split()[:2] in (["memset", "legacy"], ["memcpy", "legacy"])]
    waits = [i for i, l in enumerate(log) if l.split()[:2] == ["sync", "legacy"]]
    return bool(writes) and bool(waits) and waits[-1] > writes[-1]


@pytest.mark.parametrize("step", ["ap.SiddonProjector(*G3)", "ap.SiddonProjector(*G2)", "P.set_sampling(2, 2)",
                                  "P.set_alpha_precision(True)",
                                  "P.set_option(_lib.APIRL_OPT_ACCUMULATE, _lib.APIRL_ACC_COMPENSATED)"])
def test_tables_and_zeros_are_waited_for(gpu, step):
    """Non-blocking streams do not wait for the legacy stream, on which tables are copied and buffers cleared."""
    log = gpu(GEOMS + f"P = ap.SiddonProjector(*G3)\nfake.clear()\n{step}\ndone(fake.log())")
    assert waited(log), log


def test_second_pair_is_cleared_on_the_callers_stream(gpu):
    log = gpu(GEOMS + '''
P = ap.SiddonProjector(*G3)
fake.clear()
_lib.check(lib.apirl_backproject_and_ones(P.h, D, D, ctypes.c_void_p(1 << 42), -1, 1, S))
done(fake.log())''')
    assert any(l.startswith("memset 0x9990") for l in log)
    assert not any(l.split()[:2] == ["memset", "legacy"] for l in log), log


@pytest.mark.parametrize("nz", [1, 2])
def test_2d_passes_update_every_slice(gpu, nz):
    """The padded 2D layouts hold one slice; an image of several takes the pass that updates all its voxels."""
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom(32, 32, {nz}, 2.0, 2.0, 2.0), Sino2DGeom(16, 40, 33.0, 100.0))
fake.clear()
_lib.check(lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, None, S))
done(fake.launches())''')
    assert any("k_planar_update" in n for n in names) == (nz == 1)
    assert any("k_update" in n for n in names) == (nz == 2)


@pytest.mark.parametrize("ny", [65534 * 8, 65534 * 8 + 1, 65535 * 8 - 1])
def test_tall_2d_images_stay_within_the_grid(gpu, ny):
    """The update's grid has one row of blocks a tile row of 8 and one for the likelihood, 65535 at most."""
    log = gpu(f'''
P = ap.SiddonProjector(ImageGeom(4, {ny}, 1, 2.0, 2.0, 2.0), Sino2DGeom(3, 4, 33.0, 100.0))
fake.clear()
st = lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, D, S)
done([st] + fake.log())''')
    assert log[0] == 0 and not any(l.startswith("refused") for l in log[1:]), log


@pytest.mark.parametrize("nz", [65534 * 32, 65534 * 32 + 1])
def test_long_images_stay_within_the_grid(gpu, nz):
    """As above for the column layout's update, whose grid has a layer more than 32 slices each (images of
    more than 65535 slices that keep to the padded pair have no pass, and had none)."""
    log = gpu(f'''
P = ap.SiddonProjector(ImageGeom(8, 8, {nz}, 2.0, 2.0, 0.01), Sino3DGeom.span1(3, 4, 16, 16.0, 500.0, 100.0, 0))
fake.clear()
st = lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, D, S)
done([st] + fake.log())''')
    cols = any("k_em_cols" in l for l in log[1:])
    assert cols == (nz == 65534 * 32) and not any(l.startswith("refused") and "k_col" in l for l in log[1:]), log
