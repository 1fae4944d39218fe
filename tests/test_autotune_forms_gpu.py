"""The autotuner's cache tells meshes apart on which a variant number stands for
different kernels, and leaves records of an earlier set of kernels alone."""
import numpy as np
import pytest

import simplexfem as sf
from test_cg_patch_gpu import unstructured
from test_dg_fused_gpu import shuffled

pytestmark = pytest.mark.gpu


@pytest.fixture
def cache(tmp_path):
    path = tmp_path / "tune.jsonl"
    sf.set_autotune_cache(str(path))
    yield path
    sf.set_autotune_cache(None)


@pytest.mark.parametrize("components", [1, 3])
def test_box_and_unstructured_mesh(cuda, cache, components):
    """Equal cell counts: variant 1 is the patch form on the unstructured mesh, a thread
    per cell on the box, whose default is the block form."""
    for k, mesh in enumerate((unstructured((32, 32, 32)), sf.Mesh(32, jitter=0.1, seed=3))):
        for again in (False, True):
            op = sf.Operator(mesh, 2, "cg", "fp64", n_components=components)
            assert op.autotune(reps=3)["cached"] == again, (k, again)


def test_one_launch_and_two(cuda, cache):
    """DG P3 FP64: variant 1 is one launch, or two where most neighbours are outside a block."""
    assert not sf.Operator(sf.Mesh((6, 5, 7), jitter=0.1, seed=3), 3, "dg").autotune(reps=3)["cached"]
    mesh = shuffled((6, 5, 7))
    assert not sf.Operator(mesh, 3, "dg").autotune(reps=3)["cached"]
    ops = [sf.Operator(m, 3, "dg") for m in (sf.Mesh((6, 5, 7)), mesh)]
    assert not sf.Batch([ops[0], ops[0]]).autotune(reps=3)["cached"]
    assert not sf.Batch(ops).autotune(reps=3)["cached"]


def test_records_of_other_kernels(cuda, cache):
    import torch
    gpu = torch.cuda.get_device_name().replace(" ", "_")
    mesh = sf.Mesh(24, jitter=0.1, seed=3)
    lg = int(np.rint(np.log2(mesh.n_cells)))
    keys = [f"kind={kind},p=2,prec={prec},nc={nc},log2cells={lg},gpu={gpu}" for kind in (0, 1, 2) for prec in (0, 1)
            for nc in (1, 3)]
    cache.write_text("".join(f'{{"key": "{k}", "variant": 2, "us": []}}\n' for k in keys))
    sf.set_autotune_cache(str(cache))
    for kind in ("cg", "dg"):
        assert not sf.Operator(mesh, 2, kind).autotune(reps=3)["cached"]
