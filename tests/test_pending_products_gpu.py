"""The dense decoder on the GPU with the norms of its few-row steps inside the products around them, and without."""
import pytest
import torch

import plain_model
from util import make_model_dir, prompts, read_weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    return {n: make_model_dir(n, tmp_path_factory.mktemp(n)) for n in ("tiny_hd64", "tiny_hd128")}


@pytest.mark.parametrize("name", ["tiny_hd64", "tiny_hd128"])
@pytest.mark.parametrize("cuts", [(1,) * 12, (17, 8, 1), (33, 64, 31), (128, 1)])
def test_norms_inside_the_products_and_outside(folders, name, cuts):
    """bfloat16 steps of up to 128 rows with the norms in the products around them and in kernels of their own: one launch fewer for
    every norm behind a sublayer but the last, and logits as near to the 32-bit model's. (Two results that each round a row's
    values once, before its factor or behind it; a quarter more covers what the roundings of some hundred logits differ by.)"""
    from fusezap_core_b200 import load_model
    from fusezap_core_b200.cache import CacheManager
    from fusezap_core_b200.engine import Portion, StepRunner
    d, cfg, opts = folders[name]
    w = {k: v.to(torch.bfloat16) for k, v in read_weights(d).items()}
    model = load_model(d, "bfloat16", "cuda:0", max_len=256)
    ids = prompts(cfg, (sum(cuts),), seed=3)[0]
    ref = plain_model.forward(cfg, w, ids)
    error, launches = {}, {}
    for fused in (True, False):
        model.ops.fuse_norm = fused
        try:
            cache = CacheManager(model.cache_needs(), model.state_needs(), 16, 20, 1, 256, model.ops.dtype, "cuda:0")
            runner, out, at = StepRunner(model, cache, max_rows=128, max_segments=1), [], 0
            before = model.ops.launches
            for n in cuts:
                out.append(runner.run([Portion(0, ids[at: at + n], list(range(n)))]).clone())
                at += n
            launches[fused] = model.ops.launches - before
            model.ops.check_errors()
        finally:
            model.ops.fuse_norm = True
        error[fused] = float((torch.cat(out).cpu() - ref).norm() / ref.norm())
    assert launches[False] - launches[True] == len(cuts) * (2 * cfg["num_hidden_layers"] - 1)
    assert error[True] <= 1.25 * error[False] and error[False] < 0.03, error
