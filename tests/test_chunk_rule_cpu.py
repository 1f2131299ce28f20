"""The choice between a recurrence's one-pass and chunk forms, at steps whose times are known on both sides -- all of chunks of 64 rows by
FMAs, which the rule was fitted to (linear attention and mLSTM run theirs on the tensor cores, where more steps would gain)."""
import pytest

from gpustack_b200 import config, ops
from gpustack_b200.lib import load

WIDTHS = {"linear": (128, 128), "mlstm": (128, 128), "gated_linear": (64, 128), "state_space": (128, 64)}


# kind, heads, portions (rows), one-pass us, chunk us (L2 cold)
@pytest.mark.parametrize("kind,H,lens,one,chunk", [
    ("linear", 8, [64], 34.8, 40.0), ("linear", 8, [128], 57.3, 42.0), ("linear", 32, [2048], 761.9, 205.7),
    ("linear", 8, [32] * 16, 55.3, 74.8), ("linear", 8, [64] * 16, 92.2, 80.9), ("linear", 8, [2048] + [16] * 30, 1252.4, 126.0),
    ("linear", 8, [128] * 4 + [1] * 100, 198.7, 178.8), ("mlstm", 8, [64] * 16, 113.5, 126.0), ("mlstm", 8, [128] * 16, 200.7, 131.9),
    ("mlstm", 16, [512] * 4 + [1] * 100, 845.8, 617.5), ("mlstm", 8, [2048] + [1] * 64, 840.5, 230.4),
    ("gated_linear", 8, [256], 47.1, 50.2), ("gated_linear", 8, [512], 84.0, 52.2), ("gated_linear", 8, [128] * 16, 69.6, 82.9),
    ("gated_linear", 8, [128] * 4 + [1] * 100, 96.2, 134.2), ("gated_linear", 8, [2048] + [16] * 30, 448.5, 107.5),
    ("gated_linear", 16, [512] * 4, 118.8, 130.0), ("state_space", 32, [1024], 108.5, 87.0), ("state_space", 32, [512] * 4, 120.8, 148.5),
    ("state_space", 32, [512] * 16, 399.4, 531.5), ("state_space", 32, [2048] + [16] * 30, 477.2, 195.3)], ids=str)
def test_the_faster_form_is_chosen(kind, H, lens, one, chunk):
    dk, dv = WIDTHS[kind]
    pays = lambda longest: ops.chunk_scan_pays(kind, sum(lens), len(lens), H, dk, dv, longest)   # noqa: E731
    assert pays(max(lens)) == (chunk < one)
    if len(set(lens)) == 1:
        assert pays(sum(lens)) == (chunk < one)                # all rows as the bound: portions are taken for equal


@pytest.mark.parametrize("kind", sorted(WIDTHS))
def test_single_rows_and_other_widths_stay_one_pass(kind):
    dk, dv = WIDTHS[kind]
    for n in (1, 7, 256, 4096):
        assert not ops.chunk_scan_pays(kind, n, n, 128, dk, dv, 1)
    assert ops.chunk_scan_pays(kind, 4096, 2, 8, dk, dv, 2048)
    for a, b in ((96, dv), (dk, dv + 2), (256, dv)):
        assert not ops.chunk_scan_pays(kind, 4096, 2, 8, a, b, 2048)


def test_the_runner_states_the_longest_portion():
    """A prompt step hands its scans the longest portion, not the sum of the portions."""
    from pathlib import Path

    root = Path(ops.__file__).parent
    assert "self.longest_portion = max(lens" in (root / "runner.py").read_text()
    text = (root / "layer_list_runner.py").read_text()
    for scan in ("linattn_scan", "mlstm_scan", "gla_scan"):
        call = text[text.index("ops." + scan):]
        assert "max_len=self.longest_portion" in call[:call.index("ops.", 4)]


@pytest.mark.parametrize("rows,n", [(1, 1), (17, 3), (63, 1), (64, 64), (8192, 256), (100000, 5)])
def test_the_workspace_has_one_size(rows, n):
    for H, dk, dv, per_channel in ((1, 64, 36, False), (8, 64, 128, True), (32, 128, 64, False)):
        size = (rows // 64 + min(n, rows // 17)) * H * (dk * dv + dk + 4 + (128 * dk if per_channel else 0))    # as the header has it
        assert config.chunk_scan_floats(rows, n, H, dk, dv, per_channel) == load().b200_chunk_scan_floats(rows, n, H, dk, dv, int(per_channel)) == size


def test_the_workspace_is_in_the_memory_estimate():
    """The estimate of a model with such a recurrence counts what the runner allocates for the chunks."""
    from gpustack_b200 import resource_fit
    from gpustack_b200.config import EngineConfig, LinearAttentionSpec

    class Layer:
        mlp = None

        def __init__(self, dim):
            self.mixer = LinearAttentionSpec(heads=8, dim=dim, vdim=128, decay=(0.9,) * 8)

    class Model:
        family, hidden_size, vocab_size, residual, max_position_embeddings = "layer_list", 1024, 1000, "parallel", 4096
        loop_times, n_streams = 1, 1

        def __init__(self, dim):
            self.layers = [Layer(dim)]

        def state_bytes_per_seq(self):
            return 0

    e = EngineConfig(max_num_seqs=64, max_num_batched_tokens=8192)
    with_chunks, without = (resource_fit._layer_list_workspace(Model(d), e) for d in (128, 96))
    ws = 4 * config.chunk_scan_workspace_floats(Model(128).layers, 8192, 64)
    assert ws == 4 * (128 + 64) * 8 * (128 * 128 + 132)
    assert config.chunk_scan_workspace_floats(Model(96).layers, 8192, 64) == 0
    assert with_chunks - without > ws
    assert config.chunk_scan_workspace_floats(Model(128).layers, 10 ** 7, 256) * 4 == config.CHUNK_SCAN_MAX_BYTES
