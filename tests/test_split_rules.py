"""Split counts where the rows' lengths are known, and where the caller has no more than a bound on them: the rules, and what the calls hand to the library."""
import types
import pytest
from gaac_b200.kernel import choose_flat256, choose_nsplit256, choose_nsplit_sm100


class _Tensor:
    """What the calls ask a tensor for before the library is called."""
    def __init__(self, *shape): self.shape, self.device, self.is_cuda = shape, types.SimpleNamespace(type="cuda", index=0), True
    def size(self, i): return self.shape[i]
    def stride(self, i): return self.shape[-1] if i == 0 else 1
    def numel(self): return 1 << 20
    def data_ptr(self): return 0


@pytest.fixture
def calls(monkeypatch):
    """The calls that reach the native module: (name, arguments)."""
    from gaac_b200 import _lib, kernel
    from gaac_b200.vllm import paged_kernel, paged_kernel256
    made = []

    class Recording:
        def __getattr__(self, name): return lambda *a: made.append((name, a)) or 0
    monkeypatch.setattr(_lib, "host", Recording)
    monkeypatch.setattr(_lib, "stream_ptr", lambda dev: 0)
    for module in (kernel, paged_kernel, paged_kernel256): monkeypatch.setattr(module, "workspace", lambda *a: _Tensor(1))
    return made


def _paged(calls, B, n_kv, G, blocks, wide=False, bases=(1, 2, 3, 4)):
    from gaac_b200.vllm.paged_kernel import paged_attention
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    call = paged_attention256 if wide else paged_attention
    call(_Tensor(B, n_kv * G, 256 if wide else 128), "out", "buf", "raw", "mt", _Tensor(B, blocks), "seq_lens", bases, 3008, n_kv * G, n_kv)
    return calls.pop()


@pytest.mark.parametrize("tiles", [1, 9, 10, 12, 13, 16, 17, 28])
@pytest.mark.parametrize("B,n_kv", [(1, 1), (1, 8), (2, 8), (9, 2), (40, 1)])
def test_rows_of_one_cta_are_no_teams(calls, B, n_kv, tiles):
    """Up to 16 tiles a row takes one CTA wherever its length is read on the GPU: a count above one would only make a cluster of it."""
    name, a = _paged(calls, B, n_kv, 4, tiles)
    assert name == "gaac_paged_decode_attn" and (a[8] == 1) == (tiles <= 16)
    assert (choose_nsplit_sm100(B, n_kv, 16 * tiles, bound=True) == 1) == (tiles <= 16)
    if B * n_kv <= 22: assert (choose_nsplit_sm100(B, n_kv, 16 * tiles) == 1) == (tiles <= 12)              # lengths known


@pytest.mark.parametrize("rows,most", [(15, 8), (16, 6), (22, 6), (23, 5), (24, 5), (25, 4), (26, 4), (33, 4), (34, 3), (43, 3), (44, 2), (45, 2), (74, 2), (75, 1)])
def test_teams_of_three_and_five_are_not_packed_to_the_last(rows, most):
    for bound in (False, True): assert choose_nsplit_sm100(rows, 1, 16 * 28, bound=bound) == (most if most > 1 else 1)


@pytest.mark.parametrize("B,n_kv", [(2, 8), (3, 4), (8, 2), (16, 1), (9, 4)])
def test_equal_ranges_up_to_a_tile_per_warp(calls, B, n_kv):
    wave = 148 // (B * n_kv)
    for tiles, name in ((16 * wave, "gaac_paged_decode_attn"), (16 * wave + 1, "gaac_paged_decode_attn_balanced")):
        made = _paged(calls, B, n_kv, 4, tiles)
        assert made[0] == name and (name.endswith("balanced") or made[1][8] == wave)


@pytest.mark.parametrize("B,n_kv,tiles,G,splits", [
    (1, 8, 8, 4, 1), (1, 8, 9, 4, 3), (1, 8, 9, 8, 1), (1, 8, 16, 8, 1), (1, 8, 17, 8, 5), (27, 2, 18, 4, 2), (27, 2, 18, 8, 1), (27, 2, 25, 8, 2), (40, 1, 18, 8, 3),
    (1, 1, 64, 4, 16), (1, 1, 70, 4, 16), (1, 1, 128, 4, 16), (1, 1, 150, 4, 19), (1, 8, 150, 4, 16), (1, 4, 250, 8, 32), (1, 8, 256, 8, 16), (1, 8, 400, 8, 18), (1, 2, 600, 4, 32), (1, 1, 5000, 4, 143)])
def test_counts_of_head_dim_256(calls, B, n_kv, tiles, G, splits):
    name, a = _paged(calls, B, n_kv, G, tiles, wide=True)
    assert name == "gaac_paged_decode_attn256" and a[8] == splits == choose_nsplit256(B, n_kv, 16 * tiles, group=G)


@pytest.mark.parametrize("B,n_kv,tiles,G,flat", [(20, 8, 70, 4, False), (20, 8, 159, 8, False), (20, 8, 160, 4, True), (27, 2, 47, 4, False), (27, 2, 48, 4, True), (27, 2, 48, 8, False), (27, 2, 49, 8, True),
                                                 (2, 1, 600, 4, True), (2, 1, 600, 8, False), (16, 2, 64, 4, False), (16, 2, 65, 4, True), (1, 8, 600, 4, False)])
def test_flat_launches_of_head_dim_256(calls, B, n_kv, tiles, G, flat):
    name, a = _paged(calls, B, n_kv, G, tiles, wide=True)
    assert (name == "gaac_paged_decode_attn256_flat") == flat == (choose_flat256(B, n_kv, 16 * tiles, group=G) > 0)
