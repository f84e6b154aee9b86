"""The encoder's launch of many steps, which rules candidates and lines out by bounds of their error (csrc/encode.cu), against single steps,
which evaluate them: the same encoding bit for bit, over scales at which squares are subnormal or large, ranges that bounds are not
made for, repeated values, lists longer than the kernel's tables, and several windows of groups."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _same(W, conf):
    from sbvr import encoder
    one = encoder.encode(W, conf, progress=lambda done, of: None)
    many = encoder.encode(W, conf)
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one[:3], many[:3])) and one[3] == many[3]
    return many[3]


def _values(kind, rows, cols, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((rows, cols), device="cuda", generator=g)
    if kind == "normal":
        x = x * 0.02 * torch.exp(0.3 * torch.randn((rows, 1), device="cuda", generator=g))
    elif kind == "tiny":                           # squares of the errors are subnormal
        x = x * 4e-4
    elif kind == "large":
        x = x * 2.5
    elif kind == "beyond":                         # above the range that bounds are made for
        x = x * 12.0
    elif kind == "mean":
        x = x * 0.02 + 0.1
    elif kind == "levels":                         # few different values, many of them equal
        x = torch.round(x * 3) * 0.01
    elif kind == "sparse":
        x = x * 0.05 * (torch.rand((rows, cols), device="cuda", generator=g) < 0.2)
    elif kind == "outlier":
        x = x * 0.01
        x[:, ::256] *= 40
    elif kind == "uniform":
        x = (torch.rand((rows, cols), device="cuda", generator=g) - 0.3) * 0.2
    return x.half()


@pytest.mark.parametrize("S", [2, 3, 4])
@pytest.mark.parametrize("kind", ["normal", "tiny", "large", "beyond", "mean", "levels", "sparse", "outlier", "uniform"])
def test_bounds_leave_the_encoding_as_it_is(kind, S):
    from sbvr import encoder
    stats = _same(_values(kind, 12, 1024, S), encoder.EncoderConfig(num_sums=S))
    assert stats["cache_lines"] >= 1


@pytest.mark.parametrize("settings", [
    {"r_search_num": 300, "b_search_num": 6, "s_search_num": 8},       # more ratios than the tables in shared memory hold
    {"r_search_num": 6, "b_search_num": 5, "s_search_num": 3},         # fewer candidates than threads
    {"r_search_num": 1000, "b_search_num": 60, "s_search_num": 40},    # more candidates than quotients by reciprocals are exact for
])
def test_other_search_spaces(settings):
    from sbvr import encoder
    _same(_values("normal", 4, 1024, 7), encoder.EncoderConfig(num_sums=3, **settings))


def test_several_windows_of_groups():
    """8192 groups: more than a window has warps, so that later windows meet many lines at once, bounded 32 at a time."""
    from sbvr import encoder
    stats = _same(_values("normal", 512, 4096, 3), encoder.EncoderConfig(num_sums=2))
    assert stats["groups"] == 8192 and stats["cache_lines"] > 16
