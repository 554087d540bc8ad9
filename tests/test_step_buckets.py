"""Which steps replay a captured graph, and padded to what: the runner's decisions, which need no GPU."""
import types

from vllm_cpp_b200.engine.step import ModelRunner, StepEntry


def fake_runner(graphs=True, page_size=16):
    r = types.SimpleNamespace(cuda_graphs=graphs, page_size=page_size, page_sizes=[page_size])
    for name in ("GRAPH_BUCKETS", "PORTION_BUCKETS", "MIXED_SINGLES", "MIXED_PORTIONS", "MIXED_TOKENS"):
        setattr(r, name, getattr(ModelRunner, name))
    for name in ("capture_size", "portion_size", "mixed_size", "rows_capacity", "_mixed_updates", "_portion_updates"):
        setattr(r, name, types.MethodType(getattr(ModelRunner, name), r))
    return r


def entry(n, want="last", slot=0, start=0):
    return StepEntry(slot, start, list(range(n)), [[0] * 64], {"last": [n - 1], "none": [], "all": list(range(n))}[want])


def test_single_tokens_round_up_to_a_power_of_two():
    r = fake_runner()
    assert r.capture_size([entry(1, slot=i) for i in range(5)]) == 8
    assert r.capture_size([entry(1)]) == 1
    assert r.capture_size([entry(1, slot=i) for i in range(257)]) is None
    assert r.capture_size([entry(1), entry(2, slot=1)]) is None
    assert r.capture_size([entry(1, want="none")]) is None            # no logits wanted: not a decoding step
    assert fake_runner(graphs=False).capture_size([entry(1)]) is None


def test_a_lone_portion_rounds_up_to_its_bucket():
    r = fake_runner()
    assert r.portion_size([entry(2)]) == 16
    assert r.portion_size([entry(16, want="none")]) == 16
    assert r.portion_size([entry(17)]) == 32
    assert r.portion_size([entry(512)]) == 512
    assert r.portion_size([entry(513)]) is None
    assert r.portion_size([entry(40, want="all")]) is None            # logits wanted at other places than the last
    assert r.portion_size([entry(40), entry(1, slot=1)]) is None
    assert r.portion_size([entry(1)]) is None
    assert r._portion_updates(64) == 64 // 16 + 2


def test_single_tokens_beside_portions():
    r = fake_runner()
    singles = [entry(1, slot=i) for i in range(5)]
    assert r.mixed_size(singles + [entry(60, slot=9)]) == (8, 96)
    assert r.mixed_size(singles + [entry(56, slot=9)]) == (8, 64)      # 8 slots + 56 tokens fill 64 rows exactly
    assert r.mixed_size([entry(30, slot=1), entry(20, slot=2)]) == (0, 64)     # portions only
    assert r.mixed_size([entry(1, slot=i) for i in range(40)] + [entry(100, slot=50)]) == (64, 192)
    assert r.mixed_size(singles + [entry(300, slot=9)]) is None        # more than 256 rows: kernel by kernel
    assert r.mixed_size([entry(1, slot=i) for i in range(65)] + [entry(10, slot=70)]) is None
    assert r.mixed_size(singles + [entry(10, slot=10 + i) for i in range(5)]) is None   # five portions
    assert r.mixed_size([entry(60, slot=9)] + singles) is None         # single tokens must come first
    assert r.mixed_size(singles + [entry(60, slot=9, want="all")]) is None
    assert r.mixed_size(singles) is None                               # that is a decoding step
    assert r.mixed_size([entry(60)]) is None                           # and that a lone portion
    # a one-token entry without logits (the last token of a portion cut by the budget) takes a single-token slot
    assert r.mixed_size([entry(1, want="none")] + [entry(30, slot=3)]) == (8, 64)


def test_rows_of_logits_a_step_computes():
    r = fake_runner()
    singles = [entry(1, slot=i) for i in range(5)]
    assert r.rows_capacity(singles) == 8
    assert r.rows_capacity(singles + [entry(60, slot=9)]) == 8 + ModelRunner.MIXED_PORTIONS
    assert r.rows_capacity([entry(60)]) == 1
    assert r.rows_capacity([entry(600), entry(700, slot=1, want="none")]) == 1
    assert fake_runner(graphs=False).rows_capacity(singles) == 5


def test_portions_pad_to_half_way_steps_from_64_on():
    r = fake_runner()
    assert [r.portion_size([entry(n)]) for n in (64, 65, 96, 97, 129, 193, 257, 385)] == [64, 96, 96, 128, 192, 256, 384, 512]


def test_portions_whose_launches_hide_run_kernel_by_kernel():
    """A 32-bit engine's portions beyond its limit are not padded: neither alone nor beside single tokens."""
    r = fake_runner()
    r.capture_limit = 44
    assert r.portion_size([entry(44)]) == 64 and r.portion_size([entry(45)]) is None
    singles = [entry(1, slot=i) for i in range(5)]
    assert r.mixed_size(singles + [entry(39, slot=9)]) == (8, 64) and r.mixed_size(singles + [entry(40, slot=9)]) is None
    assert r.capture_size(singles) == 8                     # single tokens stay captured
    from vllm_cpp_b200.engine.step import _launches_hide_from
    spec = lambda *shape, role="matrix": types.SimpleNamespace(shape=shape, role=role)
    part = lambda *specs, **kw: types.SimpleNamespace(tensor_specs=lambda: list(specs), **kw)
    layer = types.SimpleNamespace(parts=dict(a=part(spec(6144, 2560), spec(2560, role="vector")), b=part(spec(9728 * 3, 2560), spec(4096, 2560)),
                                             c=part(spec(100, 1000, 1000), spec(1 << 20, 1 << 10), top=2)))
    model = types.SimpleNamespace(layers=[layer], order=[types.SimpleNamespace(layer=0)] * 36)
    assert 30 < _launches_hide_from(model) < 60
    assert _launches_hide_from(types.SimpleNamespace()) is None


def test_portions_that_fill_their_bucket_stay_captured_beyond_the_limit():
    """Beyond the limit a 32-bit engine's portions run kernel by kernel only where their bucket has more rows of products, in whole
    tiles of 32 to 64 rows, than would make up for the launches."""
    r = fake_runner()
    r.capture_limit = 44
    sizes = {n: r.portion_size([entry(n)]) for n in range(2, 513)}
    for low, high, padded in ((2, 44, (16, 32, 64)), (57, 64, (64,)), (81, 96, (96,)), (121, 128, (128,)), (169, 192, (192,)), (241, 256, (256,)),
                              (361, 384, (384,)), (505, 512, (512,))):
        assert all(sizes[n] in padded for n in range(low, high + 1)), (low, high)
    for low, high in ((45, 56), (65, 80), (97, 120), (129, 168), (193, 240), (257, 320), (385, 448)):
        assert all(sizes[n] is None for n in range(low, high + 1)), (low, high)
    singles = [entry(1, slot=i) for i in range(8)]
    assert r.mixed_size(singles + [entry(56, slot=9)]) == (8, 64) and r.mixed_size(singles + [entry(88, slot=9)]) == (8, 96)
    assert r.mixed_size(singles + [entry(40, slot=9)]) is None
    r.capture_limit = 23
    assert [r.portion_size([entry(n)]) for n in (24, 28, 32, 33, 40, 64)] == [32, 32, 32, None, None, 64]
    r.capture_limit = None
    assert all(r.portion_size([entry(n)]) is not None for n in range(2, 513))
