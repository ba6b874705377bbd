"""The plain GEMM of few output tiles, split over K by the CTAs of a cluster, against fp64."""
import pytest
import torch

from flashoverlap_b200 import ops
from flashoverlap_b200.utils import config, layout

pytestmark = pytest.mark.gpu
HALF_ULP = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}


@pytest.fixture(scope="module")
def impl(cuda):
    i = ops.OverlapImpl()
    i.nccl_init(0, 1, [0] * 16)
    i.cutlass_init()
    return i


def _check(c, a, b, dt):
    """One rounding to the storage type, and fp32 sums of K products: their error is below
    K * 2^-24 * sum |a b| and, for random signs, far below 2^-18 * sum |a b|."""
    ref = a.double() @ b.double().t()
    bound = 2.02 * HALF_ULP[dt] * ref.abs() + 2.0 ** -18 * (a.double().abs() @ b.double().abs().t()) + 2.0 ** -24
    assert ((c.double() - ref).abs() <= bound).all()


# smallest K, a K that no split divides, K with a partial k-block, one tile, the largest tile counts of
# each split, N that only 128-wide tiles divide
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,algo", [(128, 256, 256, 0), (128, 1024, 1000, 1), (128, 8192, 3584, 0), (256, 4096, 1096, 1),
                                        (128, 1152, 4096, 2), (384, 1280, 72 * 64 + 8, 24), (512, 512, 2048, 3),
                                        (2176, 1024, 520, 0)])
def test_split_gemm_natural(cuda, impl, dt, M, N, K, algo):
    algo = config.default_solution(M, N, algo)["Algo"]
    a = (torch.randn(M, K, device=cuda) * 0.5).to(dt)
    b = (torch.randn(N, K, device=cuda) * 0.5).to(dt)
    try:
        for split in (-1, 0, 2, 4, 8):
            impl.set_option("split_k", split)
            c = torch.full((M, N), float("nan"), device=cuda, dtype=dt)
            impl.cutlass_gemm(a, b, c, algo)
            _check(c, a, b, dt)
            ran = impl.get_option("last_split")
            if split >= 0:       # a forced split runs wherever K has that many k-blocks and the clusters fit at once
                ctas = (M // 128) * (N // 128) * split
                if split == 0 or (K + 63) // 64 < split or ctas > impl.get_option("sm_count"):
                    assert ran == 0
                elif ctas <= impl.get_option("sm_count") * 3 // 4:
                    assert ran == split
            elif (M, N, K) == (128, 8192, 3584):
                assert ran == 2          # the decode batch: 64 tiles, bound by one SM's share of the loads
            again = torch.empty_like(c)
            impl.cutlass_gemm(a, b, again, algo)
            assert torch.equal(c, again)             # the partial sums are added in a fixed order
    finally:
        impl.set_option("split_k", -1)
    impl.check_status()


@pytest.mark.parametrize("M,N,K,algo,rldn", [(128, 2048, 1024, 0, 1), (256, 1024, 520, 2, 2), (256, 512, 4096, 1, 1)])
def test_split_gemm_reordered(cuda, impl, M, N, K, algo, rldn):
    p = config.algo_params(algo)
    tm, tn = M // p["BM"], N // p["BN"]
    dt = torch.bfloat16
    a = (torch.randn(M, K, device=cuda) * 0.5).to(dt)
    b = (torch.randn(N, K, device=cuda) * 0.5).to(dt)
    RA = torch.randperm(tm * tn, device=cuda, dtype=torch.int32)
    e = torch.empty(0, dtype=torch.int32)
    mm = torch.zeros(tm + 1, tn, device=cuda, dtype=torch.int32)
    try:
        for split in (-1, 2, 4, 8):
            impl.set_option("split_k", split)
            c = torch.full((M, N), float("nan"), device=cuda, dtype=dt)
            impl.gemm_allreduce_overlap(a, b, c, mm, RA, rldn, e, e.to(cuda), algo, False)
            small = (M // 128) * (N // 128) * split <= impl.get_option("sm_count") * 3 // 4
            assert split == -1 or (K + 63) // 64 < split or not small or impl.get_option("last_split") == split
            _check(layout.from_reordered(c.cpu(), M, N, p["BM"], p["BN"], RA.cpu(), rldn).to(cuda), a, b, dt)
    finally:
        impl.set_option("split_k", -1)
    impl.check_status()


def _ran(impl):
    """(Algo whose kernel the last GEMM ran, its split, its units computed as halves)"""
    return tuple(impl.get_option(name) for name in ("last_algo", "last_split", "last_tail"))


# odd row tiles on pairs, 512-row units with nothing to fill them, 256-wide tiles computed as 128-wide ones
@pytest.mark.parametrize("M,N,K,algo", [(1920, 5376, 1000, 0), (512, 4096, 520, 3), (256, 8192, 320, 1), (640, 1152, 200, 2)])
def test_stand_in_kernels(cuda, impl, M, N, K, algo):
    """A small or ragged problem may run on another kernel than its Algo's: same values, same layout."""
    dt = torch.bfloat16
    a = (torch.randn(M, K, device=cuda) * 0.5).to(dt)
    b = (torch.randn(N, K, device=cuda) * 0.5).to(dt)
    p = config.algo_params(algo)
    tm, tn = M // p["BM"], N // p["BN"]
    RA = torch.randperm(tm * tn, device=cuda, dtype=torch.int32)
    rldn = 2 if tm * tn % 2 == 0 else 1
    e = torch.empty(0, dtype=torch.int32)
    mm = torch.zeros(tm + 1, tn, device=cuda, dtype=torch.int32)
    try:
        for exact, tma in ((1, -1), (0, -1), (0, 0)):
            impl.set_option("exact_algo", exact)
            impl.set_option("tma_out", tma)
            c = torch.full((M, N), float("nan"), device=cuda, dtype=dt)
            impl.cutlass_gemm(a, b, c, algo)
            _check(c, a, b, dt)
            if exact:
                assert _ran(impl) == (algo, 0, 0)
            else:
                assert _ran(impl)[:2] != (algo, 0)
                if M == 1920:                            # 168 pair units on 74 pairs: the last 20 in halves
                    assert _ran(impl)[:2] == (1, 0) and _ran(impl)[2] > 0
            c.fill_(float("nan"))
            impl.gemm_allreduce_overlap(a, b, c, mm, RA, rldn, e, e.to(cuda), algo, False)
            assert not exact or _ran(impl) == (algo, 0, 0)
            _check(layout.from_reordered(c.cpu(), M, N, p["BM"], p["BN"], RA.cpu(), rldn).to(cuda), a, b, dt)
    finally:
        impl.set_option("exact_algo", 0)
        impl.set_option("tma_out", -1)
    impl.check_status()


# the last wave in halves (80 units on 74 pairs), in a layout whose tiles are twice as wide as the halves; odd row
# tiles on pairs; 128-wide stand-ins for 256-wide tiles; a split: both types, one and two tiles to a row of the layout
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,algo,rldn", [(2560, 2048, 264, 1, 2), (1920, 5376, 136, 0, 1), (256, 8192, 320, 1, 2),
                                             (512, 4096, 520, 3, 2), (128, 2048, 4096, 0, 2)])
def test_stand_ins_in_the_tile_contiguous_layout(cuda, impl, dt, M, N, K, algo, rldn):
    a = (torch.randn(M, K, device=cuda) * 0.5).to(dt)
    b = (torch.randn(N, K, device=cuda) * 0.5).to(dt)
    p = config.algo_params(algo)
    tiles = (M // p["BM"]) * (N // p["BN"])
    RA = torch.randperm(tiles, device=cuda, dtype=torch.int32)
    e = torch.empty(0, dtype=torch.int32)
    mm = torch.zeros(M // p["BM"] + 1, N // p["BN"], device=cuda, dtype=torch.int32)
    for tma in (-1, 0):
        impl.set_option("tma_out", tma)
        c = torch.full((M, N), float("nan"), device=cuda, dtype=dt)
        impl.gemm_allreduce_overlap(a, b, c, mm, RA, rldn, e, e.to(cuda), algo, False)
        ran = _ran(impl)
        assert ran != (algo, 0, 0)
        if M == 2560:
            assert ran == (1, 0, 80 % (impl.get_option("sm_count") // 2))
        _check(layout.from_reordered(c.cpu(), M, N, p["BM"], p["BN"], RA.cpu(), rldn).to(cuda), a, b, dt)
    impl.set_option("tma_out", -1)
    impl.check_status()


def test_dependent_launches_across_streams(cuda, impl):
    """The early launch waits for its own stream's predecessor and for what an event makes it wait for, and a
    plain kernel behind it for all of it."""
    dt = torch.bfloat16
    M = N = K = 2048
    a, b = (torch.randn(M, K, device=cuda).to(dt) for _ in range(2))
    w = torch.ones(N, device=cuda, dtype=dt)
    c, y, z, out = (torch.empty(M, N, device=cuda, dtype=dt) for _ in range(4))
    side = torch.cuda.Stream()
    main = torch.cuda.current_stream()
    impl.cutlass_gemm(a, b, c, 1)
    ref = ops.rmsnorm(c, w, 1e-5)
    impl.cutlass_gemm(ref, b, z, 1)
    expect = z + z
    for _ in range(20):
        for t in (c, y, z, out):
            t.fill_(float("nan"))
        impl.cutlass_gemm(a, b, c, 1)                             # main: writes c
        done = torch.cuda.Event()
        done.record()
        with torch.cuda.stream(side):
            side.wait_event(done)
            torch.ops.flashoverlap_op.rmsnorm(c, y, w, 1e-5)      # side: behind the event
            impl.cutlass_gemm(y, b, z, 1)                         # side: behind the norm, launched early
            torch.add(z, z, out=out)
            back = torch.cuda.Event()
            back.record()
        main.wait_event(back)
        assert torch.equal(out, expect)
    impl.check_status()
