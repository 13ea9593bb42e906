"""Which GEMM kernel takes a product (csrc/gemm_sm100.cu, gemm_route): a function of sizes, options and addresses that needs no
device.  Epilogue operands that start off a 16-byte boundary may only reach the kernel that moves them by elements."""
import pytest

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

native._load()
pytestmark = pytest.mark.skipif(native._mod is None, reason="native extension not built")
SMS = 148
EVEN, ODD = 0x1000, 0x1008            # addresses on and off a 16-byte boundary
ONE_CTA, PAIR, CLUSTER, REFUSED = 0, 1, 2, -4


def route(M, N, K, *, act=F.ACT_NONE, bias=0, aux=0, preact_out=0, residual=0, fp32=False, accumulate=False, sms=SMS):
    return native.ext().gemm_route(M, N, K, fp32, accumulate, act, bias, aux, preact_out, residual, 0.0, sms)


@pytest.mark.parametrize("operand,act", [("residual", F.ACT_NONE), ("preact_out", F.ACT_GELU), ("aux", F.ACT_DGELU),
                                         ("aux", F.ACT_DRELU)])
@pytest.mark.parametrize("M,N,K", [(16, 8, 64), (300, 24, 2000), (4096, 31, 512), (300, 32, 2000), (512, 1024, 1024),
                                   (200, 72, 64), (4096, 4096, 1024), (30000, 40, 64)])
def test_row_operands_off_a_boundary(operand, act, M, N, K):
    kernel, bn, slices = route(M, N, K, act=act, **{operand: EVEN})
    assert kernel in (ONE_CTA, PAIR, CLUSTER) and (kernel != CLUSTER or (bn in (64, 128) and slices in (1, 2, 4, 8)))
    for start in range(EVEN + 2, EVEN + 16, 2):
        assert route(M, N, K, act=act, **{operand: start})[0] == (ONE_CTA if N < 32 else REFUSED)


def test_narrow_outputs_do_take_the_cluster_kernel():
    """(what makes the test above one of the addresses, not of the sizes)"""
    assert route(300, 24, 2000, residual=EVEN)[0] == CLUSTER


def test_an_operand_that_is_not_read_may_lie_anywhere():
    assert route(512, 1024, 1024, aux=ODD)[0] == route(512, 1024, 1024, aux=EVEN)[0]


@pytest.mark.parametrize("M,N,K,odd", [(300, 24, 2000, None), (200, 31, 64, None), (512, 1024, 1024, None),
                                       (4096, 4096, 1024, REFUSED), (30000, 40, 64, REFUSED)])
def test_bias_off_a_boundary(M, N, K, odd):
    """The cluster kernel reads the bias by elements, the others 32 (16) columns at a time in 16-byte pieces."""
    even = route(M, N, K, bias=EVEN)
    assert even[0] >= 0
    assert route(M, N, K, bias=ODD) == (even if odd is None else (odd, 0, 0))


PLAIN, GELU = {}, dict(act=F.ACT_GELU, bias=EVEN, preact_out=EVEN)
RESIDUAL, DGELU, WGRAD = dict(bias=EVEN, residual=EVEN), dict(act=F.ACT_DGELU, aux=EVEN), dict(fp32=True, accumulate=True)


@pytest.mark.parametrize("M,N,K,call,one_cta,cluster", [       # microseconds with either kernel, captured
    (2048, 8, 200, PLAIN, 5.4, 6.4), (64, 4096, 512, PLAIN, 7.1, 8.4), (512, 2048, 512, PLAIN, 7.4, 8.2),
    (1000, 8, 64, GELU, 5.4, 6.0), (200, 32, 64, GELU, 5.4, 6.4), (200, 32, 128, DGELU, 5.7, 6.6),
    (512, 4096, 16384, GELU, 68.7, 89.9), (2048, 1024, 12288, GELU, 54.2, 69.8), (2048, 1024, 16384, RESIDUAL, 69.8, 91.2),
    (512, 1024, 1024, RESIDUAL, 12.7, 9.1), (512, 1024, 4096, RESIDUAL, 23.0, 12.0), (512, 4096, 1024, GELU, 13.1, 11.4),
    (1024, 512, 512, WGRAD, 15.0, 8.6), (1000, 8, 8192, PLAIN, 32.4, 9.1), (1024, 1024, 512, WGRAD, 15.0, 8.6),
])
def test_the_faster_kernel_takes_the_call(M, N, K, call, one_cta, cluster):
    assert route(M, N, K, **call)[0] == (CLUSTER if cluster < one_cta else ONE_CTA)


@pytest.mark.parametrize("M,N,K,b_mn,lines,columns", [
    # rounds a fifth shorter and more, in either layout
    (2048, 3072, 2048, False, True, 192), (2560, 2048, 4096, False, True, 160), (2560, 4096, 4096, True, True, 192),
    (4096, 1280, 4096, True, True, 160), (4096, 768, 512, False, True, 192),
    # an eighth shorter: less of the output is padding, or B is read K-major
    (12544, 640, 5760, False, True, 224), (12544, 640, 5760, True, True, 224), (4096, 5120, 4096, False, True, 224),
    (4096, 5120, 4096, True, True, 256), (2048, 8192, 4096, True, True, 256),
    # more rounds of narrower tiles, which move more for each operation
    (8192, 2560, 2048, False, True, 256), (16384, 1280, 4096, True, True, 256), (4096, 6144, 4096, False, True, 256),
    (8192, 3072, 4096, True, True, 256), (16384, 1536, 2048, False, True, 256),
    # a reduction that ends before the epilogue does, over several rounds
    (4096, 5120, 512, False, True, 256), (2048, 10240, 512, False, True, 256),
    # operands whose rows start off 128 bytes
    (2560, 4096, 4096, True, False, 256), (2560, 2048, 4096, False, False, 160), (12536, 640, 4096, True, False, 256),
])
def test_columns_of_a_tile_on_pairs(M, N, K, b_mn, lines, columns):
    """Narrower tiles only where they are the faster ones, also under the power cap (times in csrc/gemm2_sm100.cu)."""
    assert native.ext().gemm_pair_columns(M, N, K, False, SMS, b_mn, lines) == columns
