"""CPU: the rules that decide which calls run on the few-token integer kernel (qgemm_unit.cu), and how, over the forms they
accept.  They are plain host functions of the library."""
import ctypes

import pytest

from ubridge_b200 import _lib

Q4_0, Q8_0, Q4_K, Q5_K, Q6_K = 2, 8, 12, 13, 14
ROWS = [256 * i for i in range(1, 113)] + [30720, 32768, 40960]


def rule(name, types):
    f = getattr(_lib.lib(), "_ZN2ub%d%sE%s" % (len(name), name, types))
    f.restype = ctypes.c_bool
    return f


def early(tag, M, K, y_f32):
    return rule("unit_early", "iiib")(tag, M, K, ctypes.c_bool(y_f32))


def test_no_request_ahead_where_plain_launches_took_the_call():
    """A call whose kernels waited for the one in front in full may have its weights written by that one, without a flag."""
    for K in ROWS:
        odd = K % 2048 != 0
        for M in range(1, 17):
            # f32 results of Q4_K: token pairs of a whole row fit the integer kernel's 219 KB, or K has a kernel of its own
            if M >= 2 and not (K in (2048, 4096) or (K == 8192 and M > 4)):
                pairs = 1 if M == 2 else 2 if M <= 4 else 4
                if pairs * (K // 256) > 70:
                    assert not early(Q4_K, M, K, True), (M, K)
            # Q8_0: whole 64-block chunks whose token quads fit; two-piece weights otherwise for 16-bit results, but CUDA cores
            # for one token, and for two and four where they were the faster ones
            quads = 1 if M <= 4 else 2
            if odd or quads * (K // 32) > 568:
                assert not early(Q8_0, M, K, True), (M, K)
            if odd and M in (1, 2, 4):
                assert not early(Q8_0, M, K, False), (M, K)
        for tag in (Q4_0, Q5_K, Q6_K):
            for M in (1, 2, 3, 4, 5, 16, 17, 200):
                if odd:
                    assert not early(tag, M, K, True) and not early(tag, M, K, False), (tag, M, K)
                # longer than any staged plan: one token 14336 (Q6_K), four 10240 (Q6_K) and fewer
                if K > 16384 or (M >= 4 and K > 12288):
                    assert not early(tag, M, K, True), (tag, M, K)
                    assert M > 4 or not early(tag, M, K, False), (tag, M, K)


@pytest.mark.parametrize("tag,M,K,y_f32", [
    (Q4_K, 4, 14336, False), (Q4_K, 2, 14336, True), (Q4_K, 8, 4096, True), (Q8_0, 4, 6144, True), (Q8_0, 16, 14336, False),
    (Q5_K, 2, 4096, True), (Q6_K, 4, 4096, True), (Q4_0, 8, 14336, False), (Q6_K, 16, 4096, True),
])
def test_weights_are_requested_ahead_where_they_always_were(tag, M, K, y_f32):
    assert early(tag, M, K, y_f32)


def takes(tag, M, N, K, x_f32, y_f32):
    """Which kernel has the call: 1 the integer kernel, 2 two-piece weights, 0 another one."""
    b = ctypes.c_bool
    if tag in (Q8_0, Q4_K):
        f = rule("few_tokens_route", "iiiibb")
        f.restype = ctypes.c_int
        return f(tag, M, N, K, b(x_f32), b(y_f32))
    return int(rule("unit_takes", "iiiibb")(tag, M, N, K, b(x_f32), b(y_f32)))


@pytest.mark.parametrize("tag,M,N,K,x_f32,y_f32", [
    # B200, us, the other kernel / this one: 2.0 / 5.5, 2.6 / 5.5, 20.8 / 24, 10.3 / 13.9; 2.3 / 4.2 (CUDA cores), 6.9 / 10.9 (two pieces)
    (Q6_K, 1, 1024, 512, False, False), (Q6_K, 4, 1024, 512, False, False), (Q6_K, 1, 14336, 3328, False, False),
    (Q6_K, 2, 512, 12288, True, False), (Q8_0, 1, 2048, 512, False, True), (Q4_K, 16, 4096, 512, True, False),
])
def test_calls_that_other_kernels_do_faster(tag, M, N, K, x_f32, y_f32):
    assert takes(tag, M, N, K, x_f32, y_f32) != 1


@pytest.mark.parametrize("tag,M,N,K,x_f32,y_f32", [
    (Q4_K, 4, 4096, 14336, False, False), (Q8_0, 4, 6144, 5120, False, False), (Q4_0, 1, 4096, 4352, False, False),
    (Q5_K, 4, 14336, 3328, False, True), (Q6_K, 8, 16384, 5120, False, False), (Q5_K, 1, 8192, 28672, False, False),
])
def test_calls_that_this_kernel_does_faster(tag, M, N, K, x_f32, y_f32):
    assert takes(tag, M, N, K, x_f32, y_f32) == 1


def test_two_piece_weights_only_for_f32_tokens_in_a_second_pass():
    for tag in (Q8_0, Q4_K):
        for M in range(1, 17):
            for N in (1, 300, 1200, 4096, 28672):
                for K in ROWS:
                    for y_f32 in (False, True):
                        assert takes(tag, M, N, K, False, y_f32) != 2
                        assert M > 8 or takes(tag, M, N, K, True, y_f32) != 2
