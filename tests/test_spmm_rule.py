"""The built-in choice of the product kernel: it names a kernel that the
operator has at that width, and at the sizes where one was measured well
ahead of the others it is that one."""

import ctypes

import pytest

import native

CSR, GROUPS, TMA = 0, 1, 2


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    lib = native.load("rule", tmp_path_factory.mktemp("rule"))

    def pick(f64, rows, per_row, G, b, have_map=True):
        out = (ctypes.c_int * 2)()
        lib.rule(int(f64), ctypes.c_longlong(rows), ctypes.c_double(per_row),
                 G, b, int(have_map), out)
        return tuple(out)
    return pick


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("G", [0, 4, 8, 16])
def test_choices_exist_for_the_operator(rule, f64, G):
    for b in [2**i for i in range(11)]:
        for rows in (1, 500, 16383, 16384, 24000, 49152, 65536, 131072,
                     200000, 2000000):
            for per_row in (0.0, 8.0, 48.0, 500.0):
                kind, rpw = rule(f64, rows, per_row, G, b)
                assert rule(f64, rows, per_row, G, b, False)[0] != TMA
                if kind == CSR:
                    continue
                assert G and b >= 32
                if kind == TMA:
                    assert not f64 and G == 16 and b in (128, 256)
                else:
                    assert kind == GROUPS and not (f64 and G == 16)
                    assert rpw in ((0, 4, 8) if b <= 64 and G <= 8
                                   else (4, 8))
                    assert rpw <= G


@pytest.mark.parametrize("f64,rows,per_row,G,b,want", [
    # whole groups: 223 us against 366 (CSR) and 372 (parts), 55 against 81,
    # 27 against 37, 183 against 250
    (True, 200000, 60.5, 8, 64, (GROUPS, 0)),
    (True, 40009, 59.9, 8, 64, (GROUPS, 0)),
    (True, 16400, 59.2, 8, 64, (GROUPS, 0)),
    (True, 300000, 25.9, 4, 64, (GROUPS, 0)),
    (False, 32768, 98.3, 4, 64, (GROUPS, 0)),
    (False, 32768, 98.3, 8, 32, (GROUPS, 0)),
    # CSR: 18 against 34, 25 against 37
    (True, 12000, 39.8, 8, 32, (CSR, 0)),
    (False, 8000, 30.3, 8, 256, (CSR, 0)),
    # parts: 152 against 208
    (False, 65537, 60.1, 8, 256, (GROUPS, 8)),
    # CSR: 121 against 133 (TMA)
    (False, 65537, 60.1, 16, 128, (CSR, 0)),
    # TMA: 205 against 222
    (False, 80000, 99.3, 16, 128, (TMA, 0)),
])
def test_measured_choices(rule, f64, rows, per_row, G, b, want):
    assert rule(f64, rows, per_row, G, b) == want


@pytest.mark.parametrize("rows,b,want", [
    # parts where the TMA form has no map: 748 us against 1,124, 626 against
    # 748; CSR below: 227 against 288
    (262144, 128, (GROUPS, 8)), (262144, 256, (GROUPS, 8)),
    (220000, 256, (GROUPS, 8)), (150000, 256, (CSR, 0))])
def test_choice_without_a_tensor_map(rule, rows, b, want):
    assert rule(False, rows, 60.0, 16, b, False) == want
