"""The oracle's entry points are declared per call, so that threads which declare
and call one function at the same time do not replace each other's signatures."""
import ctypes as C
import threading

import numpy as np

import oracle


def test_each_declaration_is_an_object_of_its_own():
    O = oracle.oracle()
    f = O._fn("or_adaptive_stopping", C.c_int, C.c_int)
    g = O._fn("or_adaptive_stopping", C.c_int64, C.c_void_p, C.c_double)
    assert f.argtypes == [C.c_int] and f.restype is C.c_int
    assert g.argtypes == [C.c_void_p, C.c_double] and g.restype is C.c_int64


def test_one_function_from_many_threads():
    O = oracle.oracle()
    x = np.random.default_rng(1).standard_normal(2000).astype(np.float32)
    want = O.encode("negabinary", x, 3, 32, True)
    errors = []

    def work():
        try:
            for _ in range(100):
                got = O.encode("negabinary", x, 3, 32, True)
                assert all(np.array_equal(a, b) for a, b in zip(got, want))
        except Exception as e:
            errors.append(repr(e))

    ths = [threading.Thread(target=work) for _ in range(8)]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    assert not errors
