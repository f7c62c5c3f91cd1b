"""CPU: the autotuner's answer for the library's own choice is accepted back, and only it."""


def test_default_is_accepted():
    import bigint_gb300 as B

    B.build()
    L = B.lib()
    for m, full in ((4, 1), (64, 1), (250, 0), (4096, 1)):
        assert L.bi_mul_set_tuning_u64(m, full, B.MUL_DEFAULT, 1) == 0
        assert L.bi_mul_set_tuning_u32(m, full, B.MUL_DEFAULT, 1) == 0
        assert L.bi_mul_set_tuning_u64(m, full, B.MUL_DEFAULT, 2) == 1
        assert L.bi_mul_set_tuning_u64(m, full, B.MUL_DEFAULT + 1, 1) == 1
    assert L.bi_mul_set_tuning_u64(0, 1, B.MUL_DEFAULT, 1) == 1
