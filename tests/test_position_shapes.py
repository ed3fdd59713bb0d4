"""Launch shapes of the position pass: those of earlier builds keep their names, so that a program
that picks one by name still finds it.  CPU only."""


def test_named_shapes_stay():
    from mmnorm_b200 import ops
    names = ops.position_variants()
    assert names[0] == "interp_local_t4_n128"
    for name in ("interp_t2_n128_s24", "interp_t2_n256_s24", "interp_t1_n256_s48",
                 "interp_t1_n128_s16"):
        assert name in names
    assert len(set(names)) == len(names)
