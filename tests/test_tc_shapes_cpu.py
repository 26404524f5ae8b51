"""Shapes of the streamed tensor-core form that a model description may ask for (no device)."""
import pytest


# With one 128-walker sub-tile and up to 256 features the library's own choice is 6 stages: the
# tuner answers with it, so it can be asked for.  Other counts go by what fits beside a walker
# operand in shared memory (at most 4 stages up to 192 features, 3 up to 256).
@pytest.mark.parametrize("features,fits,refused", [(129, (2, 4, 6), (1, 5, 7)), (192, (4, 6), (5,)),
                                                   (193, (2, 3, 6), (4, 5)), (256, (3, 6), (4, 5)),
                                                   (257, (2,), (3, 6)), (320, (2,), (3, 6))])
def test_stages_of_one_subtile(features, fits, refused):
    from bayadera_gb300 import _native as N, build, models as M
    from bayadera_gb300.engine import check_model
    build.build()
    for st in fits:
        check_model(M.logistic_model(features), "gemm", tensor=True, tc_subtiles=1, tc_stages=st)
    for st in refused:
        with pytest.raises(N.IllegalArgument):
            check_model(M.logistic_model(features), "gemm", tensor=True, tc_subtiles=1, tc_stages=st)
