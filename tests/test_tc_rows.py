"""Order of instructions in the batched Q8_0 GEMV on tcgen05, as for the kernels of test_kernel_order.py."""
from test_kernel_order import test_copies_in_flight_are_waited_for as check


def test_copies_of_the_batched_q8_0_gemv_are_waited_for():
    check("gemv_tc.cu")
