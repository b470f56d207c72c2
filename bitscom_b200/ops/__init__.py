"""Python entry points of the hand-written sm_100a kernels (ctypes over C symbols)."""


def check_status(device) -> None:
    """Raise if a GEMM, cross-entropy or attention kernel gave up on one of its bounded waits since
    the last check: it then returned early and its output is not valid.  Synchronises the device;
    nothing to do on CPU ranks."""
    if device.type != "cuda":
        return
    from . import attention, gemm, nn

    if gemm.available():
        gemm.check_status()
        nn.check_status()
    if attention.available():
        attention.check_status()
