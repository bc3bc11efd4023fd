#pragma once
#include <torch/python.h>

/** Adds adamw_ready and adamw_update to the extension module; 0, or -1 with a Python error set. */
int add_adamw_step(PyObject* module);
