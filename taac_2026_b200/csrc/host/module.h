// Parts of the host module.
#pragma once
#include <Python.h>

namespace tb200_host {
void bind_engine(PyObject* module);
}
