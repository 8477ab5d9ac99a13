// jsh_forms_ft.cu -- jsh_forms.cu built with the Faraday-thick mode of the IQUV
// pass compiled in (requests with JSH_FLAG_FARADAY_THICK).
#define JSH_FARADAY_THICK_BUILD 1
#include "jsh_forms.cu"
